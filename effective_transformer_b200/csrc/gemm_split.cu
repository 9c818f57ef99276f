// Projections of small batches: C[M,N] = epilogue(A[M,K] * W[N,K]^T), the K range of a tile split over
// the CTAs of a cluster.
//
// The persistent kernels (gemm_tcgen05.cu, gemm_tf32x3.cu) give a CTA (pair) whole 256-wide tiles with all
// of K: right when there are tiles for every SM, but a batch of a few hundred tokens has 3 to 24 of them,
// and each walks K alone (48 dependent 64-wide steps for K = 3072) while most of the GPU idles.  What
// bounds such a projection is the latency of that chain and how many SMs pull on the weights (1 to 5 MB).
// So here a tile is 128 x 64 (fp32 also 128 x 128: a third less to fetch per output, where the number of CTAs
// that run at once, one per SM, is the limit) and its K range is cut into `splits` (1 to 8) parts, one CTA each:
//   warp 0      TMA producer: A [128 x BK] and W [64 or 128 x BK] boxes into a ring of shared-memory stages
//   warp 1      tcgen05.mma (M = 128, N = 64 or 128) into TMEM, one accumulator block per accumulation unit
//   warps 2-5   read the partial sums from TMEM and send row r to the CTA r % splits of the cluster through
//               distributed shared memory; behind a cluster barrier each CTA adds the parts of its rows
//               in rank order (the result does not depend on timing), applies the epilogue and stores
// Rows are dealt to the CTAs by r % splits, so a last tile with few rows still keeps all of them busy.
// The shared memory of an fp16 CTA is below half an SM's, so the next projection's CTAs are resident while this
// one runs, and the producer requests their W boxes before it waits for this kernel
// (`weights_ready`: W was complete before the preceding kernel began): a weight's trip from HBM then lies
// under the kernel before.  Every mbarrier wait is bounded.
#include "common.cuh"
#include "ptx_sm100.cuh"

#include <type_traits>

namespace etb {

namespace {

using namespace ptx;

constexpr int BM = 128;
constexpr int kRowBytes = 128;        // one swizzle row of an operand tile: 64 fp16 or 32 tf32
constexpr int kThreads = 192;
constexpr int kEpThreads = 128;
constexpr int kMaxSplits = 8;

enum Site : int { kSiteProducer = 1, kSiteDrain = 2, kSiteMma = 3, kSiteMmaDrain = 4, kSiteEpilogue = 5, kSiteAlign = 6 };

template <bool kTf32, int BN>
struct Cfg {
  static constexpr bool kWide = BN == 128;
  static constexpr int BK = kTf32 ? 32 : 64;
  static constexpr int kParts = kTf32 ? 2 : 1;  // tf32: hi and lo halves of both operands
  static constexpr int kABytes = BM * kRowBytes;
  static constexpr int kWBytes = BN * kRowBytes;
  static constexpr int kStageBytes = kParts * (kABytes + kWBytes);
  static constexpr int kStages = 3;
  // tf32: the tensor core adds into its accumulator with truncation, so a chain is cut every six k-blocks
  // (see gemm_tf32x3.cu); every unit has a TMEM block of its own here.  fp16: one unit.
  static constexpr int kUnitKb = kTf32 ? 6 : 1 << 20;
  static constexpr int kBlocks = kTf32 ? 512 / BN : 1;
  static constexpr int kTmemCols = kBlocks * BN;
  // partial sums of this CTA's rows from every CTA of the cluster: splits * ceil(128 / splits) rows.  The 128-wide
  // tiles receive them where their operand stages were: both would not fit an SM.
  static constexpr int kRecvBytes = (BM + kMaxSplits) * BN * 4;
  static constexpr int kRecvAt = kWide ? 0 : kStages * kStageBytes;
  static_assert(!kWide || kRecvBytes <= kStages * kStageBytes, "the partial sums must fit the stages");
  static constexpr int kBarsAt = kWide ? kStages * kStageBytes : kRecvAt + kRecvBytes;
  static constexpr int kPieces = BN / 8;                // eight-column pieces of a row
  static constexpr int kRowsPass = kEpThreads / kPieces;  // rows the epilogue threads cover at once
  static constexpr int kNumBars = 2 * kStages + 2;
  static constexpr int kSmemBytes = kBarsAt + 128;
};

__device__ __forceinline__ void umma_tf32_ss(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void st_cluster_v4(uint32_t addr, float a, float b, float c, float d) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d)
               : "memory");
}
__device__ __forceinline__ float4 ld_shared_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

__device__ __forceinline__ void load8(const __half* p, float* f) { VecTraits<__half>::unpack(ld_global_nc_v4(p), f); }
__device__ __forceinline__ void load8(const float* p, float* f) {
  VecTraits<float>::unpack(ld_global_nc_v4(p), f);
  VecTraits<float>::unpack(ld_global_nc_v4(p + 4), f + 4);
}

struct Maps {
  CUtensorMap a, w, a_lo, w_lo;  // the lo halves only for tf32
};

template <bool kTf32, int BN, int EPI>
__global__ void __launch_bounds__(kThreads, kTf32 ? 1 : 2)
gemm_split_kernel(const __grid_constant__ Maps maps, void* __restrict__ c_ptr, float* __restrict__ c_lo,
                  const void* __restrict__ bias_ptr, const void* res_ptr, const int* m_ptr,
                  int max_m, int N, int num_kb, int weights_ready, int* status_word, const GemmLayerNorm ln) {
  using cfg = Cfg<kTf32, BN>;
  using T = typename std::conditional<kTf32, float, __half>::type;
  constexpr int S = cfg::kStages;
  constexpr bool kNormIn = EPI == kEpiNormIn || EPI == kEpiNormInGelu;
  constexpr bool kResidual = EPI == kEpiBiasResidual || EPI == kEpiNormResidual;

  pdl_trigger();
  const int splits = gridDim.x, rank = blockIdx.x;  // the cluster covers gridDim.x
  const int m0 = blockIdx.z * BM, n0 = blockIdx.y * BN;
  const int kb0 = num_kb * rank / splits, kb1 = num_kb * (rank + 1) / splits;
  const int units = (kb1 - kb0 + cfg::kUnitKb - 1) / cfg::kUnitKb;

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = smem_u32(smem_raw);
  const bool aligned = (base & 1023u) == 0u;  // the same in every CTA of the grid
  const uint32_t recv = base + cfg::kRecvAt;
  const int slots = (BM + splits - 1) / splits;  // rows of the tile that are this CTA's
  const uint32_t bar0 = base + cfg::kBarsAt;
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (S + s); };
  const uint32_t acc_bar = bar0 + 8u * (2 * S), drain_bar = acc_bar + 8u;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_raw + cfg::kBarsAt + 8 * cfg::kNumBars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(acc_bar, 1);
    mbar_init(drain_bar, 1);
    *abort_flag = 0;
    fence_mbar_init();
    fence_proxy_async_smem();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), cfg::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // First arrival at the cluster's barrier, behind which the shared memory of its CTAs may be written: every CTA
  // runs from here on; where the partial sums take the place of the stages, only when its MMAs are done.
  if (!cfg::kWide && splits > 1) cluster_arrive();

  auto fail = [&](int site) {
    *abort_flag = 1;
    report_timeout(status_word, kKernelGemmTc, 16 + site);
  };
  auto valid_rows = [&]() {  // behind pdl_wait()
    const int M = *m_ptr;
    return (M < 0 ? 0 : (M > max_m ? max_m : M)) - m0;  // of this tile, <= 0: nothing to do
  };

  if (warp == 0) {
    // ------------------------- TMA producer -------------------------
    if (lane == 0 && aligned) {
      const CUtensorMap* map_a[2] = {&maps.a, &maps.a_lo};
      const CUtensorMap* map_w[2] = {&maps.w, &maps.w_lo};
      auto load_w = [&](int kb, int s) {
        mbar_arrive_expect_tx(full_bar(s), cfg::kStageBytes);
        const uint32_t dst = base + s * cfg::kStageBytes + cfg::kParts * cfg::kABytes;
#pragma unroll
        for (int h = 0; h < cfg::kParts; ++h) tma_load_2d(dst + h * cfg::kWBytes, map_w[h], kb * cfg::BK, n0, full_bar(s));
      };
      auto load_a = [&](int kb, int s) {
        const uint32_t dst = base + s * cfg::kStageBytes;
#pragma unroll
        for (int h = 0; h < cfg::kParts; ++h) tma_load_2d(dst + h * cfg::kABytes, map_a[h], kb * cfg::BK, m0, full_bar(s));
      };
      const int first = min(kb1 - kb0, S);
      if (weights_ready) {
        for (int i = 0; i < first; ++i) load_w(kb0 + i, i);
        pdl_wait();
        for (int i = 0; i < first; ++i) load_a(kb0 + i, i);
      } else {
        pdl_wait();
        for (int i = 0; i < first; ++i) {
          load_w(kb0 + i, i);
          load_a(kb0 + i, i);
        }
      }
      int issued = first;
      // a tile beyond the valid rows stops here (the first tile needs no look: it has rows unless M is 0)
      const bool live = blockIdx.z == 0 || valid_rows() > 0;
      if (live) {
        for (; issued < kb1 - kb0; ++issued) {
          const int s = issued % S;
          if (!mbar_wait(empty_bar(s), static_cast<uint32_t>((issued / S - 1) & 1), abort_flag)) {
            fail(kSiteProducer);
            break;
          }
          load_w(kb0 + issued, s);
          load_a(kb0 + issued, s);
        }
      }
      // the issuer's commits on the empty barriers are asynchronous arrivals: the last of them land before the
      // barriers go away
      if (live)
        for (int i = max(0, issued - S); i < issued; ++i)
          if (!mbar_wait(empty_bar(i % S), static_cast<uint32_t>((i / S) & 1), abort_flag) && *abort_flag == 0)
            fail(kSiteDrain);
      // copies in flight must land before the CTA's shared memory goes away
      for (int i = max(0, issued - S); i < issued; ++i)
        if (!mbar_drain(full_bar(i % S), static_cast<uint32_t>((i / S) & 1)) && *abort_flag == 0)
          fail(kSiteDrain);
    } else {
      pdl_wait();
      if (lane == 0) report_timeout(status_word, kKernelGemmTc, 16 + kSiteAlign);
    }
    __syncwarp();
    if (splits > 1) {
      if (cfg::kWide) cluster_arrive();
      cluster_wait();
      cluster_arrive();
      cluster_wait();
    }
  } else if (warp == 1) {
    // ------------------------- MMA issuer -------------------------
    pdl_wait();
    if (lane == 0 && aligned && (blockIdx.z == 0 || valid_rows() > 0)) {
      constexpr uint32_t idesc = make_idesc_f16_f32acc(BM, BN) | (kTf32 ? (2u << 7) | (2u << 10) : 0u);
      bool ok = true;
      for (int i = 0; i < kb1 - kb0; ++i) {
        const int s = i % S;
        if (!mbar_wait(full_bar(s), static_cast<uint32_t>((i / S) & 1), abort_flag)) {
          fail(kSiteMma);
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t a = base + s * cfg::kStageBytes, w = a + cfg::kParts * cfg::kABytes;
        const uint32_t d = tmem_base + (i / cfg::kUnitKb) * BN;
        const bool fresh = i % cfg::kUnitKb == 0;
        const uint64_t ad = make_kmajor_sw128_desc(a), wd = make_kmajor_sw128_desc(w);
        if constexpr (kTf32) {
          const uint64_t ad2 = make_kmajor_sw128_desc(a + cfg::kABytes), wd2 = make_kmajor_sw128_desc(w + cfg::kWBytes);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_tf32_ss(d, ad + 2u * k, wd + 2u * k, idesc, (!fresh || k > 0) ? 1u : 0u);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_tf32_ss(d, ad + 2u * k, wd2 + 2u * k, idesc, 1u);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_tf32_ss(d, ad2 + 2u * k, wd + 2u * k, idesc, 1u);
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_f16_ss(d, ad + 2u * k, wd + 2u * k, idesc, (!fresh || k > 0) ? 1u : 0u);
        }
        umma_commit(empty_bar(s));
      }
      if (ok) umma_commit(acc_bar);
      umma_commit(drain_bar);
      if (!mbar_drain(drain_bar, 0u) && *abort_flag == 0) fail(kSiteMmaDrain);
    }
    __syncwarp();
    if (splits > 1) {
      if (cfg::kWide) cluster_arrive();
      cluster_wait();
      cluster_arrive();
      cluster_wait();
    }
  } else {
    // ------------------------- partial sums, reduction, epilogue -------------------------
    pdl_wait();
    const int rows = min(valid_rows(), BM);
    const bool live = rows > 0 && aligned;
    const int quad = warp & 3;
    const int t = threadIdx.x - 64;      // 0..127
    const int piece = t % cfg::kPieces;  // this thread's eight columns
    const int col = n0 + piece * 8;
    // slots (rows) of this thread, at most eight: a 128-wide tile has two CTAs at least
    const int items = (slots + cfg::kRowsPass - 1) / cfg::kRowsPass;
    auto slot_of = [&](int j) { return t / cfg::kPieces + cfg::kRowsPass * j; };
    auto row_of = [&](int j) { return rank + splits * slot_of(j); };
    T* C = static_cast<T*>(c_ptr);
    const T* bias = static_cast<const T*>(bias_ptr);
    const T* residual = static_cast<const T*>(res_ptr);

    // what the epilogue needs beside the sums is requested before the accumulator is waited for
    float fb[8], fg[8], fe[8];
    Vec16 res[8];
    float2 st[8][2];
#pragma unroll
    for (int e = 0; e < 8; ++e) fb[e] = 0.f, fg[e] = 1.f, fe[e] = 0.f;
    if (live) {
      if (EPI != kEpiNone) load8(bias + col, fb);
      if constexpr (EPI == kEpiNormResidual) {
        if (ln.gamma != nullptr) {
          load8(ln.gamma + col, fg);
          load8(ln.beta + col, fe);
        }
      }
      if constexpr (kNormIn) load8(ln.csum + col, fg);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j < items && row_of(j) < rows) {
          if constexpr (kResidual) res[j] = ld_activation_v4(residual + static_cast<size_t>(m0 + row_of(j)) * N + col);
          if constexpr (is_deferred_norm(EPI)) {
            st[j][0] = st[j][1] = make_float2(0.f, 0.f);
            if (ln.stats_in != nullptr) {
              const float2* sp = reinterpret_cast<const float2*>(ln.stats_in) + static_cast<size_t>(m0 + row_of(j)) * ln.stat_slots;
              if ((piece & 7) < ln.stat_slots) st[j][0] = sp[piece & 7];
              if ((piece & 7) + 8 < ln.stat_slots) st[j][1] = sp[(piece & 7) + 8];
            }
          }
        }
    }

    bool got = live;
    if (live) {
      got = __all_sync(0xffffffffu, mbar_wait(acc_bar, 0u, abort_flag));
      if (!got && lane == 0) fail(kSiteEpilogue);
    }
    if (splits > 1) {
      if (cfg::kWide) cluster_arrive();
      cluster_wait();
    }
    if (got && quad * 32 < rows) {
      tc_fence_after();
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
      const int r = quad * 32 + lane;
      const int slot = r / splits;
      const uint32_t dst0 = recv + ((rank * slots + slot) * BN) * 4;
      const uint32_t dst = splits > 1 ? mapa_shared(dst0, r % splits) : dst0;
#pragma unroll
      for (int hcol = 0; hcol < BN / 32; ++hcol) {
        float sum[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) sum[e] = 0.f;
        for (int u = 0; u < units; ++u) {
          uint32_t v[32];
          tmem_ld_32x32b_x32(t_row + u * BN + hcol * 32, v);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; ++e) sum[e] += __uint_as_float(v[e]);
        }
        if (r < rows) {
#pragma unroll
          for (int g = 0; g < 8; ++g) {
            // 16-byte groups swizzled by the row's slot: the readers' and the writers' banks are spread
            const uint32_t at = dst + (((hcol * 8 + g) ^ (slot & 15)) << 4);
            if (splits > 1) st_cluster_v4(at, sum[4 * g], sum[4 * g + 1], sum[4 * g + 2], sum[4 * g + 3]);
            else asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(at), "f"(sum[4 * g]), "f"(sum[4 * g + 1]),
                              "f"(sum[4 * g + 2]), "f"(sum[4 * g + 3]) : "memory");
          }
        }
      }
      tc_fence_before();
    }
    __syncwarp();
    if (splits > 1) {
      cluster_arrive();
      cluster_wait();
    } else {
      asm volatile("bar.sync 1, %0;" ::"n"(kEpThreads) : "memory");
    }
    if (live && *abort_flag == 0) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (j >= items) break;           // uniform
        const int r = row_of(j);
        const int slot = slot_of(j);
        const bool mine = r < rows;      // uniform in the lanes of a row
        float f[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = 0.f;
        if (mine) {
          for (int src = 0; src < splits; ++src) {
            const uint32_t rowp = recv + ((src * slots + slot) * BN) * 4;
            const float4 p0 = ld_shared_f4(rowp + (((2 * piece) ^ (slot & 15)) << 4));
            const float4 p1 = ld_shared_f4(rowp + (((2 * piece + 1) ^ (slot & 15)) << 4));
            f[0] += p0.x, f[1] += p0.y, f[2] += p0.z, f[3] += p0.w;
            f[4] += p1.x, f[5] += p1.y, f[6] += p1.z, f[7] += p1.w;
          }
        }
        float mu = 0.f, rstd = 1.f;
        if constexpr (is_deferred_norm(EPI)) {
          float a = mine ? st[j][0].x + st[j][1].x : 0.f, b = mine ? st[j][0].y + st[j][1].y : 0.f;
#pragma unroll
          for (int o = 1; o < 8; o <<= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            b += __shfl_xor_sync(0xffffffffu, b, o);
          }
          if (ln.stats_in != nullptr) {
            const float inv = 1.0f / static_cast<float>(ln.stat_slots * 64);
            mu = a * inv;
            rstd = rsqrtf(fmaxf(b * inv - mu * mu, 0.f) + ln.eps);
          }
        }
        const size_t at = static_cast<size_t>(m0 + r) * N + col;
        if constexpr (kTf32) {
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            if (EPI != kEpiNone) f[e] += fb[e];
            if (EPI == kEpiBiasGelu) f[e] = gelu_tanh(f[e]);
            if (EPI == kEpiBiasTanh) f[e] = tanhf(f[e]);
          }
          if (mine) {
            if (c_lo != nullptr) {
              float lo[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) {
                const float hi = rn_tf32(f[e]);
                lo[e] = f[e] - hi;
                f[e] = hi;
              }
              st_global_v4(c_lo + at, VecTraits<float>::pack(lo));
              st_global_v4(c_lo + at + 4, VecTraits<float>::pack(lo + 4));
            }
            st_global_v4(C + at, VecTraits<float>::pack(f));
            st_global_v4(C + at + 4, VecTraits<float>::pack(f + 4));
          }
        } else {
          if constexpr (kNormIn) {
            // rstd * (acc - mu * csum[n]) + bias[n]
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = fmaf(rstd, fmaf(-mu, fg[e], f[e]), fb[e]);
          } else if constexpr (EPI == kEpiNormResidual) {
            // (res - mu) * rstd in fp32: see epilogue_warp_tile in gemm_tcgen05.cu
            float fr[8];
            VecTraits<__half>::unpack(res[j], fr);
            const float nmr = -mu * rstd;
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] += fb[e] + fmaf(fmaf(fr[e], rstd, nmr), fg[e], fe[e]);
          } else if constexpr (EPI != kEpiNone) {
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] += fb[e];
          }
          if constexpr (EPI == kEpiBiasResidual) {
            float fr[8];
            VecTraits<__half>::unpack(res[j], fr);
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] += fr[e];
          }
          if constexpr (EPI == kEpiBiasTanh) {
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = tanhf(f[e]);
          }
          Vec16 o = VecTraits<__half>::pack(f);
          if constexpr (EPI == kEpiBiasGelu || EPI == kEpiNormInGelu) {
            o.x = gelu_tanh_half2(o.x);
            o.y = gelu_tanh_half2(o.y);
            o.z = gelu_tanh_half2(o.z);
            o.w = gelu_tanh_half2(o.w);
          }
          if (mine) st_global_v4(C + at, o);
          if constexpr (EPI == kEpiNormResidual) {
            // statistics of the row's 64-column piece as stored
            float y[8], a = 0.f, b = 0.f;
            VecTraits<__half>::unpack(o, y);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              a += y[e];
              b = fmaf(y[e], y[e], b);
            }
#pragma unroll
            for (int o2 = 1; o2 < 8; o2 <<= 1) {
              a += __shfl_xor_sync(0xffffffffu, a, o2);
              b += __shfl_xor_sync(0xffffffffu, b, o2);
            }
            if (mine && (piece & 7) == 0)
              reinterpret_cast<float2*>(ln.stats_out)[static_cast<size_t>(m0 + r) * (N / 64) + col / 64] = make_float2(a, b);
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, cfg::kTmemCols);
  }
}

template <bool kTf32, int BN, int EPI>
cudaError_t launch_split_bn(const Maps& maps, const SplitGemm& g, int splits, cudaStream_t stream) {
  using cfg = Cfg<kTf32, BN>;
  static PerDeviceOnce once;  // function attributes are per device
  const cudaError_t once_err = once.run([] {
    return cudaFuncSetAttribute(gemm_split_kernel<kTf32, BN, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                cfg::kSmemBytes);
  });
  if (once_err != cudaSuccess) return once_err;
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(splits, g.n / BN, (g.max_m + BM - 1) / BM);
  lc.blockDim = dim3(kThreads);
  lc.dynamicSmemBytes = cfg::kSmemBytes;
  lc.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = splits;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  lc.attrs = attr;
  lc.numAttrs = pdl_enabled() ? 2 : 1;
  return cudaLaunchKernelEx(&lc, gemm_split_kernel<kTf32, BN, EPI>, maps, g.c, g.c_lo, g.bias, g.residual, g.m_ptr,
                            g.max_m, g.n, (g.k + cfg::BK - 1) / cfg::BK, g.hints.weights_ready ? 1 : 0, g.status_word, g.ln);
}

template <bool kTf32, int EPI>
cudaError_t launch_split(const Maps& maps, const SplitGemm& g, const SplitPlan& p, cudaStream_t stream) {
  if constexpr (kTf32)
    if (p.bn == 128) return launch_split_bn<kTf32, 128, EPI>(maps, g, p.splits, stream);
  return launch_split_bn<kTf32, 64, EPI>(maps, g, p.splits, stream);
}

bool encode_split(CUtensorMap* map, bool tf32, const void* base, int rows, int k, int box_rows, TensorMapCache* cache) {
  return tf32 ? encode_2d_f32_sw128(map, base, rows, k, box_rows, cache)
              : encode_2d_fp16_sw128(map, base, rows, k, k, box_rows, 64, cache);
}

}  // namespace

// Where a cluster's split pays, from the capacity in rows (the valid rows are only known on the device).
// Measured where it counts, inside a replayed pass, whose kernels overlap and whose weights come from HBM: us per
// pass on one B200 with one projection's plan changed and the others at their best ("64x4" = tiles 64 wide, 4 CTAs
// per tile; "-" = the persistent kernels).  BERT-base fp16, capacity 64 / 256 / 512 / 1024 / 2048 (60 to 70 % valid):
//   QKV       64x1 426  64x2 463  - 452    64x2 515 - 489            64x2 543 - 521   64x1 635 - 587   - 706
//   out       64x4 426  64x2 460  - 467    64x4 490 - 542            64x2 526 - 555   64x2 591 - 608   64x2 733 - 707
//   FFN1      64x2 425  64x4 471  - 460    64x2 488 - 504            64x2 561 - 517   64x1 638 - 592   - 706
//   FFN2      64x8 425  64x4 489  - 638    64x8 489 64x4 525 - 647   64x4 530 - 660   64x2 587 - 660   64x2 707 - 734
// and with every row of 2048 valid FFN2 64x2 919, - 839.  BERT-large fp16, capacity 128 / 256 / 512 / 768 / 1024 /
// 1280 (55 to 65 % valid; the rule's plan first, then the best other one and the persistent kernels):
//   QKV       64x3 944 64x5 927 - 980   - 1129 64x2 1115   - 1206 64x2 1226   - 1339   - 1441   - 1612
//   out       64x5 939 64x4 921 - 1073   64x3 1127 64x5 1116 - 1250   64x3 1206 64x4 1199 - 1271
//             64x2 1338 64x3 1314 - 1377   - 1441 64x2 1392   - 1611
//   FFN1      64x3 943 - 988   - 1128 64x2 1144   - 1205   - 1340   - 1441   - 1611
//   FFN2      64x8 939 - 1363   64x6 1127 - 1503   64x3 1206 64x4 1176 - 1502   64x2 1339 64x3 1289 - 1526
//             64x2 1441 - 1625   - 1611 64x2 1416
// It holds there, but stops early for K = 4096 (1536 rows: - 1664, 64x2 1530).  fp32, BERT-base, capacity 64 / 256 / 512:
//   QKV       64x3 755  - 853              64x2 949 128x2 981 - 1001  128x2 1223 - 1170
//   out       64x8 754  - 876              64x5 949 64x4 962 - 1064   128x5 1170 64x2 1173 - 1342
//   FFN1      128x5 755 64x2 767 - 856     128x2 949 64x2 1005 - 965  128x2 1162 - 1155
//   FFN2      64x8 755  - 1269             128x8 951 64x4 978 - 1401  128x5 1186 64x2 1295 - 1669
// fp32, BERT-large, capacity 128 / 256 / 512: QKV 128x5 2175 64x2 2086 - 2217, 128x2 2666 - 2601, - 4048 128x2 3924; out
// 64x6 2188 - 2529, 64x4 2665 - 2959, 128x4 4047 - 4191; FFN1 128x4 2177 64x2 2090 - 2293, - 2659, - 4046; FFN2 64x6
// 2183 - 3470, 64x4 2668 - 3833, - 4047 128x6 3237 (384 rows: - 3899, 128x6 2730: its clusters are counted out below).
// fp16: the most CTAs per tile with five 64-wide steps of K each to hide the load latency, or three where the grid
// is small enough (two thirds of the SMs) not to share L2 bandwidth.  Two CTAs fit an SM, but clusters of more
// than two stop finding places on a third more CTAs than SMs, and a short K does not pay for more either.
// The rule goes by capacity; a mostly empty batch pays for CTAs that find no rows.
// The projection in front of the attention gains least: up to one row tile only, three CTAs per tile, none of them with
// less than two steps of K (384, 6 steps: three 432 and 448, persistent 411 and 434).  us per pass at capacity 64 and
// 128 with one / three CTAs / the persistent kernels, by hidden size:
//   512   441 385 401,  481 435 439      640   513 483 481,  496 459 462      768   426 448 454,  447 470 474
//   896   611 569 580,  652 607 603      1024  501 453 474,  572 517 526      1152  629 576 589,  646 598 600
// One CTA without a cluster wins at 768 alone (with a feed-forward width of 2048 too: 393 423 420), by 5 %; why is not
// known, so that line lies between the neighbours that were measured, K = 640 and 896.
// fp32: one CTA fits an SM; among the plans whose clusters all find one the one whose CTA fetches the least, 64
// or 48 KB per 32-wide step, a 128-wide tile's longer reduction counted as another 128 KB.  From six row tiles on a
// third more CTAs than SMs is taken where K is long: a batch has padding, and the tiles it leaves empty cost next
// to nothing (N = 768, K = 3072, capacity 1024: 1591 against 1727; full, the launch alone 44 us against 54).
static SplitPlan gemm_split_plan(int max_m, int n, int k, bool tf32, bool feeds_attention) {
  SplitPlan best;
  if (max_m <= 0) return best;
  const int num_kb = (k + (tf32 ? 31 : 63)) / (tf32 ? 32 : 64);
  const long long m_tiles = (max_m + BM - 1) / BM, sms = sm_count();
  constexpr int kCounts[] = {8, 6, 5, 4, 3, 2};
  if (!tf32) {
    const long long tiles = m_tiles * (n / 64);
    if (n % 64 != 0 || (feeds_attention && m_tiles > 1)) return best;
    if (feeds_attention) {
      if (num_kb < 8) return best;
      if (num_kb > 10 && num_kb <= 12 && 4 * tiles <= sms) best.splits = 1;
      else if (9 * tiles <= 4 * sms) best.splits = 3;
      if (best.splits != 0) return best;
    }
    for (const int splits : kCounts) {
      const int share = num_kb / splits;
      const long long ctas = tiles * splits;
      if (share < 3 || (share < 5 && 3 * ctas > 2 * sms)) continue;
      if (splits == 2 && share >= 12 ? ctas > 2 * sms : 3 * ctas > 4 * sms) continue;
      best.splits = splits;
      return best;
    }
    return best;
  }
  const bool padded = m_tiles >= 6;
  for (const bool second_try : {false, true}) {
    int least = 0;
    for (const int bn : {64, 128}) {
      if (n % bn != 0) continue;
      for (const int splits : kCounts) {
        const int share = (num_kb + splits - 1) / splits;
        const long long ctas = m_tiles * (n / bn) * splits;
        const int most = bn == 64 ? Cfg<true, 64>::kBlocks * Cfg<true, 64>::kUnitKb
                                  : Cfg<true, 128>::kBlocks * Cfg<true, 128>::kUnitKb;  // what TMEM holds
        if (num_kb / splits < 3 || share > most) continue;
        if (second_try) {
          if (!(padded && share >= 24 && 3 * ctas <= 4 * sms)) continue;
        } else {
          // percent of the SMs the clusters of this size can count on
          const int places = splits > 5 ? 66 : splits > 2 ? 88 : bn == 128 ? (padded ? 0 : 66) : 100;
          if (100 * ctas > places * sms) continue;
        }
        const int fetched = bn == 64 ? share * 48 : share * 64 + 128;
        if (best.splits == 0 || fetched < least) best.bn = bn, best.splits = splits, least = fetched;
      }
    }
    if (best.splits != 0) break;
  }
  return best;
}

SplitPlan gemm_route(bool tf32, int rows, int n, int k, int epilogue) {
  // the LayerNorm inside the GEMM kernel is the persistent kernel's
  if (epilogue == kEpiResidualLayerNorm || epilogue == kEpiLayerNorm) return SplitPlan();
  // the QKV projection is the one without activation or residual behind its bias
  return gemm_split_plan(rows, n, k, tf32, !tf32 && (epilogue == kEpiBias || epilogue == kEpiNormIn));
}

cudaError_t launch_gemm_split(const SplitGemm& g, int epilogue, const SplitPlan& plan, TensorMapCache* maps, cudaStream_t stream) {
  const bool tf32 = g.a_lo != nullptr;
  Maps m;
  if (!encode_split(&m.a, tf32, g.a, g.max_m, g.k, BM, maps) || !encode_split(&m.w, tf32, g.w, g.n, g.k, plan.bn, maps))
    return cudaErrorInvalidValue;
  m.a_lo = m.a, m.w_lo = m.w;
  if (tf32 && (!encode_split(&m.a_lo, true, g.a_lo, g.max_m, g.k, BM, maps) ||
               !encode_split(&m.w_lo, true, g.w_lo, g.n, g.k, plan.bn, maps)))
    return cudaErrorInvalidValue;
#define ETB_CASE(TF, E) \
  case E:               \
    return launch_split<TF, E>(m, g, plan, stream)
  if (tf32) {
    switch (epilogue) {
      ETB_CASE(true, kEpiNone);
      ETB_CASE(true, kEpiBias);
      ETB_CASE(true, kEpiBiasGelu);
      ETB_CASE(true, kEpiBiasTanh);
      default:
        return cudaErrorInvalidValue;
    }
  }
  switch (epilogue) {
    ETB_CASE(false, kEpiNone);
    ETB_CASE(false, kEpiBias);
    ETB_CASE(false, kEpiBiasGelu);
    ETB_CASE(false, kEpiBiasTanh);
    ETB_CASE(false, kEpiBiasResidual);
    ETB_CASE(false, kEpiNormIn);
    ETB_CASE(false, kEpiNormInGelu);
    ETB_CASE(false, kEpiNormResidual);
    default:
      return cudaErrorInvalidValue;
  }
#undef ETB_CASE
}

}  // namespace etb
