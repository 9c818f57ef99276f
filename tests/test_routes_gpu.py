"""GPU tests that name the kernel they reach."""
import numpy as np
import pytest
import torch

from effective_transformer_b200 import _capi
from oracle import bert_encoder as O
from routes import SPLIT_ROUTES, route
from test_kernels_gpu import (LONG_LEN_CASES, _deferred_consumer_case, _deferred_producer_case, _gemm_case,
                              _gemm_fused_case, test_gemm_fp32_on_tensor_cores_keeps_fp32_accuracy as fp32_gemm_case)
from util import dev, iptr, lib, ok, status_word, stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,m,cap,n,k,epi,plan", SPLIT_ROUTES)
def test_split_projection_of_every_plan(dtype, m, cap, n, k, epi, plan):
    """Every number of CTAs per tile the rule picks, with the epilogues the layers use."""
    assert route(dtype, cap, n, k, epi) == plan
    if dtype == "fp32":
        fp32_gemm_case(m, cap, n, k, epi)
        return
    if epi == 4:
        _gemm_fused_case(m, cap, n, k, 4)
    else:
        _gemm_case(torch.float16, m, cap, n, k, epi, use_simt=False)
    if n <= 1024:
        assert route(dtype, cap, n, k, 9) == plan
        _deferred_producer_case(m, cap, n, k, True)
    if k <= 1024 and route(dtype, cap, n, k, 8) == plan:
        _deferred_consumer_case(m, cap, n, k, True, True)


@pytest.mark.parametrize("lens", LONG_LEN_CASES)
def test_attention_of_long_sequences_into_a_context_off_the_32_byte_boundary(lens):
    """Such a context is the mma.sync kernel's at any length; an aligned one goes to the tcgen05 kernel."""
    heads, d = 2, 64
    h = heads * d
    lens = np.asarray(lens, np.int32)
    cu = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    t = int(cu[-1])
    qkv = dev(np.random.RandomState(t).randn(t, 3 * h).astype(np.float32), torch.float16)
    buf = torch.full((t * h + 16,), 2.0, dtype=torch.float16, device="cuda")
    assert buf.data_ptr() % 32 == 0
    st = status_word()
    es = qkv.element_size()
    ok(lib().et_attention(_capi.ET_FP16, qkv.data_ptr(), qkv.data_ptr() + h * es, qkv.data_ptr() + 2 * h * es, 3 * h, d,
                          buf.data_ptr() + 16, iptr(dev(cu)), len(lens), int(lens.max()), t, heads, d, 0, iptr(st),
                          stream()))
    torch.cuda.synchronize()
    assert int(st[0]) == 0
    q, k, v = (qkv[:, i * h:(i + 1) * h].double().cpu() for i in range(3))
    ref = O.packed_attention(q, k, v, cu, heads, d)
    torch.testing.assert_close(buf[8:8 + t * h].view(t, h).double().cpu(), ref, rtol=3e-3, atol=3e-3)
    assert torch.all(buf[:8] == 2.0) and torch.all(buf[8 + t * h:] == 2.0)
