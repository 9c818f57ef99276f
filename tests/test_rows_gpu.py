"""GPU tests that look at every row of a whole pass.

A mean over a batch hides one wrong row, and a wrong row of an early layer is diluted by the later ones; so the
largest relative error of any row is taken, on batches whose contents change from call to call.
"""
import ctypes as C

import numpy as np
import pytest
import torch

import effective_transformer_b200 as et
from effective_transformer_b200 import _capi
from effective_transformer_b200 import workloads as W

pytestmark = pytest.mark.gpu

LARGE = dict(heads=16, ffn=4096)


def make_weights(layers, h, ffn, seed=1):
    """Sixteen tensors per layer, fp16 values whatever the handle; gamma around one, beta around zero."""
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape):
        return (0.02 * torch.randn(*shape, generator=gen, device="cuda")).half()

    for _ in range(layers):
        w = [normal(h, h) if i % 2 == 0 else normal(h) for i in range(8)]
        yield w + [normal(h), 1 + 5 * normal(h), normal(h, ffn), normal(ffn), normal(ffn, h), normal(h), normal(h),
                   1 + 5 * normal(h)]


def make_engine(layers, batch, seq, heads, ffn, dtype=torch.float16, seed=1):
    h = heads * 64
    eng = et.EffectiveTransformer(layers, heads, 64, ffn, batch, seq, dtype=dtype)
    for layer, w in enumerate(make_weights(layers, h, ffn, seed)):
        eng.set_layer_weights(layer, [t.to(dtype).cpu() for t in w])
    return eng


# An fp16 row differs from the fp32 stack's by the roundings of its way: two stored sums per layer of relative error
# 2^-11 / sqrt(3), 48 of them at random add up to 2e-3; seen 1.3e-3 (a sequence of one token 3.7e-3) and 0.015 of the
# RMS in the worst single value.  One wrong 64-column piece of one row is 1/16 of its energy: 0.25.
ROW_BOUND, VALUE_BOUND = 8e-3, 0.04


@pytest.mark.parametrize("layers,heads,ffn", [(24, 16, 4096), (12, 12, 3072)], ids=["large", "base"])
def test_every_row_of_batches_whose_contents_change(layers, heads, ffn):
    """Batches of 60 to 4000 positions, short ragged sequences: every number of CTAs per tile, the split and the
    persistent kernels in turn.  Two batches of one shape alternate back to back (a count, a plan or a row left over
    from the batch before would show), and each row is held against the fp32 handle's."""
    h, cap_batch, cap_seq = heads * 64, 256, 64
    eng = make_engine(layers, cap_batch, cap_seq, heads, ffn)
    exact = make_engine(layers, cap_batch, cap_seq, heads, ffn, dtype=torch.float32)
    rng = np.random.RandomState(heads)
    for trial in range(24):
        seq = int(rng.choice([16, 20, 31, 32, 53, 64]))
        batch = max(1, min(cap_batch, int(np.exp(rng.uniform(np.log(60), np.log(4000)))) // seq))
        pair = []
        for _ in range(2):
            lens = rng.randint(1, seq + 1, size=batch).astype(np.int32)
            mask = torch.from_numpy(W.prefix_mask(lens, seq)).cuda()
            x = torch.from_numpy(rng.randn(batch, seq, h).astype(np.float16)).cuda()
            pair.append((x, mask, eng.forward(x, mask)))
            torch.cuda.synchronize()
        outs = [torch.empty_like(pair[0][0]) for _ in range(6)]
        for i, out in enumerate(outs):
            eng.forward(pair[i % 2][0], pair[i % 2][1], out)
        torch.cuda.synchronize()
        for i, out in enumerate(outs):
            assert torch.equal(out, pair[i % 2][2]), f"trial {trial}, {batch} x {seq}, pass {i}"
        x, mask, got = pair[1]
        rows = mask.bool()
        want = exact.forward(x.float(), mask)[rows]
        diff = got[rows].float() - want
        err = diff.norm(dim=1) / want.norm(dim=1)
        assert float(err.max()) < ROW_BOUND, f"{batch} x {seq}: row {int(err.argmax())} off by {float(err.max())}"
        assert float(diff.abs().max() / want.pow(2).mean().sqrt()) < VALUE_BOUND, f"{batch} x {seq}"
    assert eng.device_status() == 0
    eng.close()
    exact.close()


@pytest.mark.parametrize("dtype,seq", [("fp16", 32), ("fp16", 144), ("fp32", 16)])
def test_host_call_rows_do_not_depend_on_the_chunk_shares(monkeypatch, dtype, seq):
    """The shares follow measured times.  Chunks of a few hundred positions would run other GEMM kernels than the
    whole batch; they are held to the whole batch's.  Lengths are multiples of 16, so that a sequence meets the
    attention's 16-key steps alike wherever it stands in a tile: the rows are the same bits, whatever the shares."""
    layers, tdt = 4, torch.float16 if dtype == "fp16" else torch.float32
    batch = 6400 // seq
    rng = np.random.RandomState(seq)
    lens = (16 * rng.randint(1, seq // 16 + 1, size=batch)).astype(np.int32)
    mask = W.prefix_mask(lens, seq)
    x = rng.randn(batch, seq, 1024).astype(np.float16 if dtype == "fp16" else np.float32)
    monkeypatch.setenv("ETB_HOST_CHUNKS", "3")
    want = None
    for share in ("6", "1", "16"):
        monkeypatch.setenv("ETB_HOST_MID_SHARE", share)
        eng = make_engine(layers, batch, seq, dtype=tdt, **LARGE)
        if want is None:
            want = eng.forward(torch.from_numpy(x).cuda(), torch.from_numpy(mask).cuda()).cpu().numpy()
        for call in range(3):  # eager, eager and recorded, replayed
            got, tokens = eng.forward_host(x, mask)
            assert tokens == int(lens.sum())
            rows = np.flatnonzero((got != want).reshape(batch * seq, -1).any(axis=1))
            assert rows.size == 0, f"share {share}, call {call}: {rows.size} rows differ, the first is {rows[0]}"
        assert eng.device_status() == 0
        eng.close()


@pytest.mark.parametrize("heads,ffn", [(4, 1024), (12, 3072)])
def test_weights_given_to_the_layer_op_reach_whole_stack_calls(heads, ffn):
    """A layer op that brings its own weights replaces the handle's.  The whole-stack calls run on weights with the
    LayerNorms folded in: those have to follow, in passes recorded before as well, and also when only one layer of
    the stack is replaced."""
    layers, batch, seq, h = 3, 5, 24, heads * 64
    rng = np.random.RandomState(3)
    mask = torch.from_numpy(W.prefix_mask(rng.randint(1, seq + 1, size=batch).astype(np.int32), seq)).cuda()
    x = torch.from_numpy(rng.randn(batch, seq, h).astype(np.float16)).cuda()
    old, new = list(make_weights(layers, h, ffn, 1)), list(make_weights(layers, h, ffn, 2))

    def engine(weights):
        eng = et.EffectiveTransformer(layers, heads, 64, ffn, batch, seq, dtype=torch.float16)
        for layer, w in enumerate(weights):
            eng.set_layer_weights(layer, [t.cpu() for t in w])
        return eng

    def layer_op(eng, layer, w, packed, count, batch_idx, word_idx):
        out = torch.empty_like(packed)
        names = ["attr_kernel_Q", "attr_bias_Q", "attr_kernel_K", "attr_bias_K", "attr_kernel_V", "attr_bias_V",
                 "attr_output_kernel", "attr_output_bias", "attr_output_layernorm_beta", "attr_output_layernorm_gamma",
                 "inter_kernel", "inter_bias", "output_kernel", "output_bias", "output_layernorm_beta",
                 "output_layernorm_gamma"]
        p = _capi.EncoderParam()
        for name, t in zip(names, w):
            setattr(p, name, t.data_ptr())
        p.from_tensor, p.to_tensor, p.transformer_out = packed.data_ptr(), packed.data_ptr(), out.data_ptr()
        p.batch_idx, p.word_idx = batch_idx.data_ptr(), word_idx.data_ptr()
        p.valid_word_num, p.stream = count.data_ptr(), torch.cuda.current_stream().cuda_stream
        tp = _capi.TransformerParam(batch, seq, seq, heads, 64)
        _capi.check(_capi.load().et_layer(eng._h, layer, C.byref(p), C.byref(tp)), eng._h)
        return out

    fresh = engine(new)
    mixed = engine([old[0], new[1], old[2]])
    want_new, want_mixed = fresh.forward(x, mask), mixed.forward(x, mask)
    eng = engine(old)
    out = torch.empty_like(x)
    eng.capture(x, mask, out)
    packed = eng.effective_transformer_input(x, mask)
    layer_op(eng, 1, new[1], *packed)
    assert torch.equal(eng.forward(x, mask), want_mixed)
    eng.replay()
    assert torch.equal(out, want_mixed)
    for layer in (0, 2):
        layer_op(eng, layer, new[layer], *packed)
    assert torch.equal(eng.forward(x, mask), want_new)
    eng.replay()
    assert torch.equal(out, want_new)
    for e in (fresh, mixed, eng):
        e.close()


@pytest.mark.parametrize("batch", [8190, 8191, 8192, 8193])
def test_attention_plan_of_thousands_of_short_sequences(batch):
    """Up to 8192 sequences the boundaries and the packing chain are kept in shared memory (from 8191 on more of it
    than a kernel has without asking); beyond, in global memory."""
    seq, heads = 2, 2
    lens = np.random.RandomState(batch).randint(0, seq + 1, size=batch).astype(np.int32)
    lens[0], lens[-1] = 0, 1
    mask = torch.from_numpy(W.prefix_mask(lens, seq)).cuda()
    gen = torch.Generator(device="cuda").manual_seed(batch)
    x = torch.randn(batch, seq, heads * 64, device="cuda", dtype=torch.float16, generator=gen)
    eng = make_engine(1, batch, seq, heads, 256)
    exact = make_engine(1, batch, seq, heads, 256, dtype=torch.float32)
    got = eng.forward(x, mask)
    ops = et.get_sequence_output(et.BertConfig(heads * 64, 1, heads, 256), batch, seq, None, mask, x, None, engine=eng)
    want = exact.forward(x.float(), mask)
    rows = mask.bool()
    for y in (got, ops):
        err = (y.float() - want)[rows].norm(dim=1) / want[rows].norm(dim=1)
        assert float(err.max()) < 4e-3  # one layer of fp16 roundings (2^-11 each) on rows of LayerNorm outputs
        assert not y[~rows].any()
    assert eng.device_status() == 0
    eng.close()
    exact.close()


def test_no_workspace_is_held_for_general_masks():
    """The bits of a general mask lie in a buffer that only the host-buffer calls use otherwise: a handle pays
    nothing for them, and the two kinds of calls on one handle do not disturb each other."""
    batch, seq, heads, ffn = 24, 40, 4, 1024
    h = heads * 64
    eng = make_engine(2, batch, seq, heads, ffn)
    per_position = (eng.workspace_bytes(batch, 128 * seq) - eng.workspace_bytes(batch, 64 * seq)) / (batch * 64 * seq)
    activations = 2 * (8 * h + ffn)             # x, qkv, ctx, att, two staging buffers; ffn
    indices = 4 * 10                            # masks, ids, types, four index arrays, two plan labels, position rows
    statistics = 2 * 8 * (h // 64) + 0.125      # deferred LayerNorm; row counters
    assert per_position <= activations + indices + statistics + 1
    rng = np.random.RandomState(4)
    lens = rng.randint(1, seq + 1, size=batch).astype(np.int32)
    mask_np = W.prefix_mask(lens, seq)
    x_np = rng.randn(batch, seq, h).astype(np.float16)
    x, mask = torch.from_numpy(x_np).cuda(), torch.from_numpy(mask_np).cuda()
    causal = torch.tril(torch.ones(batch, seq, seq, device="cuda", dtype=torch.float16))
    masked, plain = eng.forward_general_mask(x, mask, causal).clone(), eng.forward(x, mask).cpu().numpy()
    for _ in range(3):
        got, _ = eng.forward_host(x_np, mask_np)
        assert np.array_equal(got, plain)
        again = eng.forward_general_mask(x, mask, causal)
        torch.cuda.synchronize()  # (a host call runs on the handle's own stream)
        assert torch.equal(again, masked)
    eng.close()
