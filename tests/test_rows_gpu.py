"""GPU tests that look at every row of a whole pass.

A mean over a batch hides one wrong row, and a wrong row of an early layer is diluted by the later ones; so the
largest relative error of any row is taken, on batches whose contents change from call to call.
"""
import numpy as np
import pytest
import torch

import effective_transformer_b200 as et
from effective_transformer_b200 import workloads as W

pytestmark = pytest.mark.gpu

LARGE = dict(heads=16, ffn=4096)


def make_engine(layers, batch, seq, heads, ffn, dtype=torch.float16, seed=1):
    h = heads * 64
    eng = et.EffectiveTransformer(layers, heads, 64, ffn, batch, seq, dtype=dtype)
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, scale=0.02):  # fp16 values in every handle
        return (scale * torch.randn(*shape, generator=gen, device="cuda")).half()

    for layer in range(layers):
        w = [normal(h, h) if i % 2 == 0 else normal(h) for i in range(8)]
        w += [normal(h), 1 + normal(h), normal(h, ffn), normal(ffn), normal(ffn, h), normal(h), normal(h), 1 + normal(h)]
        eng.set_layer_weights(layer, [t.to(dtype).cpu() for t in w])
    return eng


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
