"""The work that users of this framework have it do, as cases that can be timed.

A case is one call (or one short sequence of calls) of the public API on one batch: BERT-base or
BERT-large encoder stacks, fp16 and fp32 handles, from a single request to the largest batch of the
benchmark configurations (effective_transformer_b200/workloads.py).  Calls that appear:

  forward   EffectiveTransformer.forward            device tensors in, device tensors out
  replay    EffectiveTransformer.replay             the same pass recorded once on fixed buffers
  ops       get_sequence_output(..., engine=...)    the reference's wiring: input op, N layer ops, output op
  mask      EffectiveTransformer.forward_general_mask   causal attention on top of the padding mask
  host      EffectiveTransformer.forward_host       host arrays in and out (pinned buffers)
  ids_host  EffectiveTransformer.forward_ids_host   token ids on the host -> pooled rows on the host

Inputs follow the benchmark's recipe: N(0,1) activations, 0.02 * N(0,1) weights and biases, LayerNorm
gamma = 1 and beta = 0, lengths drawn uniformly between two bounds ("skewed": 90 % short sequences and
10 % long ones), a prefix mask.  Everything is drawn on the GPU from the seed.
"""
import math

import torch

import effective_transformer_b200 as et

BASE = {"layers": 12, "heads": 12, "ffn": 3072}
LARGE = {"layers": 24, "heads": 16, "ffn": 4096}
VOCAB, TYPES, POSITIONS = 30522, 2, 512


def _case(name, api, dtype, model, batch, seq, low, high, skewed=False):
    return dict(name=name, api=api, dtype=dtype, batch=batch, seq=seq, low=low, high=high, skewed=skewed, **model)


def listed():
    return [
        # one request at a time: a query of a search or chat front end, no batching, latency counts
        _case("request_fp16_b1_s64", "forward", "fp16", BASE, 1, 64, 8, 64),
        # a small dynamic batch of an online service that records its pass once and replays it
        _case("online_replay_fp16_b8_s64", "replay", "fp16", BASE, 8, 64, 16, 64),
        # a causal (decoder-style) encoder on an odd-sized ragged batch: the general-mask option
        _case("causal_fp16_b37_s53", "mask", "fp16", BASE, 37, 53, 1, 53),
        # benchmark configuration 0: a small fp32 batch, for users who need fp32 results
        _case("base_fp32_b8_s32", "forward", "fp32", BASE, 8, 32, 8, 32),
        # benchmark configuration 1 through the op-by-op API, the wiring a user of the reference has
        _case("ops_fp16_b100_s32", "ops", "fp16", BASE, 100, 32, 8, 32),
        # one rank's eighth of benchmark configuration 2, replayed: what every GPU of an 8-GPU box runs
        _case("shard_replay_fp16_b125_s64", "replay", "fp16", BASE, 125, 64, 16, 64),
        # benchmark configuration 2, the headline: offline / high-throughput scoring
        _case("base_fp16_b1000_s64", "forward", "fp16", BASE, 1000, 64, 16, 64),
        # benchmark configuration 3: the large fp32 batch
        _case("base_fp32_b500_s64", "forward", "fp32", BASE, 500, 64, 16, 64),
        # benchmark configuration 4: BERT-large on skewed lengths, the largest batch
        _case("large_fp16_b4096_s128", "forward", "fp16", LARGE, 4096, 128, 1, 128, skewed=True),
        # documents: sequences up to BERT's 512 positions
        _case("long_fp16_b32_s512", "forward", "fp16", BASE, 32, 512, 64, 512),
        # classification service: token ids arrive on the host, pooled rows go back
        _case("classify_host_fp16_b64_s128", "ids_host", "fp16", BASE, 64, 128, 16, 128),
        # the headline batch end to end with host buffers
        _case("host_fp16_b1000_s64", "host", "fp16", BASE, 1000, 64, 16, 64),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """One more case: any of the calls, both types and models, 1 to 4096 sequences of up to 512 positions, at
    most as many positions (and as much arithmetic) as the largest listed case of the same kind."""
    api = rng.choice(["forward", "forward", "replay", "ops", "mask", "host", "ids_host"])
    dtype = "fp32" if api in ("forward", "replay", "ops") and rng.random() < 0.3 else "fp16"
    model = LARGE if rng.random() < 0.25 else BASE
    # a general mask is [B, S, S]: short sequences; half of the rest up to 128 positions, as most requests are
    seq = _log_int(rng, 16, 128) if api == "mask" or rng.random() < 0.6 else _log_int(rng, 96, 512)
    positions = 32000 if dtype == "fp32" or api == "mask" else 64000
    if model is LARGE:
        positions //= 4
    batch = _log_int(rng, 1, max(2, min(2048, positions // seq)))
    skewed = seq >= 64 and batch >= 16 and rng.random() < 0.3
    low = 1 if skewed else rng.choice([1, max(1, seq // 4), max(1, seq // 2)])
    return dict(api=api, dtype=dtype, batch=batch, seq=seq, low=low, high=seq, skewed=skewed, **model)


def _hidden(case):
    return case["heads"] * 64


def _lengths(case, gen):
    b, low, high = case["batch"], case["low"], case["high"]
    u = torch.rand(b, generator=gen, device="cuda")
    if not case["skewed"]:
        return (low + (u * (high - low + 1)).floor()).clamp(low, high).to(torch.int32)
    # 90 % in [1, S/8], 10 % in [0.78 S, S] (configuration 4: 1..16 and 100..128)
    s = case["seq"]
    short, long_low = s // 8, int(0.78 * s)
    is_long = torch.rand(b, generator=gen, device="cuda") < 0.10
    long_ = (long_low + (u * (s - long_low + 1)).floor()).clamp(max=s)
    return torch.where(is_long, long_, (1 + (u * short).floor()).clamp(max=short)).to(torch.int32)


def _expected(case):
    """Expected number of valid tokens and expected sum of squared lengths of a batch."""

    def uniform(a, b):
        return (a + b) / 2, (2 * b * b + 2 * a * b + 2 * a * a + b - a) / 6

    b, s = case["batch"], case["seq"]
    if case["skewed"]:
        m1, q1 = uniform(1, s // 8)
        m2, q2 = uniform(int(0.78 * s), s)
        return b * (0.9 * m1 + 0.1 * m2), b * (0.9 * q1 + 0.1 * q2)
    m, q = uniform(case["low"], case["high"])
    return b * m, b * q


def prepare(case, seed):
    h, f, b, s = _hidden(case), case["ffn"], case["batch"], case["seq"]
    dtype = torch.float16 if case["dtype"] == "fp16" else torch.float32
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, scale=1.0):
        return (scale * torch.randn(*shape, generator=gen, device="cuda")).to(dtype)

    engine = et.EffectiveTransformer(case["layers"], case["heads"], 64, f, b, s, dtype=dtype)
    zeros, ones = torch.zeros(h, dtype=dtype), torch.ones(h, dtype=dtype)
    for layer in range(case["layers"]):
        kernels = normal(4 * h * h + 2 * h * f, scale=0.02).cpu()
        biases = normal(5 * h + f, scale=0.02).cpu()
        k = [kernels[i * h * h:(i + 1) * h * h].view(h, h) for i in range(4)]
        k1 = kernels[4 * h * h:4 * h * h + h * f].view(h, f)
        k2 = kernels[4 * h * h + h * f:].view(f, h)
        v = [biases[i * h:(i + 1) * h] for i in range(5)]
        engine.set_layer_weights(layer, [k[0], v[0], k[1], v[1], k[2], v[2], k[3], v[3], zeros, ones,
                                         k1, biases[5 * h:], k2, v[4], zeros, ones])
    lengths = _lengths(case, gen)
    mask = (torch.arange(s, device="cuda", dtype=torch.int32)[None, :] < lengths[:, None]).to(torch.int32)
    state = {"api": case["api"], "engine": engine, "mask": mask}
    if case["api"] == "ids_host":
        engine.set_embeddings(normal(VOCAB, h, scale=0.02), normal(TYPES, h, scale=0.02),
                              normal(POSITIONS, h, scale=0.02), torch.ones(h), torch.zeros(h))
        engine.set_pooler(normal(h, h, scale=0.02), normal(h, scale=0.02))
        ids = torch.randint(0, VOCAB, (b, s), generator=gen, device="cuda", dtype=torch.int32)
        split = (torch.rand(b, generator=gen, device="cuda") * (lengths + 1)).to(torch.int32)
        types = (torch.arange(s, device="cuda", dtype=torch.int32)[None, :] >= split[:, None]).to(torch.int32)
        state.update(ids=ids.cpu().numpy(), types=types.cpu().numpy(), mask=mask.cpu().numpy())
        return state
    x = normal(b, s, h)
    if case["api"] == "host":
        pin = lambda t: t.cpu().pin_memory().numpy()  # noqa: E731
        state.update(x=pin(x), mask=pin(mask), out=torch.empty(b, s, h, dtype=dtype).pin_memory().numpy())
        return state
    state.update(x=x, out=torch.empty_like(x))
    if case["api"] == "replay":
        engine.capture(x, mask, state["out"])
    elif case["api"] == "mask":
        causal = torch.tril(torch.ones(s, s, device="cuda", dtype=dtype))
        state["attention_mask"] = (mask[:, None, :].to(dtype) * causal[None]).contiguous()
    elif case["api"] == "ops":
        state["config"] = et.BertConfig(hidden_size=h, num_hidden_layers=case["layers"],
                                        num_attention_heads=case["heads"], intermediate_size=f)
    return state


def run(state):
    api, engine = state["api"], state["engine"]
    if api == "forward":
        return engine.forward(state["x"], state["mask"], state["out"])
    if api == "replay":
        engine.replay()
        return state["out"]
    if api == "ops":
        b, s, _ = state["x"].shape
        return et.get_sequence_output(state["config"], b, s, None, state["mask"], state["x"], None, engine=engine)
    if api == "mask":
        return engine.forward_general_mask(state["x"], state["mask"], state["attention_mask"], state["out"])
    if api == "host":
        out, tokens = engine.forward_host(state["x"], state["mask"], state["out"])
        return {"sequence": out, "tokens": tokens}
    _, pooled, tokens = engine.forward_ids_host(state["ids"], state["mask"], state["types"], sequence_output=False,
                                                pooled_output=True)
    return {"pooled": pooled, "tokens": tokens}


def work(case):
    """Weights read once, the valid input rows read, the padded output written, the mask (and ids) read; the
    projections' and the attention's arithmetic on valid tokens."""
    h, f, n, b, s = _hidden(case), case["ffn"], case["layers"], case["batch"], case["seq"]
    e = 2 if case["dtype"] == "fp16" else 4
    tokens, squares = _expected(case)
    weights = n * (4 * h * h + 2 * h * f + 9 * h + f) * e
    moved = weights + 4 * b * s
    if case["api"] == "ids_host":
        moved += tokens * (8 + h * e) + (POSITIONS + TYPES) * h * e + h * h * e + b * h * e
    else:
        moved += tokens * h * e + b * s * h * e
    if case["api"] == "mask":
        moved += b * s * s * e
    flops = n * (2 * tokens * h * (4 * h + 2 * f) + 4 * h * squares)
    if case["api"] == "ids_host":
        flops += 2 * b * h * h
    return {"bytes": float(moved), "flops": float(flops)}


def tolerance(case):
    """About four times what two correct paths of the same precision were seen to differ by: the default fp16 path
    against the one with LayerNorm kernels and against the CUDA-core path 1.9e-3 in norm and up to 0.017 of the RMS
    after 12 layers, 2.3e-3 and 0.035 after 24; the fp32 path against fp32 FMA arithmetic 4.3e-6 and 3.2e-5."""
    if case["dtype"] == "fp16":
        return {"rel": 7.5e-3, "max": 0.07} if case["layers"] <= 12 else {"rel": 9e-3, "max": 0.14}
    return {"rel": 1.6e-5, "max": 1.3e-4}
