"""Rules that every kernel of a pass keeps, checked on its source.

A kernel launched while its predecessors still run (programmatic dependent launch) may not read what they write
through the non-coherent path: ld.global.nc, and const T* __restrict__, which lets the compiler choose it and move
the load in front of griddepcontrol.wait.  No run shows such a load reliably, so the sources are read instead.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "effective_transformer_b200", "csrc")
FILES = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))
# complete before a pass begins: weights and what is worked out from them
CONSTANT = {"bias", "bias_ptr", "gamma", "beta", "word_table", "type_table", "pos_table"}
CONSTANT_VECTOR = re.compile(r"ld_global_nc_v4\((p\b|\(lane < 8 \? nc\.bias_g : nc\.csum_g\)|ln\.gamma|ln\.beta|wrow)")


def kernels(text):
    """(name, parameter list, body) of every __global__ function."""
    for m in re.finditer(r"__global__", text):
        name = re.compile(r"(\w+_kernel)\(").search(text, m.end())
        depth, i = 1, name.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        params = text[name.end():i - 1]
        start = text.index("{", i)
        depth, j = 1, start + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
        yield name.group(1), params, text[start:j]


def read(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_the_parser_sees_the_kernels():
    names = [k for f in FILES for k, _, _ in kernels(read(f))]
    assert {"gemm_split_kernel", "gemm_tcgen05_pair_kernel", "gemm_tf32x3_pair_kernel", "attention_tcgen05_kernel",
            "attention_tcgen05_long_kernel", "restore_padding_kernel", "add_bias_input_layernorm_kernel"} <= set(names)


@pytest.mark.parametrize("name", FILES)
def test_what_an_earlier_kernel_writes_is_read_coherently(name):
    for kernel, params, body in kernels(read(name)):
        if "pdl_wait()" not in body:
            continue  # launched in plain stream order
        restrict = re.findall(r"const\s+[\w:]+\s*\*\s*__restrict__\s+(\w+)", params)
        assert set(restrict) <= CONSTANT, f"{name}: {kernel}: {sorted(set(restrict) - CONSTANT)}"
    text = read(name)
    if "pdl_wait()" in text:
        for call in re.findall(r"ld_global_nc_v4\([^;]*", text):
            # (the standalone bias + transpose kernel is launched in plain stream order)
            assert CONSTANT_VECTOR.match(call) or "srcs[w]" in call, f"{name}: {call}"


def test_ring_commits_are_waited_for_before_the_barriers_go_away():
    """tcgen05.commit arrives on a barrier asynchronously, in the CTA-pair kernels on the peer's.  A kernel that frees
    its ring with such arrivals outstanding could have them land in another CTA's shared memory: the producer waits
    for its stages once inside the loop and once behind it."""
    seen = 0
    for name in FILES:
        for kernel, _, body in kernels(read(name)):
            if re.search(r"umma_commit(_pair)?\(empty_bar", body):
                seen += 1
                assert body.count("mbar_wait(empty_bar(") == 2, f"{name}: {kernel}"
    assert seen == 5


def test_what_is_in_flight_lands_even_when_a_role_has_given_up():
    """mbar_wait returns at once behind the abort flag, so it cannot be the wait that keeps shared memory and TMEM
    until copies and MMAs in flight have landed."""
    for name in FILES:
        text = read(name)
        for site in re.findall(r"if \(!(mbar_\w+)\((full_bar|drain_bar)[^;]*?fail\(kSite\w*Drain\)", text):
            assert site[0] == "mbar_drain", f"{name}: {site}"
    attention = dict((k, b) for k, _, b in kernels(read("attention_tcgen05.cu")))
    for kernel in ("attention_tcgen05_kernel", "attention_tcgen05_long_kernel"):
        body = attention[kernel]
        assert "drain_attention(bar_qk, qk_issued, bar_v, v_issued, bar_mma, mma_issued)" in body
        assert body.count("umma_commit(bar_mma);") == body.count("++mma_issued;") == 2


def test_only_a_ready_row_count_is_read_in_front_of_the_wait():
    """The row count may come in under the wait where the launch says so (GemmHints); otherwise a kernel reads nothing
    that a kernel of the pass writes in front of its first wait."""
    with open(os.path.join(CSRC, "common.cuh")) as f:
        helper = re.search(r"int pdl_wait_row_count\(.*?\n\}", f.read(), re.S).group(0)
    load = r"v = ld_\w+\(p\);"
    assert re.search(rf"if \(ready != 0\) {load}\s*pdl_wait\(\);\s*if \(ready == 0\) {load}", helper)
    for name in FILES:
        for kernel, params, body in kernels(read(name)):
            if "pdl_wait" not in body:
                continue
            front = body[:body.index("pdl_wait")]
            # (a lambda that loads is called behind the wait in gemm_split.cu; producers and epilogues wait themselves)
            front = re.sub(r"auto valid_rows = .*?\n  \};", "", front, flags=re.S)
            assert not re.search(r"\*m_ptr|\*t_ptr|\*rows_ptr|cu_seqlens\[|plan\[|ld_l2_s32|ld_row_count|ld_activation", front), \
                f"{name}: {kernel}"
