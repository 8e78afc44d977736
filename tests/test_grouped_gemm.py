"""The tcgen05 grouped GEMM at the sizes where it can go wrong, against the oracle: every format, one and two activation rows per
token, one token, tiles of one column more or less than a block of 16 and than a full tile (the shared expert's tiles hold T
tokens), several tiles per expert. Needs a B200."""
import numpy as np
import pytest
import torch

import moe_b200 as m
from oracle import oracle as o
from parity import check_ffn

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("lib_built")]
DEV, E, K = "cuda:0", 32, 8


@pytest.mark.parametrize("fmt", [m.FMT_SYM_F16, m.FMT_SYM_F32, m.FMT_ZP])
@pytest.mark.parametrize("block", [False, True])
def test_grouped_gemm_edges(fmt, block):
    c = m.Context(0, max_tokens=300, max_experts=E, top_k=K)
    c.set_prefill_min_tokens(1)
    L = m.Layer(c, fmt, E)
    L.fill_synth(3, 0)
    rng = np.random.default_rng(5)
    W = (rng.standard_normal((E + 1, 2048)) * 0.02).astype(np.float32)
    L.set_router(W)
    host = [m.synth_expert_host(fmt, 3, 0, e) for e in range(E + 1)]
    try:
        for T in (1, 15, 17, 48, 49, 80, 81, 300):
            X = torch.from_numpy(rng.standard_normal((T, 2048)).astype(np.float32))
            for x in (X, X.to(torch.bfloat16)):
                idx = torch.empty(T, K, dtype=torch.int32, device=DEV)
                xf = x.float().numpy()
                got = L.forward(x.to(DEV), T, K, idx=idx, flags=2 if block else 0).cpu().numpy()
                assert c.status() == 0
                ref, ri, _, _ = o.layer_forward(fmt, host, W, o.rmsnorm(xf) if block else xf, K)
                assert np.array_equal(idx.cpu().numpy(), ri)
                check_ffn(got, xf + ref if block else ref, fmt, f"grouped GEMM T={T} {x.dtype} block={block}")
    finally:
        L.close(); c.close()


@pytest.mark.parametrize("fmt", [m.FMT_SYM_F16, m.FMT_ZP])
def test_a_threshold_of_any_size_keeps_batches_on_the_streaming_kernels(fmt):
    """Thresholds whose third, rounded up, would pass the largest int: the outputs are those of the streaming kernels bit for bit. (The
    grouped GEMM adds the products of a group in another order, so its outputs differ somewhere; that is checked first.)"""
    T = 40
    c = m.Context(0, max_tokens=T, max_experts=E, top_k=K)
    L = m.Layer(c, fmt, E)
    L.fill_synth(3, 0)
    rng = np.random.default_rng(7)
    L.set_router((rng.standard_normal((E + 1, 2048)) * 0.02).astype(np.float32))
    X = torch.from_numpy(rng.standard_normal((T, 2048)).astype(np.float32)).to(DEV)
    try:
        streaming = L.forward(X, T, K).clone()   # 40 tokens: below the default threshold of either format
        c.set_prefill_min_tokens(1)
        assert not torch.equal(L.forward(X, T, K), streaming)
        for tokens in (2**31 - 1, 2**31 - 2, 2**31 - 3, 3 * T + 1):
            c.set_prefill_min_tokens(tokens)
            assert torch.equal(L.forward(X, T, K), streaming), tokens
        for tokens in (3 * T, 3 * T - 2) if fmt == m.FMT_ZP else (T,):   # the smallest batch that the grouped GEMM takes
            c.set_prefill_min_tokens(tokens)
            assert not torch.equal(L.forward(X, T, K), streaming), tokens
        assert c.status() == 0
    finally:
        L.close(); c.close()


@pytest.mark.parametrize("fmt", [m.FMT_SYM_F16, m.FMT_SYM_F32, m.FMT_ZP])
@pytest.mark.parametrize("x_type", [torch.float32, torch.bfloat16])
def test_grouped_gemm_repeats_bit_for_bit(fmt, x_type):
    """Tiles of 6 to 30 tokens over every expert, with two activation rows a token and, of bf16 tokens, one, where the weight ring turns over
    as fast as it can. The streaming kernels' results within the bars, and a pair's result does not depend on its place in a tile, so
    every run gives the same bits; weights that are overwritten before they are read do not."""
    T, E = 512, 256
    c = m.Context(0, max_tokens=T, max_experts=E, top_k=K)
    L = m.Layer(c, fmt, E)
    L.fill_synth(3, 0)
    rng = np.random.default_rng(11)
    L.set_router((rng.standard_normal((E + 1, 2048)) * 0.02).astype(np.float32))
    X = torch.from_numpy(rng.standard_normal((T, 2048)).astype(np.float32)).to(DEV).to(x_type)
    try:
        c.set_prefill_min_tokens(1 << 20)
        want = L.forward(X, T, K).cpu().numpy()
        c.set_prefill_min_tokens(1)
        first = L.forward(X, T, K).clone()
        check_ffn(first.cpu().numpy(), want, fmt, f"grouped GEMM against the streaming kernels, {T} {x_type} tokens")
        for _ in range(40):
            assert torch.equal(L.forward(X, T, K), first)
        assert c.status() == 0
    finally:
        L.close(); c.close()


def test_the_branch_free_silu_is_the_division():
    """Every float gate value, the infinities, NaN and the quotients near the end of the range among them: the bits of CUDA's correctly
    rounded division, but for the sign of zero."""
    c = m.Context(0, max_tokens=1, max_experts=E, top_k=K)
    try:
        assert c.selftest_swiglu() == (0, 0, 0)
    finally:
        c.close()


def test_an_overflowed_gate_row_marks_its_tokens():
    """One gate row of an expert overflows to +inf or -inf: silu of either is no finite number, so every token that selected the expert
    has an output of none, as in the oracle and on the streaming kernels; the other tokens' outputs are those without the overflow."""
    T, fmt = 40, m.FMT_SYM_F32
    c = m.Context(0, max_tokens=T, max_experts=E, top_k=K)
    L = m.Layer(c, fmt, E)
    L.fill_synth(3, 0)
    rng = np.random.default_rng(23)
    W = (rng.standard_normal((E + 1, 2048)) * 0.02).astype(np.float32)
    L.set_router(W)
    host = [m.synth_expert_host(fmt, 3, 0, e) for e in range(E + 1)]
    X = rng.standard_normal((T, 2048)).astype(np.float32)
    idx = torch.empty(T, K, dtype=torch.int32, device=DEV)
    x = torch.from_numpy(X).to(DEV)
    try:
        c.set_prefill_min_tokens(1)
        want = L.forward(x, T, K, idx=idx).cpu().numpy()
        expert = int(np.bincount(idx.cpu().numpy().ravel(), minlength=E).argmax())
        hit = (idx.cpu().numpy() == expert).any(axis=1)
        row, group = 100, 5   # the scale of 64 inputs of one gate row: 32 groups a row
        blob = host[expert].copy()
        blob[m.Q_BYTES + (row * 32 + group) * 4:][:4] = np.frombuffer(np.float32(3e38).tobytes(), np.uint8)
        host[expert] = blob
        L.upload_blob(expert, blob)
        with np.errstate(all="ignore"):
            ref, _, _, _ = o.layer_forward(fmt, host, W, X, K)
            assert np.array_equal(~np.isfinite(ref).all(axis=1), hit) and 0 < hit.sum() < T
            for min_tokens in (1, 1 << 20):   # the grouped GEMM, the streaming kernels
                c.set_prefill_min_tokens(min_tokens)
                got = L.forward(x, T, K).cpu().numpy()
                assert np.array_equal(~np.isfinite(got).any(axis=1), hit), min_tokens
                if min_tokens == 1:
                    assert np.array_equal(got[~hit], want[~hit])
        assert c.status() == 0
    finally:
        L.close(); c.close()
