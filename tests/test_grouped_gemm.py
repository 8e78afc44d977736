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
def test_grouped_gemm_repeats_bit_for_bit(fmt):
    """Tiles of 6 to 30 tokens over every expert: the weight ring turns over as fast as it can. A pair's result does not depend on its
    place in a tile, so every run gives the same bits; weights that are overwritten before they are read do not."""
    T, E = 512, 256
    c = m.Context(0, max_tokens=T, max_experts=E, top_k=K)
    c.set_prefill_min_tokens(1)
    L = m.Layer(c, fmt, E)
    L.fill_synth(3, 0)
    rng = np.random.default_rng(11)
    L.set_router((rng.standard_normal((E + 1, 2048)) * 0.02).astype(np.float32))
    X = torch.from_numpy(rng.standard_normal((T, 2048)).astype(np.float32)).to(DEV)
    try:
        first = L.forward(X, T, K).clone()
        for _ in range(40):
            assert torch.equal(L.forward(X, T, K), first)
        assert c.status() == 0
    finally:
        L.close(); c.close()
