"""Activation rows that do not begin on a 16-byte boundary, as a view into a larger buffer gives them: the calls take them and give the
results of aligned rows bit for bit. Needs a B200."""
import numpy as np
import pytest
import torch

import moe_b200 as m

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("lib_built")]
DEV, E, K = "cuda:0", 32, 8


def shifted(x, elements):
    """The same values, `elements` places behind an aligned address."""
    buf = torch.empty(x.numel() + elements, device=x.device, dtype=x.dtype)
    view = buf[elements:].view(x.shape)
    view.copy_(x)
    assert view.data_ptr() % 16 == elements * x.element_size() % 16
    return view


@pytest.fixture(scope="module")
def blobs():
    """A context and a layer of every format in the reference layout."""
    c = m.Context(0, max_tokens=16, max_experts=E, top_k=K)
    layers = {}
    for fmt in (m.FMT_SYM_F16, m.FMT_SYM_F32, m.FMT_ZP):
        layers[fmt] = m.Layer(c, fmt, E, layout=m.LAYOUT_REFERENCE)
        layers[fmt].fill_synth(6, 0)
    yield c, layers
    for L in layers.values():
        L.close()
    c.close()


@pytest.mark.parametrize("fmt", [m.FMT_SYM_F16, m.FMT_SYM_F32, m.FMT_ZP])
def test_pairs_and_one_token_calls(blobs, fmt):
    c, layers = blobs
    L, T = layers[fmt], 5
    g = torch.Generator(device=DEV).manual_seed(1)
    X = torch.randn(T, 2048, device=DEV, generator=g)
    idx = torch.rand(T, E, device=DEV, generator=g).topk(K, dim=1).indices.to(torch.int32).contiguous()
    w = torch.rand(T, K, device=DEV, generator=g)
    items, pairs, _ = m.group_pairs(idx, w, T, K, E, L.slot_table())
    slots = torch.tensor([L.blob_ptr(int(e)) for e in idx[0]], dtype=torch.int64, device=DEV)

    def both(x):
        y = c.pairs_forward_tc(fmt, items, E, pairs, x, T, T * K, None, torch.zeros(T * K, 2048, device=DEV))
        return y.cpu().numpy(), m.experts_forward(fmt, slots, w[0].contiguous(), K, x[0]).cpu().numpy()

    c.make_default()
    try:
        want = both(X)
        for elements in (1, 2, 3):
            for a, b in zip(both(shifted(X, elements)), want):
                assert np.array_equal(a, b), elements
        assert c.status() == 0
    finally:
        c.make_default(False)


@pytest.mark.parametrize("fmt,min_tokens", [(m.FMT_SYM_F16, 1 << 20), (m.FMT_ZP, 1 << 20), (m.FMT_SYM_F16, 1), (m.FMT_ZP, 1)])
@pytest.mark.parametrize("flags", [0, 2])
def test_bf16_rows_of_a_layer(fmt, min_tokens, flags):
    """bf16 rows on a 4-byte boundary, through the routing kernel (1 and 3 tokens, and blocks of 16) and the kernel that prepares the rows."""
    c = m.Context(0, max_tokens=16, max_experts=E, top_k=K)
    c.set_prefill_min_tokens(min_tokens)
    L = m.Layer(c, fmt, E)
    L.fill_synth(6, 0)
    rng = np.random.default_rng(2)
    L.set_router((rng.standard_normal((E + 1, 2048)) * 0.02).astype(np.float32))
    try:
        for T in (1, 3, 16):
            X = torch.from_numpy(rng.standard_normal((T, 2048)).astype(np.float32)).to(DEV).to(torch.bfloat16)
            want = L.forward(X, T, K, flags=flags).cpu().numpy()
            for elements in (2, 4, 6):
                assert np.array_equal(L.forward(shifted(X, elements), T, K, flags=flags).cpu().numpy(), want), (T, elements)
        assert c.status() == 0
    finally:
        L.close(); c.close()


@pytest.mark.parametrize("residual", [True, False])
@pytest.mark.parametrize("min_tokens", [1 << 20, 1])
def test_rows_of_an_expert_parallel_step(residual, min_tokens):
    """f32 rows at any float and bf16 rows on a 4-byte boundary as the input of a step (one rank)."""
    T = 9
    c = m.Context(0, max_tokens=T, max_experts=E, top_k=K)
    c.set_prefill_min_tokens(min_tokens)
    L = m.Layer(c, m.FMT_SYM_F16, E)
    L.fill_synth(6, 0)
    rng = np.random.default_rng(3)
    L.set_router((rng.standard_normal((E + 1, 2048)) * 0.02).astype(np.float32))
    buf = m.ExchangeBuffer(T, K, 1)
    ep = m.EP(c, 0, 1, T, K, E, [buf.ptr])
    try:
        X = torch.from_numpy(rng.standard_normal((T, 2048)).astype(np.float32)).to(DEV)
        for x, places in ((X, (1, 2, 3)), (X.to(torch.bfloat16), (2, 4, 6))):
            def step(rows):
                ep.begin_step()
                ep.dispatch(L, 0, rows, residual)
                ep.experts(L, 0)
                out = torch.empty(T, 2048, device=DEV)
                ep.finish(1, out, residual)
                return out.cpu().numpy()
            want = step(x)
            assert np.isfinite(want).all() and want.any()
            for elements in places:
                assert np.array_equal(step(shifted(x, elements)), want), (x.dtype, elements)
        assert c.status() == 0
    finally:
        ep.close(); L.close(); c.close(); buf.close()
