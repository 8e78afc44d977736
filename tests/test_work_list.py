"""The work list where its size changes the path: the grouping kernel over several passes of 1024 pairs, and layers whose experts are too
many for the router's buckets (a planning launch instead). Needs a B200."""
import numpy as np
import pytest
import torch

import moe_b200 as m
from oracle import oracle as o
from parity import check_ffn

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("lib_built")]
DEV = "cuda:0"
ITEM_DT = np.dtype([("slot", "<u8"), ("start", "<i4"), ("count", "<i4")])
PAIR_DT = np.dtype([("t", "<i4"), ("p", "<i4"), ("w", "<f4")])


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


@pytest.mark.parametrize("T", [128, 129, 300])
def test_group_pairs_in_several_passes(T):
    E, K = 64, 8
    rng = np.random.default_rng(T)
    idx = np.stack([rng.choice(E, size=K, replace=False) for _ in range(T)]).astype(np.int32)
    w = rng.uniform(0, 1, (T, K)).astype(np.float32)
    table = np.arange(1, E + 2, dtype=np.int64) * 4096
    held = np.ones(E, np.uint8)
    held[7:11] = 0
    table[7:11] = 0
    items, pairs, nitems = m.group_pairs(dev(idx), dev(w), T, K, E, dev(table))
    ri, pt, pp, pw = o.group_pairs(idx, w, E, held)
    gi = items.cpu().numpy().view(ITEM_DT); gp = pairs.cpu().numpy().view(PAIR_DT)
    assert int(nitems.item()) == len(ri)
    assert [(int(table[e]), s, c) for e, s, c in ri] == [(int(a), int(b), int(c)) for a, b, c in gi[:len(ri)]]
    assert not gi["count"][len(ri):].any() and not gp["w"][len(pt):].any()
    assert np.array_equal(gp["t"][:len(pt)], pt) and np.array_equal(gp["p"][:len(pt)], pp) and np.array_equal(gp["w"][:len(pt)], pw)


def test_layer_with_more_experts_than_the_buckets_take():
    E, K = 288, 8
    c = m.Context(0, max_tokens=20, max_experts=E, top_k=K)
    L = m.Layer(c, m.FMT_SYM_F16, E)
    L.fill_synth(4, 0)
    rng = np.random.default_rng(6)
    W = (rng.standard_normal((E + 1, 2048)) * 0.02).astype(np.float32)
    L.set_router(W)
    host = [m.synth_expert_host(m.FMT_SYM_F16, 4, 0, e) for e in range(E + 1)]
    try:
        for T, min_tokens in ((5, 256), (20, 256), (20, 1)):
            c.set_prefill_min_tokens(min_tokens)
            X = rng.standard_normal((T, 2048)).astype(np.float32)
            idx = torch.empty(T, K, dtype=torch.int32, device=DEV)
            out = L.forward(dev(X), T, K, idx=idx).cpu().numpy()
            assert c.status() == 0
            ref, ri, _, _ = o.layer_forward(m.FMT_SYM_F16, host, W, X, K)
            assert np.array_equal(idx.cpu().numpy(), ri)
            check_ffn(out, ref, m.FMT_SYM_F16, f"{E} experts, {T} tokens")
    finally:
        L.close(); c.close()


@pytest.mark.parametrize("fmt,T", [(m.FMT_SYM_F16, 5), (m.FMT_ZP, 24), (m.FMT_SYM_F16, 24)])
def test_a_call_that_failed_after_its_router_leaves_nothing_behind(fmt, T):
    """The pairs that the router of a failed call put into the buckets must not be there for the next call, nor for the replay of a
    stack captured before. 64 places a bucket: the pairs of both calls fit."""
    E, K = 32, 8
    c = m.Context(0, max_tokens=64, max_experts=E, top_k=K)
    L = m.Layer(c, fmt, E)
    L.fill_synth(5, 0)
    rng = np.random.default_rng(T)
    W = (rng.standard_normal((E + 1, 2048)) * 0.02).astype(np.float32)
    L.set_router(W)
    X = rng.standard_normal((T, 2048)).astype(np.float32)
    stack = m.Stack(c, [L], T, K, m.F32, residual=False)
    try:
        before = stack.run(dev(X)).cpu().numpy()
        for again in range(3):
            c.selftest_fail()
            with pytest.raises(m.MoexbError, match="self-test"):
                L.forward(dev(rng.standard_normal((T, 2048)).astype(np.float32)), T, K)
            if again == 1:
                assert np.array_equal(stack.run(dev(X)).cpu().numpy(), before)
        assert np.array_equal(L.forward(dev(X), T, K).cpu().numpy(), before)
        assert c.status() == 0
        ref, _, _, _ = o.layer_forward(fmt, [m.synth_expert_host(fmt, 5, 0, e) for e in range(E + 1)], W, X, K)
        check_ffn(before, ref, fmt, f"{T} tokens before and after failed calls")
    finally:
        stack.close(); L.close(); c.close()


@pytest.mark.parametrize("fmt", [m.FMT_SYM_F16, m.FMT_SYM_F32, m.FMT_ZP])
@pytest.mark.parametrize("layout", [m.LAYOUT_TILED, m.LAYOUT_REFERENCE])
def test_the_expert_kernels_are_resident_as_often_as_their_grids_assume(fmt, layout):
    """Work list from the buckets, from a planning launch (288 experts) and one token's own; both widths of a pass; the grouped GEMM."""
    K = 8
    for E in (32, 288):
        c = m.Context(0, max_tokens=16, max_experts=E, top_k=K)
        L = m.Layer(c, fmt, E, layout=layout)
        L.fill_synth(1, 0)
        L.set_router(np.zeros((E + 1, 2048), np.float32))
        try:
            for T, pairs, min_tokens in ((1, 8, 256), (3, 8, 256), (16, 8, 256), (16, 4, 256), (16, 8, 1)):
                c.set_pairs_per_pass(pairs)
                c.set_prefill_min_tokens(min_tokens)
                L.forward(torch.zeros(T, 2048, device=DEV), T, K)
            assert c.status() == 0
        finally:
            L.close(); c.close()
    assert m.short_residency() == 0


@pytest.mark.parametrize("fmt, tokens", [(m.FMT_ZP, (1,)), (m.FMT_SYM_F16, (8, 9, 15, 16)), (m.FMT_SYM_F32, (8, 15))])
def test_k_slices_on_four_warps(fmt, tokens):
    """Gate/up with the K slices of a row tile on four warps: few experts (CTAs without a round, ranges that begin inside a sub-item) and
    many, narrow and wide sub-items. Against the oracle; 4 and 8 pairs a pass agree bit for bit."""
    for E in (32, 96):
        c = m.Context(0, max_tokens=16, max_experts=E, top_k=8)
        L = m.Layer(c, fmt, E)
        L.fill_synth(3, 0)
        rng = np.random.default_rng(13)
        W = (rng.standard_normal((E + 1, 2048)) * 0.02).astype(np.float32)
        L.set_router(W)
        host = [m.synth_expert_host(fmt, 3, 0, e) for e in range(E + 1)]
        try:
            for T in tokens:
                X = rng.standard_normal((T, 2048)).astype(np.float32)
                ref, ids, _, _ = o.layer_forward(fmt, host, W, X, 8)
                idx = torch.empty(T, 8, dtype=torch.int32, device=DEV)
                outs = []
                for p in (4, 8):
                    c.set_pairs_per_pass(p)
                    outs.append(L.forward(torch.from_numpy(X).to(DEV), T, 8, idx=idx).cpu().numpy())
                assert c.status() == 0 and np.array_equal(idx.cpu().numpy(), ids)
                assert np.array_equal(outs[0], outs[1])
                check_ffn(outs[1], ref, fmt, f"K slices on four warps, T={T} E={E}")
        finally:
            L.close(); c.close()


@pytest.mark.parametrize("fmt", [m.FMT_SYM_F16, m.FMT_ZP])
@pytest.mark.parametrize("router, x_type", [(m.F32, torch.float32), (m.F16, torch.bfloat16)])
def test_small_stack_equals_chained_layers(fmt, router, x_type):
    """A stack of 2 to 12 tokens, in which the end of a layer and the routing of the next are one kernel (13: two): the bits of the layers
    called one after the other, on the first run and on a repeated one, and the context takes plain calls afterwards."""
    E, NL = 64, 4
    c = m.Context(0, max_tokens=13, max_experts=E, top_k=8)
    rng = np.random.default_rng(17)
    layers = []
    for l in range(NL):
        L = m.Layer(c, fmt, E, router_dtype=router)
        L.fill_synth(3, l)
        L.set_router((rng.standard_normal((E + 1, 2048)) * 0.02).astype(np.float32 if router == m.F32 else np.float16))
        layers.append(L)
    try:
        for T in (2, 7, 8, 9, 12, 13):
            X = torch.from_numpy(rng.standard_normal((T, 2048)).astype(np.float32)).to(DEV).to(x_type)
            s = m.Stack(c, layers, T, 8, m.F32 if x_type == torch.float32 else m.BF16)
            want = X
            for L in layers:
                want = L.forward(want, T, 8, flags=2)
            for _ in range(3):
                assert torch.equal(s.run(X), want)
            assert torch.equal(layers[0].forward(X, T, 8, flags=2), layers[0].forward(X, T, 8, flags=2))
            assert c.status() == 0
            s.close()
    finally:
        for L in layers:
            L.close()
        c.close()


@pytest.mark.parametrize("fmt, layout", [(m.FMT_SYM_F16, m.LAYOUT_TILED), (m.FMT_ZP, m.LAYOUT_TILED), (m.FMT_SYM_F32, m.LAYOUT_REFERENCE)])
@pytest.mark.parametrize("x_type", [torch.float32, torch.bfloat16])
def test_blocks_of_a_few_tokens(fmt, layout, x_type):
    """Residual blocks whose norm and split are made by the routing kernel (1 to 16 tokens; 17: by a launch before it), against the oracle; a
    bf16 row that begins on 4 bytes gives the same bits."""
    E = 32
    c = m.Context(0, max_tokens=17, max_experts=E, top_k=8)
    L = m.Layer(c, fmt, E, layout=layout)
    L.fill_synth(3, 0)
    rng = np.random.default_rng(19)
    W = (rng.standard_normal((E + 1, 2048)) * 0.02).astype(np.float32)
    L.set_router(W)
    host = [m.synth_expert_host(fmt, 3, 0, e) for e in range(E + 1)]
    try:
        for T in (1, 2, 8, 9, 16, 17):
            X = torch.from_numpy(rng.standard_normal((T, 2048)).astype(np.float32)).to(x_type)
            xf = X.float().numpy()
            idx = torch.empty(T, 8, dtype=torch.int32, device=DEV)
            got = L.forward(X.to(DEV), T, 8, idx=idx, flags=2)
            assert c.status() == 0
            ref, ids, _, _ = o.layer_forward(fmt, host, W, o.rmsnorm(xf), 8)
            assert np.array_equal(idx.cpu().numpy(), ids)
            check_ffn(got.cpu().numpy(), xf + ref, fmt, f"block of {T} {x_type} tokens")
            if x_type == torch.bfloat16:
                at2 = torch.empty(T * 2048 + 2, dtype=x_type, device=DEV)[2:]
                at2.copy_(X.view(-1))
                assert torch.equal(L.forward(at2.view(T, 2048), T, 8, flags=2), got)
    finally:
        L.close(); c.close()


# experts, tokens, residual block; kernels of a call: routing, gate/up, down and combine, one more where a launch before the routing prepares
# the rows, and one more for the work list of layers whose experts are too many for the buckets
ROUTES = [(256, 8, False, m.F32, 4), (288, 8, False, m.F32, 5), (320, 8, False, m.F32, 6), (1024, 7, False, m.F32, 5), (1024, 8, False, m.F32, 6),
          (256, 16, True, m.F32, 4), (512, 15, True, m.F32, 5), (512, 16, True, m.F32, 6), (1024, 8, True, m.F32, 5), (1024, 9, True, m.F32, 6),
          (1024, 12, True, m.F16, 5), (1024, 13, True, m.F16, 6)]


@pytest.mark.parametrize("E, T, block, router, kernels", ROUTES)
def test_the_rows_of_a_few_tokens_by_the_number_of_routing_blocks(E, T, block, router, kernels):
    """Whether the routing kernel or a launch before it prepares the rows depends on the experts as well as on the tokens. The selected
    experts are the oracle's on either side of the line, and the outputs those of calls of fewer tokens, which always leave it to the
    routing kernel."""
    c = m.Context(0, max_tokens=16, max_experts=E, top_k=8)
    L = m.Layer(c, m.FMT_SYM_F16, E, router_dtype=router)
    L.fill_synth(3, 0)
    rng = np.random.default_rng(E + T)
    W = (rng.standard_normal((E + 1, 2048)) * 0.02).astype(np.float32 if router == m.F32 else np.float16)
    L.set_router(W)
    X = rng.standard_normal((T, 2048)).astype(np.float32)
    x, flags = dev(X), 2 if block else 0
    idx = torch.empty(T, 8, dtype=torch.int32, device=DEV)
    try:
        before = m.launch_count()
        got = L.forward(x, T, 8, idx=idx, flags=flags).cpu().numpy()
        assert m.launch_count() - before == kernels
        ids, _ = o.router_topk(o.router_logits(W, o.rmsnorm(X) if block else X, T), E, 8, True, T, E + 1)
        assert np.array_equal(idx.cpu().numpy(), ids)
        parts = [L.forward(x[t:t + 4].contiguous(), min(4, T - t), 8, flags=flags).cpu().numpy() for t in range(0, T, 4)]
        check_ffn(got, np.concatenate(parts), m.FMT_SYM_F16, f"{T} tokens of {E} experts against calls of 4")
        assert c.status() == 0
    finally:
        L.close(); c.close()


@pytest.mark.parametrize("K", [1, 11, 12, 15])
def test_one_zero_point_token_by_its_number_of_experts(K):
    """The K slices of a row tile on four warps up to 11 experts, on one warp beyond, against the oracle."""
    E = 32
    c = m.Context(0, max_tokens=1, max_experts=E, top_k=15)
    L = m.Layer(c, m.FMT_ZP, E)
    L.fill_synth(3, 0)
    rng = np.random.default_rng(K)
    W = (rng.standard_normal((E + 1, 2048)) * 0.02).astype(np.float32)
    L.set_router(W)
    X = rng.standard_normal((1, 2048)).astype(np.float32)
    idx = torch.empty(1, K, dtype=torch.int32, device=DEV)
    try:
        got = L.forward(dev(X), 1, K, idx=idx).cpu().numpy()
        ref, ids, _, _ = o.layer_forward(m.FMT_ZP, [m.synth_expert_host(m.FMT_ZP, 3, 0, e) for e in range(E + 1)], W, X, K)
        assert c.status() == 0 and np.array_equal(idx.cpu().numpy(), ids)
        check_ffn(got, ref, m.FMT_ZP, f"one zero-point token through {K} experts")
    finally:
        L.close(); c.close()


@pytest.mark.parametrize("fmt", [m.FMT_SYM_F16, m.FMT_SYM_F32])
def test_k_slices_on_four_warps_of_a_planned_list(fmt):
    """The same form with the work list of a planning launch (288 experts): the partial sums lie behind a list of another size. 4 and 8 pairs a
    pass agree bit for bit, and the kernels are resident as often as their grids assume."""
    E, K = 288, 8
    c = m.Context(0, max_tokens=15, max_experts=E, top_k=K)
    L = m.Layer(c, fmt, E)
    L.fill_synth(4, 0)
    rng = np.random.default_rng(29)
    W = (rng.standard_normal((E + 1, 2048)) * 0.02).astype(np.float32)
    W[40:] *= 0.2   # most pairs go to 40 experts: wide sub-items too
    L.set_router(W)
    host = [m.synth_expert_host(fmt, 4, 0, e) for e in range(E + 1)]
    try:
        for T in (8, 15):
            X = rng.standard_normal((T, 2048)).astype(np.float32)
            idx = torch.empty(T, K, dtype=torch.int32, device=DEV)
            outs = []
            for p in (4, 8):
                c.set_pairs_per_pass(p)
                outs.append(L.forward(dev(X), T, K, idx=idx).cpu().numpy())
            ref, ids, _, _ = o.layer_forward(fmt, host, W, X, K)
            assert c.status() == 0 and np.array_equal(idx.cpu().numpy(), ids)
            assert np.array_equal(outs[0], outs[1])
            check_ffn(outs[1], ref, fmt, f"K slices on four warps, planned list, {T} tokens")
    finally:
        L.close(); c.close()
    assert m.short_residency() == 0


@pytest.mark.parametrize("x_type", [torch.float32, torch.bfloat16])
def test_blocks_of_a_few_tokens_with_more_than_256_experts(x_type):
    """The routing kernel that makes the norm, in its form for up to 1024 experts, against the oracle."""
    E, K, fmt = 288, 8, m.FMT_SYM_F16
    c = m.Context(0, max_tokens=16, max_experts=E, top_k=K)
    L = m.Layer(c, fmt, E, router_dtype=m.F16)
    L.fill_synth(4, 0)
    rng = np.random.default_rng(31)
    W = (rng.standard_normal((E + 1, 2048)) * 0.02).astype(np.float16)
    L.set_router(W)
    host = [m.synth_expert_host(fmt, 4, 0, e) for e in range(E + 1)]
    try:
        for T in (1, 8, 16):
            X = torch.from_numpy(rng.standard_normal((T, 2048)).astype(np.float32)).to(x_type)
            xf = X.float().numpy()
            idx = torch.empty(T, K, dtype=torch.int32, device=DEV)
            got = L.forward(X.to(DEV), T, K, idx=idx, flags=2).cpu().numpy()
            ref, ids, _, _ = o.layer_forward(fmt, host, W, o.rmsnorm(xf), K)
            assert c.status() == 0 and np.array_equal(idx.cpu().numpy(), ids)
            check_ffn(got, xf + ref, fmt, f"block of {T} {x_type} tokens, {E} experts")
    finally:
        L.close(); c.close()


@pytest.mark.parametrize("fmt, K", [(m.FMT_SYM_F32, 8), (m.FMT_SYM_F16, 3), (m.FMT_SYM_F16, 15), (m.FMT_ZP, 9)])
def test_small_stack_of_other_numbers_of_experts(fmt, K):
    """Stacks whose layers' ends and routings are one kernel, with fewer and more ranks than the eight it requests at once: the bits of the
    layers called one after the other. A stack whose capture fails between leaves nothing behind."""
    E, NL, T = 64, 3, 6
    c = m.Context(0, max_tokens=T, max_experts=E, top_k=15)
    rng = np.random.default_rng(K)
    layers = []
    for l in range(NL):
        L = m.Layer(c, fmt, E)
        L.fill_synth(3, l)
        L.set_router((rng.standard_normal((E + 1, 2048)) * 0.02).astype(np.float32))
        layers.append(L)
    stacks = []
    try:
        X = dev(rng.standard_normal((T, 2048)).astype(np.float32))
        want = X
        for L in layers:
            want = L.forward(want, T, K, flags=2)
        stacks.append(m.Stack(c, layers, T, K))
        assert stacks[0].kernel_count == 3 * NL + 1
        assert torch.equal(stacks[0].run(X), want)
        c.selftest_fail()
        with pytest.raises(m.MoexbError, match="self-test"):
            m.Stack(c, layers, T, K)
        assert torch.equal(stacks[0].run(X), want)
        stacks.append(m.Stack(c, layers, T, K))
        assert torch.equal(stacks[1].run(X), want) and torch.equal(layers[0].forward(X, T, K, flags=2), layers[0].forward(X, T, K, flags=2))
        assert c.status() == 0
    finally:
        for s in stacks:
            s.close()
        for L in layers:
            L.close()
        c.close()
