"""The gradient GEMM with its fused accumulation and ReLU, the BF16 message gradient and the clustered edge-weight gradient
against float64 references, at the edges of the 128-row tiles."""
import numpy as np
import pytest

from conftest import grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 127, 128, 129, 128 * 1500 + 3])
@pytest.mark.parametrize("k,n", [(64, 128), (128, 64)])
def test_gradient_gemm_matches_float64(engine_lib, k, n, M):
    """accum += A W[:, :64] in FP32, second = A W[:, 64:], dz = the new accum where z > 0.  FP32 sums of k BF16 products:
    k * 2^-24 relative to the largest, 1e-5 leaves a margin; dz adds BF16's 2^-9."""
    import torch
    from olfgpu import gnn
    rng = np.random.default_rng(M + k)
    A = torch.from_numpy(rng.standard_normal((M, k)).astype(np.float32)).cuda().to(torch.bfloat16)
    W = torch.from_numpy((rng.standard_normal((k, n)) / 8).astype(np.float32)).cuda().to(torch.bfloat16)
    z = torch.from_numpy(rng.standard_normal((M, 64)).astype(np.float32)).cuda().to(torch.bfloat16)
    acc0 = torch.from_numpy(rng.standard_normal((M, 64)).astype(np.float32)).cuda()
    acc, dz = acc0.clone(), torch.empty((M, 64), dtype=torch.bfloat16, device="cuda")
    second = torch.empty((M, 64), dtype=torch.float32, device="cuda") if n == 128 else None
    gnn._call("olfgpu_gnn_gemm_grad", M, k, n, gnn._ptr(A), gnn._ptr(W), gnn._ptr(acc), gnn._ptr(second), gnn._ptr(z),
              gnn._ptr(dz), gnn._stream())
    y = A.double() @ W.double()
    ref = acc0.double() + y[:, :64]
    scale = float(ref.abs().max())
    assert float((acc.double() - ref).abs().max()) / scale < 1e-5
    if n == 128:
        assert float((second.double() - y[:, 64:]).abs().max()) / float(y.abs().max()) < 1e-5
    want = torch.where(z > 0, acc, torch.zeros_like(acc)).to(torch.bfloat16)
    assert torch.equal(dz, want)
    assert gnn.tc_timeouts() == 0


@pytest.mark.parametrize("M", [1, 33, 128 * 5 + 7])
@pytest.mark.parametrize("k1,k2,n", [(16, 0, 64), (64, 0, 128), (64, 64, 64), (64, 0, 16)])
def test_weight_gradient_with_partials_off_the_pair_alignment(engine_lib, k1, k2, n, M):
    """A scratch array that starts at an odd element gives the bits of an aligned one.  Against float64: FP32 sums of M products
    of BF16 values, M * 2^-24 of the products' magnitudes."""
    import torch
    from olfgpu import gnn
    rng = np.random.default_rng(M + k1 + n)
    draw = lambda *s: torch.from_numpy(rng.standard_normal(s).astype(np.float32)).cuda().to(torch.bfloat16)  # noqa: E731
    a1, a2, dz = draw(M, k1), draw(M, k2) if k2 else None, draw(M, n)
    chunks, k = 3, k1 + k2
    got = []
    for first in (0, 1):
        partial = torch.full((chunks * (k * n + n) + 1,), float("nan"), device="cuda")[first:]
        dw, db = torch.empty((k, n), device="cuda"), torch.empty(n, device="cuda")
        gnn._call("olfgpu_gnn_gemm_dw", M, k1, k2, n, gnn._ptr(a1), gnn._ptr(a2), gnn._ptr(dz), gnn._ptr(dw), gnn._ptr(db),
                  gnn._ptr(partial), chunks, gnn._stream())
        got.append((dw, db))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    a = torch.cat([a1, a2], 1).double() if k2 else a1.double()
    assert bool((torch.abs(got[0][0] - a.T @ dz.double()) <= (M + 8) * 2.0 ** -24 * (a.abs().T @ dz.double().abs())).all())
    assert bool((torch.abs(got[0][1] - dz.double().sum(0)) <= (M + 8) * 2.0 ** -24 * dz.double().abs().sum(0)).all())


@pytest.mark.parametrize("B", [1, 3, 9])
def test_message_gradients_match(engine_lib, B):
    """dPQ rounded to BF16 is the FP32 entry's dPQ rounded; the edge-weight gradient is the float64 product."""
    import torch
    from olfgpu import gnn
    g, _ = grid("grid118")
    gd = gnn.GraphData.from_grid(g)
    gen = torch.Generator(device="cuda").manual_seed(B)
    M = B * gd.nb
    rnd = lambda *s: torch.randn(s, device="cuda", generator=gen)  # noqa: E731
    pq, C, bm, dagg = rnd(M, 128).to(torch.bfloat16), rnd(gd.n_edges, 64), rnd(64), rnd(M, 64)
    outage = torch.arange(B, dtype=torch.int32, device="cuda") * 5
    d32 = torch.empty((M, 128), device="cuda")
    d16 = torch.empty((M, 128), dtype=torch.bfloat16, device="cuda")
    dc32, dc16 = torch.empty((gd.n_edges, 64), device="cuda"), torch.empty((gd.n_edges, 64), device="cuda")
    for name, out, dc in (("olfgpu_gnn_message_backward", d32, dc32), ("olfgpu_gnn_message_backward_bf16", d16, dc16)):
        gnn._call(name, B, gd.nb, gd.n_edges, *[gnn._ptr(t) for t in (gd.in_ptr, gd.in_edge, gd.out_ptr, gd.out_edge, gd.src,
                  gd.dst, gd.branch, outage, pq, C, bm, dagg, out, dc)], gnn._stream())
    assert torch.equal(d16, d32.to(torch.bfloat16)) and torch.equal(dc16, dc32)
    # arrays off the vector accesses' alignment (one element in): the same values
    off = lambda x: torch.cat([x.reshape(-1)[:1], x.reshape(-1)])[1:]  # noqa: E731
    agg, agg1 = torch.empty((M, 64), dtype=torch.bfloat16, device="cuda"), torch.empty(M * 64 + 1, dtype=torch.bfloat16, device="cuda")[1:]
    pq1, c1, bm1, da1 = off(pq), off(C), off(bm), off(dagg)
    d1, dc1 = torch.empty(M * 128 + 1, device="cuda")[1:], torch.empty(gd.n_edges * 64 + 1, device="cuda")[1:]
    gnn._call("olfgpu_gnn_message_backward", B, gd.nb, gd.n_edges, *[gnn._ptr(t) for t in (gd.in_ptr, gd.in_edge, gd.out_ptr,
              gd.out_edge, gd.src, gd.dst, gd.branch, outage, pq1, c1, bm1, da1, d1, dc1)], gnn._stream())
    assert torch.equal(d1.reshape(M, 128), d32) and torch.equal(dc1.reshape(-1, 64), dc32)
    for p_, c_, b_, a_ in ((pq, C, bm, agg), (pq1, c1, bm1, agg1)):
        gnn._call("olfgpu_gnn_message_forward", B, gd.nb, *[gnn._ptr(t) for t in (gd.in_ptr, gd.in_edge, gd.src, gd.branch,
                  outage, p_, c_, b_, a_)], gnn._stream())
    assert torch.equal(agg1.reshape(M, 64), agg)
    we, db = torch.empty((4, 64), device="cuda"), torch.empty((1, 64), device="cuda")
    gnn._call("olfgpu_gnn_edge_project_backward", gd.n_edges, gnn._ptr(gd.es), gnn._ptr(dc32), gnn._ptr(we), gnn._ptr(db),
              gnn._stream())
    ref, refb = gd.es.double().T @ dc32.double(), dc32.double().sum(0)
    # FP32 sums over n_edges terms: n_edges * 2^-24 of the terms' magnitudes
    bound = gd.n_edges * 2.0 ** -24
    assert float((we - ref).abs().max()) <= bound * float((gd.es.abs().T @ dc32.abs()).max())
    assert float((db[0] - refb).abs().max()) <= bound * float(dc32.abs().sum(0).max())


@pytest.mark.parametrize("B", [1, 3, 9])
def test_message_gradients_match_float64(engine_lib, B):
    """dPQ and dC of both entries against sums over the edges in float64, the outaged branch's edges left out.  The inputs are
    such that no pre-activation is near zero (a ReLU's side does not hang on rounding): FP32 sums of as many terms as a bus has
    edges or an edge has samples, 16 * 2^-24 of the terms' magnitudes; BF16, of eight significant bits, adds half a unit in the last, 2^-8 of the result."""
    import torch
    from olfgpu import gnn
    g, _ = grid("grid118")
    gd = gnn.GraphData.from_grid(g)
    gen = torch.Generator(device="cuda").manual_seed(40 + B)
    nb, M = gd.nb, B * gd.nb
    # multiples of 1/4, and an odd multiple of 1/8 in the bias: exact in BF16 and FP32, and never a sum of zero
    quarter = lambda *s: torch.randint(-8, 9, s, device="cuda", generator=gen).float() / 4  # noqa: E731
    pq, C, bm = quarter(M, 128).to(torch.bfloat16), quarter(gd.n_edges, 64), quarter(64) + 0.125
    dagg = torch.randn((M, 64), device="cuda", generator=gen)
    outage = torch.arange(B, dtype=torch.int32, device="cuda") * 7
    src, dst, branch = gd.src.long(), gd.dst.long(), gd.branch.long()
    PQ, D = pq.double().reshape(B, nb, 128), dagg.double().reshape(B, nb, 64)
    pre = PQ[:, src, :64] + PQ[:, dst, 64:] + C.double() + bm.double()
    on = (pre > 0) & (branch[None, :] != outage.long()[:, None])[..., None]
    ge = torch.where(on, D[:, dst], torch.zeros_like(pre))
    want = torch.zeros((B, nb, 128), dtype=torch.float64, device="cuda")
    want[:, :, :64].index_add_(1, src, ge)
    want[:, :, 64:].index_add_(1, dst, ge)
    size = torch.zeros_like(want)
    size[:, :, :64].index_add_(1, src, ge.abs())
    size[:, :, 64:].index_add_(1, dst, ge.abs())
    want, size = want.reshape(M, 128), size.reshape(M, 128)
    for name, dtype, ulp in (("olfgpu_gnn_message_backward", torch.float32, 0.0),
                             ("olfgpu_gnn_message_backward_bf16", torch.bfloat16, 2.0 ** -8)):
        out, dc = torch.full((M, 128), 7.0, dtype=dtype, device="cuda"), torch.full((gd.n_edges, 64), 7.0, device="cuda")
        gnn._call(name, B, nb, gd.n_edges, *[gnn._ptr(t) for t in (gd.in_ptr, gd.in_edge, gd.out_ptr, gd.out_edge, gd.src,
                  gd.dst, gd.branch, outage, pq, C, bm, dagg, out, dc)], gnn._stream())
        bound = 16 * 2.0 ** -24 * size
        assert bool(((out.double() - want).abs() <= bound + ulp * (want.abs() + bound)).all())
        assert bool(((dc.double() - ge.sum(0)).abs() <= 16 * 2.0 ** -24 * ge.abs().sum(0)).all())
