"""The adjoint kernels at every way their feature rows are walked: 16-byte
groups and single columns, 16 and 32 lanes per row, one pass and several, K on
both sides of 16 and 32.

The oracle is FP64 autograd at the same neighbours.  Tolerance: every output is
a sum of products of FP32 factors, each with at most 40 roundings (keys 20,
__expf about 4, the rest of the entry's geometry 16) and n terms added in FP32;
relative to the sum of the terms' magnitudes that is (40 + n) 2^-24, with n at
most F (dot products), K and the longest point row, here below 1700 in all, so
1.1e-4 of the output's largest value bounds what cancellation leaves; the
repository's bar for gradients, 1e-4, is used."""
import pytest
import torch

import oracle as O
from conftest import rel_err

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("F", [1, 15, 16, 33, 37, 64, 65, 68, 128, 132, 256, 300, 516])
@pytest.mark.parametrize("K,dtype", [(5, torch.float32), (17, torch.float32), (40, torch.float32),
                                     (9, torch.float64)])
def test_both_orders_match_fp64_autograd(F, K, dtype):
    from cuda_knn_aggregate import knn_aggregate_aniso, workloads as W

    _, t = W.make("small", B=2, Q=61, P=150, F=F, K=K, seed=1000 * K + F, dtype=dtype)
    x = [a.to(DEV).requires_grad_(True) for a in t]
    g = torch.Generator().manual_seed(F)
    gfo = torch.randn(2, 61, F, generator=g, dtype=torch.float64)
    ggq = torch.randn(2, 61, 3, generator=g, dtype=torch.float64)
    gfo_d = gfo.to(DEV, dtype).requires_grad_(True)
    f_out, _, _, idxs = knn_aggregate_aniso(*x, K)
    first = torch.autograd.grad(f_out, x, grad_outputs=gfo_d, create_graph=True)
    second = torch.autograd.grad(first[0], [gfo_d] + x, grad_outputs=ggq.to(DEV, dtype))

    y = [a.double().requires_grad_(True) for a in t]
    gfo.requires_grad_(True)
    fo, _ = O.aggregate64(*y, idxs.cpu())
    want = torch.autograd.grad(fo, y, grad_outputs=gfo, create_graph=True)
    want2 = torch.autograd.grad(want[0], [gfo] + y, grad_outputs=ggq)
    tol = 1e-4 if dtype == torch.float32 else 1e-10
    for a, b in zip(list(first) + list(second), list(want) + list(want2)):
        assert rel_err(a.detach().cpu().numpy(), b.detach().numpy()) < tol


@pytest.mark.parametrize("B,Q,P,K", [(1, 1, 1, 1), (3, 5, 40, 3), (1, 33, 200, 15), (2, 77, 300, 16), (1, 61, 90, 17),
                                     (1, 9, 70, 33)])
def test_broadcast_gradient_query_sides(B, Q, P, K):
    """The Eikonal step's query sides (a broadcast f_out gradient, then dq's
    own gradient) where quads of lanes that share their record loads are cut:
    K around multiples of 4, of a half-warp and a warp, an odd number of
    queries, indices out of range beside good ones.  FP64 autograd of the plain
    formula, tolerance as for every gradient here."""
    from cuda_knn_aggregate import _C

    g = torch.Generator().manual_seed(Q + K)
    r = lambda *s: torch.rand(*s, generator=g)  # noqa: E731
    x = [r(B, Q, 3), r(B, P, 3), r(B, P, 6), r(B, P, 3), r(B, P, 3, 3)]
    idx = torch.randint(0, P, (B, Q, K), generator=g)
    ggq = torch.randn(B, Q, 3, generator=g)
    gfo = torch.ones(B, Q, 6)
    first, second = O.grads64(*[t.double() for t in x], idx, gfo.double(), ggq.double())
    dev = [t.cuda() for t in x]
    need = _C.NEED_DQ | 64  # KNNAG_GFO_SCALAR
    one = torch.ones(1, device="cuda").expand(B, Q, 6)  # one value, broadcast
    out = _C.backward_ex(one, *dev, idx.cuda(), None, None, need)
    assert _rel(out[0], first[0]) < 1e-4
    two = _C.backward2_ex(ggq.cuda(), one, *dev, idx.cuda(), None, None, out[5], need)
    assert _rel(two[1], second[1]) < 1e-4
    if K > 1:  # an entry that is out of range counts for nothing
        bad = idx.clone()
        bad[:, :, 1] = P
        part = _C.backward_ex(one, *dev, bad.cuda(), None, None, need)
        alone = _C.backward_ex(one, *dev, idx[:, :, 1:2].contiguous().cuda(), None, None, need)
        assert _rel(part[0] + alone[0], first[0]) < 1e-4


def _rel(a, b):
    return float((a.cpu().double() - b).norm() / b.norm())


@pytest.mark.parametrize("F", [64, 512, 5, 70])  # 16 and 32 lanes a query, 16-byte columns; the same with single ones
def test_ragged_gradients_of_a_given_grad_f_out(F):
    """Segments of K 3, 17 and 32 over clouds of different sizes, odd query
    counts, so that a warp serves queries of two segments; a query's sums do not
    depend on its neighbour in the warp: equal to the uniform op's to the bit."""
    from cuda_knn_aggregate import knn_aggregate_aniso
    from cuda_knn_aggregate.ragged import CloudSet, ragged_forward

    g = torch.Generator().manual_seed(F)
    sizes = [300, 33, 1000, 70]
    P = sum(sizes)
    p, sigma, f = (torch.rand(P, n, generator=g).cuda() for n in (3, 3, F))
    R = torch.linalg.qr(torch.randn(P, 3, 3, generator=g))[0].contiguous().cuda()
    clouds = CloudSet(p, sigma, R, f, sizes)
    order, Qs, Ks = [0, 1, 2, 3, 1, 0], [7, 5, 41, 1, 33, 9], [17, 32, 3, 32, 3, 17]
    q = torch.rand(sum(Qs), 3, generator=g).cuda()
    gfo = torch.randn(sum(Qs), F, generator=g).cuda()
    res = ragged_forward(clouds, q, order, Qs, Ks, grad_q=[True] * 5 + [False], grad_f_out=gfo)
    q0 = 0
    for i, (c, Q, K) in enumerate(zip(order, Qs, Ks)):
        rows = slice(sum(sizes[:c]), sum(sizes[:c + 1]))
        qi = q[q0:q0 + Q].clone()[None].requires_grad_(True)
        f_out = knn_aggregate_aniso(qi, *(t[rows].clone()[None] for t in (p, f, sigma, R)), K)[0]
        assert torch.equal(res.f_out[q0:q0 + Q], f_out[0].detach())
        if i < 5:
            (dq,) = torch.autograd.grad(f_out, qi, gfo[q0:q0 + Q].clone()[None])
            assert torch.equal(res.dq[q0:q0 + Q], dq[0])
        q0 += Q


@pytest.mark.parametrize("scale", [1, 19, 160])  # one, two and eight rows a warp's turn
def test_ragged_gradients_of_the_sum(scale):
    """grad_f_out of ones: a warp takes one to eight consecutive rows, of
    several segments where these are short, some without a gradient at the end;
    equal to the uniform op's to the bit."""
    from cuda_knn_aggregate import knn_aggregate_aniso
    from cuda_knn_aggregate.ragged import CloudSet, ragged_forward

    g = torch.Generator().manual_seed(scale)
    sizes = [300, 33, 1000, 70]
    P = sum(sizes)
    p, sigma, f = (torch.rand(P, n, generator=g).cuda() for n in (3, 3, 8))
    R = torch.linalg.qr(torch.randn(P, 3, 3, generator=g))[0].contiguous().cuda()
    clouds = CloudSet(p, sigma, R, f, sizes)
    order, Ks = [0, 1, 2, 3, 1, 2, 3, 0], [17, 32, 3, 32, 3, 16, 1, 8]
    Qs = [7, 1, 41 * scale + 1, 2, 3, 211 * scale, 5, 9]
    q = torch.rand(sum(Qs), 3, generator=g).cuda()
    res = ragged_forward(clouds, q, order, Qs, Ks, grad_q=[True] * 7 + [False])
    q0 = 0
    for i, (c, Q, K) in enumerate(zip(order, Qs, Ks)):
        if i < 7:
            rows = slice(sum(sizes[:c]), sum(sizes[:c + 1]))
            qi = q[q0:q0 + Q].clone()[None].requires_grad_(True)
            f_out = knn_aggregate_aniso(qi, *(t[rows].clone()[None] for t in (p, f, sigma, R)), K)[0]
            (dq,) = torch.autograd.grad(f_out.sum(), qi)
            assert torch.equal(res.dq[q0:q0 + Q], dq[0])
        q0 += Q
