"""The point -> entry adjacency at its row lengths (one warp's registers, the
CTA's shared memory, several runs) and row counts (the scan folded into the
fill, and not), built from scratch, on the forward's counts, and again on the
same counts.  Integers: compared exactly with a stable sort on the CPU."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _expect(idxs, P):
    B, Q, K = idxs.shape
    rows = (idxs + P * torch.arange(B)[:, None, None]).reshape(-1)
    rowptr = torch.zeros(B * P + 1, dtype=torch.int64)
    rowptr[1:] = torch.bincount(rows, minlength=B * P).cumsum(0)
    return rowptr, torch.argsort(rows, stable=True)


def _check(adj, idxs, P):
    from cuda_knn_aggregate import _C

    B, Q, K = idxs.shape
    rowptr, entries = _C.adjacency_views(adj, B, Q, P, K)
    want_ptr, want = _expect(idxs, P)
    assert torch.equal(rowptr.cpu().long(), want_ptr)
    assert torch.equal(entries.cpu().long(), want)


@pytest.mark.parametrize("B,Q,P,K,power", [
    (1, 3, 1, 1, 1), (2, 100, 7, 3, 1),
    (1, 4000, 64, 9, 4),       # rows of up to some thousand entries: shared memory
    (1, 9000, 4, 2, 2),        # several thousand each
    (2, 21000, 3, 2, 3),       # more than one run of 8192
    (1, 2000, 16384, 5, 3),    # the most rows of the folded scan
    (3, 900, 5500, 6, 1),      # one more CTA's worth: the scan by itself
])
def test_rows_are_sorted_entries(B, Q, P, K, power):
    from cuda_knn_aggregate import _C

    g = torch.Generator().manual_seed(Q + P)
    score = torch.rand(B, Q, P, generator=g) * torch.linspace(0.05, 1, P) ** power  # low points are picked most
    idxs = score.topk(K, largest=False).indices.contiguous()
    _check(_C.build_adjacency(idxs.to(DEV), P), idxs, P)


@pytest.mark.parametrize("P,dtype,K", [(300, torch.float32, 12), (300, torch.float64, 12), (9000, torch.float32, 5),
                                       (9000, torch.float32, 40), (100, torch.float64, 7)])
def test_counted_forward_and_a_second_backward(P, dtype, K):
    """Gradients of the same graph twice: the second pass builds the adjacency
    on the counts the forward left and must give the same bits."""
    from cuda_knn_aggregate import knn_aggregate_aniso, workloads as W

    _, t = W.make("small", B=2, Q=700, P=P, F=8, K=K, seed=P + K, dtype=dtype)
    x = [a.to(DEV).requires_grad_(True) for a in t]
    f_out = knn_aggregate_aniso(*x, K)[0]
    g = torch.randn_like(f_out)
    first = torch.autograd.grad(f_out, x, grad_outputs=g, retain_graph=True)
    for _ in range(2):
        again = torch.autograd.grad(f_out, x, grad_outputs=g, retain_graph=True)
        assert all(torch.equal(a, b) for a, b in zip(first, again))


@pytest.mark.parametrize("P", [50, 20000])  # the scan folded into the fill, and not
def test_no_queries(P):
    """A forward of no queries counts nothing; its adjacency has empty rows
    whatever the buffer held before."""
    from cuda_knn_aggregate import _C, capi, knn_aggregate_aniso

    lib, K = capi.lib(), 3
    adj = torch.full((lib.knnag_adjacency_bytes(2, 0, P, K),), 0x11, dtype=torch.uint8, device=DEV)
    idxs = torch.empty(2, 0, K, dtype=torch.int64, device=DEV)
    assert lib.knnag_build_adjacency_counted(capi._p(idxs), 2, 0, P, K, capi._p(adj), capi._stream(DEV)) == 0
    assert not _C.adjacency_views(adj, 2, 0, P, K)[0].any()
    x = [torch.rand(2, n, *s, device=DEV).requires_grad_(True) for n, s in ((0, (3,)), (P, (3,)), (P, (4,)), (P, (3,)),
                                                                            (P, (3, 3)))]
    f_out = knn_aggregate_aniso(*x, K)[0]
    assert f_out.shape == (2, 0, 4)
    with pytest.raises(RuntimeError, match="invalid argument"):  # no gradients of nothing, as before
        torch.autograd.grad(f_out.sum(), x)
    torch.cuda.synchronize()
