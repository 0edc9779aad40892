"""The one-warp-per-query search at the sizes where it can go wrong: list
lengths around 32, 64 and 128, FP64, clouds of one point around a tile, a
group of tiles and the finer grid, queries that fill no unit, tied, negative
and non-finite keys.

Two oracles, both exact (every output must be equal bit for bit, so there is
no tolerance): the CPU oracle for FP32 indices and keys, and the exact MinK
kernel, which serves FP64 and K > 32 when the workspace has no room for the
search index."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _inputs(kind, B, Q, P, F, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    q = torch.rand(B, Q, 3, generator=g, dtype=torch.float64)
    p = torch.rand(B, P, 3, generator=g, dtype=torch.float64)
    f = torch.rand(B, P, F, generator=g, dtype=torch.float64)
    sigma = torch.rand(B, P, 3, generator=g, dtype=torch.float64)
    R = torch.rand(B, P, 3, 3, generator=g, dtype=torch.float64)
    if kind == "ties":  # a coarse lattice, unit Gaussians: most keys are shared
        p, q = (p * 5).round() / 4, (q * 9).round() / 8
        sigma, R = torch.ones_like(sigma), torch.eye(3, dtype=torch.float64).expand(B, P, 3, 3).clone()
    elif kind == "twins":  # a few points of the same place and shape, most of them far apart in the order
        to = torch.arange(7, P, 41)
        at = torch.randint(0, P, (len(to),), generator=g)
        for v in (p, sigma, R):
            v[:, to] = v[:, at]
    elif kind == "negative":
        sigma = sigma - 0.5
    elif kind == "nan":
        p[:, 1::97] = float("nan")
        sigma[:, 3::89] = float("inf")
    elif kind == "far":  # queries outside the points' box, where windows tell little
        q = q * 6 - 3
    return [t.to(dtype).contiguous().to(DEV) for t in (q, p, f, sigma, R)]


def _call(x, K, ws_bytes):
    from cuda_knn_aggregate import capi

    q, p, f, sigma, R = x
    B, Q, P, F = q.shape[0], q.shape[1], p.shape[1], f.shape[2]
    o = dict(dtype=q.dtype, device=DEV)
    out = [torch.full((B, Q, F), -7.0, **o), torch.full((B, Q, K), -7.0, **o), torch.full((B, Q, K), -7.0, **o),
           torch.full((B, Q, K), -7, dtype=torch.int64, device=DEV)]
    ws = torch.empty(ws_bytes, dtype=torch.uint8, device=DEV)
    code = capi.F64 if q.dtype == torch.float64 else capi.F32
    rc = capi.lib().knnag_forward(*[capi._p(t) for t in x], B, Q, P, F, K, code, *[capi._p(t) for t in out], None,
                                  capi._p(ws), ws_bytes, capi._stream(DEV))
    assert rc == 0 and capi.read_device_status(ws, DEV) == 0
    return out


def _bits(t):
    return t.view(torch.int32) if t.dtype == torch.float32 else t.view(torch.int64)


@pytest.mark.parametrize("kind,dtype,B,Q,P,F,K", [
    ("rand", torch.float64, 2, 131, 128, 6, 1),       # one tile; units of 4 with 3 left over
    ("rand", torch.float64, 1, 257, 4097, 5, 32),     # full list; past a group of tiles, finer grid, odd F
    ("rand", torch.float64, 1, 60, 700, 4, 33),       # second list register
    ("rand", torch.float64, 1, 30, 700, 4, 128),      # fourth
    ("rand", torch.float32, 2, 101, 129, 8, 33),
    ("rand", torch.float32, 1, 203, 8193, 12, 64),    # full two-register list; three groups of tiles
    ("rand", torch.float32, 1, 45, 1000, 4, 65),
    ("rand", torch.float32, 1, 33, 128, 4, 128),      # K == P
    ("ties", torch.float64, 1, 90, 600, 4, 9),
    ("ties", torch.float32, 1, 90, 600, 4, 64),
    ("twins", torch.float64, 1, 300, 3000, 4, 1),      # replays: one slot,
    ("twins", torch.float64, 1, 200, 4097, 4, 32),     # two CTAs a query, unmerged tails
    ("twins", torch.float64, 1, 60, 33000, 4, 64),     # eight CTAs, three lengths of ranges
    ("twins", torch.float32, 1, 200, 8193, 4, 33),
    ("twins", torch.float32, 1, 60, 66000, 4, 128),    # every slot of the longest list
    ("negative", torch.float64, 1, 70, 900, 4, 12),
    ("negative", torch.float32, 1, 70, 900, 4, 40),
    ("nan", torch.float64, 1, 70, 900, 4, 12),
    ("nan", torch.float32, 1, 70, 900, 4, 40),
    ("far", torch.float64, 1, 300, 9000, 4, 16),
    ("far", torch.float32, 1, 300, 9000, 4, 48),
])
def test_indexed_calls_equal_the_exact_kernel(kind, dtype, B, Q, P, F, K):
    _compare(_inputs(kind, B, Q, P, F, dtype, seed=P + K), K)


def _compare(x, K):
    from cuda_knn_aggregate import capi

    B, Q, P, F, dtype = x[0].shape[0], x[0].shape[1], x[1].shape[1], x[2].shape[2], x[0].dtype
    size = 8 if dtype == torch.float64 else 4
    r256 = lambda n: (n + 255) // 256 * 256  # noqa: E731
    lean = 256 + r256(B * Q * 4) + r256(B * P * 16 * size)
    full = capi.lib().knnag_forward_workspace_bytes(B, Q, P, F, K, capi.F64 if size == 8 else capi.F32)
    assert full > lean
    got, want = _call(x, K, full), _call(x, K, lean)
    for a, b in zip(got, want):
        assert torch.equal(_bits(a), _bits(b))


@pytest.mark.parametrize("kind,dtype,B,Q,P", [
    ("rand", torch.float32, 1, 1, 128),         # the fewest points that are indexed: one tile
    ("rand", torch.float32, 3, 1023, 1025),     # tiles for all eight, one with two
    ("rand", torch.float32, 1, 32768, 4096),    # the largest element of the one-launch index
    ("rand", torch.float32, 1, 32769, 4096),    # past it by a query,
    ("rand", torch.float32, 1, 500, 4097),      # by a point,
    ("rand", torch.float32, 8, 40, 200),        # the most elements,
    ("rand", torch.float32, 9, 40, 200),        # and one more
    ("rand", torch.float32, 17, 40, 200),
    ("rand", torch.float64, 16, 65, 300),
    ("rand", torch.float64, 1, 9000, 4096),
    ("nan", torch.float64, 2, 40, 4096),
    ("far", torch.float32, 2, 700, 4000),
])
def test_index_sizes(kind, dtype, B, Q, P):
    _compare(_inputs(kind, B, Q, P, 4, dtype, seed=Q + P), 33)


@pytest.mark.parametrize("kind,B,Q,P,K", [
    ("rand", 1, 1, 1, 1), ("rand", 3, 5, 31, 31), ("rand", 1, 6, 64, 32), ("rand", 1, 9, 65, 32),
    ("rand", 1, 4750, 127, 7),     # two queries a warp
    ("rand", 1, 9501, 300, 3),     # four a warp, one left over
    ("far", 1, 700, 4096, 16), ("far", 1, 700, 4097, 32), ("far", 2, 300, 12500, 8),
    ("ties", 1, 500, 4200, 32), ("negative", 1, 200, 5000, 32), ("nan", 1, 200, 5000, 32),
])
def test_forward_matches_the_cpu_oracle(kind, B, Q, P, K):
    from cuda_knn_aggregate import capi

    x = _inputs(kind, B, Q, P, 4, torch.float32, seed=Q + P)
    out = _call(x, K, capi.lib().knnag_forward_workspace_bytes(B, Q, P, 4, K, capi.F32))
    _, _, d_ref, i_ref = O.forward_f32(*[t.cpu() for t in x], K, with_features=False)
    assert np.array_equal(out[3].cpu().numpy(), i_ref)
    d = out[2].cpu().numpy()
    assert np.array_equal(np.isnan(d), np.isnan(d_ref))  # the GPU's and the CPU's NaN differ in their payload
    assert np.array_equal(d.view(np.int32)[~np.isnan(d)], d_ref.view(np.int32)[~np.isnan(d)])


@pytest.mark.parametrize("B,Q,P,K", [
    (9, 7, 3, 2),        # 128 chunks of an element's points, most of them empty
    (10, 5, 200, 3),     # 64
    (75, 5, 70, 5),      # 8
    (593, 3, 33, 4),     # 1
    (1200, 2, 300, 3),   # 1, and more of them than run at a time
])
def test_many_elements_match_the_cpu_oracle(B, Q, P, K):
    from cuda_knn_aggregate import capi

    x = _inputs("rand", B, Q, P, 4, torch.float32, seed=B)
    out = _call(x, K, capi.lib().knnag_forward_workspace_bytes(B, Q, P, 4, K, capi.F32))
    _, _, d_ref, i_ref = O.forward_f32(*[t.cpu() for t in x], K, with_features=False)
    assert np.array_equal(out[3].cpu().numpy(), i_ref)
    assert np.array_equal(out[2].cpu().numpy().view(np.int32), d_ref.view(np.int32))


@pytest.mark.parametrize("P,K,order", [
    (700, 12, "lattice"),       # one CTA per query, first ranges only
    (9000, 32, "lattice"),      # two CTAs, two ranges per warp
    (70000, 16, "lattice"),     # eight CTAs
    (70000, 24, "descending"),  # every key is below all before it: more points kept than are merged at a time
])
def test_flagged_queries_replay_as_the_cpu_oracle(P, K, order):
    """Tied keys everywhere (every query is replayed): MinK's order of equal
    keys depends on the whole history of its slots."""
    from cuda_knn_aggregate import capi

    g = torch.Generator().manual_seed(P)
    Q = 23
    q = (torch.rand(1, Q, 3, generator=g) * 8).round() / 8
    p = (torch.rand(1, P, 3, generator=g) * 12).round() / 8
    if order == "descending":
        p = 2 + (torch.arange(P, 0, -1, dtype=torch.float64) / P).to(torch.float32)[None, :, None].expand(1, P, 3)
        p = torch.cat([p, p[:, -K:]], 1).contiguous()  # the nearest ones twice
    P = p.shape[1]
    x = [t.contiguous() for t in (q, p, torch.rand(1, P, 4, generator=g), torch.ones(1, P, 3),
                                  torch.eye(3).expand(1, P, 3, 3))]
    out = _call([t.to(DEV) for t in x], K, capi.lib().knnag_forward_workspace_bytes(1, Q, P, 4, K, capi.F32))
    _, _, d_ref, i_ref = O.forward_f32(*x, K, with_features=False)
    assert np.array_equal(out[3].cpu().numpy(), i_ref)
    assert np.array_equal(out[2].cpu().numpy().view(np.int32), d_ref.view(np.int32))


def _scaled(dtype, Q, P, at, row, sig, seed):
    """Unit-cube clouds with rotations, coordinates times `at`, rows of R times `row`, sigma times `sig`."""
    g = torch.Generator().manual_seed(seed)
    q = torch.rand(1, Q, 3, generator=g, dtype=torch.float64) * at
    p = torch.rand(1, P, 3, generator=g, dtype=torch.float64) * at
    f = torch.rand(1, P, 4, generator=g, dtype=torch.float64)
    sigma = (torch.rand(1, P, 3, generator=g, dtype=torch.float64) + 0.5) * sig
    R = torch.linalg.qr(torch.randn(1, P, 3, 3, generator=g, dtype=torch.float64))[0] * row
    return [t.to(dtype).contiguous() for t in (q, p, f, sigma, R)]


# Scales at which the bounds that cull tiles leave the range of FP32 (they are
# FP32 for FP64 calls too) while every key is finite and almost all differ.
@pytest.mark.parametrize("dtype,K,at,row,sig", [
    (torch.float64, 16, 1e21, 1, 1),         # squared distances above the largest float
    (torch.float64, 16, 1e21, 1, 1e-42),     # and the bound factor below the normal ones
    (torch.float64, 16, 1e21, 1, 1e-44),
    (torch.float64, 16, 1, 1, 1e39),         # the bound factor above the largest float
    (torch.float64, 33, 1e10, 1, 1e25),      # the product
    (torch.float64, 16, 3e-22, 1, 1),        # squared distances among the subnormal ones
    (torch.float64, 16, 3e-20, 1, 1e30),
    (torch.float64, 65, 1e-160, 1, 1),       # below them
    (torch.float64, 16, 1e40, 1, 1),         # coordinates above the largest float
    (torch.float64, 16, 1, 1e-7, 1),         # short rows
    (torch.float32, 40, 1e21, 1e-3, 1),
    (torch.float32, 40, 1e-4, 1e10, 1e20),
    (torch.float32, 40, 3e-20, 1, 1),        # subnormal keys
    (torch.float32, 40, 3e-20, 1, 1e30),
    (torch.float32, 40, 1e-18, 1e-3, 1e30),  # squares of rotated offsets among the subnormal ones
    (torch.float32, 40, 1e-14, 1e-7, 1e30),
])
def test_bounds_at_scales_beyond_the_floats_range(dtype, K, at, row, sig):
    x = [t.to(DEV) for t in _scaled(dtype, 200, 4096, at, row, sig, seed=K)]
    _compare(x, K)


@pytest.mark.parametrize("at,row,sig", [
    (1e21, 1e-3, 1), (1e-4, 1e10, 1e20), (3e-20, 1, 1), (3e-20, 1, 1e30), (1e-18, 1e-3, 1e30), (1e-14, 1e-7, 1e30),
])
def test_scaled_forward_matches_the_cpu_oracle(at, row, sig):
    from cuda_knn_aggregate import capi

    x = _scaled(torch.float32, 200, 4096, at, row, sig, seed=5)
    out = _call([t.to(DEV) for t in x], 16, capi.lib().knnag_forward_workspace_bytes(1, 200, 4096, 4, 16, capi.F32))
    _, _, d_ref, i_ref = O.forward_f32(*x, 16, with_features=False)
    assert np.isfinite(d_ref).all()
    assert np.array_equal(out[3].cpu().numpy(), i_ref)
    assert np.array_equal(out[2].cpu().numpy().view(np.int32), d_ref.view(np.int32))


@pytest.mark.parametrize("dtype,P,K", [
    (torch.float32, 64, 32), (torch.float32, 128, 64), (torch.float64, 200, 128), (torch.float32, 256, 128),
])
def test_zeros_of_either_sign_tie(dtype, P, K):
    """K - 1 negative keys, then +0 and -0: equal, so the first of the two
    points in index order takes the last place of a full list."""
    from cuda_knn_aggregate import capi

    q, p, f, _, R = _scaled(dtype, 9, P, 1, 1, 1, seed=K)
    sigma = torch.ones(1, P, 3, dtype=dtype)
    sigma[:, 1:K] = -1
    sigma[:, 0], sigma[:, K] = 0.0, -0.0
    x = [q, p, f, sigma, R]
    if P >= 128:
        _compare([t.to(DEV) for t in x], K)
    if dtype == torch.float32:
        out = _call([t.to(DEV) for t in x], K, capi.lib().knnag_forward_workspace_bytes(1, 9, P, 4, K, capi.F32))
        assert np.array_equal(out[3].cpu().numpy(), O.forward_f32(*x, K, with_features=False)[3])


@pytest.mark.parametrize("dtype,B,Q,P,F,K", [
    (torch.float64, 1, 400, 128, 5, 1),      # one chunk of points
    (torch.float64, 1, 400, 512, 4, 32),     # K <= 32: a whole one,
    (torch.float64, 3, 160, 513, 4, 9),      # and a point more; several clouds
    (torch.float64, 1, 170, 385, 4, 64),     # K <= 64,
    (torch.float64, 1, 170, 1537, 4, 65),    # K <= 128
    (torch.float32, 1, 400, 768, 4, 33), (torch.float32, 2, 300, 1537, 4, 64), (torch.float32, 1, 200, 1025, 4, 128),
    (torch.float32, 1, 500, 33000, 4, 40),   # clusters of eight CTAs
    (torch.float64, 90, 11, 150, 4, 3),      # sixteen queries of two or three clouds
    (torch.float64, 2, 2100000, 128, 1, 2),  # more rows than are put in order
])
def test_many_flagged_queries(dtype, B, Q, P, F, K):
    _compare(_inputs("ties", B, Q, P, F, dtype, seed=P + K), K)


@pytest.mark.parametrize("B,Q,P,K", [(1, 400, 1024, 32), (5, 100, 1025, 7), (1, 190, 12000, 16), (2, 160000, 130, 3)])
def test_many_flagged_queries_match_the_cpu_oracle(B, Q, P, K):
    from cuda_knn_aggregate import capi

    x = _inputs("ties", B, Q, P, 4, torch.float32, seed=Q + P)
    out = _call(x, K, capi.lib().knnag_forward_workspace_bytes(B, Q, P, 4, K, capi.F32))
    _, _, d_ref, i_ref = O.forward_f32(*[t.cpu() for t in x], K, with_features=False)
    assert np.array_equal(out[3].cpu().numpy(), i_ref)
    assert np.array_equal(out[2].cpu().numpy().view(np.int32), d_ref.view(np.int32))


def test_many_flagged_queries_of_ragged_clouds():
    """Segments of tied clouds of very different sizes, each equal to the uniform op's call."""
    from cuda_knn_aggregate import knn_aggregate_aniso
    from cuda_knn_aggregate.ragged import CloudSet, ragged_forward

    sizes = [40, 700, 5, 20000, 1025, 3000, 64]
    xs = [_inputs("ties", 1, 1, P, 4, torch.float32, seed=P) for P in sizes]
    cloud = lambda k: torch.cat([x[k][0] for x in xs]).contiguous()  # noqa: E731
    clouds = CloudSet(cloud(1), cloud(3), cloud(4), cloud(2), sizes)
    order = [3, 0, 1, 2, 1, 4, 5, 6, 3, 5]
    Qs = [90, 33, 301, 7, 1, 160, 200, 64, 45, 500]
    Ks = [16, 32, 3, 5, 1, 12, 8, 32, 9, 31]
    qs = [_inputs("ties", 1, Q, 1, 1, torch.float32, seed=Q)[0][0] for Q in Qs]
    out = ragged_forward(clouds, torch.cat(qs).contiguous(), order, Qs, Ks)
    q0 = e0 = 0
    for c, Q, K, q in zip(order, Qs, Ks, qs):
        _, p, f, sigma, R = xs[c]
        f_out, w, dists, idxs = knn_aggregate_aniso(q[None], p, f, sigma, R, K)
        for got, want in ((out.f_out[q0:q0 + Q], f_out[0]), (out.w_out[e0:e0 + Q * K], w[0].reshape(-1)),
                          (out.dists[e0:e0 + Q * K], dists[0].reshape(-1))):
            assert torch.equal(_bits(got), _bits(want))
        assert torch.equal(out.idxs[e0:e0 + Q * K], idxs[0].reshape(-1))
        q0, e0 = q0 + Q, e0 + Q * K


def test_group_boxes_of_ragged_clouds():
    """Boxes of groups of 32 tiles are built where a cloud has more than two
    groups, and only there: a launch less with at most 8192 points."""
    from cuda_knn_aggregate import capi, knn_aggregate_aniso
    from cuda_knn_aggregate.ragged import CloudSet, ragged_forward

    launches = []
    for sizes in ([8192, 300], [8193, 300]):
        xs = [_inputs("rand", 1, 60, P, 4, torch.float32, seed=P) for P in sizes]
        cloud = lambda k: torch.cat([x[k][0] for x in xs]).contiguous()  # noqa: E731
        clouds = CloudSet(cloud(1), cloud(3), cloud(4), cloud(2), sizes)
        before = capi.launch_count()
        clouds.build()
        launches.append(capi.launch_count() - before)
        out = ragged_forward(clouds, cloud(0), [0, 1], [60, 60], [24, 24])
        for i, x in enumerate(xs):
            f_out, w, dists, idxs = knn_aggregate_aniso(*x, 24)
            assert torch.equal(out.f_out[60 * i:60 * i + 60], f_out[0])
            assert torch.equal(out.idxs[1440 * i:1440 * i + 1440], idxs[0].reshape(-1))
    assert launches[0] == launches[1] - 1
