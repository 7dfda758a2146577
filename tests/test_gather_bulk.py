"""The gather's bulk launch (one thread sets a query up) against its launch for few
queries (a warp does), bit for bit, and against exhaustive search.  From 18,944
queries on a call takes the bulk form, with 16 queries a block; 2.5M queries come
256 a block."""
import numpy as np
import pytest

from test_gather_paths import BOX, _exhaustive

FIRST_BULK = 18_944


def _inputs(layout, photons=6000):
    rng = np.random.default_rng(11)
    pos = rng.uniform(-1, 1, (photons, 3)).astype(np.float32)
    pos[:, 1] = np.where(rng.random(photons) < 0.7, -0.98, pos[:, 1])
    if layout == "lattice":      # many equal distances
        pos = (np.round(pos * 8) / 8).astype(np.float32)
    if layout == "clump":        # full stores, empty cells elsewhere
        pos = np.where(rng.random((photons, 1)) < 0.6, pos * 0.02 + 0.3, pos).astype(np.float32)
    if layout == "outside":      # photons beyond the grid's box, kept in its outermost cells
        pos = np.where(rng.random((photons, 1)) < 0.3, pos * 1.5, pos).astype(np.float32)
    q = np.concatenate([pos[rng.integers(0, photons, 40)] + rng.normal(0, 0.01, (40, 3)),
                        rng.uniform(-1.6, 1.6, (29, 3)), pos[:2]]).astype(np.float32)
    return (pos, rng.uniform(0.1, 1, (photons, 3)).astype(np.float32), rng.standard_normal((photons, 3)).astype(np.float32),
            q, rng.standard_normal(q.shape).astype(np.float32))


def _bulk_equals_few(ctx, q, qn, n, k, radius):
    import torch
    m = q.shape[0]
    at = torch.arange(n, device="cuda") % m
    many, many_n = q[at], qn[at]
    torch.cuda.synchronize()                                   # the context has a stream of its own
    few = ctx.gather(q, qn, k, radius, want_ids=True)
    bulk = ctx.gather(many, many_n, k, radius, want_ids=True)
    for a, b in zip(few, bulk):
        # bits: a photon at its query alone gives 0 / 0
        a, b = (x.reshape(-1, x.numel() // r).view(torch.int32) for x, r in ((a, m), (b, n)))
        assert torch.equal(b, a[at]), (n, k, radius)
    return few


@pytest.mark.gpu
@pytest.mark.parametrize("sub_div", [1, 2, 4, 8])
@pytest.mark.parametrize("layout", ["surface", "lattice", "clump", "outside"])
def test_bulk_equals_few_and_exhaustive_search(sub_div, layout):
    import torch
    import photonmap
    pos, power, inc, q, qn = _inputs(layout)
    ctx = photonmap.Context(0)
    ctx.set_photons(0, pos, power, inc)
    ctx.build_grid(0, aabb=BOX, sub_div=sub_div, desired=50)
    tq, tn = torch.from_numpy(q).cuda(), torch.from_numpy(qn).cuda()
    for k, r in ((1, 0.5), (64, 0.03), (65, 0.2), (97, 0.2), (161, 0.6), (256, 0.05), (256, 4.0)):
        for n in (FIRST_BULK - 1, FIRST_BULK, FIRST_BULK + 77):
            rad, ids, cnt = _bulk_equals_few(ctx, tq, tn, n, k, r)
        want, ref = _exhaustive(pos, power, inc, q, qn, k, r)
        assert np.array_equal(ids.cpu().numpy(), want), (k, r)
        assert np.array_equal(cnt.cpu().numpy(), (want >= 0).sum(1)), (k, r)
        # as in test_gather_paths: sums of at most 256 positive float32 terms
        ok = ref.sum(1) > 0
        np.testing.assert_allclose(rad.cpu().numpy()[ok], ref[ok], rtol=1e-5)
    assert ctx.status() == 0
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [200_003, 2_500_001])
def test_larger_blocks_of_queries(n):
    import torch
    import photonmap
    pos, power, inc, q, qn = _inputs("surface")
    ctx = photonmap.Context(0)
    ctx.set_photons(0, pos, power, inc)
    ctx.build_grid(0, aabb=BOX, sub_div=4, desired=50)
    for k, r in ((1, 0.1), (16, 0.6)):
        _bulk_equals_few(ctx, torch.from_numpy(q).cuda(), torch.from_numpy(qn).cuda(), n, k, r)
    assert ctx.status() == 0
    ctx.close()
