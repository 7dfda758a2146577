"""The gather's choice of the k-th distance where many candidates share a bin of its
histogram: shells of nearly equal distances (steps of one float), few distinct
distances, exact duplicates, and dense places that fill the store over and over,
against exhaustive search."""
import numpy as np
import pytest

from test_gather_paths import BOX, _exhaustive


def _photons(layout, rng):
    u = rng.standard_normal((3000, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    if layout == "shell":            # squared distances from the origin within some 40 floats
        return (0.25 * u * (1 + 1e-6 * rng.standard_normal((3000, 1)))).astype(np.float32)
    if layout == "steps":            # nine distances, each hundreds of times
        return (u * (0.05 * rng.integers(1, 10, (3000, 1)))).astype(np.float32)
    if layout == "copies":           # 60 places, 50 photons in each
        return np.repeat((0.3 * u[:60]).astype(np.float32), 50, 0)[rng.permutation(3000)]
    r = 10 ** rng.uniform(-7, 0, (3000, 1))   # "scales": distances over seven decades
    return (u * r).astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("sub_div", [1, 4])
@pytest.mark.parametrize("layout", ["shell", "steps", "copies", "scales"])
def test_full_bins(sub_div, layout):
    import torch
    import photonmap
    rng = np.random.default_rng(7)
    pos = _photons(layout, rng)
    one = np.ones_like(pos)
    q = np.concatenate([np.zeros((1, 3)), 1e-4 * rng.standard_normal((5, 3)), pos[:3],
                        rng.uniform(-1, 1, (4, 3))]).astype(np.float32)
    qn = np.tile(np.array([[0, 0, -1]], np.float32), (len(q), 1))
    ctx = photonmap.Context(0)
    ctx.set_photons(0, pos, one, one)
    ctx.build_grid(0, aabb=BOX, sub_div=sub_div, desired=500)
    for k in (1, 31, 33, 64, 65, 97, 200, 256):
        for r in (0.25, 0.6, 4.0, 1e6):
            rad, ids, cnt = ctx.gather(torch.from_numpy(q), torch.from_numpy(qn), k, r, want_ids=True)
            want, ref = _exhaustive(pos, one, one, q, qn, k, r)
            assert np.array_equal(ids.cpu().numpy(), want), (k, r)
            assert np.array_equal(cnt.cpu().numpy(), (want >= 0).sum(1)), (k, r)
            # as in test_gather_paths: sums of at most 256 positive float32 terms
            ok = ref.sum(1) > 0
            np.testing.assert_allclose(rad.cpu().numpy()[ok], ref[ok], rtol=1e-5)
    assert ctx.status() == 0
    ctx.close()
