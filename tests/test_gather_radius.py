"""The kNN gather with radii far beyond the map, infinity among them, against
exhaustive search."""
import numpy as np
import pytest

from test_gather_paths import BOX, _exhaustive


def _map(photons, seed=5):
    rng = np.random.default_rng(seed)
    pos = rng.uniform(-1, 1, (photons, 3)).astype(np.float32)
    pos[:, 1] = np.where(rng.random(photons) < 0.7, -0.98, pos[:, 1])
    return pos, rng.uniform(0.1, 1, (photons, 3)).astype(np.float32), rng.standard_normal((photons, 3)).astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("sub_div", [1, 4])
@pytest.mark.parametrize("photons", [1, 10, 64, 65, 999])
@pytest.mark.parametrize("radius", [1e9, 1e30, np.inf])
def test_radius_beyond_the_map(sub_div, photons, radius):
    import torch
    import photonmap
    pos, power, inc = _map(photons)
    rng = np.random.default_rng(6)
    q = np.concatenate([rng.uniform(-1.3, 1.3, (21, 3)), pos[:1] + 0.001]).astype(np.float32)
    qn = rng.standard_normal(q.shape).astype(np.float32)
    ctx = photonmap.Context(0)
    ctx.set_photons(0, pos, power, inc)
    ctx.build_grid(0, aabb=BOX, sub_div=sub_div, desired=10)
    for k in (10, 64, 256):
        rad, ids, cnt = ctx.gather(torch.from_numpy(q), torch.from_numpy(qn), k, radius, want_ids=True)
        want, ref = _exhaustive(pos, power, inc, q, qn, k, radius)
        assert np.array_equal(ids.cpu().numpy(), want), k
        assert np.array_equal(cnt.cpu().numpy(), (want >= 0).sum(1)), k
        # at most 256 positive float32 terms, as in test_gather_paths
        ok = ref.sum(1) > 0
        np.testing.assert_allclose(rad.cpu().numpy()[ok], ref[ok], rtol=1e-5)
    assert ctx.status() == 0
    ctx.close()


@pytest.mark.gpu
def test_box_of_ten_million_rows():
    """A sphere that covers a grid of 3 x 400 x 400 cells, each cut 8 ways: 10.24M
    rows of sub-cells in 3 runs each."""
    import torch
    import photonmap
    rng = np.random.default_rng(2)
    size = np.array([3, 400, 400], np.float32)
    pos = (rng.random((480_000, 3)) * size).astype(np.float32)
    pos[-3:] = size - np.float32(0.01)      # the last sub-cell of the last row holds photons
    ctx = photonmap.Context(0)
    ctx.set_photons(0, pos, np.ones_like(pos), np.ones_like(pos))
    ctx.build_grid(0, aabb=np.concatenate([0 * size, size]), sub_div=8, desired=1)
    assert ctx.photons(0)["dims"] == (3, 400, 400)
    q = np.array([[-2000, 200, 200], [1.5, 200, 3000], [1.5, 900, 900]], np.float32)
    qn = np.zeros_like(q)
    for k in (8, 256):
        _, ids, cnt = ctx.gather(torch.from_numpy(q), torch.from_numpy(qn), k, 1e4, want_ids=True)
        want, _ = _exhaustive(pos, np.ones_like(pos), np.ones_like(pos), q, qn, k, 1e4)
        assert np.array_equal(ids.cpu().numpy(), want), k
    assert ctx.status() == 0
    ctx.close()
