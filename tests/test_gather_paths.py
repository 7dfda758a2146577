"""The kNN gather at the edges of its paths (few photons, full stores, ties,
sparse cubes, every sub-cell split and store size) against exhaustive search."""
import numpy as np
import pytest

BOX = np.array([-1, -1, -1, 1, 1, 1], np.float32)


def _exhaustive(pos, power, inc, q, qn, k, r):
    """ids ascending by (float32 distance, index), and the estimate in float64."""
    ids = np.full((len(q), k), -1, np.int32)
    rad = np.zeros((len(q), 3))
    for i, (p, n) in enumerate(zip(q, qn)):
        d = pos - p
        dist = np.sqrt((d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2])   # float32, the kernel's order
        near = np.flatnonzero(dist <= np.float32(r))
        near = near[np.lexsort((near, dist[near]))][:k]
        ids[i, :len(near)] = near
        if len(near) == 0 or dist[near[-1]] == 0:
            continue
        rk = float(dist[near[-1]])
        f = 1.818 * (1 - (1 - np.exp(-1.953 * dist[near].astype(np.float64) ** 2 / (2 * rk * rk))) / (1 - np.exp(-1.953)))
        f *= (inc[near].astype(np.float64) @ n.astype(np.float64)) < 0
        rad[i] = (power[near] * f[:, None]).sum(0) / (np.pi * rk * rk)
    return ids, rad


@pytest.mark.gpu
@pytest.mark.parametrize("sub_div", [1, 2, 4, 8])
@pytest.mark.parametrize("photons", [1, 33, 6000])
@pytest.mark.parametrize("layout", ["surface", "lattice", "clump"])
def test_gather_equals_exhaustive_search(sub_div, photons, layout):
    import torch
    import photonmap
    rng = np.random.default_rng(photons)
    pos = rng.uniform(-1, 1, (photons, 3)).astype(np.float32)
    pos[:, 1] = np.where(rng.random(photons) < 0.7, -0.98, pos[:, 1])
    if layout == "lattice":      # many equal distances: ties by index
        pos = (np.round(pos * 8) / 8).astype(np.float32)
    if layout == "clump":        # full stores and bins, empty cells elsewhere
        pos = np.where(rng.random((photons, 1)) < 0.6, pos * 0.02 + 0.3, pos).astype(np.float32)
    inc = rng.standard_normal((photons, 3)).astype(np.float32)
    power = rng.uniform(0.1, 1, (photons, 3)).astype(np.float32)
    q = np.concatenate([pos[rng.integers(0, photons, 24)] + rng.normal(0, 0.01, (24, 3)),
                        rng.uniform(-1.3, 1.3, (17, 3)), pos[:1]]).astype(np.float32)
    qn = rng.standard_normal(q.shape).astype(np.float32)
    ctx = photonmap.Context(0)
    ctx.set_photons(0, pos, power, inc)
    ctx.build_grid(0, aabb=BOX, sub_div=sub_div, desired=50)
    for k, r in ((1, 0.5), (64, 0.03), (65, 0.2), (97, 0.2), (161, 0.6), (256, 0.05), (256, 4.0)):
        rad, ids, cnt = ctx.gather(torch.from_numpy(q), torch.from_numpy(qn), k, r, want_ids=True)
        want, ref = _exhaustive(pos, power, inc, q, qn, k, r)
        assert np.array_equal(ids.cpu().numpy(), want), (k, r)
        assert np.array_equal(cnt.cpu().numpy(), (want >= 0).sum(1)), (k, r)
        # sums of at most 256 positive float32 terms in 8 + 5 additions, each term
        # a few roundings and an exponential: 1e-5 is over ten times their bound
        ok = ref.sum(1) > 0
        np.testing.assert_allclose(rad.cpu().numpy()[ok], ref[ok], rtol=1e-5)
    ctx.close()
