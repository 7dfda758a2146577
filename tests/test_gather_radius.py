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


def _tied(target):
    """(x, y) with x * x + y * y == target in float32."""
    for x in np.linspace(0.6, 0.9, 4001, dtype=np.float32) * np.sqrt(target):
        y = np.sqrt(target - x * x)
        for _ in range(8):
            y = np.nextafter(y, np.float32(0))
        for _ in range(16):
            if np.float32(x * x) + np.float32(y * y) == target:
                return x, y
            y = np.nextafter(y, np.float32(1))
    raise AssertionError("no such point")


@pytest.mark.gpu
@pytest.mark.parametrize("first", ["sphere", "guess"])
def test_equal_distances_on_either_side_of_the_first_bound(first):
    """The two farthest of k + 1 photons have one rounded distance, their squares
    lie on either side of the walk's first bound: the smaller index stays."""
    import torch
    import photonmap
    if first == "sphere":        # nothing in the 27 sub-cells of edge 1 / 8: (8 / 8)^2
        k, S, lo, bound = 4, 8, 0.0, np.float32(1)
        near = 0.5 * np.eye(3)
        far = np.zeros((0, 3))
    else:                        # the density guess of 1.6 k photons among N in a plane of 9 sub-cells of edge 1 / 4
        k, S, lo = 8, 4, -0.5
        for N in range(30, 60):
            bound = np.float32(0.5625) * (np.float32(1.6) * np.float32(k)) / (np.float32(3.14159265) * np.float32(N))
            if np.sqrt(bound) == np.sqrt(np.nextafter(bound, np.float32(1))):
                break
        near = np.stack([np.linspace(0.01, 0.1, k - 1), np.zeros(k - 1), np.zeros(k - 1)], 1)
        far = np.stack([np.linspace(0.4, 0.45, N - k - 1), np.zeros(N - k - 1), np.zeros(N - k - 1)], 1)
    beyond = np.nextafter(bound, np.float32(2))
    assert np.sqrt(beyond) == np.sqrt(bound)
    inside, outside = _tied(bound), _tied(beyond)
    pos = np.concatenate([[[outside[0], outside[1], 0]], near, far, [[inside[0], inside[1], 0]]]).astype(np.float32)
    one = np.ones_like(pos)
    ctx = photonmap.Context(0)
    ctx.set_photons(0, pos, one, one)
    ctx.build_grid(0, aabb=np.array([lo] * 3 + [lo + 1] * 3, np.float32), sub_div=S, desired=1000)
    q = np.zeros((1, 3), np.float32)
    _, ids, _ = ctx.gather(torch.from_numpy(q), torch.from_numpy(q), k, 2.0, want_ids=True)
    want, _ = _exhaustive(pos, one, one, q, q, k, 2.0)
    assert 0 in want and len(pos) - 1 not in want
    assert np.array_equal(ids.cpu().numpy(), want)
    ctx.close()


def _time(ctx, q, qn, k, radius):
    import torch
    best = float("inf")
    for _ in range(6):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        ctx.gather(q, qn, k, radius)
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b))
    return best


@pytest.mark.gpu
@pytest.mark.parametrize("k", [16, 200])
def test_time_does_not_grow_with_a_radius_that_holds_more_than_k(k):
    """Photons on the walls of a box and on a ball that lies on its floor; the radius
    stops mattering once it holds k photons.  Near the ball the density guess
    holds too few (such walks, their next bound the radius itself, made the calls
    take several times as long with a radius of 100 boxes)."""
    import torch
    import photonmap
    gen = torch.Generator(device="cuda")
    gen.manual_seed(4)

    def photons(n):
        p = torch.rand((n, 3), generator=gen, device="cuda") * 2 - 1
        axis = torch.randint(0, 3, (n, 1), generator=gen, device="cuda")
        p = p.scatter(1, axis, torch.where(torch.rand((n, 1), generator=gen, device="cuda") < 0.5, -1.0, 1.0))
        ball = torch.nn.functional.normalize(torch.randn((n, 3), generator=gen, device="cuda")) * 0.3
        ball[:, 1] -= 0.7
        return torch.where(torch.rand((n, 1), generator=gen, device="cuda") < 0.3, ball, p).contiguous()

    pos, q = photons(1_000_000), photons(20_000)
    one = torch.ones_like(pos)
    torch.cuda.synchronize()                             # the context has a stream of its own
    ctx = photonmap.Context(0)
    ctx.set_photons(0, pos, one, one)
    ctx.build_grid(0, aabb=BOX)
    qn = -q
    torch.cuda.synchronize()
    near, far = (ctx.gather(q, qn, k, r, want_ids=True) for r in (0.5, 200.0))
    for a, b in zip(near, far):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    assert bool((near[2] == k).all())
    assert _time(ctx, q, qn, k, 200.0) < 2 * _time(ctx, q, qn, k, 0.5)
    ctx.close()


@pytest.mark.gpu
def test_time_does_not_grow_with_a_radius_beyond_few_photons():
    """Fewer than k photons in a grid of many sub-cells: the walk ends soon after its
    sphere has passed the grid, however large the radius."""
    import torch
    import photonmap
    pos, power, inc = _map(255)
    half = np.array([0.0625, 1, 1], np.float32)          # 1 x 16 x 16 cells, each cut 8 ways: 16,384 rows
    pos *= half
    q = torch.from_numpy(np.random.default_rng(3).uniform(-half, half, (500, 3)).astype(np.float32)).cuda()
    ctx = photonmap.Context(0)
    ctx.set_photons(0, pos, power, inc)
    ctx.build_grid(0, aabb=np.concatenate([-half, half]), sub_div=8, desired=1)
    assert ctx.photons(0)["dims"] == (1, 16, 16)
    near, far = (ctx.gather(q, q, 256, r, want_ids=True) for r in (4.0, 1e18))
    for a, b in zip(near, far):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    assert bool((near[2] == 255).all())
    assert _time(ctx, q, q, 256, 1e18) < 3 * _time(ctx, q, q, 256, 4.0)
    ctx.close()
