"""The radix sort behind the grid's photon order and the device BVH: stable at the
edges of its tiles and of its two forms (look-back up to 444 tiles of 4096 keys,
runs of tiles beyond)."""
import numpy as np
import pytest

BOX = np.array([0, 0, 0, 1, 1, 1], np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 4095, 4096, 4097, 444 * 4096 - 1, 444 * 4096, 444 * 4096 + 1, 2 * 444 * 4096 + 4099])
@pytest.mark.parametrize("spread", [1.0, 0.01])
def test_grid_order_is_a_stable_sort(n, spread):
    import torch
    import photonmap
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    pos = torch.rand((n, 3), generator=gen, device="cuda") * spread
    pw, d = torch.full_like(pos, 0.5), torch.full_like(pos, 1.0)
    ctx = photonmap.Context(0)
    ctx.set_photons(0, pos, pw, d)
    ctx.build_grid(0, aabb=BOX, sub_div=4, desired=200)
    g = ctx.photons(0)
    order = g["sorted_pos"][:, 3].contiguous().view(torch.int32).long()
    starts = g["key_starts"].long()
    assert torch.equal(torch.sort(order).values, torch.arange(n, device="cuda"))
    assert torch.equal(g["sorted_pos"][:, :3], pos[order])
    assert int(starts[0]) == 0 and int(starts[-1]) == n and bool((starts[1:] >= starts[:-1]).all())
    # the key of every slot, from the ranges; the source order is kept inside a key
    key = torch.searchsorted(starts, torch.arange(n, device="cuda"), right=True) - 1
    same = key[1:] == key[:-1]
    assert bool((order[1:] > order[:-1])[same].all())
    # ... and every photon lies in its key's sub-cell
    S, (gx, gy, _), cell = g["sub_div"], g["dims"], g["cell"]
    u = pos[order] / torch.tensor(cell, device="cuda")
    c = torch.minimum(u.int().clamp_min(0), torch.tensor(g["dims"], device="cuda").int() - 1)
    s = ((u - c) * S).int().clamp(0, S - 1)
    want = (c[:, 0] + c[:, 1] * gx + c[:, 2] * gx * gy).long() * S ** 3 + (s[:, 0] + S * (s[:, 1] + S * s[:, 2])).long()
    assert torch.equal(key, want)
    counts = torch.bincount(key // S ** 3, minlength=g["cells"])
    assert torch.equal(g["cell_sizes"].long(), counts)
    assert torch.equal(g["cell_starts"].long(), torch.cumsum(counts, 0) - counts)
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("m", [1, 2, 3, 31, 32, 33])
@pytest.mark.parametrize("n", [512 * 9 - 5, 512 * 3600 - 13])        # look-back, runs
def test_running_counts_pass_from_lane_to_lane(n, m):
    """Keys whose leader lane moves from one step of 32 to the next, so that each
    step reads the running count that another lane wrote."""
    import torch
    import photonmap
    i = torch.arange(n, device="cuda")
    lane, step = i & 31, i >> 5
    key = (lane + step) % m                                 # m sub-cells along x, rotated by one lane a step
    pos = torch.zeros((n, 3), device="cuda")
    pos[:, 0] = (key.float() + 0.5) / 64
    pw = torch.full_like(pos, 0.5)
    torch.cuda.synchronize()                                # the context has a stream of its own
    ctx = photonmap.Context(0)
    ctx.set_photons(0, pos, pw, pw)
    ctx.build_grid(0, aabb=BOX, sub_div=8, desired=-(-n // 512), regrid_mult=1000)   # 64 sub-cells along x
    g = ctx.photons(0)
    assert g["dims"] == (8, 8, 8) and g["cell"] == 0.125
    order = g["sorted_pos"][:, 3].contiguous().view(torch.int32).long()
    assert torch.equal(order, torch.sort(key, stable=True).indices)
    ctx.close()
