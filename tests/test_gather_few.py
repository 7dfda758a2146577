"""The gather's launch for few queries (one per warp, set up by the warp) against its
bulk launch, and the order of its ids, where many distances tie, against an
exhaustive search: the ids, counts and estimates are the same bits."""
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("k", [1, 31, 33, 200, 256])
@pytest.mark.parametrize("radius", [0.02, 0.1, 0.6])
def test_few_queries_equal_many_and_ids_are_ordered(k, radius):
    import torch
    import photonmap
    gen = torch.Generator(device="cuda")
    gen.manual_seed(k)
    # photons on a plane and in a corner of it, every position three times
    p = torch.rand((6000, 3), generator=gen, device="cuda")
    p[:, 2] = 0.5
    p[4500:, :2] *= 0.05
    pos = p.repeat(3, 1)[torch.randperm(18000, generator=gen, device="cuda")].contiguous()
    pw, d = torch.full_like(pos, 0.25), torch.randn((18000, 3), generator=gen, device="cuda")
    ctx = photonmap.Context(0)
    ctx.set_photons(0, pos, pw, d)
    import numpy as np
    ctx.build_grid(0, aabb=np.array([0, 0, 0, 1, 1, 1], np.float32), sub_div=4, desired=200)
    q = torch.rand((9600, 3), generator=gen, device="cuda")
    q[:, 2] = 0.5
    q[:100] = p[:100]
    q[100:150] = p[5000:5050]
    nrm = torch.zeros_like(q)
    nrm[:, 2] = 1
    few = ctx.gather(q[:203].contiguous(), nrm[:203].contiguous(), k, radius, want_ids=True)
    many = ctx.gather(q, nrm, k, radius, want_ids=True)
    for a, b in zip(few, many):
        # bits: a photon at its query alone gives 0 / 0
        assert torch.equal(a.view(torch.int32), b.reshape((9600,) + tuple(a.shape[1:]))[:203].view(torch.int32))
    v = q[:203, None, :] - pos[None]
    dist = torch.sqrt(v[..., 0] * v[..., 0] + v[..., 1] * v[..., 1] + v[..., 2] * v[..., 2])
    key = dist.view(torch.int32).long() << 32 | torch.arange(18000, device="cuda")
    key = torch.where(dist <= radius, key, torch.full_like(key, 1 << 62)).sort(1).values[:, :k]
    want = torch.where(key < 1 << 62, key & 0xffffffff, torch.full_like(key, 0xffffffff))
    got = few[1].reshape(203, k).to(torch.int64) & 0xffffffff
    assert torch.equal(got, want)
    assert torch.equal(few[2].long().reshape(-1), (key < 1 << 62).sum(1))
    assert ctx.status() == 0
    ctx.close()
