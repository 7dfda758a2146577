"""The eye pass's pixel order (tiles of 32 x 4 in bands of 4 rows, the last columns
and rows row by row): frames whose sizes leave whole tiles, remainders of either
kind or nothing but remainders, against the oracle; bands of rows that start and
end inside a band of 4 are the full frame's, bit for bit, and 0 outside."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("W,H", [(32, 4), (31, 3), (33, 5), (64, 9), (100, 7), (3, 50)])
def test_ragged_frames_and_row_bands(orc, W, H):
    import photonmap
    from photonmap import scenes
    sc, _, _ = scenes.workload("cornell_small")
    ctx = photonmap.Context(0)
    ctx.set_scene(sc)
    s = orc.scene(sc)
    ctx.trace_photons(3, 8, 20_000)
    ctx.build_grid(0)
    tr = s.trace_photons(3, 8, 20_000)
    g = orc.grid_build(tr["g_pos"], tr["g_pow"], tr["g_dir"], s.aabb(), sub_div=ctx.photons(0)["sub_div"])
    cam = photonmap.camera_setup((0, 0, 3.5), (0, 0, -1), (0, 1, 0), 45.0, W, H)
    _, rad = ctx.render(cam, 40, 0.2, 4)
    full = rad.cpu().numpy()
    # estimates of up to 40 terms in the same order: the bound of the parity tests
    np.testing.assert_allclose(full, s.render(cam.as_vector(), W, H, g, 40, 0.2, 4)["radiance"], rtol=1e-4, atol=1e-7)
    for y0, y1 in [(0, 1), (1, H), (H // 2, H // 2 + 1), (max(0, H - 2), H), (0, H)]:
        _, band = ctx.render_rows(cam, 40, 0.2, 4, y0, y1)
        band = band.cpu().numpy()
        assert np.array_equal(band[y0 * W:y1 * W], full[y0 * W:y1 * W])
        assert not band[:y0 * W].any() and not band[y1 * W:].any()
    assert ctx.status() == 0
    ctx.close()
