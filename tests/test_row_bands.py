"""Bands of rows of frames whose pixel blocks straddle the eye pass's bands of 4
rows: every single row and bands of all phases are the full frame's, 0 outside."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("W,H", [(641, 38), (50, 61), (129, 17)])
def test_every_row_and_phase(W, H):
    import photonmap
    from photonmap import scenes
    sc, _, _ = scenes.workload("cornell_small")
    ctx = photonmap.Context(0)
    ctx.set_scene(sc)
    ctx.trace_photons(3, 8, 20_000)
    ctx.build_grid(0)
    cam = photonmap.camera_setup((0, 0, 3.5), (0, 0, -1), (0, 1, 0), 45.0, W, H)
    full = ctx.render(cam, 40, 0.2, 4)[1].cpu().numpy()
    assert full.any()
    for y0, y1 in [(y, y + 1) for y in range(H)] + [(a, H - b) for a in range(5) for b in range(5)]:
        band = ctx.render_rows(cam, 40, 0.2, 4, y0, y1)[1].cpu().numpy()
        assert np.array_equal(band[y0 * W:y1 * W], full[y0 * W:y1 * W]), (y0, y1)
        assert not band[:y0 * W].any() and not band[y1 * W:].any(), (y0, y1)
    assert ctx.status() == 0
    ctx.close()
