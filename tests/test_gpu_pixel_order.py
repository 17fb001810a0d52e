"""Paths follow blocks of 32 x 32 pixels where a segment holds 32 full rows, row order elsewhere.
Waves of 37 paths have no full rows, so they give the row order: the image must be that of one
wave, at sizes around the block edges.  A pixel's sum of three positive samples is grouped by
wave (two roundings of 2^-24 each way)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shader", [5, 3])
@pytest.mark.parametrize("w,h", [(31, 33), (32, 31), (32, 32), (33, 64), (64, 65), (95, 40), (1, 70)])
def test_blocked_order_equals_row_order(rg, w, h, shader):
    images = []
    for paths in (0, 37):
        r = rg.RayRenderer(rg.RendererSettings(resolutionWidth=w, resolutionHeight=h, samples=3, maxDepth=5, seed=5,
                                               pathsPerWave=paths, shaderProvider=shader))
        r.set_scene(rg.Scene.builtin(1, 1))
        r.render()
        assert (r.get_sample_counts() == 3).all()
        images.append(r.get_hdr_result())
        r.close()
    np.testing.assert_allclose(images[0], images[1], rtol=1e-6)
