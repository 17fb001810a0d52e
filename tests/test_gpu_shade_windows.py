"""The shade kernel's windows shrink when a wave holds few rays, so that all SMs share them: from one
ray to more than the resident blocks' full windows (148 SMs, two blocks each, 32 to 896 rays a
window), around the sizes where the window grows.  The image must be that of waves of other sizes,
whose windows lie elsewhere: a pixel's path does not depend on the window that shades it."""
import json

import numpy as np
import pytest

import scenes
from test_gpu_media import LAMP, ROOM, box

pytestmark = pytest.mark.gpu
BLOCKS = 2 * 148


def image(rg, scene, w, h, paths):
    r = rg.RayRenderer(rg.RendererSettings(resolutionWidth=w, resolutionHeight=h, samples=1, maxDepth=6, rrDepth=3, seed=7,
                                           pathsPerWave=paths))
    r.set_scene(scene)
    r.render()
    out = r.get_hdr_result()
    r.close()
    return out


@pytest.mark.parametrize("n", [1, 31, 33, 32 * BLOCKS - 1, 32 * BLOCKS + 1, 64 * BLOCKS + 1, 448 * BLOCKS + 1,
                               896 * BLOCKS - 1, 896 * BLOCKS + 1])
def test_any_number_of_rays(rg, n):
    w = max(k for k in range(1, 700) if n % k == 0)
    scene = rg.Scene.builtin(4, 2, [3000, 6])
    got = image(rg, scene, w, n // w, 0)
    other = image(rg, scene, w, n // w, max(1, n // 3 + 5))
    scene.close()
    assert got.shape == (n // w, w, 4) and (got[..., :3] > 0).any()
    np.testing.assert_allclose(got, other, rtol=1e-6)


@pytest.mark.parametrize("w,h", [(40, 25), (160, 90)])
def test_media_under_an_environment(rg, tmp_path, w, h):
    """The kernel with the longest vertices: delta tracking in a cloud, rays bent by heat haze."""
    scenes.write_hdr(tmp_path / "sky.hdr", scenes.sky_image(64, 32, seed=5))
    doc = {"mainCamera": {"location": [0, 1.0, 6.0], "angle": [-8, 0, 0], "fieldOfView": 45},
           "envmap": {"texture": "sky.hdr", "intensity": 1.0}}
    doc.update(ROOM, **LAMP)
    doc["cloud"] = box([0, 0.6, 0], [2.4, 1.6, 2.4], {"sigma_a": [0.05] * 3, "sigma_s": [2.5] * 3, "densityField": "fbm",
                                                      "noiseFrequency": 1.6, "noiseOctaves": 3})
    doc["haze"] = box([0, 0.5, 1], [3, 2, 1], {"heatHaze": True, "iorAmplitude": 0.02, "iorMarchSteps": 8})
    (tmp_path / "s.json").write_text(json.dumps(doc))
    scene = rg.Scene.from_json(str(tmp_path / "s.json"))
    np.testing.assert_allclose(image(rg, scene, w, h, 0), image(rg, scene, w, h, w * h // 3 + 5), rtol=1e-6)
    scene.close()
