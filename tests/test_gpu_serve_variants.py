"""The server's wave graphs: jobs with area lights only (no media, environment or point-light
code), and the same job sharing waves with a point-light scene and with fog.  The image does not
depend on the graph that ran it (the tolerance of the other server tests)."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


def point_light_scene(rg):
    base, _ = scenes.lit_floor_scene(rg)
    d = base.desc
    pos, nrm, tm = (np.array(a) for a in base.arrays())
    light = rg.rg_point_light()
    light.position[:] = [0.5, 0.5, -1.0]
    light.normal[:] = [0.0, -1.0, 0.0]
    light.material = 1
    return rg.Scene.from_arrays(pos, nrm, tm, [d.mesh_object[i] for i in range(d.num_meshes)],
                                [d.objects[i] for i in range(d.num_objects)],
                                [d.materials[i] for i in range(d.num_materials)], d.camera, point_lights=[light])


def test_plain_job_alone_and_beside_others(rg):
    plain = rg.Scene.builtin(4, 11, [3000, 5])
    others = [point_light_scene(rg), rg.Scene.builtin(3, 2, [500])]
    st = rg.RendererSettings(resolutionWidth=90, resolutionHeight=70, samples=9, maxDepth=6, rrDepth=3, seed=8)
    r = rg.RayRenderer(st)
    images = []
    for sc in [plain] + others:
        r.set_scene(sc)
        r.render()
        images.append(r.get_hdr_result())
    r.close()
    for mix in ([0], [0, 1], [0, 2], [1], [2], [0, 1, 2]):
        srv = rg.RenderServer(rg.RendererSettings(rrDepth=3))
        ids = [srv.submit(([plain] + others)[k], 90, 70, 9, max_depth=6, seed=8) for k in mix]
        for k, j in zip(mix, ids):
            srv.wait(j)
            np.testing.assert_allclose(srv.result(j), images[k], rtol=1e-4, atol=1e-6)
        srv.close()
