"""Scenes that carry SBS arrays no geometry names, against the oracle."""
import numpy as np
import pytest

import pyoracle as po
from graphic_lab_task_b200 import SceneRT, workloads as wl
from helpers import MISS, bit_equal, hit_summary

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("others", ["triangles", "triangles and voxels"])
def test_new_values_leave_other_geometry_alone(cuda, others):
    """lrt_sbs_update_values on a scene without brick geometry: the values are
    taken, and later traces hit what they hit before."""
    torch = cuda

    def build(bricks):
        sc = SceneRT()
        sc.AddInstance(sc.AddGeom_Triangles3f(*wl.noisy_sphere(20, seed=3)), wl.similarity(0.6, (-0.5, 0, 0)))
        if "voxels" in others:
            sc.AddInstance(sc.AddGeom_SdfSVS(wl.svs_from_spheres(wl.spheres(8, seed=2), 4)), wl.similarity(0.5, (0.6, 0, 0)))
        if bricks:
            sc.AddInstance(sc.AddGeom_SdfSBS(*wl.sbs_from_spheres(wl.spheres(6, seed=5), grid_res=32)), wl.IDENTITY)
        sc.CommitScene(host_only=True)
        return {k: v.copy() for k, v in sc.export_arrays().items()}

    a, with_bricks = build(False), build(True)
    a.update({k: v for k, v in with_bricks.items() if k.startswith("sdfSBS")})
    rays = wl.eye_rays_host(wl.camera((0.3, 0.4, 3.2), width=80, height=60))
    want = po.port_trace(a, rays)
    sc = SceneRT()
    sc.upload_arrays(a)
    r = torch.from_numpy(rays).cuda()
    h = torch.zeros(len(rays) * 8, dtype=torch.float32, device="cuda")
    values = torch.from_numpy(a["sdfSBSDataF"] + np.float32(0.25)).cuda()
    for updates in range(3):
        if updates:
            sc.update_sbs_values(values.data_ptr(), len(values))
        h.zero_()
        sc.trace_image(r.data_ptr(), h.data_ptr(), 80, 60)
        sc.sync()
        got = np.ascontiguousarray(h.cpu().numpy()).view(want.dtype).reshape(-1)
        assert bit_equal(got, want).all(), (updates, hit_summary(got, want))
    assert (want["primId"] != MISS).mean() > 0.05
    sc.close()
