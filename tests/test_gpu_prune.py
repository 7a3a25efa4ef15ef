"""Pruning of the SBS node pairs on the device after new values, and the
device-made triangle records, against the oracle bit for bit."""
import numpy as np
import pytest

import pyoracle as po
from graphic_lab_task_b200 import BUILD_LOW, SceneRT, workloads as wl
from graphic_lab_task_b200._abi import SBS_LAYOUT_DX
from helpers import MISS, bit_equal, hit_summary

pytestmark = pytest.mark.gpu


def _dx(model):
    """The model with 16-bit distances in the plain layout."""
    hdr, nodes, vals, vf = (None if m is None else m.copy() for m in model)
    v3 = 11 ** 3
    v = vf[vals.reshape(len(nodes), -1)[:, :v3]]
    dmax = np.sqrt(3.0) * 2.0 / float(nodes["pos_z_lod_size"][0] & 0xFFFF)
    q = np.zeros((len(nodes), 1332), np.uint16)
    q[:, :v3] = np.clip(np.rint((v + dmax) / (2 * dmax) * 65535.0), 0, 65535)
    hdr["bytes_per_value"], hdr["aux_data"] = 2, SBS_LAYOUT_DX
    nodes["data_offset"] = np.arange(len(nodes)) * 666
    return hdr, nodes, q.reshape(-1).view(np.uint32), None


@pytest.mark.parametrize("others", ["alone", "with a mesh", "with a quantised model and a mesh"])
def test_updates_prune_like_an_upload(cuda, others):
    """Bricks that lose their surface, bricks that gain one, all of them, none
    of them: hits after each update equal the oracle's on a scene built with
    those values."""
    torch = cuda
    hdr, nodes, vals, vf = wl.sbs_from_spheres(wl.spheres(10, seed=3), grid_res=48)
    first = 3 * 10
    shifts = [np.zeros(len(vf), np.float32) for _ in range(4)]
    v3 = 11 ** 3 * np.arange(len(nodes))[:, None] + np.arange(11 ** 3)
    half = (nodes["pos_xy"] >> 16) >= 3
    shifts[0][first + v3[half]] = 1.0      # half the bricks lose their surface
    shifts[1][first + v3[~half]] = 0.02    # the others shrink
    shifts[2][first:] = 1.0                # nothing is left
    rays = wl.eye_rays_host(wl.camera((0.5, 0.8, 3.0), width=97, height=83))
    r = torch.from_numpy(rays).cuda()
    h = torch.zeros(len(rays) * 8, dtype=torch.float32, device="cuda")

    def build(values):
        sc = SceneRT()
        sc.AddInstance(sc.AddGeom_SdfSBS(hdr, nodes, vals, values), wl.IDENTITY)
        if others != "alone":
            sc.AddInstance(sc.AddGeom_Triangles3f(*wl.noisy_sphere(12, seed=4)), wl.similarity(0.3, (1.0, 0, 0.4)))
        if "quantised" in others:
            sc.AddInstance(sc.AddGeom_SdfSBS(*_dx((hdr, nodes, vals, vf))), wl.similarity(0.4, (-0.8, 0.6, 0.3)))
        return sc

    sc = build(vf)
    sc.CommitScene()
    hit_counts = []
    for s in shifts + [shifts[0]]:
        values = vf + s
        sc.update_sbs_values(torch.from_numpy(values).cuda().data_ptr(), len(values))
        for image in (True, False):
            h.zero_()
            if image:
                sc.trace_image(r.data_ptr(), h.data_ptr(), 97, 83)
            else:
                sc.trace_device(r.data_ptr(), h.data_ptr(), len(rays))
            sc.sync()
            got = h.cpu().numpy().view(np.dtype([("w", "<f4", 8)])).view(np.uint8).reshape(len(rays), 32)
            want_sc = build(values)
            want_sc.CommitScene(host_only=True)
            want = po.port_trace(want_sc.export_arrays(), rays)
            got = np.ascontiguousarray(got).view(want.dtype).reshape(-1)
            assert bit_equal(got, want).all(), hit_summary(got, want)
        hit_counts.append(int((want["primId"] != MISS).sum()))
    assert hit_counts[3] > hit_counts[0] > hit_counts[2]
    sc.close()


@pytest.mark.parametrize("build", [0, BUILD_LOW])
def test_triangle_records_of_odd_meshes(cuda, build):
    """Several meshes, signed zeros, repeated and unused vertices, a wide
    vertex stride, remainders of a block of 256: the device-made boxes and
    records trace like the oracle on the exported arrays."""
    rng = np.random.default_rng(8)
    sc = SceneRT()
    for k, n in enumerate((1, 2, 3, 257, 1000)):
        v = rng.uniform(-1, 1, (n + 7, 5)).astype(np.float32)
        v[rng.integers(0, n + 7, 5), rng.integers(0, 3, 5)] = -0.0
        v[rng.integers(0, n + 7, 5), rng.integers(0, 3, 5)] = 0.0
        t = rng.integers(0, n + 3, (n, 3)).astype(np.uint32)
        g = sc.AddGeom_Triangles3f(v, t, flags=build or 4, vByteStride=20)
        sc.AddInstance(g, wl.similarity(0.5, (0.7 * k - 1.4, 0.1, 0)))
    sc.CommitScene()
    rays = wl.eye_rays_host(wl.camera((0.3, 0.5, 4.0), width=120, height=90))
    got = sc.RayQuery_NearestHitBatch(rays)
    want = po.port_trace(sc.export_arrays(), rays)
    assert bit_equal(got, want).all(), hit_summary(got, want)
    assert (want["primId"] != MISS).mean() > 0.03
