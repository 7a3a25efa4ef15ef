"""The trace kernels compiled per geometry kind, in both launch sizes, and the
brick march's reach test, against the oracle bit for bit."""
import numpy as np
import pytest

import pyoracle as po
from graphic_lab_task_b200 import SceneRT, parity_preset, workloads as wl
from graphic_lab_task_b200._abi import HIT_DTYPE
from helpers import MISS, bit_equal, hit_summary

pytestmark = pytest.mark.gpu

KINDS = {"triangles": "t", "nodes": "ov", "triangles+nodes": "tov", "bricks": "b", "bricks twice": "bb",
         "bricks+triangles": "bt", "all": "tovb"}


def _scene(letters, preset=None, count=None):
    sc = SceneRT(preset=preset or parity_preset())
    sph = wl.spheres(12, seed=4)
    make = {"t": lambda: sc.AddGeom_Triangles3f(*wl.noisy_sphere(24, seed=2)),
            "o": lambda: sc.AddGeom_SdfFrameOctree(wl.frame_octree_from_spheres(sph, 4)),
            "v": lambda: sc.AddGeom_SdfSVS(wl.svs_from_spheres(sph, 4)),
            "b": lambda: sc.AddGeom_SdfSBS(*wl.sbs_from_spheres(sph, grid_res=32))}
    geoms = [make[k]() for k in letters]
    small = (0.05, 0.1) if count else (0.3, 0.6)
    for i, m in enumerate(wl.random_instances(count or 3 * len(geoms), seed=6, scale=small, trans=1.0)):
        sc.AddInstance(geoms[i % len(geoms)], m)
    sc.CommitScene()
    return sc


def _trace(torch, sc, rays, width, height, row, repeat=2):
    r = torch.from_numpy(rays).cuda()
    h = torch.zeros(len(rays) * 8, dtype=torch.float32, device="cuda")
    for _ in range(repeat):
        h.zero_()
        if row:
            sc.trace_device(r.data_ptr(), h.data_ptr(), len(rays))
        else:
            sc.trace_image(r.data_ptr(), h.data_ptr(), width, height)
    sc.sync()
    return h.cpu().numpy().view(HIT_DTYPE).reshape(-1)


@pytest.mark.parametrize("kind", sorted(KINDS))
@pytest.mark.parametrize("width,height,row", [(53, 41, False), (53, 41, True), (1537, 1237, False), (1537, 1237, True)])
def test_kinds_match_oracle(cuda, kind, width, height, row):
    """Ragged frames of one wave and of many; every pixel of the small frame,
    every 61st of the large one."""
    sc = _scene(KINDS[kind])
    rays = wl.eye_rays_host(wl.camera((0.4, 0.6, 3.2), width=width, height=height))
    got = _trace(cuda, sc, rays, width, height, row)
    pick = slice(None) if width < 100 else slice(7, None, 61)
    want = po.port_trace(sc.export_arrays(), rays[pick])
    got = np.ascontiguousarray(got[pick])
    assert bit_equal(got, want).all(), hit_summary(got, want)
    assert (want["primId"] != MISS).mean() > 0.02
    sc.close()


@pytest.mark.parametrize("surface", [False, True])
@pytest.mark.parametrize("noise,distance", [(0.0, 3.0), (0.002, 3.0), (0.05, 3.0), (0.002, 7.0)])
def test_reach_test_keeps_every_hit(cuda, surface, noise, distance):
    """Grazing and noisy bricks, in both representation modes, and from as far
    as the march's step of 1e-6 still moves the ray."""
    p = parity_preset()
    p.representation_mode = 0 if surface else 1
    hdr, nodes, vals, vf = wl.sbs_from_spheres(wl.spheres(24, seed=9), grid_res=64)
    vf = vf.copy()
    vf[3 * 24:] += np.random.default_rng(1).normal(0, noise, len(vf) - 3 * 24).astype(np.float32)
    sc = SceneRT(preset=p)
    sc.AddInstance(sc.AddGeom_SdfSBS(hdr, nodes, vals, vf), wl.IDENTITY)
    sc.CommitScene()
    w, h = 211, 157
    rays = wl.eye_rays_host(wl.camera((0.2 * distance, 0.3 * distance, 0.93 * distance), width=w, height=h,
                                      fovy=60.0 if distance < 5 else 25.0))
    got = _trace(cuda, sc, rays, w, h, False)
    want = po.port_trace(sc.export_arrays(), rays, preset=p)
    assert bit_equal(got, want).all(), hit_summary(got, want)
    assert (want["primId"] != MISS).mean() > 0.05
    sc.close()


@pytest.mark.parametrize("kind", ["triangles", "nodes", "bricks", "all"])
@pytest.mark.parametrize("width,height", [(61, 43), (333, 251)])
def test_split_tiles_of_repeated_frames_match_oracle(cuda, kind, width, height):
    """Repeated small frames, whose slowest tiles go out in the parts that the
    launch before makes of them (planted levels: test_gpu_schedule.py): every
    pixel of every repeat, and of the fused Lambert image, stays what it was."""
    torch = cuda
    sc = _scene(KINDS[kind])
    rays = wl.eye_rays_host(wl.camera((0.4, 0.6, 3.2), width=width, height=height))
    want = po.port_trace(sc.export_arrays(), rays)
    for repeat in (3, 4, 7):
        got = _trace(torch, sc, rays, width, height, False, repeat)
        assert bit_equal(got, want).all(), (repeat, hit_summary(got, want))
    r = torch.from_numpy(rays).cuda()
    image = torch.zeros(len(rays), dtype=torch.float32, device="cuda")
    shade = po.port_render_lambert(sc.export_arrays(), rays, wl.LIGHT)
    for _ in range(5):
        image.zero_()
        sc.render_lambert(r.data_ptr(), len(rays), wl.LIGHT, image.data_ptr(), image_size=(width, height))
        sc.sync()
        assert np.array_equal(image.cpu().numpy(), shade)
    sc.close()


@pytest.mark.parametrize("rays", [47361, 52001, 66305])
def test_rows_around_a_wave_match_oracle(cuda, rays):
    """Rows on scenes of all kinds whose warps of 16 rays are more than a wave
    of the frames' kernel, and the first size of 32 rays to a warp."""
    sc = _scene(KINDS["all"])
    r = wl.eye_rays_host(wl.camera((0.4, 0.6, 3.2), width=320, height=240))[:rays]
    got = _trace(cuda, sc, r, 0, 0, True, 1)
    want = po.port_trace(sc.export_arrays(), r)
    assert bit_equal(got, want).all(), hit_summary(got, want)
    sc.close()


def test_mixed_batches_match_oracle(cuda):
    """Cameras and Lambert passes of a scene of all kinds, whose kernels keep
    the ray and its inverse in shared memory."""
    torch = cuda
    from graphic_lab_task_b200.lrt import CameraBatch
    sc = _scene(KINDS["all"])
    cams = wl.sphere_cameras(5, radius=3.2, res_min=17, res_max=90, seed=8)
    b = CameraBatch(sc, cams)
    h = torch.zeros(b.total_rays * 8, dtype=torch.float32, device="cuda")
    b.trace(h.data_ptr())
    b.sync()
    rays = np.concatenate([wl.eye_rays_host(c) for c in cams])
    want = po.port_trace(sc.export_arrays(), rays)
    got = h.cpu().numpy().view(HIT_DTYPE).reshape(-1)
    assert bit_equal(got, want).all(), hit_summary(got, want)
    image = torch.zeros(len(rays), dtype=torch.float32, device="cuda")
    r = torch.from_numpy(rays).cuda()
    sc.render_lambert(r.data_ptr(), len(rays), wl.LIGHT, image.data_ptr())
    sc.sync()
    assert np.array_equal(image.cpu().numpy(), po.port_render_lambert(sc.export_arrays(), rays, wl.LIGHT))
    b.close()
    sc.close()


@pytest.mark.parametrize("instances", [255, 256])
@pytest.mark.parametrize("row", [False, True])
def test_many_waves_of_many_instances_match_oracle(cuda, instances, row):
    """Scenes without bricks around the instance count from which launches of
    this size take the kernel for many waves; every 61st ray."""
    sc = _scene(KINDS["triangles+nodes"], count=instances)
    width, height = 2051, 1489  # over 20 waves of 8 blocks on 148 SMs
    assert (width + 7) // 8 * ((height + 3) // 4) > 4 * 20 * 8 * 148
    rays = wl.eye_rays_host(wl.camera((0.4, 0.6, 3.2), width=width, height=height))
    got = _trace(cuda, sc, rays, width, height, row)[7::61]
    want = po.port_trace(sc.export_arrays(), rays[7::61])
    got = np.ascontiguousarray(got)
    assert bit_equal(got, want).all(), hit_summary(got, want)
    assert (want["primId"] != MISS).mean() > 0.02
    sc.close()
