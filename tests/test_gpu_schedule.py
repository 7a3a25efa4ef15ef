"""Frames whose tile schedule is planted: every split level, against the oracle
bit for bit."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import pyoracle as po
from conftest import ROOT
from graphic_lab_task_b200 import SceneRT, build as b, parity_preset, workloads as wl
from graphic_lab_task_b200._abi import HIT_DTYPE
from helpers import MISS, bit_equal, hit_summary

pytestmark = pytest.mark.gpu

HEADER, WARPS, LEVEL, BUSY = 8, 4, 5, 6  # words of the schedule's header


@pytest.fixture(scope="module")
def buffers(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("schedule") / "schedule_buffers.so")
    subprocess.run(["g++"] + b.CXX_COMMON + ["-shared", os.path.join(ROOT, "tests", "schedule_buffers.cpp"), "-o", so],
                   check=True)
    f = C.CDLL(so).schedule_buffers
    f.argtypes = [C.c_void_p, C.c_uint32, C.c_uint32, C.POINTER(C.c_uint64)]

    def get(torch, sc, w, h):
        out = (C.c_uint64 * 5)()
        assert f(sc.h, w, h, out) == 0

        def words(ptr):
            mem = type("mem", (), {"__cuda_array_interface__": {
                "shape": (out[2],), "typestr": "<i4", "data": (ptr, False), "version": 3}})()
            return torch.as_tensor(mem, device="cuda")
        return words(out[0]), words(out[1]), int(out[4])
    return get


def _scene(kind):
    sc = SceneRT(preset=parity_preset())
    if kind != "bricks":
        sc.AddInstance(sc.AddGeom_Triangles3f(*wl.noisy_sphere(24, seed=2)), wl.similarity(0.6, (-0.5, 0.1, 0)))
    if kind != "triangles":
        sc.AddInstance(sc.AddGeom_SdfSBS(*wl.sbs_from_spheres(wl.spheres(12, seed=4), grid_res=32)),
                       wl.similarity(0.7, (0.4, 0, 0)))
    sc.CommitScene()
    return sc


@pytest.mark.parametrize("kind,most", [("triangles", 3), ("bricks", 1), ("mixed", 1)])
@pytest.mark.parametrize("width,height", [(61, 43), (333, 251)])
def test_planted_levels_match_oracle(cuda, buffers, kind, most, width, height):
    torch = cuda
    sc = _scene(kind)
    rays = wl.eye_rays_host(wl.camera((0.4, 0.6, 3.2), width=width, height=height))
    want = po.port_trace(sc.export_arrays(), rays)
    shade = po.port_render_lambert(sc.export_arrays(), rays, wl.LIGHT)
    r = torch.from_numpy(rays).cuda()
    h = torch.zeros(len(rays) * 8, dtype=torch.float32, device="cuda")
    image = torch.zeros(len(rays), dtype=torch.float32, device="cuda")
    sc.trace_image(r.data_ptr(), h.data_ptr(), width, height)
    sc.sync()
    tiles = ((width + 7) // 8) * ((height + 3) // 4)
    for level in range(4):
        for which in ("trace", "lambert"):
            rd, _, lists = buffers(torch, sc, width, height)
            plan = np.zeros(len(rd), np.int32)
            plan[0] = level + 1            # the longest tile, in mean busy times of one warp
            plan[1] = (tiles + 1) // 2     # every other tile in class 0, last first
            plan[WARPS] = plan[BUSY] = 1
            listed = np.arange(tiles)[::2]
            plan[lists:lists + len(listed)] = listed[::-1]
            np.bitwise_or.at(plan[HEADER:], listed >> 5, (np.uint32(1) << (listed & 31).astype(np.uint32)).view(np.int32))
            rd.copy_(torch.from_numpy(plan))
            h.zero_()
            image.zero_()
            if which == "trace":
                sc.trace_image(r.data_ptr(), h.data_ptr(), width, height)
            else:
                sc.render_lambert(r.data_ptr(), len(rays), wl.LIGHT, image.data_ptr(), image_size=(width, height))
            sc.sync()
            told = buffers(torch, sc, width, height)[0].cpu().numpy()  # what that launch wrote
            assert told[LEVEL] == min(level, most)
            if which == "trace":
                got = np.ascontiguousarray(h.cpu().numpy()).view(HIT_DTYPE).reshape(-1)
                assert bit_equal(got, want).all(), (level, hit_summary(got, want))
            else:
                assert np.array_equal(image.cpu().numpy(), shade), level
    assert (want["primId"] != MISS).mean() > 0.02
    sc.close()


def test_image_of_many_tiles(cuda):
    """More than 2^24 tiles: a column of rays that miss but for its last rows,
    in natural and in scheduled launches."""
    torch = cuda
    sc = _scene("triangles")
    tail = wl.eye_rays_host(wl.camera((0.4, 0.6, 3.2), width=40, height=30))
    want = po.port_trace(sc.export_arrays(), tail)
    height = 4 * ((1 << 24) + 3) + 1
    rays = torch.empty((height, 8), dtype=torch.float32, device="cuda")
    rays[:] = torch.tensor([0.0, 50.0, 0.0, 1e-4, 0.0, 1.0, 0.0, 9.0], device="cuda")
    rays[-len(tail):] = torch.from_numpy(tail).cuda()
    hits = torch.empty((height, 8), dtype=torch.int32, device="cuda")
    for natural in (True, False, False):
        hits.fill_(7)
        sc.trace_image(rays.data_ptr(), hits.data_ptr(), 1, height, natural_order=natural)
        sc.sync()
        assert bool((hits[:-len(tail), 1] == -1).all())
        got = np.ascontiguousarray(hits[-len(tail):].cpu().numpy()).view(HIT_DTYPE).reshape(-1)
        assert bit_equal(got, want).all(), hit_summary(got, want)
    assert (want["primId"] != MISS).mean() > 0.02
    sc.close()


def test_deep_trees_launch_one_wave(cuda, buffers):
    """A tree as deep as the traversal stack: its launches start the blocks
    that its stacks leave room for, and every pixel is the oracle's."""
    torch = cuda
    sc = SceneRT(preset=parity_preset())
    sc.AddInstance(sc.AddGeom_Triangles3f(*wl.noisy_sphere(24, seed=2)), wl.IDENTITY)
    sc.CommitScene(host_only=True)
    a = {k: v.copy() for k, v in sc.export_arrays().items()}
    tree = a["allNodePairs"]
    depth, todo = 0, [(0, 1)]
    while todo:
        k, d = todo.pop()
        depth = max(depth, d)
        todo += [(int(tree[side]["leftOffset"][k]), d + 1) for side in ("left", "right")
                 if tree[side]["leftOffset"][k] < 0x80000000]
    n = 80 - depth
    chain = np.repeat(tree[:1], n)  # pairs that lead from one to the next and then to the mesh's root
    for side in ("left", "right"):
        chain[side]["boxMin"], chain[side]["boxMax"] = -2.0, 2.0
        lo = tree[side]["leftOffset"]
        tree[side]["leftOffset"] = np.where(lo < 0x80000000, lo + n, lo)
    chain["left"]["leftOffset"], chain["right"]["leftOffset"] = np.arange(1, n + 1), 0xFFFFFFFF
    a["allNodePairs"] = np.concatenate([chain, tree])
    w, h = 640, 480
    rays = wl.eye_rays_host(wl.camera((0.4, 0.6, 3.2), width=w, height=h))
    want = po.port_trace(a, rays)
    sc = SceneRT(preset=parity_preset())
    sc.upload_arrays(a)
    r = torch.from_numpy(rays).cuda()
    hits = torch.zeros(len(rays) * 8, dtype=torch.float32, device="cuda")
    for _ in range(3):
        hits.zero_()
        sc.trace_image(r.data_ptr(), hits.data_ptr(), w, h)
        sc.sync()
        got = np.ascontiguousarray(hits.cpu().numpy()).view(HIT_DTYPE).reshape(-1)
        assert bit_equal(got, want).all(), hit_summary(got, want)
    # 81 + 16 words a thread, and 1 KB a block of the system's own
    blocks = (228 * 1024) // ((81 + 16) * 128 * 4 + 1024)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert buffers(torch, sc, w, h)[0].cpu().numpy()[WARPS] == blocks * sms * 4
    sc.close()
