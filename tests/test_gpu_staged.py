"""Host-pointer traces of fewer rays than the pipeline takes (page-locked
staging that the kernel reads and writes over the bus, and above its size
buffers on the device) equal device traces."""
import numpy as np
import pytest

from graphic_lab_task_b200 import LrtError, SceneRT, workloads as wl
from graphic_lab_task_b200._abi import HIT_DTYPE
from helpers import MISS, bit_equal, hit_summary

pytestmark = pytest.mark.gpu


def test_staged_sizes_match_device_trace(cuda):
    """One ray, remainders, the sizes where the buffer grows, launches within
    one wave (groups by warp index) and beyond (a counter), then small again."""
    torch = cuda
    sc = SceneRT()
    sc.AddInstance(sc.AddGeom_Triangles3f(*wl.noisy_sphere(40, seed=3)), wl.IDENTITY)
    sc.AddInstance(sc.AddGeom_SdfSBS(*wl.sbs_from_spheres(wl.spheres(8, seed=2), grid_res=32)),
                   wl.similarity(0.5, (1.0, 0.5, 0.2)))
    sc.CommitScene()
    rng = np.random.default_rng(5)
    for n in (1, 2, 37, 4096, 4097, 20000, 32768, 32769, 94719, 94721, 150001, 262143, 3):
        o = rng.normal(size=(n, 3))
        o *= 3.0 / np.linalg.norm(o, axis=1, keepdims=True)
        d = rng.uniform(-1.2, 1.2, (n, 3)) - o
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        rays = np.concatenate([o, np.full((n, 1), 1e-4), d, np.full((n, 1), 1e9)], axis=1).astype(np.float32)
        got = sc.RayQuery_NearestHitBatch(rays)
        r = torch.from_numpy(rays).cuda()
        h = torch.zeros(n * 8, dtype=torch.float32, device="cuda")
        sc.trace_device(r.data_ptr(), h.data_ptr(), n)
        sc.sync()
        want = h.cpu().numpy().view(HIT_DTYPE).reshape(-1)
        assert bit_equal(got, want).all(), (n, hit_summary(got, want))
        if n > 1000:
            assert 0.02 < (want["primId"] != MISS).mean() < 1.0


def test_page_locked_rays_are_read_in_stream_order(cuda):
    """Rays that an earlier copy on the stream brings into page-locked memory
    are traced as they are once that copy has run."""
    torch = cuda
    sc = SceneRT()
    sc.AddInstance(sc.AddGeom_Triangles3f(*wl.noisy_sphere(40, seed=3)), wl.IDENTITY)
    sc.CommitScene()
    n = 64 * 64
    rays = wl.eye_rays_host(wl.camera((0.1, 0.2, 3), width=64, height=64))
    want = sc.RayQuery_NearestHitBatch(rays)
    src = torch.from_numpy(rays).cuda()
    busy = torch.empty(1 << 28, dtype=torch.uint8, device="cuda")
    host = torch.zeros(n * 8, dtype=torch.float32).pin_memory()
    hits = torch.zeros(n * 8, dtype=torch.float32).pin_memory()
    for _ in range(20):
        busy.add_(1)  # the copy below is still to come when the call is made
    host.copy_(src.view(-1), non_blocking=True)
    sc.trace_host(host.data_ptr(), hits.data_ptr(), n)
    got = hits.numpy().view(HIT_DTYPE).reshape(-1)
    assert bit_equal(got, want).all(), hit_summary(got, want)


def test_staged_error_is_reported_once(cuda):
    sc = SceneRT()
    sc.AddInstance(sc.AddGeom_SdfSBS(*wl.sbs_from_spheres(wl.spheres(8, seed=2), grid_res=32)), wl.IDENTITY)
    sc.CommitScene()
    rays = wl.eye_rays_host(wl.camera((0, 0, 3), width=64, height=64))
    want = sc.RayQuery_NearestHitBatch(rays)
    sc.set_voxel_step_limit(1)
    with pytest.raises(LrtError) as e:
        sc.RayQuery_NearestHitBatch(rays)
    assert e.value.status == 5
    sc.set_voxel_step_limit(0)
    assert bit_equal(sc.RayQuery_NearestHitBatch(rays), want).all()
