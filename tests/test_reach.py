"""The brick march's test for voxels whose sphere trace cannot hit (out_of_reach
in trace_impl.cuh), restated in float32 and compared with the trace itself."""
import numpy as np
import pytest

F = np.float32


def trilinear(v, p):
    """eval_dist_trilinear in float32, in its operation order (v: (n, 8), p: (n, 3))."""
    x, y, z = p[:, 0], p[:, 1], p[:, 2]
    one = F(1)
    out = None
    for k in range(8):
        t = (x if k & 4 else one - x) * (y if k & 2 else one - y)
        t = t * (z if k & 1 else one - z) * v[:, k]
        out = t if out is None else out + t
    return out


def trace_hits(v, q, d, q_far, surface):
    """LocalSurfaceIntersection's march (BVH2Common.cpp:364-390) past its early hits."""
    t = np.zeros(len(v), F)
    dist = trilinear(v, q)
    sign = np.where(surface, np.sign(dist), 1).astype(F)
    dist = dist * sign
    early = dist <= F(1e-6)
    scale = F(37.0)  # d_inv: voxels per unit
    for _ in range(256):
        go = (t < q_far) & (dist > F(1e-6))
        if not go.any():
            break
        t = np.where(go, t + dist * scale, t)
        nd = sign * trilinear(v, q + t[:, None] * d)
        dist = np.where(go, nd, dist)
    return early, (dist <= F(1e-6)) & (t <= q_far)


def out_of_reach(v, q, d, q_far, surface):
    """The Bernstein bound (numpy has no fused multiply-add: float64 products, rounded once, in its place)."""
    fma = lambda a, b, c: (a.astype(np.float64) * b + c).astype(F)  # noqa: E731
    start = trilinear(v, q)
    sign = np.where(surface, np.sign(start), 1).astype(F)
    e = np.stack([fma(q_far, d[:, k], q[:, k]) for k in range(3)], 1)
    ends = (q, e)
    f = [[fma(p[:, 0], v[:, k + 4] - v[:, k], v[:, k]) for k in range(4)] for p in ends]
    g = [[[fma(p[:, 1], f[i][k + 2] - f[i][k], f[i][k]) for k in range(2)] for p in ends] for i in range(2)]
    h = [[[fma(p[:, 2], g[i][j][1] - g[i][j][0], g[i][j][0]) for p in ends] for j in range(2)] for i in range(2)]
    b1 = sign * (h[1][0][0] + h[0][1][0] + h[0][0][1])
    b2 = sign * (h[1][1][0] + h[1][0][1] + h[0][1][1])
    b3 = sign * h[1][1][1]
    out = np.maximum(np.abs(q - F(0.5)).max(1), np.abs(e - F(0.5)).max(1))
    m = F(4e-5) * np.abs(v).max(1) + F(1e-6)
    return (out <= 1) & (start * sign > m) & (b1 > 3 * m) & (b2 > 3 * m) & (b3 > m)


@pytest.mark.parametrize("amplitude", [1e-6, 1e-4, 0.01, 1.0, 1e4])
@pytest.mark.parametrize("surface", [False, True])
def test_rejected_voxels_never_hit(amplitude, surface):
    rng = np.random.default_rng(int(amplitude * 1e6) + surface)
    n = 8000
    # near-planar fields that graze zero, and plain noise; rays that cross the voxel, also a little outside of it
    nrm = rng.normal(size=(n, 3))
    corners = np.array([[(k >> 2) & 1, (k >> 1) & 1, k & 1] for k in range(8)], float)
    v = nrm @ corners.T + rng.normal(size=(n, 1)) + rng.normal(size=(n, 8)) * rng.choice([0, 0.1, 1.0], size=(n, 1))
    v = (v * amplitude).astype(F)
    v[: n // 4] -= v[: n // 4].min(1, keepdims=True)  # lowest corner exactly zero
    q = rng.uniform(-0.1, 1.1, size=(n, 3)).astype(F)
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(F)
    q_far = (rng.uniform(-0.1, 1.5, size=n)).astype(F)
    with np.errstate(all="ignore"):
        reject = out_of_reach(v, q, d, q_far, surface)
        early, hit = trace_hits(v, q, d, q_far, surface)
    assert not (reject & early).any()
    assert not (reject & hit).any()
    if amplitude >= 1e-4:
        missed = ~early & ~hit & (q_far > 0) & (np.abs(q + q_far[:, None] * d - 0.5).max(1) <= 1)
        assert reject[missed].mean() > 0.5  # the test is worth having


def test_rejects_no_nan_or_infinite_field():
    v = np.full((4, 8), 1, F)
    v[0, 3], v[1, 5], v[2, 0] = np.nan, np.inf, -np.inf
    q = np.full((4, 3), 0.25, F)
    d = np.tile(np.array([[1, 0, 0]], F), (4, 1))
    with np.errstate(all="ignore"):
        r = out_of_reach(v, q, d, np.full(4, 0.5, F), False)
    assert r.tolist() == [False, False, False, True]
