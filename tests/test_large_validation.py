"""Validation of trees large enough for the walk on all cores: faults are
found and named as by the sequential walk."""
import os
import subprocess
import time

import numpy as np
import pytest

from conftest import ROOT
from graphic_lab_task_b200 import LrtError, SceneRT, build as b, workloads as wl


def _arrays():
    sc = SceneRT()
    sc.AddInstance(sc.AddGeom_Triangles3f(*wl.noisy_sphere(24, seed=1)), wl.IDENTITY)
    sc.AddInstance(sc.AddGeom_Triangles3f(*wl.noisy_sphere(260, seed=2)), wl.similarity(0.5, (1, 0, 0)))
    sc.CommitScene(host_only=True)
    return sc.export_arrays()


@pytest.fixture(scope="module")
def arrays():
    a = _arrays()
    assert len(a["allNodePairs"]) > 2 * 32768
    return a


@pytest.mark.parametrize("what,message", [
    ("duplicate", "reached twice"), ("shared", "reached twice"), ("backward", "not a later pair"), ("beyond", "beyond allNodePairs"),
    ("leaf", "outside its"), ("vertex", "vertex beyond vertPos"), ("prims", "triangles beyond indices")])
def test_faults_are_named(arrays, what, message):
    a = {k: v.copy() for k, v in arrays.items()}
    base = int(a["geomData"]["bvhOffset"][1])
    pairs = a["allNodePairs"]
    inner = np.nonzero(pairs["left"]["leftOffset"][base:] < 0x80000000)[0]
    k = base + int(inner[len(inner) * 3 // 4])  # deep in the large tree
    if what == "duplicate":
        first = base + int(inner[len(inner) // 2])
        pairs["left"]["leftOffset"][first] = max(int(pairs["left"]["leftOffset"][first]), k - base + 1)
    elif what == "shared":  # the small mesh's tree runs into the large one's
        small = np.nonzero(pairs["left"]["leftOffset"][:base] < 0x80000000)[0]
        both = (pairs["left"]["leftOffset"][base:] >= 0x80000000) & (pairs["right"]["leftOffset"][base:] >= 0x80000000)
        pairs["left"]["leftOffset"][int(small[-1])] = base + int(np.nonzero(both)[0][0])
    elif what == "backward":
        pairs["left"]["leftOffset"][k] = k - base
    elif what == "beyond":
        pairs["left"]["leftOffset"][k] = len(pairs)
    elif what == "leaf":
        leaf = base + int(np.nonzero(pairs["right"]["leftOffset"][base:] >= 0x80000000)[0][-1])
        pairs["right"]["leftOffset"][leaf] = 0x80000000 | 0x0FFFFFF0
    elif what == "vertex":
        a["indices"][-1] = len(a["vertPos"])
    else:
        a["primIdCount"][-1] = 0x80000000 | (1 << 28) | (len(a["indices"]) // 3)
    sc = SceneRT()
    with pytest.raises(LrtError) as e:
        sc.upload_arrays(a)
    assert e.value.status == 2 and message in str(e.value)


def test_depth_of_a_large_tree(arrays):
    """The parallel walk's depth is the tree's: the traversal stack is sized by it."""
    pairs = arrays["allNodePairs"]
    base = int(arrays["geomData"]["bvhOffset"][1])
    deepest, todo = 0, [(0, 1)]
    while todo:
        k, d = todo.pop()
        deepest = max(deepest, d)
        for side in ("left", "right"):
            lo = int(pairs[side]["leftOffset"][base + k])
            if lo < 0x80000000:
                todo.append((lo, d + 1))
    a = {k: v.copy() for k, v in arrays.items()}
    last = base + int(np.nonzero(pairs["right"]["leftOffset"][base:] < 0x80000000)[0][-1])
    assert 10 < deepest <= 80 and last > base
    sc = SceneRT()
    chain = a["allNodePairs"][:1].copy()
    n = 90  # a chain deeper than the 80-entry stack, appended as a third geometry, is refused
    extra = np.repeat(chain, n)
    extra["left"]["leftOffset"] = np.arange(1, n + 1)
    extra["left"]["leftOffset"][-1] = 0x90000000
    extra["right"]["leftOffset"] = 0x90000000
    a["allNodePairs"] = np.concatenate([a["allNodePairs"], extra])
    g = a["geomData"][:1].copy()
    g["bvhOffset"] = len(pairs)
    a["geomData"] = np.concatenate([a["geomData"], g])
    a["geomTags"] = np.concatenate([a["geomTags"], a["geomTags"][:1]])
    a["startEnd"] = np.concatenate([a["startEnd"], a["startEnd"][:1]])
    with pytest.raises(LrtError) as e:
        sc.upload_arrays(a)
    assert e.value.status == 2 and "depth 90" in str(e.value)


def test_many_small_meshes_are_validated_by_one_core():
    """4,000 meshes of 12 triangles: starting all cores for each of them made
    the commit take a tenth of the time that the adders take (0.5% without; the
    bound is six times that)."""
    v, t = wl.noisy_sphere(3, seed=1)
    ratio = []
    for _ in range(5):
        sc = SceneRT()
        t0 = time.perf_counter()
        for _ in range(4000):
            g = sc.AddGeom_Triangles3f(v, t)
        sc.AddInstance(g, wl.IDENTITY)
        t1 = time.perf_counter()
        sc.CommitScene(host_only=True)
        ratio.append((time.perf_counter() - t1) / (t1 - t0))
        sc.close()
    assert min(ratio) < 0.03, ratio


def test_cores_without_memory_leave_the_walk_to_the_caller(tmp_path):
    exe, so = str(tmp_path / "host_alloc_failure"), os.path.dirname(b.LIB)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + b.INCLUDE, os.path.join(ROOT, "tests", "host_alloc_failure.cpp"),
                    "-o", exe, b.LIB, "-Wl,-rpath," + so, "-lpthread"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, env=dict(os.environ, OMP_NUM_THREADS="4"))
    assert r.returncode == 0 and "status 0" in r.stdout, (r.returncode, r.stdout, r.stderr)
    assert int(r.stdout.split()[-1]) > 0  # cores were refused memory
