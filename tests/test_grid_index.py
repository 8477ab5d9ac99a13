"""The bucket index of gridded fields on the CPU (tests/cpp/grid_index_check.cpp):
against a search of all triangles, in the arithmetic of both lookups, for even
and strongly graded grids, slivers, rows of buckets, vertices, edge points and
points at the end of the last bucket; lists longer than the seven inline ids, and the
lean form's lists;
and its build on several threads: the same index, in the time of a serial one
or less."""
import os
import subprocess
import time

import numpy as np
import pytest

from jetshow_gb300.runtime import triangulate

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "jetshow_gb300", "csrc")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    d = tmp_path_factory.mktemp("index")
    exe = str(d / "check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", CSRC, "-I", os.path.join(REPO, "include"),
                    os.path.join(REPO, "tests", "cpp", "grid_index_check.cpp"), os.path.join(CSRC, "jsh_grid_index.cpp"),
                    "-o", exe, "-lpthread"], check=True)

    def run(xy, tri, q, lean=False):
        path = str(d / "grid.bin")
        with open(path, "wb") as f:
            f.write(np.array([len(xy), len(tri), len(q)], np.int64).tobytes())
            f.write(np.ascontiguousarray(xy, np.float64).tobytes())
            f.write(np.ascontiguousarray(tri, np.int32).tobytes())
            f.write(np.ascontiguousarray(q, np.float64).tobytes())
        r = subprocess.run([exe, path] + ["lean"] * lean, capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stdout + r.stderr
        w = r.stdout.split()
        return dict(buckets=int(w[0]), entries=int(w[2]), longest=int(w[5].rstrip(",")), inside=int(w[6]))

    return run


def grids():
    rng = np.random.default_rng(7)
    even = rng.random((3000, 2)) * [20.0, 0.5]
    graded = np.column_stack([20.0 * rng.random(3000) ** 6, 0.5 * rng.random(3000) ** 6])
    box = np.array([[0.0, 0.0], [20.0, 0.0], [0.0, 0.5], [20.0, 0.5]])
    strip = np.vstack([np.column_stack([np.linspace(0.0, 20.0, 1500), np.zeros(1500)]),
                       np.column_stack([np.linspace(0.0, 20.0, 1499), np.full(1499, 1e-4)])])
    fan = np.vstack([[[0.0, 0.0]], np.column_stack([np.full(400, 20.0), np.linspace(0.0, 0.5, 400)])])
    far = rng.random((2000, 2)) + [300.0, 0.0]
    return {"even": even, "graded": np.vstack([graded, box]), "strip": strip, "fan": fan, "far": far, "box": box}


@pytest.mark.parametrize("lean", [False, True])
@pytest.mark.parametrize("kind", ["even", "graded", "strip", "fan", "far", "box"])
def test_finds_what_all_triangles_hold(check, kind, lean):
    xy = grids()[kind]
    tri = triangulate(xy)
    rng = np.random.default_rng(11)
    lo, hi = xy.min(0), xy.max(0)
    # points of random triangles (few, whatever their size), and of the rectangle
    w = rng.dirichlet([1.0, 1.0, 1.0], 600)
    pick = tri[rng.integers(len(tri), size=600)]
    edge = xy[pick[:200, 0]] + rng.random((200, 1)) * (xy[pick[:200, 1]] - xy[pick[:200, 0]])
    q = np.vstack([(w[:, :, None] * xy[pick]).sum(1), edge, xy[:200], lo + (hi - lo) * rng.uniform(-0.05, 1.05, (300, 2)),
                   [hi, [hi[0], lo[1]], [lo[0], hi[1]], lo], np.column_stack([np.full(50, hi[0]), rng.uniform(lo[1], hi[1], 50)])])
    s = check(xy, tri, q, lean)
    assert s["inside"] > 500
    if kind in ("graded", "fan"):
        assert s["longest"] > 7


def test_build_time(lib):
    """The index on several threads is under a third of the time of the same
    grid's triangulation on one (about a tenth on 16 cores; the serial build of
    two passes was about half)."""
    import ctypes as C
    rng = np.random.default_rng(2)
    xy = rng.random((200_000, 2)) * [20.0, 0.5]
    t_tri = time.perf_counter()
    tri = triangulate(xy)
    t_tri = time.perf_counter() - t_tri
    src = r"""
#include <stdio.h>
#include <stdarg.h>
#include "jsh_grid_index.h"
void jsh_set_error(const char*, ...) {}
extern "C" long long build(const double* xy, long long n, const int* tri, long long m) {
  JshGridIndex X;
  return jsh_grid_index(xy, n, tri, m, false, &X) ? -1 : (long long)X.more.n;
}
"""
    import tempfile
    with tempfile.TemporaryDirectory() as d:
        open(os.path.join(d, "b.cpp"), "w").write(src)
        so = os.path.join(d, "b.so")
        subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-ffp-contract=off", "-I", CSRC, "-I",
                        os.path.join(REPO, "include"), os.path.join(d, "b.cpp"),
                        os.path.join(CSRC, "jsh_grid_index.cpp"), "-o", so, "-lpthread"], check=True)
        L = C.CDLL(so)
        L.build.restype = C.c_longlong
        L.build.argtypes = [C.c_void_p, C.c_longlong, C.c_void_p, C.c_longlong]
        best = 1e9
        for _ in range(5):
            t0 = time.perf_counter()
            assert L.build(xy.ctypes.data, len(xy), tri.ctypes.data, len(tri)) >= 0
            best = min(best, time.perf_counter() - t0)
    if (os.cpu_count() or 1) >= 4:
        assert best < t_tri / 3
