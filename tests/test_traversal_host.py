"""The traversal code of the CUDA kernels compiled for the host
(traversal_host.cpp): the box tests against the exact slab test in 64 bits, and
the traversal stack at and past its capacity."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import PKG


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    out = str(tmp_path_factory.mktemp("traversal") / "libtraversal_host.so")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "traversal_host.cpp")
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.check_call([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-w", "-I" + cuda,
                           "-I" + os.path.join(PKG, "csrc"), src, "-o", out])
    return ctypes.CDLL(out)


def _p(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def _boxes(scale, zeros, rng, n=20000):
    """Rays and boxes of a scene with coordinates up to `scale`: `zeros` of the
    direction's components exactly 0, +0 and -0 alike (or, for `tiny`, too small
    for a finite reciprocal times a coordinate)."""
    o = rng.uniform(-1, 1, (n, 3))
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    small = np.array([0.0, -0.0, 1e-45, -1e-40, 1e-38, -1e-37, 3e-30, -1e-20])
    for k in range(n):
        for a in rng.permutation(3)[:zeros]:
            d[k, a] = small[rng.integers(0, 2 if k % 2 else len(small))]
    size = rng.uniform(0, 1, (n, 3)) * 10.0 ** rng.uniform(-3, 0, (n, 1))
    # half the boxes around a point of the ray, half anywhere
    c = np.where(rng.random((n, 1)) < 0.5, o + d * rng.uniform(0, 1, (n, 1)) + size * rng.uniform(-1, 1, (n, 3)),
                 rng.uniform(-1, 1, (n, 3)))
    lo, hi = c - size, c + size
    return [np.ascontiguousarray(x, np.float32) for x in (o * scale, d, lo * scale, hi * scale)]


@pytest.mark.parametrize("zeros", [0, 1, 2])
@pytest.mark.parametrize("scale", [1e-3, 1.0, 300.0, 1e6])
def test_box_tests_never_lose_a_box_the_ray_meets(host, scale, zeros):
    rng = np.random.default_rng(zeros * 10 + int(np.log10(scale)) + 3)
    o, d, lo, hi = _boxes(scale, zeros, rng)
    tmin, tmax = np.float32(1e-4), np.float32(1e30)
    # the exact test of the box, in 64 bits
    O, D, L, H = (x.astype(np.float64) for x in (o, d, lo, hi))
    with np.errstate(divide="ignore", invalid="ignore", over="ignore"):
        ta, tb = (L - O) / D, (H - O) / D
    t0, t1 = np.minimum(ta, tb), np.maximum(ta, tb)
    inside = (L <= O) & (O <= H)
    t0 = np.where(D == 0, np.where(inside, -np.inf, np.inf), t0)
    t1 = np.where(D == 0, np.where(inside, np.inf, -np.inf), t1)
    meets = np.maximum(t0.max(1), float(tmin)) <= np.minimum(t1.min(1), float(tmax))
    assert 0.3 < meets.mean() < 0.95
    # a BVH's boxes are padded by 2^-20 of the largest coordinate
    pad = np.float32(max(np.abs(o).max(), np.abs(lo).max(), np.abs(hi).max()) * 2.0 ** -20 + 1e-30)
    lo, hi = np.ascontiguousarray(lo - pad), np.ascontiguousarray(hi + pad)
    n = len(o)
    got = [np.zeros(n, np.uint8) for _ in range(2)]
    host.host_box_tests(n, _p(o), _p(d), _p(lo), _p(hi), ctypes.c_float(tmin), ctypes.c_float(tmax), *(_p(g) for g in got))
    for g in got:
        assert not (meets & (g == 0)).any()
        # and it rejects: at most the margins' share of the boxes beside the ray
        assert ((g != 0) & ~meets).mean() < 0.02


@pytest.mark.parametrize("any_hit", [0, 1])
@pytest.mark.parametrize("extra", [-90, -1, 0, 1, 2, 40])
def test_stack_at_and_past_its_capacity(host, any_hit, extra):
    # the top entry is in registers: kStack + 1 entries fit, what comes after is
    # dropped and reported, and no pop reads past the stack
    room = host.host_stack_size() + 1
    pushes = room + extra
    codes, ok = (ctypes.c_int * 1024)(), ctypes.c_int()
    n = host.host_push_pop(any_hit, pushes, 0x7eadbee, codes, ctypes.byref(ok))
    kept = min(pushes, room)
    assert list(codes[:n]) == list(range(kept, 0, -1))
    assert bool(ok.value) == (pushes <= room)
