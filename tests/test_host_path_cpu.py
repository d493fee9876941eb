"""The library's host path without a GPU: what it allocates, copies and launches.

Child processes load a stand-in for the CUDA runtime (fake_cudart.cpp: host memory, kernels that do
not run, two devices, the shared-memory limit of a launch as the runtime enforces it) ahead of
libcudart.  Its values are zeros; the tests look at the calls."""
import functools
import os
import shutil
import subprocess
import sys
import tempfile
import textwrap

import pytest

from tests.conftest import ROOT

HEAD = """
import ctypes as C, os, sys, threading, time
import numpy as np
F = C.CDLL(os.environ["FAKE_CUDART"])
from jse_gb300 import nnap as J, workloads as W
def log():
    b = C.create_string_buffer(1 << 22)
    assert F.fake_log(b, 1 << 22) < 1 << 22
    return b.value.decode().splitlines()
def launches(part):
    return [l.split() for l in log() if l.startswith("launch") and part in l]
def atoms(n, T=2, density=0.05):
    return W.random_liquid(n, density, [1.0 / T] * T, 1.9, n)
def sph(T, hidden, nmax=8, lmax=6, wtype="default"):
    return W.write_model(["S%d" % t for t in range(T)],
                         {"type": "spherical_chebyshev", "nmax": nmax, "lmax": lmax, "rcut": 6.0, "wtype": wtype}, hidden, 1)
"""


@functools.lru_cache(None)
def _fake():
    inc = [d for d in (os.environ.get("CUDA_HOME", ""), "/usr/local/cuda") if os.path.exists(os.path.join(d, "include", "cuda_runtime_api.h"))]
    if not inc or not shutil.which("g++"):
        pytest.skip("no CUDA headers or no g++")
    from jse_gb300 import build, nnap
    if not os.path.exists(nnap.LIB_PATH):
        build.build()
    out = os.path.join(tempfile.mkdtemp(), "libfakecudart.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", os.path.join(inc[0], "include"),
                    os.path.join(ROOT, "tests", "fake_cudart.cpp"), "-o", out, "-lpthread"], check=True)
    return out


def _child(code):
    env = dict(os.environ, LD_PRELOAD=_fake(), FAKE_CUDART=_fake(), PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", HEAD + textwrap.dedent(code)], env=env, cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]


def test_shared_memory_limits_of_a_second_device():
    """Every launch beyond 48 KiB is allowed on each device that a handle is made for."""
    _child("""
    rng = np.random.default_rng(1)
    deep = sph(3, [64, 64])
    for device in (0, 1):
        for model, T in ((deep, 3), (sph(1, [300, 100], 5), 1), (sph(8, [32], 5), 8), (sph(2, [20], 7, 5), 2)):
            for precision in ("fp32", "mixed"):
                with J.NNAP(model, precision=precision, device=device) as p:
                    for n in (60, 4500, 50000):
                        p.calForces(atoms(n, T))
                    p.setTuning(4500, dict(p.tuning(4500), desc_fwd_warps=8, desc_bwd_warps=8, nb_warps=8))
                    p.calForces(atoms(4500, T))
                    p.calFp(atoms(60, T))
        basis = {"type": "spherical_chebyshev", "nmax": 4, "lmax": 4, "rcut": 5.0, "wtype": "fuse", "fuse_size": 2}
        fuse = W.write_model(["A", "B"], dict(basis, wtype="default"), [64, 64], 1)
        for m in fuse["models"]:
            m["basis"] = dict(basis, fuse_weight=rng.normal(0, 1, 4).tolist())
        with J.NNAP(fuse, device=device) as p:
            p.backwardEnergyForceBatch([atoms(40)], np.ones(40), np.ones((40, 3)), want_fp=True)
    big = {int(l.split()[3]) for l in log() if l.startswith("launch") and int(l.split()[4]) > 48 * 1024}
    assert big == {0, 1}, big
    """)


def test_shared_memory_limits_of_two_threads():
    """A narrow network's call between another thread's raise of the limit and its launch."""
    _child("""
    s = atoms(4000, 3)
    wide, narrow = J.NNAP(sph(3, [200, 200])), J.NNAP(sph(3, [64, 64]))
    F.fake_pause(b"k_net_warp")
    failed = []
    def work():
        try:
            wide.calForces(s)
        except Exception as e:
            failed.append(e)
    t = threading.Thread(target=work)
    t.start()
    while not F.fake_paused():
        time.sleep(0.01)
    narrow.calForces(s)
    F.fake_resume()
    t.join()
    assert not failed, failed
    """)


def test_backward_warps_of_many_species():
    """The backward's shared memory does not grow with the square of the species: eight warps or
    more stay on an SM (228 KB, of which each CTA costs 1 KB more than it asks for)."""
    _child("""
    for T, lmax in ((4, 6), (10, 6), (12, 4), (15, 4)):
        with J.NNAP(sph(T, [16], 8, lmax)) as p:
            log()
            p.calForces(atoms(600, T))
            (l,) = launches("k_sph_bwd_n")
            grid, threads, smem = int(l[1]), int(l[2]), int(l[4])
            warps = threads // 32 * (228 * 1024 // (smem + 1024))
            assert warps >= 8 and grid * threads // 32 >= 600, (T, lmax, l, warps)
    """)


def test_default_shape_of_many_species():
    """The compiled forward of the default shape serves few species, the any-shape one many; the
    radial-space backward serves them all."""
    _child("""
    for T, wtype in ((6, "default"), (7, "default"), (16, "default"), (6, "none"), (12, "none")):
        with J.NNAP(sph(T, [16], 5, 6, wtype)) as p:
            p.calForces(atoms(600, T))
            names = [l.split()[5] for l in log() if l.startswith("launch")]
            assert any("k_sph_bwd_n" in s for s in names), names
            assert any("9k_sph_fwd" in s for s in names) == (T <= 6), (T, names)
            assert any("k_sph_fwd_g" in s for s in names) == (T > 6), (T, names)
    """)


def test_any_shape_kernels_launch_after_their_predecessors():
    """Early, they would run with the split of shared memory and L1 of the kernels before them."""
    _child("""
    for basis in ({"type": "chebyshev", "nmax": 15, "rcut": 4.0}, {"type": "spherical_chebyshev", "nmax": 6, "lmax": 5, "rcut": 5.0}):
        model = W.write_model(["A", "B"], basis, [30], 1)
        for precision in ("fp32", "mixed"):
            with J.NNAP(model, precision=precision) as p:
                log()
                p.calForces(atoms(600))
                l = [l for l in log() if l.startswith("launch")]
                fwd, bwd = ([s for s in l if part in s] for part in ("fwd_g", "bwd_g"))
                assert len(fwd) == len(bwd) == 1 and not fwd[0].endswith("early") and not bwd[0].endswith("early"), l
    """)


def test_staging_by_size_and_memory():
    """Small host calls are staged; larger ones, and sooner those whose memory is pinned, copy
    straight between the caller's arrays and the device."""
    _child("""
    model = W.write_model(["A", "B"], {"type": "chebyshev", "nmax": 3, "rcut": 4.0}, [4], 1)
    cudart = F
    def host(a, pinned):
        if not pinned:
            return np.array(a)
        p = C.c_void_p()
        assert cudart.cudaMallocHost(C.byref(p), C.c_size_t(a.nbytes)) == 0
        b = np.frombuffer((C.c_char * a.nbytes).from_address(p.value), dtype=a.dtype).reshape(a.shape)
        b[...] = a
        return b
    for n, pinned, staged in ((30, False, True), (30, True, True), (4000, False, True), (4000, True, False), (8000, False, True),
                              (16000, False, False), (16000, True, False)):
        s = atoms(n)
        x, t, e, f = (host(a, pinned) for a in (s.x, s.types, np.zeros(1), np.zeros((n, 3))))
        with J.NNAP(model) as p:
            box = np.ascontiguousarray(s.box.reshape(9))
            for _ in range(2):
                log()
                p._check(p._L.nnap_compute(p._handle(), n, J._dptr(x), J._iptr(t), s.box_kind, J._dptr(box), 5, J._dptr(e), None,
                                           J._dptr(f), None, None))
                calls = log()
                ends = {int(v) for l in calls if l.startswith("copy") for v in l.split()[3:]}
                assert any("k_pack_results" in l for l in calls) == staged, (n, pinned, calls)
                for a in (x, f):
                    assert (a.ctypes.data in ends) == (not staged), (n, pinned, calls)
    """)


def test_staging_of_a_growing_structure():
    """Insertion moves: an atom more per call, and few allocations of pinned memory for all of them."""
    _child("""
    model = W.write_model(["A", "B"], {"type": "chebyshev", "nmax": 3, "rcut": 4.0}, [4], 1)
    s = atoms(400)
    with J.NNAP(model) as p:
        p.calForces(W.Structure(s.x[:100], s.types[:100], s.box, s.box_kind))
        log()
        for n in range(101, 401):
            p.calForces(W.Structure(s.x[:n], s.types[:n], s.box, s.box_kind))
        calls = log()
        assert sum("k_pack_results" in l for l in calls) == 300
        assert sum(l.startswith("host_alloc") for l in calls) <= 6, [l for l in calls if l.startswith("host_")]
    """)


def test_calls_that_alternate_share_a_captured_sequence():
    """Forces (copied directly at this size) and the energy alone (staged) in turn: the launch
    sequence of the layout is captured once."""
    _child("""
    model = W.write_model(["A", "B"], {"type": "chebyshev", "nmax": 3, "rcut": 4.0}, [4], 1)
    s = atoms(8000)
    box = np.ascontiguousarray(s.box.reshape(9))
    e, f = np.zeros(1), np.zeros((8000, 3))
    with J.NNAP(model) as p:
        log()
        for k in range(12):
            p._check(p._L.nnap_compute(p._handle(), 8000, J._dptr(s.x), J._iptr(s.types), s.box_kind, J._dptr(box), 4 if k % 2 else 1,
                                       J._dptr(e), None, J._dptr(f), None, None))
        calls = log()
        assert sum("k_pack_results" in l for l in calls) == 6, "the sizes no longer straddle the limit"
        assert calls.count("capture") == 1, calls.count("capture")
    """)


def test_autotuner_times_shapes_that_differ():
    """Two runs and a warm-up per candidate: the backward of compiled shapes runs at most four warps,
    the network has no choice of threads per row with two tiles in flight."""
    _child("""
    for model, n, precision, shapes in ((sph(2, [16], 5), 600, "fp32", 11), (sph(2, [16], 4, 5), 600, "fp32", 12),
                                        (sph(2, [16], 5), 600, "mixed", 13), (sph(2, [16], 5), 41000, "mixed", 11)):
        with J.NNAP(model, precision=precision) as p:
            p.setAutotune(True)
            log()
            p.calForces(atoms(n))
            calls = len(launches("k_neighbors"))
            assert calls == 3 * shapes + 2, (n, precision, calls)
            log()
            p.calForces(atoms(n))
            assert len(launches("k_neighbors")) == 1
    """)
