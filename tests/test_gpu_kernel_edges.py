"""Kernels at the sizes where their work split changes, against the FP64 oracle.

Backward descriptors: 32 lanes per atom below 4096 atoms and 16 from there (where two atoms' G
fits), one- and several-species fuse matrices, more than three species (the sparse fuse
tables), rows of fewer entries than a lane group, of whole groups and of one more.
Neighbour rows: the chunk of atoms per warp (1, 2, 4 or 8 by the atom count), cells of the
cutoff's width and of half of it, thin boxes with more stencil cells than are held at a time,
batches that mix them.  Sets are compared exactly.
FP32 network: see its test.
Forward descriptors on the tensor cores: rounds of four atoms with one to five atoms in them,
atoms without a neighbour, rows of more than 64.  A coefficient is the sum of up to 15 MMAs that
each truncate it (2^-23), squared: 4e-6 of a column's scale, tested at 1e-5.

Tolerances: a pair gradient is a sum of 2 N1 (lmax+1)^2, about a thousand, products of 24-bit
numbers (2^-24 sqrt(1000) = 2e-6 of its terms) whose terms cancel to about a tenth: 2e-5 of the
largest force on average, five times that at most.  Energies: the plain path's 2e-5 eV.
"""
import numpy as np
import pytest

from jse_gb300 import workloads as W
from oracle import model as OM, native as ON

pytestmark = pytest.mark.gpu


def _model(basis, T, hidden=(16, 16), seed=3):
    """A random model normalised over a small structure, so that no network saturates."""
    symbols = ["A", "B", "C", "D"][:T]
    m = W.write_model(symbols, basis, list(hidden), seed)
    s = W.random_liquid(120, 0.05, [1.0 / T] * T, 2.0, 9)
    fp = ON.compute(OM.load(m), s.x, s.types, s.box_kind, s.box, want_fp=True)["fp"]
    mu, sd = fp.mean(0), fp.std(0) + 1e-2 * np.abs(fp).max(0) + 1e-3
    return W.write_model(symbols, basis, list(hidden), seed, [mu] * T, [sd] * T)


def _check(model, s, precision="fp32", etol=2e-5, fmax=1e-4, frms=2e-5):
    from jse_gb300.nnap import NNAP
    r = ON.compute(OM.load(model), s.x, s.types, s.box_kind, s.box)
    with NNAP(model, precision=precision) as p:
        o = p.calEnergyForceVirials(s)
    assert np.abs(o["energies"] - r["energies"]).max() <= etol * max(1.0, np.abs(r["energies"]).max())
    for key in ("forces", "virials"):
        d = np.abs(o[key] - r[key])
        scale = np.abs(r[key]).max()
        assert d.max() <= fmax * scale and np.sqrt((d * d).mean()) <= frms * scale, (key, d.max() / scale)


LMAX4 = {"type": "spherical_chebyshev", "nmax": 8, "lmax": 4, "rcut": 5.5}
DEFAULT = {"type": "spherical_chebyshev", "rcut": 6.0}  # nmax 5, lmax 6
FULL = {"type": "spherical_chebyshev", "nmax": 3, "lmax": 2, "rcut": 5.0, "wtype": "full"}


@pytest.mark.parametrize("basis,T,n,density", [
    (LMAX4, 2, 4095, 0.058), (LMAX4, 2, 4097, 0.058), (LMAX4, 1, 4096, 0.023), (LMAX4, 2, 4100, 0.094),
    (DEFAULT, 2, 4101, 0.06), (DEFAULT, 2, 61, 0.035), (DEFAULT, 1, 4099, 0.018), (DEFAULT, 1, 75, 0.075),
    (FULL, 4, 4098, 0.06), (FULL, 4, 33, 0.09)])
def test_backward_lanes(basis, T, n, density):
    s = W.random_liquid(n, density, [1.0 / T] * T, 1.9, n, tilt=0.1)
    _check(_model(basis, T), s)


def _keys(off, j, img):
    i = np.repeat(np.arange(len(off) - 1), np.diff(off))
    img = np.asarray(img).reshape(-1, 3)
    return np.unique(np.stack([i, j, img[:, 0], img[:, 1], img[:, 2]], 1), axis=0), len(j)


def _same_rows(p, s, rcut):
    off, j, img = p.neighborList(s)
    nl = ON.neighbors(ON.wrap(s.x, s.box_kind, s.box), s.box_kind, s.box, rcut)
    a, na = _keys(off, j, img)
    b, nb = _keys(nl.offsets, nl.j, nl.img)
    assert na == nb == len(a) and np.array_equal(a, b)


@pytest.mark.parametrize("rcut,n,tilt", [
    (5.0, 1, None), (5.0, 9, 0.1), (5.0, 4863, None), (5.0, 14593, 0.1), (5.0, 29187, None), (5.0, 58370, 0.1),
    (8.0, 3, 0.1), (8.0, 611, None), (8.0, 14593, 0.1), (8.0, 29190, None)])
def test_neighbor_chunks(rcut, n, tilt):
    from jse_gb300.nnap import NNAP
    model = W.write_model(["A", "B"], {"type": "chebyshev", "nmax": 3, "rcut": rcut}, [4], 1)
    s = W.random_liquid(n, 0.06, [0.5, 0.5], 1.9, n + 1, tilt=tilt)
    with NNAP(model) as p:
        _same_rows(p, s, rcut)


def test_neighbor_thin_boxes():
    from jse_gb300.nnap import NNAP
    model = W.write_model(["A"], {"type": "chebyshev", "nmax": 3, "rcut": 6.0}, [4], 1)
    rng = np.random.default_rng(4)
    boxes = [np.diag([70.0, 2.3, 2.9]), np.diag([30.0, 5.0, 4.0]), np.diag([40.0, 33.0, 31.0])]
    structures = []
    for b in boxes:
        n = max(1, int(0.05 * np.linalg.det(b)))
        structures.append(W.Structure(rng.random((n, 3)) @ b, np.ones(n, dtype=np.int32), b, 0))
    with NNAP(model) as p:
        for s in structures:
            _same_rows(p, s, 6.0)
        both = p.calEnergyForceVirialsBatch(structures)
        for s, o in zip(structures, both):
            r = p.calEnergyForceVirials(s)
            assert np.array_equal(r["forces"], o["forces"]) and np.array_equal(r["energies"], o["energies"])


@pytest.mark.parametrize("precision", ["mixed", "fp32"])
@pytest.mark.parametrize("n,density", [(1, 0.001), (2, 0.003), (3, 0.06), (5, 0.012), (33, 0.06), (66, 0.083)])
def test_forward_descriptors(precision, n, density):
    from jse_gb300.nnap import NNAP
    basis = {"type": "spherical_chebyshev", "nmax": 8, "lmax": 6, "rcut": 6.0}
    model = W.write_model(["A", "B", "C"], basis, [8], 2)
    s = W.random_liquid(n, density, [0.4, 0.4, 0.2], 1.8, n, tilt=0.1)
    ref = ON.compute(OM.load(model), s.x, s.types, s.box_kind, s.box, want_fp=True)["fp"]
    with NNAP(model, precision=precision) as p:
        fp = p.calFp(s)
    scale = np.abs(ref).max(0) + 1e-6
    assert (np.abs(fp - ref) / scale).max() <= 1e-5


@pytest.mark.parametrize("T,nmax,hidden,n", [
    (1, 10, (32, 32), 5), (1, 10, (33,), 9), (2, 15, (31,), 40), (3, 20, (64, 7, 40), 1), (3, 20, (64, 7, 40), 17),
    (3, 20, (300, 20), 33), (2, 15, (64, 64), 3700)])
def test_network_slices(T, nmax, hidden, n):
    """The FP32 network by a warp, a CTA or without slices per eight atoms: layers of up to one, of
    exactly one and of several slices, more units than a CTA's threads, the last group of atoms
    short, a batch equal to its structures alone.  Sums of up to 300 products: 2^-24 sqrt(300) =
    1e-6 of the terms."""
    from jse_gb300.nnap import NNAP
    model = _model({"type": "chebyshev", "nmax": nmax, "rcut": 5.0}, T, hidden)
    s = W.random_liquid(n, 0.05, [1.0 / T] * T, 1.9, n)
    _check(model, s)
    small = W.random_liquid(13, 0.05, [1.0 / T] * T, 1.9, 2)
    with NNAP(model) as p:
        for a, b in zip(p.calEnergyForceVirialsBatch([small, s]), [p.calEnergyForceVirials(small), p.calEnergyForceVirials(s)]):
            assert np.array_equal(a["energies"], b["energies"]) and np.array_equal(a["forces"], b["forces"])


@pytest.mark.parametrize("n", [1, 31, 40, 65, 700])
def test_training_sums(n):
    """Parameter gradients with fewer partials than the final sum's rows, chunks of a few slots and
    several, against the oracle's energies: dL/d(output bias) is the sum of the upstream energy
    gradients times sigma_E, exactly (2^-24 sqrt(n) of its terms), and the radial weights' gradient
    of a batch is the sum of its structures' (the FP32 partials' 2^-22)."""
    from jse_gb300.nnap import NNAP
    rng = np.random.default_rng(n)
    basis = {"type": "spherical_chebyshev", "nmax": 4, "lmax": 4, "rcut": 5.0, "wtype": "fuse", "fuse_size": 2,
             "fuse_weight": rng.normal(0, 1, 4).tolist()}
    model = W.write_model(["A", "B"], dict(basis, wtype="default"), [8, 8], 1)
    for m in model["models"]:
        m["basis"] = basis
    ss = [W.random_liquid(n, 0.05, [0.5, 0.5], 1.9, n), W.random_liquid(12, 0.05, [0.5, 0.5], 1.9, 3)]
    N = n + 12
    be, bf = rng.normal(0, 1, N), rng.normal(0, 1, (N, 3))
    with NNAP(model) as p:
        both = p.backwardEnergyForceBatch(ss, be, bf, want_fp=True)
        one = [p.backwardEnergyForceBatch([ss[0]], be[:n], bf[:n], want_fp=True),
               p.backwardEnergyForceBatch([ss[1]], be[n:], bf[n:], want_fp=True)]
    types = np.concatenate([s.types for s in ss])
    for t in range(2):
        want = be[types == t + 1].sum()
        assert abs(both["grad_nn"][t][-1] - want) <= 1e-6 * np.abs(be).sum()
        for key in ("grad_nn", "grad_fp"):
            parts = one[0][key][t] + one[1][key][t]
            size = np.abs(one[0][key][t]) + np.abs(one[1][key][t])
            assert np.abs(both[key][t] - parts).max() <= 1e-5 * max(size.max(), 1e-30)


@pytest.mark.parametrize("n", [7, 15000, 22000])
def test_host_staging(n):
    """Host calls that go through pinned staging (up to 2 MiB in and out) and ones that copy directly
    give the same numbers for every choice of outputs, with outputs in any order, call after call."""
    import ctypes as C
    from jse_gb300 import nnap as J
    model = W.write_model(["A"], {"type": "chebyshev", "nmax": 3, "rcut": 3.0}, [4], 1)
    s = W.random_liquid(n, 0.05, [1.0], 1.6, n)
    with J.NNAP(model) as p:
        ref = p.calEnergyForceVirials(s)  # n = 22000 with per-atom virials: above the limit
        shapes = {"energy": (1,), "energies": (n,), "forces": (n, 3), "virial": (9,), "virials": (n, 9)}
        for flags in (J.WANT_ENERGY, J.WANT_FORCES, J.WANT_ENERGIES | J.WANT_VIRIAL, 31, J.WANT_VIRIALS, 31):
            out = {k: np.full(v, np.nan) for k, v in shapes.items()}
            p._check(p._L.nnap_compute(p._handle(), n, J._dptr(np.ascontiguousarray(s.x)), J._iptr(s.types), s.box_kind,
                                       J._dptr(np.ascontiguousarray(s.box.reshape(9))), flags,
                                       *[J._dptr(out[k]) for k in ("energy", "energies", "forces", "virial", "virials")]))
            for bit, k in zip((1, 2, 4, 8, 16), ("energy", "energies", "forces", "virial", "virials")):
                if flags & bit:
                    assert np.array_equal(out[k].reshape(-1), np.reshape(ref[k], -1)), (flags, k)
                else:
                    assert np.isnan(out[k]).all()
        bad = W.Structure(s.x, s.types.copy(), s.box, s.box_kind)
        bad.types[-1] = 2
        with pytest.raises(ValueError):
            p.calForces(bad)
        assert np.array_equal(p.calForces(s), ref["forces"])


@pytest.mark.parametrize("T,n,density,tilt", [
    (1, 1, 0.01, None), (3, 2, 0.02, 0.1), (16, 31, 0.05, None), (16, 33, 0.05, 0.1), (3, 1023, 0.05, None),
    (3, 1024, 0.05, 0.1), (3, 1025, 0.05, None), (2, 900, 0.0002, None), (2, 900, 0.0001, None)])
def test_one_cta_order(T, n, density, tilt):
    """Atoms ordered by one CTA (up to 1024 atoms and 4096 cells) and by the general kernels: exact
    neighbour sets, descriptors in atom order, and the structure alone equal to it in a batch too
    large for one CTA, bit for bit."""
    from jse_gb300.nnap import NNAP
    basis = {"type": "chebyshev", "nmax": 2, "rcut": 5.0, "wtype": "none"}
    model = W.write_model(["S%d" % k for k in range(T)], basis, [4], 1)
    s = W.random_liquid(n, density, [1.0 / T] * T, 1.9, n, tilt=tilt)
    other = W.random_liquid(1100, 0.05, [1.0 / T] * T, 1.9, 5)
    ref = ON.compute(OM.load(model), s.x, s.types, s.box_kind, s.box, want_fp=True)
    with NNAP(model) as p:
        _same_rows(p, s, 5.0)
        assert np.abs(p.calFp(s) - ref["fp"]).max() <= 1e-5 * max(1.0, np.abs(ref["fp"]).max())
        alone, batch = p.calEnergyForceVirials(s), p.calEnergyForceVirialsBatch([s, other], per_atom_virial=True)[0]
        for key in ("energies", "forces", "virials"):
            assert np.array_equal(alone[key], batch[key])


@pytest.mark.parametrize("T,nmax,hidden,n", [
    (1, 10, (16,), 1999), (2, 15, (64, 64), 1921), (3, 18, (32, 48, 20), 2047), (2, 12, (64, 100), 2048),
    (1, 8, (250, 96), 1700)])
def test_network_two_tiles(T, nmax, hidden, n):
    """The tensor-core network with two tiles in flight (more than two per SM): one to three hidden
    layers, descriptors and layers of odd widths, short last tiles of every species, two groups
    that fit and (250-96) do not.  The same operations in the same order as with one tile in
    flight: equal to the structures alone, bit by bit, and those to the oracle within the mixed
    path's 5e-5 eV, 1e-3 and 2e-4 of the largest force."""
    from jse_gb300.nnap import NNAP
    model = _model({"type": "chebyshev", "nmax": nmax, "rcut": 5.0}, T, hidden)
    ss = [W.random_liquid(k, 0.05, [1.0 / T] * T, 1.9, k) for k in (n, 13, 1, 130)]
    _check(model, ss[3], "mixed", 5e-5, 1e-3, 2e-4)
    with NNAP(model, precision="mixed") as p:
        alone = [p.calEnergyForceVirials(s) for s in ss]
        for k, b in enumerate(p.calEnergyForceVirialsBatch(ss * 24)):
            a = alone[k % 4]
            assert np.array_equal(a["energies"], b["energies"]) and np.array_equal(a["forces"], b["forces"])


@pytest.mark.parametrize("precision", ["mixed", "fp32"])
@pytest.mark.parametrize("basis", [
    {"type": "chebyshev", "nmax": 6, "rcut": 5.0},
    {"type": "spherical_chebyshev", "nmax": 8, "lmax": 6, "rcut": 6.0},
    {"type": "spherical_chebyshev", "nmax": 3, "lmax": 4, "l3max": 4, "l4max": 2, "rcut": 5.0},
    {"type": "merge", "basis": [{"type": "chebyshev", "nmax": 5, "rcut": 6.0},
                                {"type": "spherical_chebyshev", "nmax": 3, "lmax": 3, "rcut": 4.5, "wtype": "full"}]}])
def test_descriptors_after_another_structure(precision, basis):
    """Rows of descriptors are written whole: what an evaluation before left in the workspace does
    not show, and atoms without a neighbour have zeros.  Equal bit by bit."""
    from jse_gb300.nnap import NNAP
    from tests.golden.make_golden import _model as make
    model = make(["A", "B"], basis, [8, 8], 2)
    big, s = W.random_liquid(300, 0.06, [0.5, 0.5], 1.9, 1), W.random_liquid(7, 0.002, [0.5, 0.5], 1.9, 5)
    with NNAP(model, precision=precision) as p, NNAP(model, precision=precision) as q:
        p.calEnergyForceVirials(big)
        a, b = p.calEnergyForceVirials(s), q.calEnergyForceVirials(s)
        assert np.array_equal(p.calFp(s), q.calFp(s)) and np.isfinite(p.calFp(s)).all()
        assert all(np.array_equal(a[k], b[k]) for k in ("energies", "forces", "virials"))
