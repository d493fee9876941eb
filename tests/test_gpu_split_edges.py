"""Splits of work by size at their edges: lanes and chunks of the LAMMPS sums, totals of batches
with empty structures, host calls that grow and shrink, eight atoms per warp over half-width cells."""
import numpy as np
import pytest

from jse_gb300 import workloads as W
from oracle import native as ON

pytestmark = pytest.mark.gpu


def _radial(rcut=4.0, nmax=3):
    return W.write_model(["A", "B"], {"type": "chebyshev", "nmax": nmax, "rcut": rcut}, [8], 1)


def _cluster(n, seed):
    """Atoms of a box's interior in a vacuum that leaves no images in reach, and their full lists."""
    s = W.random_liquid(n, 0.05, [0.5, 0.5], 1.9, seed)
    box = s.box + 20.0 * np.eye(3)
    x = ON.wrap(s.x, 0, s.box) + 10.0
    d = np.linalg.norm(x[:, None] - x[None], axis=2)
    lists = [np.flatnonzero((row < 4.5) & (np.arange(n) != i)) for i, row in enumerate(d)]
    return W.Structure(x, s.types, box, 0), lists


@pytest.mark.parametrize("nall", [1, 2, 15, 17, 511, 512, 513, 1024, 1025, 1537])
def test_lammps_sums(nall):
    """Every atom local against the periodic call (other displacements and another order of FP32
    terms: 1e-5 of the largest force); half of them local: forces sum to zero, energies and virials
    to the totals, which the call adds itself in FP64."""
    from jse_gb300.nnap import NNAP
    s, lists = _cluster(nall, nall)
    with NNAP(_radial()) as p:
        ref = p.calEnergyForceVirials(s)
        for inum in {nall, (nall + 1) // 2}:
            il = np.arange(inum)
            o = p.computeLammps(il, lists[:inum], s.x, s.types)
            total = p.computeLammps(il, lists[:inum], s.x, s.types, cvflag_atom=False)
            kept = p.computeLammps(il, lists[:inum], s.x, s.types, cvflag_atom=False, nlflag=False)
            v = o["cvatom"][:, :6]
            assert np.abs(total["virial"] - v.sum(0)).max() <= 1e-12 * (np.abs(v).sum() + 1e-30)
            assert np.array_equal(total["virial"], kept["virial"]) and np.array_equal(o["forces"], kept["forces"])
            assert np.abs(o["forces"].sum(0)).max() <= 1e-6 * (np.abs(o["forces"]).sum() + 1e-30)
            assert abs(o["eng"] - o["eatom"].sum()) <= 1e-9 * nall
            if inum == nall:
                scale = max(np.abs(ref["forces"]).max(), 1e-3)
                assert np.abs(o["forces"] - ref["forces"]).max() <= 1e-5 * scale
                assert np.abs(o["eatom"] - ref["energies"]).max() <= 1e-5


def test_totals_with_empty_structures():
    """Structures of no atoms, of one chunk of the reduction and of several in one batch, in any
    order: each as by itself."""
    from jse_gb300.nnap import NNAP
    ss = [W.random_liquid(n, 0.05, [0.5, 0.5], 1.9, n) for n in (50, 1024, 1025, 3, 2100)]
    empty = W.Structure(np.zeros((0, 3)), np.zeros(0, dtype=np.int32), 9.0 * np.eye(3), 0)
    with NNAP(_radial()) as p:
        alone = [p.calEnergyForceVirials(s) for s in ss]
        for order in ([0, 3], [0, None], [None, 0, 3], [0, None, 2], [3, 1, None, 4, 0], [None, None, 1]):
            batch = p.calEnergyForceVirialsBatch([empty if k is None else ss[k] for k in order])
            for k, o in zip(order, batch):
                if k is None:
                    assert o["energy"] == 0.0 and not np.any(o["virial"])
                    continue
                for key in ("energies", "forces"):
                    assert np.array_equal(o[key], alone[k][key])
                assert abs(o["energy"] - alone[k]["energy"]) <= 1e-9 and np.allclose(o["virial"], alone[k]["virial"], rtol=1e-9)


def test_host_calls_that_grow_and_shrink():
    from jse_gb300.nnap import NNAP
    ss = [W.random_liquid(n, 0.05, [0.5, 0.5], 1.9, n) for n in (7, 900, 30, 5000, 900, 1, 17000, 64)]
    with NNAP(_radial()) as p:
        for s in ss:
            o = p.calEnergyForceVirials(s)
            with NNAP(_radial()) as q:
                fresh = q.calEnergyForceVirials(s)
            for key in ("energies", "forces", "virials"):
                assert np.array_equal(o[key], fresh[key]), s.natoms


@pytest.mark.parametrize("tilt", [None, 0.1])
def test_eight_atoms_per_warp_over_half_width_cells(tilt):
    import torch
    from jse_gb300.nnap import NNAP
    n = 8 * 48 * torch.cuda.get_device_properties(0).multi_processor_count + 2
    s = W.random_liquid(n, 0.045, [0.5, 0.5], 1.9, 5, tilt=tilt)
    with NNAP(_radial(8.0)) as p:
        off, j, img = p.neighborList(s)
    nl = ON.neighbors(ON.wrap(s.x, s.box_kind, s.box), s.box_kind, s.box, 8.0)
    assert np.array_equal(np.diff(off), np.diff(nl.offsets))

    def rows(offsets, j, img):
        i = np.repeat(np.arange(n), np.diff(offsets))
        img = np.asarray(img).reshape(-1, 3)
        order = np.lexsort((img[:, 2], img[:, 1], img[:, 0], j, i))
        return np.asarray(j)[order], img[order]
    a, b = rows(off, j, img), rows(nl.offsets, nl.j, nl.img)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
