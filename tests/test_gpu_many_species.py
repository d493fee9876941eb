"""Descriptors and forces of models with many species against the FP64 oracle: fuse tables read by
row, CTAs of three and four warps with a short last one, shapes compiled for few species beyond them.

Tolerances as in test_gpu_kernel_edges.py: descriptors 1e-5 of a column's largest, forces 1e-4 and
2e-5 (root mean square) of the largest, energies 2e-5 eV."""
import numpy as np
import pytest

from jse_gb300 import workloads as W
from oracle import model as OM, native as ON

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,nmax,lmax,wtype,n", [
    (4, 8, 6, "default", 97), (10, 8, 6, "default", 130), (15, 8, 4, "default", 61), (16, 8, 6, "none", 98), (5, 8, 4, "none", 4099),
    (6, 5, 6, "default", 64), (7, 5, 6, "default", 64), (16, 5, 6, "default", 155), (6, 5, 6, "none", 97), (12, 5, 6, "none", 36)])
def test_many_species(T, nmax, lmax, wtype, n):
    from jse_gb300.nnap import NNAP
    symbols = ["S%d" % t for t in range(T)]
    basis = {"type": "spherical_chebyshev", "nmax": nmax, "lmax": lmax, "rcut": 5.0, "wtype": wtype}
    s = W.random_liquid(n, 0.055, [1.0 / T] * T, 1.9, n, tilt=0.1)
    fp = ON.compute(OM.load(W.write_model(symbols, basis, [16], 2)), s.x, s.types, s.box_kind, s.box, want_fp=True)["fp"]
    mu, sd = fp.mean(0), fp.std(0) + 1e-2 * np.abs(fp).max(0) + 1e-3
    model = W.write_model(symbols, basis, [16], 2, [mu] * T, [sd] * T)
    r = ON.compute(OM.load(model), s.x, s.types, s.box_kind, s.box)
    with NNAP(model) as p:
        got, o = p.calFp(s), p.calEnergyForceVirials(s)
    assert (np.abs(got - fp) / (np.abs(fp).max(0) + 1e-6)).max() <= 1e-5
    assert np.abs(o["energies"] - r["energies"]).max() <= 2e-5 * max(1.0, np.abs(r["energies"]).max())
    d, scale = np.abs(o["forces"] - r["forces"]), np.abs(r["forces"]).max()
    assert d.max() <= 1e-4 * scale and np.sqrt((d * d).mean()) <= 2e-5 * scale, d.max() / scale
