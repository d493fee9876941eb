"""Kernels at the sizes where their work split changes, against the FP64 oracle.

Backward descriptors: 32 lanes per atom below 4096 atoms and 16 from there (where two atoms' G
fits), one- and several-species fuse matrices, more than three species (the sparse fuse
tables), rows of fewer entries than a lane group, of whole groups and of one more.

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
