"""Hidden units of the mixed network over the whole range of their argument.

One hidden layer whose units but the first have no output weight, and inputs that the first unit
does not see (an isolated atom has no descriptors), so an atom's energy is silu(z) of the bias z:
16 species, 16 values of z per call.  The bound is the arithmetic's: exp within 2 ulp, the sum, the
reciprocal and two products each within one rounding, 8 * 2^-24 in all; a sigmoid below 2^-126 may
be zero, which leaves 2e-36.
Pairs of atoms give silu'(z) through the force, to the mixed path's 1e-4 of the largest; far below
zero it vanishes."""
import numpy as np
import pytest

from jse_gb300 import workloads as W

pytestmark = pytest.mark.gpu
T = 16


def _potential(z, slope):
    from jse_gb300.nnap import NNAP
    model = W.write_model(["S%d" % t for t in range(T)], {"type": "chebyshev", "nmax": 3, "rcut": 5.0, "wtype": "none"}, [16], 1)
    for m, b in zip(model["models"], z):
        nn = m["nn"]
        nn["hidden_weights"] = [(slope * np.eye(16, 4, dtype=float)).tolist()]
        nn["hidden_biases"] = [[float(b)] + [0.0] * 15]
        nn["output_weight"] = [1.0] + [0.0] * 15
        nn["output_bias"] = 0.0
    return NNAP(model, precision="mixed")


def _silu(z):
    z = np.asarray(z, dtype=np.float32).astype(np.float64)
    s = np.exp(np.where(z < 0, z, 0.0)) / (np.exp(-np.abs(z)) + 1.0)  # of either sign without overflow
    return z * s, s * (1.0 + z * (1.0 - s))


@pytest.mark.parametrize("z", [
    [0.0, 1e-3, -1e-3, 0.4, -0.4, 1.3, -1.3, 4.7, -4.7, 11.0, -11.0, 20.0, -20.0, 43.0, -43.0, 1e-30],
    [60.0, -60.0, 80.0, -80.0, 86.9, -86.9, -87.2, -87.29, -87.31, -87.4, -88.0, -88.6, -88.8, -89.5, -104.0, 104.0],
    [-150.0, 150.0, -1e3, 1e3, -1e5, 1e5, -1e10, 1e10, -1e20, 1e20, -1e30, 1e30, -3e37, 3e37, -3e38, 3e38]])
def test_silu_of_the_bias(z):
    far = 40.0 * np.arange(T)
    s = W.Structure(np.stack([far, far * 0 + 1.0, far * 0 + 1.0], 1), np.arange(1, T + 1, dtype=np.int32),
                    np.diag([40.0 * T, 40.0, 40.0]), 0)
    with _potential(z, 0.0) as p:
        e = np.asarray(p.calEnergies(s))
    want = _silu(z)[0]
    assert (np.abs(e - want) <= 8 * 2.0 ** -24 * np.abs(want) + 2e-36).all(), (z, e, want)


def test_slope_far_from_zero():
    z = [0.0, 0.5, -0.5, 3.0, -3.0, 15.0, -15.0, 87.0, -87.0, -88.0, -95.0, -1e4, -1e20, -1e30, -1e37, -3e38]
    pairs = [W.Structure(np.array([[1.0, 1.0, 1.0], [3.1, 1.0, 1.0]]), np.full(2, t + 1, dtype=np.int32),
                         np.diag([40.0, 40.0, 40.0]), 0) for t in range(T)]
    with _potential(z, 1e-4) as p:
        f = np.array([o["forces"][0, 0] for o in p.calEnergyForceVirialsBatch(pairs)])
    want = _silu(z)[1] / _silu([0.0])[1]
    assert np.abs(f - f[0] * want).max() <= 1e-3 * abs(f[0])  # the inputs move z by up to 1e-3
    assert (np.abs(f[9:]) <= 1e-30).all(), f
