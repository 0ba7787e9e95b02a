"""The gas model's powers and exponential (sol_powlaw.cuh: fixed point, each
within 0.6 ulp) through the drag of planetesimals, against the oracle's libm
over the range of the indices and radii: positive, negative, zero and whole
exponents, 0.05 to 60 AU, bodies up to four scale heights off the midplane.

Tolerance, of a body's acceleration: (z / h)^2 <= 16 carries two powers of h
(0.6 ulp here, 0.5 in libm) and three roundings, 16 x 8e-16 = 1.3e-14 in the
exponential's argument; the other powers and products add 2e-15."""
import numpy as np
import pytest

import oracle
from solaris_gb300 import abi, engine, scenarios

pytestmark = pytest.mark.gpu

RTOL = 2e-14


@pytest.mark.parametrize("h_index,rho_index,eta_index,path_index", [
    (1.0, -2.5, 0.5, 2.75), (1.25, -2.75, 0.5, 2.75), (0.0, 0.0, 0.0, 0.0), (0.75, 1.0, -0.5, -1.0), (1.0, -3.0, 1.0, 1.5)])
def test_drag_over_indices_and_radii(h_index, rho_index, eta_index, path_index):
    s = scenarios.config2(seed=61, n_pl=700)
    rng = np.random.default_rng(62)
    g = s.gas
    g["scale_height"] = (g["scale_height"][0], h_index)
    g["density"] = (g["density"][0], rho_index)
    g["eta"] = (1.0e-3 * 0.5, eta_index)
    g["mean_free_path"] = (g["mean_free_path"][0], path_index)
    y = s.y0.reshape(-1, 6)
    r = np.exp(rng.uniform(np.log(0.05), np.log(60.0), 700))
    ph = rng.uniform(0, 2 * np.pi, 700)
    h = g["scale_height"][0] * r ** h_index
    y[3:, 0], y[3:, 1] = r * np.cos(ph), r * np.sin(ph)
    y[3:, 2] = rng.uniform(-4, 4, 700) * np.minimum(h, 0.2 * r)
    v = np.sqrt(abi.GAUSS2 / r)
    y[3:, 3], y[3:, 4], y[3:, 5] = -v * np.sin(ph), v * np.cos(ph), 0.02 * v
    ref = oracle.Oracle(s).compute(0.0, s.y0).reshape(-1, 6)[:, 3:]
    with engine.Context(s) as ctx:
        got = ctx.accel(0.0, s.y0)[0].reshape(-1, 6)[:, 3:]
    err = np.linalg.norm(got - ref, axis=1)[1:] / np.linalg.norm(ref, axis=1)[1:]
    assert np.isfinite(got).all() and err.max() <= RTOL, f"{err.max():.3e} at body {int(err.argmax()) + 1}"
