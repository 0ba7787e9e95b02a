"""The ensemble's stage sums and pair squares with their multiplications on
the integer pipe, bit for bit against the oracle: the default launch shapes of
one system, of a few and of more systems than SMs, and bodies whose position
or velocity components are zero or far outside the integer multiply's range
(the FP64 path of an element or a pair)."""
import numpy as np
import pytest

import oracle
from solaris_gb300 import abi, engine, scenarios

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 5, 310, 800, 1600])
def test_default_shapes_and_out_of_range_components(count):
    base = [scenarios.config1(seed=60 + k, n_tp=k) for k in (0, 1, 29, 125, 253)]
    for s in base[2:]:  # planar and nearly planar bodies, and components that square to subnormals
        y = s.y0.reshape(-1, 6)
        y[5, 2] = y[5, 5] = 0.0
        y[6, 1], y[6, 4] = 1e-160, 0.0
        y[7, 2], y[7, 5] = -1e-200, 1e-300
    systems = [base[k % len(base)] for k in range(count)]
    with engine.Ensemble(systems) as ens:
        ens.set_state([s.y0 for s in systems], [0.0] * count, [200.0 * s.h0 for s in systems])
        ens.advance(3)
        ys, lines, status = ens.get_state()
    want = {}
    for k, s in enumerate(base[:min(count, len(base))]):
        want[k] = oracle.Oracle(s).driver(abi.RUNGE_KUTTA_FEHLBERG78, s.y0, 0.0, 200.0 * s.h0, 3)
    for k in range(count):
        r = want[k % len(base)]
        assert status[k] == 0
        assert np.array_equal(ys[k].view(np.uint64), np.ascontiguousarray(r["y0"]).view(np.uint64)), f"system {k}"
        assert lines[k] == tuple(r["tl"])
