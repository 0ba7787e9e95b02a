"""k_gravity_ac_ref (the FP64 form of sinks with 224 sources or more) against
the oracle, bit for bit: source counts around whole tiles of 64, from two sinks a
CTA to ten and many CTAs an SM, sinks of different source ranges in one CTA
(Acceleration.cpp:285-289), a planar system (every z displacement zero), and
displacements whose x or y is exactly zero or far outside the integer multiply's
range (the IEEE path)."""
import numpy as np
import pytest

import oracle
from solaris_gb300 import abi, engine, scenarios

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float64).view(np.uint64)


def _check(s):
    o = oracle.Oracle(s)
    ref = o.compute(0.0, s.y0)
    rm3_o, nn_o, nd_o = o.last_eval()
    with engine.Context(s) as ctx:
        d, rm3, nn, nd = ctx.accel(0.0, s.y0)
    assert np.array_equal(bits(d), bits(ref))
    assert np.array_equal(bits(rm3), bits(rm3_o))
    assert np.array_equal(nn, nn_o) and np.array_equal(bits(nd), bits(nd_o))


@pytest.mark.parametrize("n", [224, 256, 257, 305, 1033, 1521, 1600, 3193])
def test_source_tiles_and_sinks_per_cta(n):
    _check(scenarios.config3(seed=900 + n, n=n))


def test_mixed_source_ranges():
    rng = np.random.default_rng(31)
    G = abi.GAUSS2

    def ph(k):
        return scenarios.elements_to_phase(G * np.ones(k), rng.uniform(0.5, 5, k), rng.uniform(0, 0.1, k),
                                           rng.uniform(0, 0.05, k), *rng.uniform(0, 2 * np.pi, (3, k)))

    groups = [scenarios._star(), (abi.GIANT_PLANET, dict(mass=[1e-3, 3e-4], phase=ph(2))),
              (abi.PROTO_PLANET, dict(mass=np.full(240, 1e-9), phase=ph(240))),
              (abi.SUPER_PLANETESIMAL, dict(mass=np.full(70, 1e-9), phase=ph(70))),
              (abi.PLANETESIMAL, dict(mass=np.full(90, 1e-11), phase=ph(90))),
              (abi.TEST_PARTICLE, dict(mass=np.zeros(61), phase=ph(61)))]
    _check(scenarios._assemble("ranges", groups))


def test_planar_and_degenerate_displacements():
    s = scenarios.config3(seed=77, n=700)
    y = s.y0.reshape(-1, 6)
    y[:, 2] = 0.0
    y[:, 5] = 0.0
    y[10, 0] = y[11, 0]            # x displacement exactly zero
    y[20:24, 1] = 0.0              # y displacements exactly zero, and pairs on an axis
    y[30, 1], y[31, 1] = 1e-140, -1e-150  # their y displacement squares to a subnormal
    s.mass[40] = 0.0               # a source without mass
    _check(s)
