"""The stage's input formed in the evaluation's first kernel (k_stage_prepass, 32
bodies a block; FP64, up to 16,384 bodies) against the oracle, bit for bit: RKF78
and RK4 driver calls of systems outside the group driver (more than 32 sources)
around whole blocks, a padded last block, and beyond the rule's end."""
import numpy as np
import pytest

import oracle
from solaris_gb300 import abi, engine, scenarios

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float64).view(np.uint64)


@pytest.mark.parametrize("n", [33, 63, 64, 65, 97, 255, 257])
@pytest.mark.parametrize("integrator", [abi.RUNGE_KUTTA_FEHLBERG78, abi.RUNGE_KUTTA4])
def test_driver_calls_match_the_oracle(n, integrator):
    s = scenarios.config3(seed=300 + n, n=n)
    ref = oracle.Oracle(s).driver(integrator, s.y0, 0.0, 100.0 * s.h0, 2)
    with engine.Context(s) as ctx:
        ctx.set_state(s.y0)
        r = ctx.driver(integrator, 0.0, 100.0 * s.h0, 2)
        y = ctx.get_state()
    assert np.array_equal(bits(y), bits(ref["y0"]))
    assert (r["time"], r["h_next"]) == ref["tl"][:2]


def test_both_sides_of_the_size_rule():
    """One RK4 call either side of 16,384 bodies, few of them massive (33), against
    the oracle."""
    rng = np.random.default_rng(5)
    for n in (16384, 16385):
        ang = rng.uniform(0, 2 * np.pi, (3, n - 1))
        ph = scenarios.elements_to_phase(abi.GAUSS2 * np.ones(n - 1), rng.uniform(0.5, 5.0, n - 1),
                                         rng.uniform(0, 0.05, n - 1), rng.uniform(0, 0.03, n - 1), *ang)
        s = scenarios._assemble("stage", [scenarios._star(), (abi.PROTO_PLANET, dict(mass=np.full(33, 1e-9), phase=ph[:33])),
                                          (abi.TEST_PARTICLE, dict(mass=np.zeros(n - 34), phase=ph[33:]))])
        ref = oracle.Oracle(s).driver(abi.RUNGE_KUTTA4, s.y0, 0.0, 1.0, 1)
        with engine.Context(s) as ctx:
            ctx.set_state(s.y0)
            ctx.driver(abi.RUNGE_KUTTA4, 0.0, 1.0, 1)
            assert np.array_equal(bits(ctx.get_state()), bits(ref["y0"]))
