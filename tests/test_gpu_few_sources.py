"""The two FP64 kernels of systems with fewer than 224 sources -- a thread a sink,
and tiles of 64 sources (k_gravity_ac_ref), by a rule on sources and sinks --
against the oracle, bit for bit: both sides of the rule's line, source counts
around whole tiles, one to many sinks a CTA, mixed source ranges, and gas terms
(to 1e-12: libm's powers)."""
import numpy as np
import pytest

import oracle
from solaris_gb300 import abi, engine, scenarios

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float64).view(np.uint64)


def _system(n_massive, n_spl, n_light, gas=None):
    rng = np.random.default_rng(7000 + 100 * n_massive + 10 * n_spl + n_light)

    def phases(n):
        ang = rng.uniform(0, 2 * np.pi, (3, n))
        return scenarios.elements_to_phase(abi.GAUSS2 * np.ones(n), rng.uniform(0.5, 5.0, n), rng.uniform(0, 0.1, n),
                                           rng.uniform(0, 0.05, n), ang[0], ang[1], ang[2])

    groups = [scenarios._star()]
    for kind, n, m in ((abi.PROTO_PLANET, n_massive - 1, 1e-8), (abi.SUPER_PLANETESIMAL, n_spl, 1e-9),
                       (abi.PLANETESIMAL, n_light, 1e-11)):
        if n:
            d = dict(mass=np.full(n, m), phase=phases(n))
            if gas and kind != abi.PROTO_PLANET:
                d.update(radius=np.full(n, 1e-8), density=np.full(n, 3.4e6), cd=np.ones(n))
            groups.append((kind, d))
    return scenarios._assemble("few_sources", groups, gas=gas)


@pytest.mark.parametrize("sizes", [(1, 0, 5), (2, 0, 0), (5, 0, 0), (6, 0, 30), (8, 0, 0), (8, 2, 3000), (33, 0, 0), (63, 0, 40),
                                   (64, 0, 0), (65, 0, 7), (20, 50, 400), (129, 0, 0), (180, 30, 2000), (223, 0, 0), (40, 0, 20000)])
def test_few_sources_bit_exact(sizes):
    s = _system(*sizes)
    o = oracle.Oracle(s)
    ref = o.compute(0.0, s.y0)
    rm3_o, nn_o, nd_o = o.last_eval()
    with engine.Context(s) as ctx:
        d, rm3, nn, nd = ctx.accel(0.0, s.y0)
    assert np.array_equal(bits(d), bits(ref))
    assert np.array_equal(bits(rm3), bits(rm3_o))
    assert np.array_equal(nn, nn_o) and np.array_equal(bits(nd), bits(nd_o))


def test_few_sources_with_gas():
    s = _system(40, 10, 300, gas=scenarios.default_gas())
    ref = oracle.Oracle(s).compute(0.0, s.y0).reshape(-1, 6)[1:, 3:]
    with engine.Context(s) as ctx:
        got = ctx.accel(0.0, s.y0)[0].reshape(-1, 6)[1:, 3:]
    assert (np.linalg.norm(got - ref, axis=1) <= 1e-12 * np.linalg.norm(ref, axis=1)).all()
