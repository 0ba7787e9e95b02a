"""The group driver (k_group_rkf78: few sources, whole driver calls in one
launch) against the host-driven loop of the per-stage kernels, bit for bit:
states, time line, step counts and the last evaluation.

Shapes where the division of work changes: no body but the sources, one and
five others (a partly filled CTA), 4 to 128 others a CTA (the chunk doubles
where the CTAs would outnumber the SMs), up to the 32 sources it takes, super-
planetesimals among them, and the limit of one lane a component (four lanes an
item, all items at once) against one lane an item.  One system has a body next
to the origin (|d|^2 below 2^-600: the fast square root hands over)."""
import numpy as np
import pytest

from solaris_gb300 import abi, engine, scenarios

pytestmark = pytest.mark.gpu


def _system(n_massive, n_spl, n_light, seed, coincide=False):
    rng = np.random.default_rng(seed)
    G = abi.GAUSS2

    def phases(n, lo, hi):
        ang = rng.uniform(0, 2 * np.pi, (3, n))
        return scenarios.elements_to_phase(G * np.ones(n), rng.uniform(lo, hi, n), rng.uniform(0, 0.05, n),
                                           rng.uniform(0, 0.03, n), ang[0], ang[1], ang[2])

    groups = [scenarios._star()]
    if n_massive > 1:
        groups.append((abi.GIANT_PLANET, dict(mass=np.full(n_massive - 1, 1e-6), phase=phases(n_massive - 1, 1.0, 20.0))))
    if n_spl:
        groups.append((abi.SUPER_PLANETESIMAL, dict(mass=np.full(n_spl, 1e-9), phase=phases(n_spl, 1.0, 5.0))))
    if n_light:
        ph = phases(n_light, 1.0, 5.0)
        if coincide:  # next to the origin: |r|^2 ~ 1e-200
            ph[0, :3] *= 0.0
            ph[0, 0] = 1e-100
        groups.append((abi.TEST_PARTICLE, dict(mass=np.zeros(n_light), phase=ph)))
    return scenarios._assemble("group_shapes", groups)


@pytest.mark.parametrize("sizes", [(2, 0, 0), (4, 0, 1), (3, 0, 5), (3, 0, 253), (5, 0, 608), (5, 0, 609), (3, 0, 2500),
                                   (3, 0, 9729), (2, 0, 19456), (32, 0, 40), (9, 23, 300), (12, 0, 4000), (1, 3, 100)])
def test_group_driver_matches_the_host_loop(sizes):
    s = _system(*sizes, seed=4400 + sum(sizes))
    out = []
    for loop in (1, 0):
        with engine.Context(s) as ctx:
            ctx.set_device_loop(loop)
            ctx.set_state(s.y0)
            r = ctx.driver(abi.RUNGE_KUTTA_FEHLBERG78, 0.0, 5.0, 4)
            out.append((ctx.get_state(), (r["time"], r["h_next"], r["h_did"]), r["stats"], ctx.last_eval()))
    g, h = out
    assert np.array_equal(g[0].view(np.uint64), h[0].view(np.uint64))
    assert g[1] == h[1] and g[2] == h[2]
    for a, b in zip(g[3], h[3]):
        assert np.array_equal(np.asarray(a).view(np.uint8), np.asarray(b).view(np.uint8))


@pytest.mark.parametrize("sizes", [(3, 0, 20), (12, 0, 4000)])
def test_group_driver_hands_over_tiny_distances(sizes):
    s = _system(*sizes, seed=4500, coincide=True)
    out = []
    for loop in (1, 0):
        with engine.Context(s) as ctx:
            ctx.set_device_loop(loop)
            ctx.set_state(s.y0)
            r = ctx.driver(abi.RUNGE_KUTTA4, 0.0, 1e-3, 2)
            out.append((ctx.get_state(), r["stats"], ctx.last_eval()))
    assert np.array_equal(out[0][0].view(np.uint64), out[1][0].view(np.uint64))
    assert out[0][1] == out[1][1]
    for a, b in zip(out[0][2], out[1][2]):
        assert np.array_equal(np.asarray(a).view(np.uint8), np.asarray(b).view(np.uint8))
