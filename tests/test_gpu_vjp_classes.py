"""The vector-Jacobian product (sol_adjoint.cu) over every pairing of body
classes -- massive bodies see the super-planetesimals, lighter ones do not, light
ones attract nothing -- sizes around the blocks of 32 bodies and where the form
over block pairs begins (448 bodies), against the oracle's tangent-linear model.
Bound: as the adjoint's other tests, 1e-6 of the directional derivative."""
import numpy as np
import pytest

import oracle
from solaris_gb300 import abi, engine, scenarios

pytestmark = pytest.mark.gpu


def _system(n_massive, n_spl, n_pl, n_tp):
    rng = np.random.default_rng(900 + n_massive + 10 * n_spl + 100 * n_pl)

    def phases(n):
        ang = rng.uniform(0, 2 * np.pi, (3, n))
        return scenarios.elements_to_phase(abi.GAUSS2 * np.ones(n), rng.uniform(0.8, 4.0, n), rng.uniform(0, 0.1, n),
                                           rng.uniform(0, 0.05, n), ang[0], ang[1], ang[2])

    groups = [scenarios._star()]
    for kind, n, m in ((abi.PROTO_PLANET, n_massive, 1e-5), (abi.SUPER_PLANETESIMAL, n_spl, 1e-6),
                       (abi.PLANETESIMAL, n_pl, 1e-7), (abi.TEST_PARTICLE, n_tp, 0.0)):
        if n:
            groups.append((kind, dict(mass=np.full(n, m), phase=phases(n))))
    s = scenarios._assemble("vjp_classes", groups)
    s.h0 = scenarios._shortest_period(s) / 200.0
    return s


@pytest.mark.parametrize("sizes", [(1, 0, 0, 0), (5, 3, 4, 2), (31, 0, 0, 0), (32, 0, 0, 0), (33, 7, 0, 30), (20, 11, 1, 1),
                                   (60, 5, 64, 3), (127, 0, 0, 0), (1, 0, 130, 0),
                                   (446, 0, 0, 0), (447, 0, 0, 0), (448, 0, 0, 0), (511, 0, 0, 0), (300, 40, 150, 30),
                                   (31, 480, 0, 0), (3, 9, 500, 0), (40, 24, 0, 455)])
def test_adjoint_of_mixed_classes_matches_the_tangent_linear_model(sizes):
    s = _system(*sizes)
    h, n_steps, every = s.h0, 3, 2
    rng = np.random.default_rng(12)
    with engine.Context(s) as ctx:
        y = ctx.adjoint_forward(s.y0, h, n_steps, every)
        g = rng.standard_normal(6 * s.n)
        g[:6] = 0.0
        dy0, dmass = ctx.adjoint_backward(g)
    o = oracle.Oracle(s)
    # directions near the cotangent's own sensitivity, so that the derivative does not vanish by chance
    for scale in (1.0, 0.0):
        dy = scale * dy0 / np.linalg.norm(dy0)
        dy[:6] = 0.0
        dm = dmass * (s.mass > 0) * (1.0 / np.linalg.norm(dmass[s.mass > 0]) if np.any(dmass[s.mass > 0]) else 0.0)
        _, dyf = o.rkf78_fixed(s.y0, h, n_steps, dy, dm)
        tlm = float(g @ dyf)
        adj = float(dy0 @ dy + dmass @ dm)
        assert abs(adj - tlm) <= 1e-6 * abs(tlm), (adj, tlm)
