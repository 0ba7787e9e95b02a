"""The float-float form over block pairs holds its partial sums compensated: what
is far below the last place of a running sum is not lost when the sum later
cancels.

A sink at x = 0 has a large mass 1 AU to its right and the same 1 AU to its left,
whose pulls along x are exact opposites, and small ones between the two in the
order of summation; every other body has no mass.  So the sink's acceleration
along x is that of the small masses (and their indirect terms).  Placed such
that the large ones meet in k_combine (block pairs' partials of a sink, and of a
source), in a sink's FP64 sums of one chunk, in a source's sums of the four warps,
and, with a small mass of 2^-40, in the two lanes that a source's sums are folded
from.

Bound: the small pulls are 2^-54 of a large one each.  Two of them against the
rounding of the indirect sums (a few 2^-53 of 2^-18 of a large pull, at 64 AU
from the star) are 2^-53 to ~2^-69: 3e-5.  The lanes' sum rounds to 2^-53 of the
large pull, 2^-13 of the small one: 1.3e-4.  4e-4 for all."""
import math

import numpy as np
import pytest

from solaris_gb300 import abi, engine, scenarios

pytestmark = pytest.mark.gpu

RTOL = 4e-4
BIG = 0.001005617
S = 2.0 ** -54


def _system(n, sink, bodies):
    """bodies: (index, distance to the right of the sink, mass)"""
    rng = np.random.default_rng(n + sink)
    ang = rng.uniform(0, 2 * np.pi, n)
    y = np.zeros((n, 6))
    y[:, 0], y[:, 1], y[:, 2] = 30.0 * np.cos(ang), 30.0 * np.sin(ang), rng.uniform(-20.0, 20.0, n)
    m = np.zeros(n)
    y[0], m[0] = 0.0, 1.0
    y[sink, :3] = (0.0, 64.0, 0.0)
    for i, x, mass in bodies:
        y[i, :3] = (x, 64.0, 0.0)
        m[i] = mass
    return scenarios._assemble("sums", [scenarios._star(), (abi.PROTO_PLANET, dict(mass=m[1:], phase=y[1:]))])


@pytest.mark.parametrize("n, sink, bodies", [
    # partials 4 to 7 of a sink's chunks (one warp of k_combine), blocks of 64
    (1500, 5, [(64 * 4 + 7, 1.0, BIG), (64 * 5 + 9, 2.0, 4 * S * BIG), (64 * 6 + 40, 4.0, 16 * S * BIG),
               (64 * 7 + 1, -1.0, BIG)]),
    # the same with a small one first, far below the next
    (1500, 5, [(64 * 4 + 9, 2.0, 4 * S * BIG), (64 * 5 + 7, 1.0, BIG), (64 * 6 + 40, 4.0, 16 * S * BIG),
               (64 * 7 + 1, -1.0, BIG)]),
    # partials 8 to 11 of a source
    (1500, 64 * 20 + 3, [(64 * 8 + 7, 1.0, BIG), (64 * 9 + 9, 2.0, 4 * S * BIG), (64 * 10 + 40, 4.0, 16 * S * BIG),
                         (64 * 11 + 1, -1.0, BIG)]),
    # the four folds of a chunk of two blocks of 256 sources
    (49409, 5, [(256 * 6 + 10, 1.0, BIG), (256 * 6 + 130, 2.0, 4 * S * BIG), (256 * 7 + 10, 4.0, 16 * S * BIG),
                (256 * 7 + 130, -1.0, BIG)]),
    # the four warps of a block of 256 sinks, in the order they reach a source
    (20225, 256 * 9 + 20, [(256 * 4 + 3, 1.0, BIG), (256 * 4 + 195, 2.0, 4 * S * BIG),
                           (256 * 4 + 131, 4.0, 16 * S * BIG), (256 * 4 + 67, -1.0, BIG)]),
    # both lanes of a warp's sinks: bodies l and l + 32 of a block of 64
    (1500, 64 * 20 + 3, [(64 * 8 + 7, 1.0, BIG), (64 * 8 + 40, 2.0, 4 * BIG * 2.0 ** -40), (64 * 9 + 1, -1.0, BIG)]),
])
def test_small_pulls_survive_large_ones_that_cancel(n, sink, bodies):
    s = _system(n, sink, bodies)
    with engine.Context(s, precision=abi.PRECISION_SPLIT_FF) as ctx:
        got = ctx.accel(0.0, s.y0)[0].reshape(-1, 6)[sink, 3]
    terms = []
    for i, x, mass in bodies:
        gm = abi.GAUSS2 * mass
        terms += [gm * x / abs(x) ** 3, -gm * x / math.hypot(x, 64.0) ** 3]
    want = math.fsum(terms)
    assert abs(got - want) <= RTOL * abs(want), (got, want)
