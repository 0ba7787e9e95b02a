"""k_potential_pairs over chunks of source blocks: systems just above the
exact-order size, with odd and even block counts, ragged last blocks, and
enough blocks that a chunk holds several; against an accurately summed value
(each row's terms pairwise, the rows by math.fsum).  The bound is the 1e-13 of
the accurately summed value; a pair's 1/r is within about one ulp."""
import math

import numpy as np
import pytest

from solaris_gb300 import abi, engine, scenarios

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1025, 1152, 1281, 2047, 12801, 16511])
def test_potential_energy_of_chunked_blocks(n):
    s = scenarios.config3(seed=40 + n, n=n)
    with engine.Context(s) as ctx:
        got = ctx.integrals(s.y0)[14]
    p, m = s.y0.reshape(-1, 6)[:, :3], s.mass
    rows = []
    for i in range(n - 1):
        d = p[i + 1:] - p[i]
        rows.append(m[i] * np.sum(m[i + 1:] / np.sqrt(np.einsum("ij,ij->i", d, d))))
    want = math.fsum(rows) * abi.GAUSS2
    assert abs(got - want) <= 1e-13 * abs(want)
