"""Nearest neighbours of very close pairs in the float-float form over block
pairs (k_pairs_sym), against the reference (FP64) form: index and distance are
equal, bit for bit.

Pairs from 2e-9 down to 1e-12 AU in a disk of 5 AU, inside a block, in
neighbouring blocks, in the first and the last one, and on either side of the
whole blocks where light bodies follow; and pairs of 1e-6 and 1e-7 AU beside one
body at 10,000 AU, which sets the grid of the float table.  Blocks of 64, 128
and 256 bodies."""
import numpy as np
import pytest

from solaris_gb300 import abi, engine, scenarios

pytestmark = pytest.mark.gpu

SPLIT_RTOL = 1e-12


def _plant(s, pairs):
    y = s.y0.reshape(-1, 6)
    for k, (a, b, sep) in enumerate(pairs):
        y[b] = y[a]
        u = np.array([[0.6, -0.48, 0.64], [-0.8, 0.6, 0.0], [0.0, 0.0, 1.0]])[k % 3]
        y[b, :3] += sep * u
    return s


def _light(n_massive, n_light):
    s = scenarios.config3(seed=311, n=n_massive)
    groups = [scenarios._star(), (abi.PROTO_PLANET, dict(mass=s.mass[1:], phase=s.y0.reshape(-1, 6)[1:])),
              (abi.TEST_PARTICLE, dict(mass=np.zeros(n_light), phase=1.01 * s.y0.reshape(-1, 6)[1:1 + n_light]))]
    return scenarios._assemble("close_neighbours", groups)


def _check(s, pairs):
    with engine.Context(s, precision=abi.PRECISION_FP64) as ctx:
        d64, _, nn64, nd64 = ctx.accel(0.0, s.y0)
        ctx.set_precision(abi.PRECISION_SPLIT_FF)
        dff, _, nn, nd = ctx.accel(0.0, s.y0)
    for a, b, sep in pairs:
        assert nn64[a] == b and nn64[b] == a, (a, b, sep)
    assert np.array_equal(nn, nn64)
    assert np.array_equal(nd.view(np.uint64), nd64.view(np.uint64))
    a, r = dff.reshape(-1, 6)[1:, 3:], d64.reshape(-1, 6)[1:, 3:]
    assert (np.linalg.norm(a - r, axis=1) / np.linalg.norm(r, axis=1)).max() <= SPLIT_RTOL


@pytest.mark.parametrize("sep", [2e-9, 1e-9, 1e-10, 1e-12])
@pytest.mark.parametrize("n, light", [(1500, 0), (11137, 0), (20225, 0), (7424, 900)])
def test_close_pairs(n, light, sep):
    s = _light(n, light) if light else scenarios.config3(seed=310, n=n)
    last = n - n % 256
    pairs = [(10, 11, sep), (63, 64, sep), (100, 163, sep), (255, 256, sep), (1, last - 3, sep), (400, n - 1, sep),
             (700, 1000, 3 * sep)]
    if light:
        pairs += [(900, n + 5, sep)]  # a light body beside a massive one
        s = _plant(s, pairs)
        with engine.Context(s, precision=abi.PRECISION_FP64) as ctx:
            nn64, nd64 = ctx.accel(0.0, s.y0)[2:]
            ctx.set_precision(abi.PRECISION_SPLIT_FF)
            nn, nd = ctx.accel(0.0, s.y0)[2:]
        assert nn64[n + 5] == 900
        assert np.array_equal(nn, nn64)
        assert np.array_equal(nd.view(np.uint64), nd64.view(np.uint64))
    else:
        _check(_plant(s, pairs), pairs)


@pytest.mark.parametrize("sep", [1e-6, 1e-7])
@pytest.mark.parametrize("n", [2049, 12300, 20480])
def test_close_pairs_beside_a_far_body(n, sep):
    s = scenarios.config3(seed=312, n=n)
    y = s.y0.reshape(-1, 6)
    y[n // 2, :3] *= 1.0e4 / np.linalg.norm(y[n // 2, :3])
    y[n // 2, 3:] *= 0.01
    pairs = [(10, 11, sep), (70, 200, sep), (255, 256, sep), (1, n - 300, sep), (400, n - 1, sep), (600, 610, 2 * sep),
             (1200, 1400, 3 * sep)]
    _check(_plant(s, pairs), pairs)
