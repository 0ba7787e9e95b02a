"""Host-buffer evaluations on both sides of the sizes at which dydt, and rm3 with the
neighbours, stop coming back through the pinned buffer: every combination of
outputs gives what the device holds.  And a large system's rm3 and neighbours
cost their copies, not a second pass over them on the host: with all outputs
400,000 light bodies take 1.3 times the call without them (2.6 times with that
pass)."""
import itertools
import time

import numpy as np
import pytest

from solaris_gb300 import abi, engine, scenarios

pytestmark = pytest.mark.gpu


def _call(ctx, y, want):
    d = np.full(6 * ctx.n, np.nan)
    rm3, nn, nd = np.full(ctx.n, np.nan), np.full(ctx.n, -7, np.int32), np.full(ctx.n, np.nan)
    abi.check(ctx.lib, ctx.lib.sol_accel_compute(ctx.h, 0.0, abi.f64p(y), abi.f64p(d), abi.f64p(rm3) if want[0] else None,
                                                 abi.i32p(nn) if want[1] else None, abi.f64p(nd) if want[2] else None))
    return d, rm3, nn, nd


@pytest.mark.parametrize("n", [3, 1194, 1195, 19500, 19700])
def test_every_combination_of_outputs(n):
    s = scenarios.config1(seed=17, n_tp=n - 3)
    other = scenarios.config1(seed=18, n_tp=n - 3)
    with engine.Context(s) as ctx:
        full = _call(ctx, s.y0, (1, 1, 1))
        held = ctx.last_eval()
        assert not np.isnan(full[0]).any()
        for a, b in zip(full[1:], held):
            assert np.array_equal(np.asarray(a).view(np.uint8), np.asarray(b).view(np.uint8))
        for want in itertools.product((0, 1), repeat=3):
            _call(ctx, other.y0, (1, 1, 1))
            got = _call(ctx, s.y0, want)
            assert np.array_equal(got[0].view(np.uint64), full[0].view(np.uint64))
            for k in range(3):
                if want[k]:
                    assert np.array_equal(got[1 + k].view(np.uint8), full[1 + k].view(np.uint8))


def test_large_outputs_are_copied_once():
    s = scenarios.config1(seed=19, n_tp=400000 - 3)
    with engine.Context(s) as ctx:
        d = np.zeros(6 * ctx.n)
        rm3, nn, nd = np.zeros(ctx.n), np.zeros(ctx.n, np.int32), np.zeros(ctx.n)

        def best(*outs):
            t = []
            for _ in range(20):
                t0 = time.perf_counter()
                abi.check(ctx.lib, ctx.lib.sol_accel_compute(ctx.h, 0.0, abi.f64p(s.y0), abi.f64p(d), *outs))
                t.append(time.perf_counter() - t0)
            return min(t)

        alone, all_outputs = best(None, None, None), best(abi.f64p(rm3), abi.i32p(nn), abi.f64p(nd))
    assert all_outputs <= 1.8 * alone, (all_outputs, alone)
