"""Launch shapes of an ensemble: the largest number of threads a system that the
kernel can be launched with is accepted and runs, a larger one is refused when it
is set, in both precisions."""
import time

import numpy as np
import pytest

from solaris_gb300 import abi, engine, scenarios

pytestmark = pytest.mark.gpu

LARGEST = 736


@pytest.mark.parametrize("precision", [abi.PRECISION_FP64, abi.PRECISION_SPLIT_FF])
def test_every_accepted_shape_runs(precision):
    systems = [scenarios.config1(seed=90 + k, n_tp=20 * k) for k in range(6)]

    def final(shape):
        with engine.Ensemble(systems, precision=precision) as ens:
            ens.configure(*shape)
            ens.set_state([s.y0 for s in systems], [0.0] * 6, [200.0 * s.h0 for s in systems])
            ens.advance(2)
            ys, lines, _ = ens.get_state()
        return np.concatenate(ys).view(np.uint64), lines

    want = final((128, 4))
    for shape in ((32, 1), (672, 1), (704, 2), (LARGEST, 1), (LARGEST, 32)):
        y, lines = final(shape)
        assert np.array_equal(y, want[0]) and lines == want[1], shape


@pytest.mark.parametrize("threads", [LARGEST + 32, 1024])
def test_larger_shapes_are_refused(threads):
    systems = [scenarios.config1(seed=97, n_tp=9)]
    with engine.Ensemble(systems) as ens:
        with pytest.raises(abi.SolError) as err:
            ens.configure(threads, 1)
        assert err.value.code == abi.SOL_ERR_ARG and str(LARGEST) in str(err.value)
        ens.set_state([systems[0].y0], [0.0], [systems[0].h0])
        ens.advance(1)  # with the shape it had


def test_the_tuned_shape_is_not_slower_than_the_default():
    """300 systems, about two an SM: the default shape is ~30 % faster than the
    twelve of other sizes, so a tuner that does not try it is found out."""
    rng = np.random.default_rng(9)
    systems = [scenarios.config4_system(rng, k) for k in range(300)]
    ms = {}
    for tuned in (False, True):
        with engine.Ensemble(systems) as ens:
            ens.set_state([s.y0 for s in systems], [0.0] * 300, [s.h0 for s in systems])
            before = ens.get_state()
            if tuned:
                ens.autotune(steps=1)
                after = ens.get_state()
                assert np.array_equal(np.concatenate(before[0]).view(np.uint64), np.concatenate(after[0]).view(np.uint64))
                assert before[1] == after[1]
            best = np.inf
            for _ in range(6):
                ens.set_state([s.y0 for s in systems], [0.0] * 300, [s.h0 for s in systems])
                t = time.perf_counter()
                ens.advance(1)
                best = min(best, time.perf_counter() - t)
            ms[tuned] = 1e3 * best
    assert ms[True] <= 1.15 * ms[False], ms
