"""Launch shapes of an ensemble: the largest number of threads a system that the
kernel can be launched with is accepted and runs, a larger one is refused when it
is set, in both precisions."""
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
