"""The backward pass begins with the stage states that the forward pass kept of
its last segment, and recomputes the other segments: a second backward pass,
which has to recompute the last one too, gives the same bits -- segments of one
step, a last one that is shorter, one segment that is all, and one longer than
the run.  New masses or another precision between the passes count from the
checkpoints on, whatever was kept."""
import numpy as np
import pytest

from solaris_gb300 import abi, engine, scenarios

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float64).view(np.uint64)


def _case(n_pl=30):
    s = scenarios.config5(seed=71, n_pl=n_pl)
    g = np.random.default_rng(72).standard_normal(6 * s.n)
    g[:6] = 0.0
    return s, g


@pytest.mark.parametrize("n_steps,every", [(4, 1), (5, 5), (5, 7), (7, 3), (6, 3)])
def test_kept_stages_are_the_recomputed_ones(n_steps, every):
    s, g = _case()
    with engine.Context(s) as ctx:
        ctx.adjoint_forward(s.y0, 500 * s.h0, n_steps, every)
        a = ctx.adjoint_backward(g)
        ctx.accel(0.0, s.y0)  # uses the context's other buffers
        b = ctx.adjoint_backward(g)
        c = ctx.adjoint_backward(g)
    for x, y in ((a, b), (a, c)):
        assert np.array_equal(bits(x[0]), bits(y[0])) and np.array_equal(bits(x[1]), bits(y[1]))


@pytest.mark.parametrize("change", ["masses", "precision"])
def test_a_change_between_the_passes_drops_the_kept_stages(change):
    s, g = _case()
    out = []
    for first in (False, True):
        with engine.Context(s) as ctx:
            ctx.adjoint_forward(s.y0, 500 * s.h0, 7, 3)
            if first:
                ctx.adjoint_backward(g)  # leaves the first segment's stage states
            if change == "masses":
                ctx.set_masses(s.mass * 1.25)
            else:
                ctx.set_precision(abi.PRECISION_SPLIT)
            out.append(ctx.adjoint_backward(g))
    assert np.array_equal(bits(out[0][0]), bits(out[1][0])) and np.array_equal(bits(out[0][1]), bits(out[1][1]))
    if change == "masses":  # (another precision need not change a bit of so small a system's gradient)
        with engine.Context(s) as ctx:
            ctx.adjoint_forward(s.y0, 500 * s.h0, 7, 3)
            assert not np.array_equal(bits(out[0][0]), bits(ctx.adjoint_backward(g)[0]))
