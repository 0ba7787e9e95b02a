"""RK4 driver calls of the group driver: the blocks' final exchange, after which the
start state may be overwritten.  A block that never arrives makes the others
give up after a short spin limit, with the state as it was before; the same
context then integrates bit for bit like a fresh one.  Migration's state and
buffers, written at the launch's end, equal the host loop's after launches of
one, two and five calls."""
import numpy as np
import pytest

from solaris_gb300 import abi, engine, scenarios

pytestmark = pytest.mark.gpu

RK4 = abi.RUNGE_KUTTA4


@pytest.mark.parametrize("absent", [0, 1, 63])
def test_rk4_gives_up_when_a_block_never_arrives(absent):
    s = scenarios.config1()  # 253 test particles: 64 blocks
    with engine.Context(s) as ctx, engine.Context(s) as fresh:
        ctx.set_state(s.y0)
        ctx.set_wait_test(4096, absent)
        with pytest.raises(abi.SolError) as err:
            ctx.driver(RK4, 0.0, s.h0, 3)
        assert err.value.code == abi.SOL_ERR_TIMEOUT
        ctx.set_wait_test(0, -1)
        assert np.array_equal(ctx.get_state().view(np.uint64), s.y0.view(np.uint64))
        ctx.set_state(s.y0)
        fresh.set_state(s.y0)
        r1, r2 = (c.driver(RK4, 0.0, s.h0, 7) for c in (ctx, fresh))
        assert r1["stats"] == r2["stats"] and (r1["time"], r1["h_next"]) == (r2["time"], r2["h_next"])
        assert np.array_equal(ctx.get_state().view(np.uint64), fresh.get_state().view(np.uint64))


@pytest.mark.parametrize("integrator", [RK4, abi.RUNGE_KUTTA_FEHLBERG78])
def test_migration_state_after_each_launch(integrator):
    s = scenarios.config2(seed=9, n_pl=700)
    y = s.y0.reshape(-1, 6)
    s.mig_type[1:3] = (abi.MIGRATION_TYPE_II, abi.MIGRATION_TYPE_II)
    s.mig_stop_at[1:3] = (0.5, 1.001 * np.linalg.norm(y[2, :3]))  # one goes on, one has arrived
    out = []
    for loop in (1, 0):
        with engine.Context(s) as ctx:
            ctx.set_device_loop(loop)
            ctx.set_state(s.y0)
            got = []
            t, h = 0.0, s.h0
            for calls in (1, 2, 5):
                r = ctx.driver(integrator, t, h, calls)
                t, h = r["time"], r["h_next"]
                got.append((ctx.get_state().copy(), t, h, r["stats"], ctx.mig_type().copy()))
            out.append(got)
    for g, w in zip(*out):
        assert np.array_equal(g[0].view(np.uint64), w[0].view(np.uint64))
        assert g[1:4] == w[1:4]
        assert np.array_equal(g[4], w[4])
    assert out[0][0][4][1] == abi.MIGRATION_TYPE_II and out[0][0][4][2] == abi.MIGRATION_NO
