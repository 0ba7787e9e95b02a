"""Device memory of the split forms' partials: the block pairs' (SPLIT_FF, 0.67 GB at
65,536 bodies) are reserved for the systems and the precision that use them, and
where a buffer grows the results stay those of a fresh context.

Otherwise a body has 40 bytes for every 4,096 bodies (42 MB at 65,536); the bound is
three times that, for smaller chunks and an allocator's granularity."""
import numpy as np
import pytest

from solaris_gb300 import abi, engine, scenarios

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

MB = 1 << 20


def _disk(n, light=0):
    s = scenarios.config3(seed=410, n=n)
    if not light:
        return s
    y = s.y0.reshape(-1, 6)
    rows = 1 + np.arange(light) % (n - 1)
    ph = y[rows] * (1.1 + 0.1 * (np.arange(light) // (n - 1)))[:, None]
    return scenarios._assemble("disk_light", [scenarios._star(), (abi.PROTO_PLANET, dict(mass=s.mass[1:], phase=y[1:])),
                                              (abi.TEST_PARTICLE, dict(mass=np.zeros(light), phase=ph))])


def _taken(ctx, precision):
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    ctx.set_precision(precision)
    return before - torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("n, light, precision, reserved", [
    (65536, 0, abi.PRECISION_SPLIT, False),
    (65536, 0, abi.PRECISION_SPLIT_FF, True),
    (7000, 60000, abi.PRECISION_SPLIT_FF, False),   # too few massive bodies for block pairs
    (131500, 0, abi.PRECISION_SPLIT_FF, False),     # too many
])
def test_block_pairs_are_reserved_where_they_are_used(n, light, precision, reserved):
    with engine.Context(_disk(n, light)) as ctx:
        taken = _taken(ctx, precision)
        if reserved:
            assert 600 * MB < taken < 900 * MB
        else:
            assert taken < 3 * 40 * (n + light) * -(-(n + light) // 4096)


def test_a_growing_buffer_gives_the_bits_of_a_fresh_context():
    """SPLIT, SPLIT_FF and SPLIT again with captured driver graphs in between."""
    s = _disk(20000)

    def run(ctx, precision):
        ctx.set_precision(precision)
        ctx.set_state(s.y0)
        r = ctx.driver(abi.RUNGE_KUTTA_FEHLBERG78, 0.0, 100.0 * s.h0, 2)
        return ctx.get_state().view(np.uint64), r["time"], r["h_next"]

    want = {}
    for p in (abi.PRECISION_SPLIT, abi.PRECISION_SPLIT_FF):
        with engine.Context(s) as ctx:
            want[p] = run(ctx, p)
    with engine.Context(s) as ctx:
        for p in (abi.PRECISION_SPLIT, abi.PRECISION_SPLIT_FF, abi.PRECISION_SPLIT, abi.PRECISION_SPLIT_FF):
            y, t, h = run(ctx, p)
            assert np.array_equal(y, want[p][0]) and (t, h) == want[p][1:]
        # the precision set to and fro without a run between
        ctx.set_precision(abi.PRECISION_SPLIT)
    with engine.Context(s) as ctx:
        run(ctx, abi.PRECISION_SPLIT)
        ctx.set_precision(abi.PRECISION_SPLIT_FF)
        y, t, h = run(ctx, abi.PRECISION_SPLIT)
        assert np.array_equal(y, want[abi.PRECISION_SPLIT][0]) and (t, h) == want[abi.PRECISION_SPLIT][1:]


@pytest.mark.parametrize("n", [1400, 5000, 7300])
def test_the_last_light_body_removed(n):
    """Every body left is massive: block pairs from then on, as in a fresh context."""
    s = _disk(n, 1)
    y = s.y0.reshape(-1, 6)
    y[n, :3] *= 60.0 / np.linalg.norm(y[n, :3])
    with engine.Context(s, precision=abi.PRECISION_SPLIT_FF) as ctx:
        ctx.set_state(s.y0)
        ctx.accel(0.0, s.y0)
        assert len(ctx.handle_events(1.0, 40.0, 0.0, 0.0)) == 1
        rest = ctx.get_state()
        assert rest.size == 6 * n
        got, _, nn, nd = ctx.accel(0.0, rest)
    with engine.Context(_disk(n), precision=abi.PRECISION_SPLIT_FF) as ctx:
        want, _, nn2, nd2 = ctx.accel(0.0, rest)
    assert np.array_equal(got.view(np.uint64), want.view(np.uint64))
    assert np.array_equal(nn, nn2) and np.array_equal(nd.view(np.uint64), nd2.view(np.uint64))
