"""The float-float kernel over pairs of blocks (k_pairs_sym, from 1,152 massive
bodies) against the reference (FP64) form on the device.

Sizes: where the path begins (every body massive, or light bodies besides),
whole blocks of 64, 128 and 256 bodies, the sizes at which the blocks grow, and
one more or less (the last block is padded when every body is massive, left to
k_pairs_ff when not), both sides of 192 and 256 blocks of 256 (one, two and four
blocks of sources a CTA, with and without a remainder), beyond the path's end,
and light bodies in numbers that leave the last massive block empty, nearly
empty and nearly full.  Pairs are planted closer than the grid step (FP64
arithmetic, on both bodies' sides) inside one block, in neighbouring blocks, in
the first and last block, and across the end of the whole blocks.  Bound: 1e-12
relative acceleration error per body, as the form's other kernel's; nearest
neighbours and their distances are equal.  A block of sinks alone gives the same
bits as the whole evaluation."""
import numpy as np
import pytest

from solaris_gb300 import abi, engine, scenarios

pytestmark = pytest.mark.gpu

SPLIT_RTOL = 1e-12


def _system(n_massive, n_spl=0, n_light=0, seed=91):
    rng = np.random.default_rng(seed + n_massive)
    G = abi.GAUSS2

    def phases(n):
        ang = rng.uniform(0, 2 * np.pi, (3, n))
        return scenarios.elements_to_phase(G * np.ones(n), rng.uniform(0.5, 5.0, n), rng.uniform(0, 0.05, n),
                                           rng.uniform(0, 0.03, n), ang[0], ang[1], ang[2])

    n_proto = n_massive - 1
    pp = phases(n_proto)
    # body b = index in the system; protoplanet b is row b - 1
    last = (n_massive - 1) // 256 * 256
    pairs = [(10, 11, 2.0e-9), (300, 301 + 200, 3.0e-7), (255, 256, 1.0e-8), (1, last - 3, 4.0e-8),
             (700, last, 1.5e-7), (last - 1, last - 257, 2.0e-6)]
    for a, b, sep in pairs:
        pp[b - 1] = pp[a - 1]
        pp[b - 1, :3] += sep * np.array([0.6, -0.48, 0.64])
    groups = [scenarios._star(), (abi.PROTO_PLANET, dict(mass=rng.uniform(0.5e-9, 2e-9, n_proto), phase=pp))]
    if n_spl:
        groups.append((abi.SUPER_PLANETESIMAL, dict(mass=np.full(n_spl, 1e-8), phase=phases(n_spl))))
    if n_light:
        groups.append((abi.TEST_PARTICLE, dict(mass=np.zeros(n_light), phase=phases(n_light))))
    return scenarios._assemble("sym_pairs", groups), pairs


@pytest.mark.parametrize("sizes", [(1151,), (1152,), (1153,), (1343,), (1344,), (2049,), (10007,), (10999,), (11000,), (11137,),
                                   (19999,), (20000,), (20225,), (49152,), (49153,), (49409,), (66000,), (131073,),
                                   (7167, 0, 5), (7168, 3, 0), (7423, 0, 700), (7424, 300, 1), (11008, 1, 130),
                                   (11009, 40, 600), (20224, 0, 77), (49664, 1, 130)])
def test_block_pairs_against_the_reference_form(sizes):
    s, pairs = _system(*sizes)
    with engine.Context(s, precision=abi.PRECISION_FP64) as ctx:
        d64, rm3_64, nn64, nd64 = ctx.accel(0.0, s.y0)
        ctx.set_precision(abi.PRECISION_SPLIT_FF)
        dff, rm3, nn, nd = ctx.accel(0.0, s.y0)
        again, *_ = ctx.accel(0.0, s.y0)
    a, r = dff.reshape(-1, 6)[1:, 3:], d64.reshape(-1, 6)[1:, 3:]
    err = np.linalg.norm(a - r, axis=1) / np.linalg.norm(r, axis=1)
    assert err.max() <= SPLIT_RTOL, f"max rel err {err.max():.3e} at body {int(err.argmax()) + 1}"
    assert np.array_equal(rm3.view(np.uint64), rm3_64.view(np.uint64))
    assert np.array_equal(nn, nn64)
    assert np.array_equal(nd.view(np.uint64), nd64.view(np.uint64))
    for i, j, sep in pairs:
        assert nn[i] == j and nn[j] == i
    assert np.array_equal(again.view(np.uint64), dff.view(np.uint64))


@pytest.mark.parametrize("sizes", [(1500,), (9000,), (8198, 40, 900)])
def test_sink_blocks_of_block_pairs_equal_the_whole(sizes):
    torch = pytest.importorskip("torch")
    s, _ = _system(*sizes)
    with engine.Context(s, precision=abi.PRECISION_SPLIT_FF) as ctx:
        whole, _, nn, _ = ctx.accel(0.0, s.y0)
        dev = torch.device("cuda", 0)
        y = torch.from_numpy(s.y0.copy()).to(dev)
        out = torch.full((6 * s.n,), float("nan"), dtype=torch.float64, device=dev)
        torch.cuda.synchronize()
        cuts = [c for c in (0, 1, 255, 600, 8191, 8195) if c < s.n] + [s.n]
        for lo, hi in zip(cuts, cuts[1:]):
            abi.check(ctx.lib, ctx.lib.sol_accel_sinks_device(ctx.h, 0.0, y.data_ptr(), lo, hi, out.data_ptr()))
            assert np.array_equal(ctx.last_eval()[1][lo:hi], nn[lo:hi])
        torch.cuda.synchronize()
        got = out.cpu().numpy()
    assert np.array_equal(got.view(np.uint64), whole.view(np.uint64))
