"""Order of shared-memory accesses between warps, checked in the kernels' source.

A missing order is a race that timing hides nearly always and that must not be
provoked on a GPU, so these tests read the source."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "solaris_gb300", "csrc")


def _body(name, function):
    """The text between the braces of a function's definition, without comments."""
    src = open(os.path.join(CSRC, name)).read()
    src = re.sub(r"//[^\n]*", "", src)
    at = src.index("{", re.search(r"\b%s\([^;{]*\)\s*(?=\{)" % function, src).start())
    depth = 0
    for end in range(at, len(src)):
        depth += {"{": 1, "}": -1}.get(src[end], 0)
        if depth == 0:
            return src[at + 1:end]
    raise AssertionError(function)


def test_group_workers_read_the_evaluation_between_its_two_barriers():
    """The state warps write the next evaluation's fields of Ctl (submit) after
    the block barrier that ends the present one: a worker reads them between the
    two barriers of its own evaluation only."""
    written = re.findall(r"S\.(\w+) =", _body("sol_group.cu", r"submit = \[&\]"))
    assert sorted(written) == ["cur", "factor", "flags", "last"]
    for function in ("work_by_component", "work"):
        body = _body("sol_group.cu", function)
        loop = body[body.index("for (;;) {"):]
        barriers = [m.end() for m in re.finditer(r"__syncthreads\(\);", loop)]
        assert len(barriers) == 2
        late = set(re.findall(r"\bS\.(\w+)", loop[barriers[1]:])) & set(written)
        assert not late, f"{function} reads {late} after the evaluation's last barrier"


def test_source_minima_are_ordered_between_two_steps_of_a_warp():
    """Two lanes of a warp take the same source in consecutive steps and both
    update its nearest sink in shared memory; votes and shuffles order no memory,
    so every step is followed by __syncwarp."""
    body = _body("sol_pairs_sym.cuh", "sym_part")
    steps = re.findall(r"sym_step<[^;]*;\s*(\w+)", body)
    assert len(steps) == 2
    assert steps == ["__syncwarp"] * 2


def test_group_launch_keeps_what_a_late_block_still_reads():
    """Every block of the group driver reads the start state, the control record
    and the migration state of the sources at its start, which may be late: the
    home block writes them at the launch's end only, and there (also in RK4
    calls outside the step loop, which exchange nothing) after an exchange."""
    work = _body("sol_group.cu", "work")
    migration = work[work.index("mig_compute("):work.index("part_sync(1")]
    assert "global_gas_buf" not in migration and "fc.mig_type" not in migration
    kernel = _body("sol_group.cu", "k_group_rkf78")
    end = kernel[kernel.index("pending = !P.rk4"):]
    guard = end.index("if (ran && P.rk4 && !P.sim && gridDim.x > 1 && !S.abort)")
    assert guard < end.index("exchange(P, k") < end.index("if (S.abort) return;") < end.index("P.y0[ge] = y0")
    assert end.index("if (S.abort) return;") < end.index("fc.mig_type[")
