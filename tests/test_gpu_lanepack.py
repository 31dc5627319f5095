"""The lane sweeps over packed records against the cluster wavefront (the same arithmetic, so the
same bits) at the edges of their tiles, warps and clusters, and their bounded waits."""
import threading

import numpy as np
import pytest

from dumux_gb300 import Batch, Context, NumericalProblem, newton_params, problem_device_bytes, problems

pytestmark = pytest.mark.gpu


def _solve(desc, u, prev, kind, precision, dt):
    ctx = Context(desc, precision=precision)
    ctx.set_ilu_kernel(kind)
    ctx.set_solution(u)
    if dt:
        ctx.set_prev_solution(prev)
        ctx.set_time_step(dt)
    ctx.assemble_jacobian_and_residual()
    res = ctx.linear_solve(1e-10 if precision == "fp64" else 1e-4, 400)
    return res["iterations"], ctx.update(), ctx.describe()


# lines per warp: 16 (2x2 FP64) or 32; up to three warps per CTA; 16 CTAs per cluster
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("eqs,dims", [
    (1, (1, 1)), (1, (5, 32)), (1, (40, 33)), (1, (7, 97)), (1, (300, 3)),
    (1, (3, 5, 17)), (1, (9, 33, 5)), (1, (6, 70, 18)), (1, (20, 8, 33)),
    (2, (4, 16)), (2, (30, 17)), (2, (6, 49, 3)), (2, (8, 15, 16)), (2, (5, 33, 17)), (2, (12, 97, 6)), (2, (3, 2, 40)),
])
def test_packed_lane_sweeps_equal_cluster_wavefront(eqs, dims, precision):
    if eqs == 1:
        desc, u = problems.darcy_1p(cells=dims, seed=4)
        prev, dt = u, 0.0
    else:
        desc, prev = problems.dnapl_2p(cells=dims, extent=(6.0, 4.0, 1.0)[:len(dims)], seed=4)
        u = prev.reshape(-1, 2).copy()
        u[:, 1] = np.random.default_rng(3).uniform(0.0, 0.3, len(u))
        u, dt = u.reshape(-1), 250.0
    n0, x0, _ = _solve(desc, u, prev, "wavefront", precision, dt)
    n1, x1, how = _solve(desc, u, prev, "auto", precision, dt)
    assert "packed records" in how
    assert n1 == n0
    assert np.array_equal(x1, x0)


def test_packed_lane_sweeps_wait_limit_expires_and_the_context_recovers():
    """A wait limit far below the time the last of 40 planes waits for its first value: the sweeps
    give up, the solve reports DXG_ERR_TIMEOUT, and with the limit restored the context solves to
    the same bits (the hand-off buffer between clusters is reset)."""
    desc, u0 = problems.dnapl_2p(cells=(16, 16, 40), seed=8)
    u = u0.reshape(-1, 2).copy()
    u[:, 1] = np.random.default_rng(5).uniform(0.0, 0.4, len(u))
    ctx = Context(desc)
    ctx.set_solution(u.reshape(-1))
    ctx.set_prev_solution(u0)
    ctx.set_time_step(250.0)
    ctx.assemble_jacobian_and_residual()
    first = ctx.linear_solve(1e-10, 500)
    assert first["converged"] and "packed records" in ctx.describe()
    x0 = ctx.update()
    ctx.set_wait_limit(1e-6)
    with pytest.raises(Exception, match="timed out"):
        ctx.linear_solve(1e-10, 500)
    ctx.set_wait_limit(0.5)
    again = ctx.linear_solve(1e-10, 500)
    assert again["converged"] and again["iterations"] == first["iterations"]
    assert np.array_equal(ctx.update(), x0)


# all the clusters that fit the GPU at once, or nearly (88 of 8 CTAs, several CTAs per SM), and
# clusters of odd sizes: every one of them has to be resident for the sweeps to end
_CROWD = [(1, (4, 4, 700), "fp64"), (1, (24, 200, 24), "fp64"), (2, (64, 64, 90), "fp64"), (2, (45, 37, 23), "mixed"),
          (1, (20, 20, 100), "fp64"), (2, (8, 8, 300), "fp64")]


def _crowd_context(eqs, dims, precision, kind="auto"):
    if eqs == 1:
        desc, prev = problems.darcy_1p(cells=dims, seed=4)
        u = prev
    else:
        desc, prev = problems.dnapl_2p(cells=dims, seed=4)
        u = prev.reshape(-1, 2).copy()
        u[:, 1] = np.random.default_rng(3).uniform(0.0, 0.3, len(u))
        u = u.reshape(-1)
    ctx = Context(desc, precision=precision)
    ctx.set_ilu_kernel(kind)
    ctx.set_solution(u)
    if eqs == 2:
        ctx.set_prev_solution(prev)
        ctx.set_time_step(250.0)
    ctx.assemble_jacobian_and_residual()
    return ctx


@pytest.mark.parametrize("eqs,dims,precision", _CROWD)
def test_packed_sweeps_of_many_clusters_equal_cluster_wavefront(eqs, dims, precision):
    ref = _crowd_context(eqs, dims, precision, "wavefront")
    ctx = _crowd_context(eqs, dims, precision)
    n0, n1 = (c.linear_solve(1e-4, 40)["iterations"] for c in (ref, ctx))
    assert "packed records" in ctx.describe()
    assert n1 == n0
    assert np.array_equal(ctx.update(), ref.update())


def test_packed_sweeps_of_many_clusters_give_way_to_faster_ones():
    """256 CTAs in 32 clusters of 8 take 1.5 times as long as the lane sweeps that read the factor in
    place from 8 clusters of 16: the timing at the first factorisation finds out."""
    ref, ctx, lanes = (_crowd_context(2, (5, 33, 128), "mixed", kind) for kind in ("wavefront", "auto", "lanes"))
    n0 = ref.linear_solve(1e-4, 40)["iterations"]
    for c in (ctx, lanes):
        assert c.linear_solve(1e-4, 40)["iterations"] == n0
        assert "packed records" not in c.describe()
        assert np.array_equal(c.update(), ref.update())
    # the records are given back, and another solve of the same context does without them
    ctx.assemble_jacobian_and_residual()
    assert ctx.linear_solve(1e-4, 40)["iterations"] == n0
    assert np.array_equal(ctx.update(), ref.update())


def test_packed_sweeps_of_clusters_of_many_sizes_on_several_threads():
    """Launches that leave each other no room for all their clusters (88 clusters of 8 CTAs, 5 of
    15, 6 of 15, 2 of 12, 7 of 15, 19 of 16), from streams of their own."""
    contexts = [_crowd_context(*case) for case in _CROWD]
    alone = [(c.linear_solve(1e-4, 40)["iterations"], c.update()) for c in contexts]
    together = [None] * len(contexts)

    def work(k):
        for _ in range(5):
            together[k] = (contexts[k].linear_solve(1e-4, 40)["iterations"], contexts[k].update())

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(contexts))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(alone, together):
        assert b is not None and a[0] == b[0] and np.array_equal(a[1], b[1])


# two warps of 32 lines per CTA (one on long lines); histories across warps, CTAs and remainders
@pytest.mark.parametrize("cells", [(1, 1), (5, 4), (9, 31), (3, 33), (70, 64), (6, 65), (40, 130), (33, 257), (300, 40)])
def test_packed_mpfa_sweeps_equal_level_kernel(cells):
    desc, u, _ = problems.mpfa_linear_field_problem(cells=cells, spacing_seed=3)
    n0, x0, _ = _solve(desc, u, u, "levels", "fp64", 0.0)
    n1, x1, how = _solve(desc, u, u, "auto", "fp64", 0.0)
    assert "packed records" in how
    assert n1 == n0
    assert np.array_equal(x1, x0)


def test_packed_mpfa_sweeps_wait_limit_expires_and_the_context_recovers():
    desc, u, _ = problems.mpfa_linear_field_problem(cells=(64, 192), spacing_seed=3)
    ctx = Context(desc)
    ctx.set_solution(u)
    ctx.assemble_jacobian_and_residual()
    first = ctx.linear_solve(1e-10, 500)
    assert first["converged"] and "packed records" in ctx.describe()
    x0 = ctx.update()
    ctx.set_wait_limit(1e-6)
    with pytest.raises(Exception, match="timed out"):
        ctx.linear_solve(1e-10, 500)
    ctx.set_wait_limit(0.5)
    assert ctx.linear_solve(1e-10, 500)["iterations"] == first["iterations"]
    assert np.array_equal(ctx.update(), x0)


# problems of one, two and three clusters of CTAs and of one to three sweeping warps in one launch
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("eqs,grids", [
    (2, [(16, 31, 3), (5, 33, 17), (17, 9, 33), (2, 1, 1), (6, 97, 4), (30, 16, 16)]),
    (2, [(12, 17), (40, 50), (3, 100), (9, 1)]),
    (1, [(9, 33, 5), (6, 70, 18), (20, 8, 40)]),
])
def test_batched_packed_sweeps_equal_batched_wavefront(eqs, grids, precision):
    """A memory budget that leaves no room for the packed records keeps the batch on the cluster
    wavefront; one that shrinks between iterations moves it there in mid-solve, one that is lifted
    brings the records back when the membership changes.  The solutions are the same bits."""
    probs = [problems.darcy_1p(cells=g, seed=k) if eqs == 1 else
             problems.dnapl_2p(cells=g, extent=(6.0, 4.0, 1.0)[:len(g)], seed=k) for k, g in enumerate(grids)]
    params = newton_params(linear_max_iter=500)

    def run(budget, changes=()):
        batch = Batch(precision=precision, memory_budget=budget)
        dt = 250.0 if eqs == 2 else 0.0
        ids = [batch.add(d, u0, dt=dt, t_end=2 * dt, params=params) for d, u0 in probs]
        how, n = [], 0
        while batch.iterate():
            how.append("packed" in batch.describe())
            for at, value in changes:
                if at == n:
                    batch.set_memory_budget(value)
            n += 1
        return [batch.solution(i) for i in ids], how

    tight = sum(problem_device_bytes(d, precision) for d, _ in probs)
    waves, how = run(tight)
    assert not any(how)
    packed, how = run(0)
    assert all(how)
    moved, how = run(0, [(1, tight), (3, 0)])
    assert not eqs == 2 or not all(how)
    for a, b, c in zip(waves, packed, moved):
        assert np.array_equal(a, b) and np.array_equal(a, c)


# tiles of 16 (2x2) or 32 lines, up to four; one to sixteen planes
@pytest.mark.parametrize("b,cells", [
    (1, (3, 4, 1)), (1, (5, 32, 3)), (1, (6, 33, 16)), (1, (4, 128, 2)), (1, (40, 9, 5)),
    (2, (2, 2, 2)), (2, (5, 16, 3)), (2, (8, 17, 16)), (2, (3, 33, 5)), (2, (9, 64, 2)), (2, (40, 7, 6)),
])
def test_packed_mpfa_plane_sweeps_equal_level_kernel(b, cells):
    if b == 1:
        desc, prev, _ = problems.mpfa_linear_field_problem(
            cells=cells, K=((2.0, 0.3, 0.1), (0.3, 1.0, 0.2), (0.1, 0.2, 1.5)), spacing_seed=2)
        u, dt = prev, 0.0
    else:
        desc, prev = problems.dnapl_2p_mpfa(cells=cells, seed=6)
        u = prev.reshape(-1, 2).copy()
        u[:, 1] = np.random.default_rng(9).uniform(0, 0.4, len(u))
        u, dt = u.reshape(-1), 250.0
    n0, x0, _ = _solve(desc, u, prev, "levels", "fp64", dt)
    n1, x1, how = _solve(desc, u, prev, "auto", "fp64", dt)
    assert "packed records" in how and "one z-plane per CTA" in how
    assert n1 == n0
    assert np.array_equal(x1, x0)


def test_packed_mpfa_plane_sweeps_wait_limit_expires_and_the_context_recovers():
    desc, u0 = problems.dnapl_2p_mpfa(cells=(16, 20, 16), seed=6)
    u = u0.reshape(-1, 2).copy()
    u[:, 1] = np.random.default_rng(9).uniform(0, 0.4, len(u))
    ctx = Context(desc)
    ctx.set_solution(u.reshape(-1))
    ctx.set_prev_solution(u0)
    ctx.set_time_step(250.0)
    ctx.assemble_jacobian_and_residual()
    first = ctx.linear_solve(1e-10, 500)
    assert first["converged"] and "packed records" in ctx.describe()
    x0 = ctx.update()
    ctx.set_wait_limit(1e-6)
    with pytest.raises(Exception, match="timed out"):
        ctx.linear_solve(1e-10, 500)
    ctx.set_wait_limit(0.5)
    assert ctx.linear_solve(1e-10, 500)["iterations"] == first["iterations"]
    assert np.array_equal(ctx.update(), x0)


def test_packed_sweeps_of_contexts_on_several_threads_equal_those_alone():
    """Eight contexts whose sweeps need several clusters resident at once, solving at the same time
    on streams of their own: no launch is held up half dispatched until its waits run out."""
    def context(k):
        if k % 4 == 3:
            desc, u0 = problems.dnapl_2p_mpfa(cells=(16, 20, 16), seed=k)
        else:
            desc, u0 = problems.dnapl_2p(cells=(40, 48, 30), seed=k)
        u = u0.reshape(-1, 2).copy()
        u[:, 1] = np.random.default_rng(k).uniform(0.0, 0.4, len(u))
        ctx = Context(desc, precision="fp64" if k % 2 else "mixed")
        ctx.set_solution(u.reshape(-1))
        ctx.set_prev_solution(u0)
        ctx.set_time_step(250.0)
        ctx.assemble_jacobian_and_residual()
        return ctx

    contexts = [context(k) for k in range(8)]
    alone = [(c.linear_solve(1e-6, 400)["iterations"], c.update()) for c in contexts]
    assert all("packed records" in c.describe() for c in contexts)
    together = [None] * 8

    def work(k):
        for _ in range(5):
            together[k] = (contexts[k].linear_solve(1e-6, 400)["iterations"], contexts[k].update())

    threads = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(alone, together):
        assert b is not None and a[0] == b[0] and np.array_equal(a[1], b[1])


def _status(desc, u, dt, precision, kind, spoil):
    ctx = Context(desc, precision=precision)
    ctx.set_ilu_kernel(kind)
    ctx.set_solution(u)
    if dt:
        ctx.set_prev_solution(u)
        ctx.set_time_step(dt)
    ctx.assemble_jacobian_and_residual()
    rows, cols, values = ctx.jacobian()
    rhs = ctx.residual()
    spoil(rows, values, rhs)
    ctx.set_linear_system(rows, cols, values, rhs)
    with pytest.raises(NumericalProblem) as e:
        ctx.linear_solve(1e-8, 100, raise_on_failure=True)
    return e.value.status


# what the sweeps wait for is a NaN with all bits set: neither that one in the caller's system nor
# other values that are not finite may keep them waiting
@pytest.mark.parametrize("value", [b"\xff" * 8, b"\xff" * 7 + b"\x7f", np.float64("nan").tobytes(),
                                   np.float64("-inf").tobytes()], ids=["ones", "ones but the sign", "nan", "inf"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("disc,eqs,dims", [("tpfa", 1, (20, 30)), ("tpfa", 1, (9, 10, 20)), ("tpfa", 2, (20, 30)),
                                           ("tpfa", 2, (9, 10, 20)), ("mpfa", 1, (20, 40)), ("mpfa", 1, (6, 33, 4)),
                                           ("mpfa", 2, (6, 17, 4))])
def test_values_that_are_not_finite_end_the_solve_as_on_the_other_kernels(disc, eqs, dims, precision, value):
    if disc == "mpfa" and precision == "mixed":
        pytest.skip("MPFA-O contexts solve in FP64")
    dt = 250.0 if eqs == 2 else 0.0
    if disc == "tpfa":
        desc, u = (problems.darcy_1p(cells=dims, seed=4) if eqs == 1 else
                   problems.dnapl_2p(cells=dims, extent=(6.0, 4.0, 1.0)[:len(dims)], seed=4))
    elif eqs == 2:
        desc, u = problems.dnapl_2p_mpfa(cells=dims, seed=4)
    else:
        K = ((2.0, 0.5), (0.5, 1.0)) if len(dims) == 2 else ((2.0, 0.3, 0.1), (0.3, 1.0, 0.2), (0.1, 0.2, 1.5))
        desc, u, _ = problems.mpfa_linear_field_problem(cells=dims, K=K, spacing_seed=2)
    x = np.frombuffer(value)[0]

    def in_matrix(rows, values, rhs):
        values[rows[len(rows) // 2] * eqs * eqs] = x

    def in_rhs(rows, values, rhs):
        rhs[len(rhs) // 3] = x

    other = "wavefront" if disc == "tpfa" else "levels"
    for spoil in (in_matrix, in_rhs):
        assert (_status(desc, u, dt, precision, "auto", spoil) == _status(desc, u, dt, precision, other, spoil))


@pytest.mark.parametrize("kind,limit", [("lanes", 90e-6), ("mpfa lines", 130e-6), ("mpfa planes", 120e-6)])
def test_wait_limit_is_that_of_a_single_wait(kind, limit):
    """Long lines: a launch takes 260 to 330 us, and the warps of its middle planes (lines) wait twice, at
    the start and at the turn, no wait being longer than about 80 us.  The limit is above every single
    wait and below the time between the two."""
    if kind == "mpfa lines":
        desc, u, _ = problems.mpfa_linear_field_problem(cells=(600, 128), spacing_seed=3)
        prev, dt = u, 0.0
    else:
        desc, prev = (problems.dnapl_2p(cells=(300, 16, 40), seed=8) if kind == "lanes" else
                      problems.dnapl_2p_mpfa(cells=(200, 10, 16), seed=8))
        u = prev.reshape(-1, 2).copy()
        u[:, 1] = np.random.default_rng(5).uniform(0.0, 0.4, len(u))
        u, dt = u.reshape(-1), 250.0
    ctx = Context(desc)
    ctx.set_solution(u)
    if dt:
        ctx.set_prev_solution(prev)
        ctx.set_time_step(dt)
    ctx.assemble_jacobian_and_residual()
    first = ctx.linear_solve(1e-6, 60)
    assert "packed records" in ctx.describe()
    x0 = ctx.update()
    ctx.set_wait_limit(limit)
    assert ctx.linear_solve(1e-6, 60) == first
    assert np.array_equal(ctx.update(), x0)


# the one-CTA line sweeps, which 2D grids run where their packed plan does not fit (long lines) or the
# records are not to be had: one to sixteen warps of lines
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("eqs,dims", [(1, (1, 1)), (1, (13, 11)), (1, (9, 512)), (1, (1000, 8)), (2, (13, 11)),
                                      (2, (100, 100)), (2, (37, 300)), (2, (700, 20))])
def test_line_sweeps_equal_cluster_wavefront(eqs, dims, precision):
    if eqs == 1:
        desc, u = problems.darcy_1p(cells=dims, seed=4)
        prev, dt = u, 0.0
    else:
        desc, prev = problems.dnapl_2p(cells=dims, extent=(6.0, 4.0), seed=4)
        u = prev.reshape(-1, 2).copy()
        u[:, 1] = np.random.default_rng(3).uniform(0.0, 0.3, len(u))
        u, dt = u.reshape(-1), 250.0
    n0, x0, _ = _solve(desc, u, prev, "wavefront", precision, dt)
    ctx = Context(desc, precision=precision)
    ctx.set_ilu_kernel("lanes")
    ctx.set_lane_ring("registers")
    ctx.set_solution(u)
    if dt:
        ctx.set_prev_solution(prev)
        ctx.set_time_step(dt)
    ctx.assemble_jacobian_and_residual()
    n1 = ctx.linear_solve(1e-10 if precision == "fp64" else 1e-4, 400)["iterations"]
    assert "line sweeps in one CTA" in ctx.describe()
    assert n1 == n0
    assert np.array_equal(ctx.update(), x0)


def test_long_lines_do_not_fit_the_packed_plan():
    desc, u = problems.darcy_1p(cells=(1000, 8), seed=4)
    n0, x0, _ = _solve(desc, u, u, "wavefront", "fp64", 0.0)
    for kind in ("auto", "lanes"):
        n1, x1, how = _solve(desc, u, u, kind, "fp64", 0.0)
        assert "packed records" not in how
        assert n1 == n0 and np.array_equal(x1, x0)
