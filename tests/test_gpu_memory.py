"""The packed factor records are memory that contexts and batches can do without: it is not missing
elsewhere, and the solves that go on without it give the same bits."""
import threading

import numpy as np
import pytest

from dumux_gb300 import Batch, Context, newton_params, problems

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _context(cells=(64, 64, 32), seed=5, kind="auto", mpfa=False):
    desc, prev = (problems.dnapl_2p_mpfa if mpfa else problems.dnapl_2p)(cells=cells, seed=seed)
    u = prev.reshape(-1, 2).copy()
    u[:, 1] = np.random.default_rng(seed).uniform(0.0, 0.3, len(u))
    ctx = Context(desc)
    ctx.set_ilu_kernel(kind)
    ctx.set_solution(u.reshape(-1))
    ctx.set_prev_solution(prev)
    ctx.set_time_step(250.0)
    ctx.assemble_jacobian_and_residual()
    return ctx


def _solve(ctx):
    return ctx.linear_solve(1e-4, 40)["iterations"], ctx.update()


class _Fill:
    """Takes device memory until `free` bytes are left."""

    def __init__(self, torch, free):
        self.torch = torch
        torch.cuda.empty_cache()
        have, _ = torch.cuda.mem_get_info(0)
        self.block = torch.empty((have - free) // (2 * MIB) * (2 * MIB), dtype=torch.uint8, device="cuda:0")

    def release(self):
        self.block = None
        self.torch.cuda.empty_cache()


def _same(a, b):
    assert a[0] == b[0] and np.array_equal(a[1], b[1])


def _used(torch, make):
    """The object that make() returns and the device memory it took."""
    torch.cuda.synchronize()
    before, _ = torch.cuda.mem_get_info(0)
    x = make()
    torch.cuda.synchronize()
    after, _ = torch.cuda.mem_get_info(0)
    return x, before - after


@pytest.mark.parametrize("holder", ["context", "mpfa context", "batch"])
def test_records_give_way_to_another_context(gpu_lib, holder):
    """Room for most of a second context only: it fits once the first holder's records are given back."""
    torch = pytest.importorskip("torch")
    _solve(_context(kind="wavefront"))                      # every kernel of the way back loaded
    _solve(_context((32, 32, 16), kind="levels", mpfa=True))
    probe, need = _used(torch, _context)
    probe.close()
    if holder == "batch":
        problem, u0 = problems.dnapl_2p(cells=(64, 64, 32), seed=5)

        def advance(before_the_last=lambda: None):
            batch = Batch(precision="fp64")
            i = batch.add(problem, u0, dt=250.0, t_end=250.0, params=newton_params(linear_max_iter=500))
            for _ in range(4):
                batch.iterate()
            assert "packed" in batch.describe()
            before_the_last()
            while batch.iterate():
                pass
            return batch.info(i)["linear_iterations"], batch.solution(i)

        alone = advance()
    else:
        first = _context((32, 32, 16), mpfa=True) if holder == "mpfa context" else _context()
        alone = _solve(first)
        assert "packed records" in first.describe()
    room = 24 * MIB if holder != "mpfa context" else 8 * MIB
    kept = {}

    def squeeze():
        fill = _Fill(torch, need - room)
        try:
            kept["second"] = _context()
        finally:
            fill.release()

    if holder == "batch":
        _same(advance(squeeze), alone)
    else:
        squeeze()
        _same(_solve(first), alone)
        assert "packed records" not in first.describe()
    _same(_solve(kept["second"]), _solve(_context()))


@pytest.mark.parametrize("mpfa", [False, True])
def test_records_are_not_taken_from_a_nearly_full_device(gpu_lib, mpfa):
    torch = pytest.importorskip("torch")
    cells = (32, 32, 16) if mpfa else (64, 64, 32)
    alone = _solve(_context(cells, mpfa=mpfa))
    _same(_solve(_context(cells, kind="levels" if mpfa else "wavefront", mpfa=mpfa)), alone)
    ctx = _context(cells, mpfa=mpfa)
    fill = _Fill(torch, 60 * MIB)
    try:
        _same(_solve(ctx), alone)
        assert "packed records" not in ctx.describe()
    finally:
        fill.release()


def test_settings_that_do_not_read_the_records_give_them_back(gpu_lib):
    torch = pytest.importorskip("torch")
    ctx = _context()
    alone, took = _used(torch, lambda: _solve(ctx))
    assert took >= 32 * MIB
    _, amg = _used(torch, lambda: ctx.set_linear_solver("amg"))
    assert -amg >= 32 * MIB
    ctx.set_linear_solver("ilu")
    _same(_solve(ctx), alone)                               # laid anew, and the captured chunk with them
    _, ring = _used(torch, lambda: ctx.set_lane_ring("registers"))
    assert -ring >= 32 * MIB
    _same(_solve(ctx), alone)
    m = _context((32, 32, 16), kind="levels", mpfa=True)
    levels, took = _used(torch, lambda: _solve(m))
    m.set_ilu_kernel("auto")                                # laid from the factor that is there
    auto, more = _used(torch, lambda: _solve(m))
    _same(auto, levels)
    assert "packed records" in m.describe() and more >= 8 * MIB
    _, back = _used(torch, lambda: m.set_ilu_kernel("levels"))
    assert -back >= 8 * MIB
    m.set_ilu_kernel("auto")
    _same(_solve(m), levels)


def test_records_are_given_back_between_the_calls_of_other_threads(gpu_lib):
    """Two threads solve while a third needs memory again and again: each holder loses its records at
    most once, between two of its calls."""
    torch = pytest.importorskip("torch")
    probe, need = _used(torch, _context)
    probe.close()
    _solve(_context(kind="wavefront"))
    contexts = [_context(seed=k) for k in (5, 6)]
    alone = [_solve(c) for c in contexts]
    results = [[], []]

    def work(k):
        for _ in range(12):
            results[k].append(_solve(contexts[k]))

    fill = _Fill(torch, need - 24 * MIB)
    try:
        threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
        for t in threads:
            t.start()
        made = 0
        for _ in range(40):
            try:
                _context(seed=9).close()
                made += 1
            except Exception as e:
                assert "OOM" in str(e)                      # both holders in a call of their own
        for t in threads:
            t.join()
        _context(seed=9).close()
    finally:
        fill.release()
    for k in range(2):
        for r in results[k]:
            _same(r, alone[k])
