"""Out of device memory, made to happen on the host: the context option
fail_alloc lets the n-th allocation of a call fail.  Every allocation of a
call is failed in turn; the call then either reports BEM_ERR_NOMEM or does
without, and the next calls give the results of an undisturbed context."""
import numpy as np
import pytest

from bem_mececcs_b200 import capi, meshgen
from bem_mececcs_b200.solver import BemSolver, solve_dense
from gpu_util import rel

pytestmark = pytest.mark.gpu


def _mesh(nx, ny):
    m = meshgen.enclosed_grid(nx, ny, jitter=0.10, seed=4, depth=2.5, layers=2)
    d = meshgen.traction_patch(m, radius=6.0, dam=0.02)
    d.kode[1::5] = 0
    return m, d


def _solver(m, d, ctx=None):
    sol = BemSolver(m) if ctx is None else BemSolver(m, ctx=ctx)
    sol.ghmatece()
    sol.set_bc(d.kode, d.bc, d.dam, d.rho)
    return sol


def _each_allocation(ctx, call, limit=200):
    """call() with its 1st, 2nd, ... allocation failing, until one is left
    over; yields (n, result or None)."""
    for n in range(1, limit):
        ctx.set_option("fail_alloc", n)
        try:
            out = call()
        except capi.BemError as e:
            assert e.code == capi.BEM_ERR_NOMEM, (n, e)
            out = None
        if ctx.get_option("fail_alloc"):  # fewer allocations than that
            ctx.set_option("fail_alloc", 0)
            return
        yield n, out
    raise AssertionError("too many allocations")


# a small system first, then a growing one whose buffers fail one by one, then
# the small one again: capacities must not outlive their buffers
@pytest.mark.parametrize("small,large", [(20, 90), (70, 300)])
def test_dense_solve(small, large):
    rng = np.random.default_rng(small)
    mats = {}
    for n in (small, large):
        a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 4.0 * np.sqrt(n) * np.eye(n)
        b = rng.standard_normal(n) + 1j * rng.standard_normal(n)
        mats[n] = a, b, np.linalg.solve(a, b)
    n = 1
    while True:
        ctx = capi.Context(0)
        try:
            assert rel(solve_dense(ctx, *mats[small][:2]), mats[small][2]) < 1e-12
            ctx.set_option("fail_alloc", n)
            try:
                x = solve_dense(ctx, *mats[large][:2])
                assert rel(x, mats[large][2]) < 1e-12, n
            except capi.BemError as e:
                assert e.code == capi.BEM_ERR_NOMEM, (n, e)
            left = ctx.get_option("fail_alloc")
            ctx.set_option("fail_alloc", 0)
            for size in (small, large):
                assert rel(solve_dense(ctx, *mats[size][:2]), mats[size][2]) < 1e-12, (n, size)
        finally:
            ctx.close()
        if left:
            break
        n += 1
    assert n > 3  # some allocations were failed


@pytest.mark.parametrize("nx,ny", [(3, 2), (10, 9)])
def test_first_calls_of_a_mesh(nx, ny):
    """Mesh upload, static diagonals, boundary values, assembly and solve on a
    new context, any one allocation failing; then all of it once more."""
    m, d = _mesh(nx, ny)
    with _solver(m, d) as sol:
        want = sol.solve_frequency(2.0)
    ctx = capi.Context(0)
    try:
        def call():
            sol = _solver(m, d, ctx)
            return sol.solve_frequency(2.0)
        count = 0
        for n, got in _each_allocation(ctx, call):
            count += 1
            if got is not None:
                assert rel(got[0], want[0]) < 1e-12 and rel(got[1], want[1]) < 1e-12, n
            again = call()
            assert rel(again[0], want[0]) < 1e-12 and rel(again[1], want[1]) < 1e-12, n
        assert count > 5
    finally:
        ctx.close()


# 189 unknowns: one forward step of three, 720: twelve; one refinement step:
# the solves' tables are asked for once per step
@pytest.mark.parametrize("nx,ny", [(9, 7), (16, 15)])
@pytest.mark.parametrize("refine", [1, 3])
def test_mixed_sweep_and_its_captured_step(nx, ny, refine):
    """A failure in the step that runs directly, then the captured step and its
    replays: the solutions stay those of the plain form (to the refinement's
    1e-6 after one step)."""
    m, d = _mesh(nx, ny)
    freqs = [1.0, 2.5, 4.0]
    with _solver(m, d) as sol:
        want, _ = sol.sweep(freqs, form="plain", batch=3)
    tol = 1e-6 if refine == 1 else 1e-9
    n = done = 0
    while True:
        n += 1
        with _solver(m, d) as sol:
            sol.ctx.set_option("fail_alloc", n)
            try:
                x, _ = sol.sweep(freqs, form="mixed", batch=3, refine=refine)
                assert rel(x, want) < tol, n
                done += 1
            except capi.BemError as e:
                assert e.code == capi.BEM_ERR_NOMEM, (n, e)
            left = sol.ctx.get_option("fail_alloc")
            if left:
                break
            for _ in range(4):  # directly or captured, then replayed
                x, _ = sol.sweep(freqs, form="mixed", batch=3, refine=refine)
                assert rel(x, want) < tol, n
    assert n > 10 and done >= 2  # the solves' tables, at least, are done without


# the last two sizes take lookahead, with buffers of its own
@pytest.mark.parametrize("form,nx,ny,count", [("plain", 9, 7, 5), ("mixed", 9, 7, 5), ("plain", 16, 15, 2),
                                              ("mixed", 16, 15, 2), ("plain", 25, 19, 2), ("mixed", 25, 19, 13)])
def test_sweep_goes_on_with_fewer_problems(form, nx, ny, count):
    """Whichever buffer of a lockstep step finds no memory, the sweep runs in
    smaller steps and gives every solution."""
    m, d = _mesh(nx, ny)
    freqs = np.linspace(1.0, 4.0, count)
    with _solver(m, d) as sol:
        want, _ = sol.sweep(freqs, form="plain", batch=count)
    n = 0
    while True:
        n += 1
        with _solver(m, d) as sol:
            sol.ctx.set_option("fail_alloc", n)
            x, corr = sol.sweep(freqs, form=form, batch=count, refine=3)
            assert rel(x, want) < 1e-9 and np.all(corr < 1e-7), n
            left = sol.ctx.get_option("fail_alloc")
            if left:
                break
            x, _ = sol.sweep(freqs, form=form, batch=count, refine=3)
            assert rel(x, want) < 1e-9, n
    assert n > 10


@pytest.mark.parametrize("form", ["plain", "mixed"])
def test_batch_goes_on_in_smaller_classes(form):
    """Whichever allocation of a batch call fails, on the driver or a worker,
    the call gives every solution; so does the next one."""
    from bem_mececcs_b200.solver import batch_solve
    probs = []
    want = []
    for k, (nx, ny) in enumerate([(3, 2), (9, 7), (9, 7), (9, 8), (10, 7), (16, 15)]):
        sol = _solver(*_mesh(nx, ny))
        fr = 1.0 + 0.3 * k
        want.append(sol.sweep([fr], form="plain", batch=1)[0][0])
        probs.append((sol, fr))
    n = ok = 0
    while True:
        n += 1
        ctx = capi.Context(0)
        try:
            ctx.set_option("fail_alloc", n)
            try:
                xs, _ = batch_solve(ctx, probs, form=form, refine=3)
                assert all(rel(x, w) < 1e-9 for x, w in zip(xs, want)), n
                ok += 1
            except capi.BemError as e:  # a class of one problem has nothing to give up
                assert e.code == capi.BEM_ERR_NOMEM, (n, e)
            left = ctx.get_option("fail_alloc")
            ctx.set_option("fail_alloc", 0)
            xs, _ = batch_solve(ctx, probs, form=form, refine=3)
            assert all(rel(x, w) < 1e-9 for x, w in zip(xs, want)), n
        finally:
            ctx.close()
        if left:
            break
    for sol, _ in probs:
        sol.close()
    assert n > 20 and ok == n
