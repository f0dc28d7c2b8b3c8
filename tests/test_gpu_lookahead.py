"""LU with lookahead (panels on a second stream beside the previous group's
update) against the same factorisation on one stream."""
import numpy as np
import pytest

from bem_mececcs_b200 import capi, meshgen
from bem_mececcs_b200.solver import BemSolver, solve_dense
from gpu_util import rel

pytestmark = pytest.mark.gpu


# one system: the smallest size with lookahead, a last panel of 1, 63 and 64
# columns, a right-hand side alone past the last pair
@pytest.mark.parametrize("n", [1582, 1599, 1600, 1601, 1663, 1664, 1665, 2241])
def test_fp64(n):
    """Backward error of the solve (see test_fp64_panel), new contexts and
    repeated solves alike."""
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    scale = np.linalg.norm(a, 2 if n < 500 else "fro")
    ctx = capi.Context(0)
    try:
        for _ in range(3):
            b = rng.standard_normal(n) + 1j * rng.standard_normal(n)
            x = solve_dense(ctx, a, b)
            err = np.linalg.norm(a @ x - b) / (scale * np.linalg.norm(x) + np.linalg.norm(b))
            assert err < 10 * n * np.finfo(float).eps
    finally:
        ctx.close()


# 3 nx ny unknowns, batches just large enough for lookahead: FP64 pairs and a
# last panel; FP32 groups of four, then two and one panels (1425: 145 columns
# left, 1020: 252, 1290: 10)
@pytest.mark.parametrize("form,nx,ny,batch", [
    ("plain", 10, 9, 35), ("plain", 13, 10, 17), ("plain", 17, 10, 10), ("plain", 25, 19, 2),
    ("mixed", 25, 19, 13), ("mixed", 20, 17, 25), ("mixed", 43, 10, 16), ("mixed", 29, 33, 4)])
def test_sweep(form, nx, ny, batch):
    """FP32 factors take the same operations in the same order on one stream
    or two, so mixed solutions are equal to the bit; plain ones differ by the
    shapes of the FP64 products (rounding times the growth, below 1e-11)."""
    m = meshgen.enclosed_grid(nx, ny, jitter=0.10, seed=3, depth=2.5, layers=2)
    d = meshgen.traction_patch(m, radius=6.0, dam=0.02)
    d.kode[1::5] = 0
    freqs = np.linspace(3.0, 14.0, batch)
    with BemSolver(m) as sol:
        sol.ghmatece()
        sol.set_bc(d.kode, d.bc, d.dam, d.rho)
        x = {}
        for on in (1, 0):
            sol.ctx.set_option("lu_lookahead", on)
            for _ in range(3):  # enqueued directly, captured, replayed
                x[on], _ = sol.sweep(freqs, form=form, batch=batch, refine=3)
        for i in range(len(freqs)):
            if form == "mixed":
                assert np.array_equal(x[1][i], x[0][i]), freqs[i]
            else:
                assert rel(x[1][i], x[0][i]) < 1e-11, freqs[i]


# the cases above, which lie just over the rule's lines, and one below each
@pytest.mark.parametrize("form,nx,ny,batch,used", [
    ("plain", 10, 9, 35, True), ("plain", 13, 10, 17, True), ("plain", 17, 10, 10, True), ("plain", 25, 19, 2, True),
    ("mixed", 25, 19, 13, True), ("mixed", 20, 17, 25, True), ("mixed", 43, 10, 16, True),
    ("mixed", 29, 33, 4, True), ("plain", 10, 9, 34, False), ("mixed", 25, 19, 12, False)])
def test_lookahead_is_used(form, nx, ny, batch, used):
    """The comparisons above say something only where lookahead runs with the
    option on, and does not with it off."""
    m = meshgen.enclosed_grid(nx, ny, jitter=0.10, seed=3, depth=2.5, layers=2)
    d = meshgen.traction_patch(m, radius=6.0, dam=0.02)
    with BemSolver(m) as sol:
        sol.ghmatece()
        sol.set_bc(d.kode, d.bc, d.dam, d.rho)
        freqs = np.linspace(3.0, 14.0, batch)
        for on in (1, 0):
            sol.ctx.set_option("lu_lookahead", on)
            before = sol.ctx.get_option("lookahead_runs")
            for _ in range(2):  # enqueued directly, then captured where it can be
                sol.sweep(freqs, form=form, batch=batch, refine=1)
            runs = sol.ctx.get_option("lookahead_runs") - before
            assert runs >= 2 if used and on else runs == 0


@pytest.mark.parametrize("n,used", [(1581, False), (1582, True), (2241, True)])
def test_lookahead_is_used_by_one_system(n, used):
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    b = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    x = {}
    for on in (1, 0):
        ctx = capi.Context(0)
        try:
            ctx.set_option("lu_lookahead", on)
            x[on] = solve_dense(ctx, a, b)
            assert ctx.get_option("lookahead_runs") == (1 if used and on else 0)
        finally:
            ctx.close()
    # two backward-stable solves of one system: apart by its condition, which
    # for these matrices is below n^2
    assert rel(x[1], x[0]) < 10 * n ** 2 * np.finfo(float).eps
