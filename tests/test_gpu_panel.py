"""The LU panel kernel (csrc/panel.cuh) at the edges of its row tiles, slices
and clusters, through the public solves, against numpy and the plain form."""
import numpy as np
import pytest

from bem_mececcs_b200 import capi, meshgen
from bem_mececcs_b200.solver import BemSolver, solve_dense
from gpu_util import rel

pytestmark = pytest.mark.gpu


def _matrix(kind, n, rng):
    if kind == "random":
        return rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    if kind == "dominant":  # pivots stay on the diagonal
        return 0.5 * np.eye(n) + 0.01 * (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(n)
    # every candidate of the first column has the same |re| + |im|
    a = (1j ** rng.integers(0, 4, (n, n))) * 0.5 + 0.1 * rng.standard_normal((n, n))
    a[:, 0] = 1j ** rng.integers(0, 4, n)
    return a


# one row, a sub-panel, a panel and one more, one slice of 64 (up to 200 rows a
# CTA), slices of 56 and fewer columns, clusters of 1 to 16 CTAs
@pytest.mark.parametrize("n", [1, 7, 8, 9, 64, 65, 201, 400, 1633, 2049])
@pytest.mark.parametrize("kind", ["random", "dominant", "ties"])
@pytest.mark.parametrize("clusters", [True, False], ids=["sized", "16"])
def test_fp64_panel(n, kind, clusters):
    """Backward error of the solve: LU with partial pivoting stays below
    n eps times the element growth, which for these matrices is far below 10."""
    rng = np.random.default_rng(n)
    a = _matrix(kind, n, rng)
    b = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    ctx = capi.Context(0)
    ctx.set_option("small_clusters", clusters)
    x = solve_dense(ctx, a, b)
    ctx.close()
    err = np.linalg.norm(a @ x - b) / (np.linalg.norm(a, 2 if n < 500 else "fro") * np.linalg.norm(x) + np.linalg.norm(b))
    assert err < 10 * max(n, 8) * np.finfo(float).eps


# n = 12..234: clusters of 1 to 2 CTAs and ragged last panels; 3366: slices of
# 32 columns on 8 CTAs until 3328 rows are left
@pytest.mark.parametrize("nx,ny", [(2, 2), (23, 1), (8, 8), (13, 6), (34, 33)])
def test_fp32_panel(nx, ny):
    """The mixed form reaches the plain form's solution (1e-10) whether its
    problems run alone or together."""
    m = meshgen.enclosed_grid(nx, ny, jitter=0.10, seed=3, depth=2.5, layers=2)
    d = meshgen.traction_patch(m, radius=6.0)
    with BemSolver(m) as sol:
        sol.ghmatece()
        sol.set_bc(d.kode, d.bc, d.dam, d.rho)
        freqs = [0.4, 1.1, 2.7]
        xp, _ = sol.sweep(freqs, form="plain", batch=3)
        for batch in (1, 3):
            xm, _ = sol.sweep(freqs, form="mixed", batch=batch, refine=4)
            for i in range(len(freqs)):
                assert rel(xm[i], xp[i]) < 1e-10, (batch, freqs[i])


# 1 to 17 row blocks on clusters of 1 to 16 CTAs, more steps than a CTA's 16
# value slots, a last block of 3, 21, 36 and 60 rows
@pytest.mark.parametrize("nx,ny", [(1, 1), (7, 3), (13, 5), (17, 10), (19, 18)])
@pytest.mark.parametrize("count", [1, 5, 40])
def test_fp32_solves_with_interchanges(nx, ny, count):
    """The cluster solves after factorisations that interchange many rows: at
    these frequencies the off-diagonal traction terms, of order omega, exceed
    the diagonal's 1/2.  The refinement converges only if L, its row order and
    the block inverses agree."""
    m = meshgen.enclosed_grid(nx, ny, jitter=0.10, seed=8, depth=2.5, layers=2)
    d = meshgen.traction_patch(m, radius=6.0, dam=0.02)
    d.kode[1::5] = 0
    with BemSolver(m) as sol:
        sol.ghmatece()
        sol.set_bc(d.kode, d.bc, d.dam, d.rho)
        freqs = np.linspace(12.0, 25.0, count)
        xp, _ = sol.sweep(freqs, form="plain", batch=8)
        xm, _ = sol.sweep(freqs, form="mixed", batch=count, refine=7)
        for i in range(count):
            assert rel(xm[i], xp[i]) < 1e-9, freqs[i]


def test_tournament_option_reaches_tall_panels():
    """n = 8250: the first FP32 panel has more rows than the push kernel's
    cluster holds (8192), so the option panel_tslu factors it by a tournament
    (six launches) whatever the in-place kernel could hold.  Its candidates go
    through k_panel_push with mailboxes.  The refined solution reaches the
    plain form's."""
    m = meshgen.enclosed_grid(55, 50, jitter=0.10, seed=9, depth=2.5, layers=2)
    d = meshgen.traction_patch(m, radius=2.0)
    launches = {}
    with BemSolver(m) as sol:
        sol.ghmatece()
        sol.set_bc(d.kode, d.bc, d.dam, d.rho)
        assert sol.nn == 8250
        sol.ctx.set_option("lu_lookahead", 0)  # which splits launches, and is for the in-place kernel
        xp, _ = sol.sweep([1.3], form="plain", batch=1)
        for on in (0, 1):
            sol.ctx.set_option("panel_tslu", on)
            before = sol.ctx.launches
            xm, _ = sol.sweep([1.3], form="mixed", batch=1, refine=3)
            launches[on] = sol.ctx.launches - before
            assert rel(xm[0], xp[0]) < 1e-10, on
    assert launches[1] == launches[0] + 5
