"""The Stokes kernels' own exponential, reciprocal root and radial functions
(csrc/cexp.cuh, csrc/bem_device.cuh) over small and large arguments, the
general path included, against the oracle's assembled system."""
import numpy as np
import pytest

import oracle
from bem_mececcs_b200 import meshgen
from bem_mececcs_b200.solver import BemSolver

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


# phases from 1e-3 to 4e7 (above 1e7: the general functions), exponents down
# to about -4000 (below -700: the general functions), undamped and damped
@pytest.mark.parametrize("omega,dam", [(0.01, 0.0), (0.01, 0.2), (1.0, 0.0), (7.3, 0.05), (300.0, 0.0),
                                       (300.0, 0.5), (4000.0, 0.01), (4.0e6, 0.0), (4.0e6, 1e-7)])
@pytest.mark.parametrize("npg", [2, 6])
def test_system_against_oracle(omega, dam, npg):
    m = meshgen.enclosed_grid(5, 4, jitter=0.10, seed=2, npg=npg, rnu=0.31, depth=2.5, layers=1)
    d = meshgen.traction_patch(m, radius=3.0, dam=dam)
    d.kode[::7] = 0
    p = oracle.OracleProblem(m, d)
    p.ghmatece()
    ozh, ozfi, _, _ = p.system(omega)
    with BemSolver(m) as sol:
        sol.ghmatece()
        sol.set_bc(d.kode, d.bc.astype(np.complex128), d.dam, d.rho)
        sol.ghmatecd(omega)
        zh, zfi = sol.get_system()
    # both sides round the phase k r (k r eps each) and cancel 1/(k r)^2
    # against order 1 in the radial functions; the nearest Gauss points are
    # a tenth of an element from the centroid
    far, near = 16.0 * omega, 0.1 * omega / 2.0
    tol = EPS * (50.0 + 4.0 * far + 20.0 / min(near, 1.0) ** 2)
    for a, b in ((zh.ravel(), ozh.ravel()), (zfi, ozfi)):
        assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b)
