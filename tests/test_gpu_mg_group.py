"""The multigrid-preconditioned solve as one launch, at the edges of the hierarchies it takes."""
import numpy as np
import pytest

import oracle as O
from conftest import rel_err
from test_gpu_multigrid import _charge, _solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(16, 12, 8), (24, 16, 40), (72, 64, 64), (80, 64, 64)])
def test_one_launch_solve_on_uneven_boxes(lib, cells):
    """The hierarchies the one-launch solve takes: uneven boxes, a body off the lattice's even points,
    fewer rows than threads and up to five rows a thread.  In both forms the Jacobi-CG solution to the
    bars of the other multigrid tests."""
    n = np.array(cells)
    lo = n // 3
    mesh = O.kuhn_box(cells, 0.05, body=tuple((int(a), int(a) + max(2, int(b) // 5)) for a, b in zip(lo, n)), bias=-10.0)
    rho = _charge(mesh, 9)
    for precision, rtol in ((0, 1e-13), (1, 1e-12)):
        rc_j, phi_j, E_j, _, _, _ = _solve(mesh, precision, False, rtol, rho)
        rc_m, phi_m, E_m, it_m, rel_m, levels = _solve(mesh, precision, True, rtol, rho)
        assert len(levels) >= 2 and rc_j == 0 and rc_m == 0 and rel_m <= rtol and it_m <= 40
        assert rel_err(phi_m, phi_j) < 1e-11
        assert rel_err(E_m, E_j) < 1e-9


def test_levels_without_couplings(lib):
    """Free nodes at even coordinates only: no row of the finest operator, nor of the next, has an entry
    beside its diagonal, so their rows are filling entries alone."""
    n = 24
    mesh = O.kuhn_box((n, n, n), 0.05, body=None, bias=0.0)
    at = np.rint(mesh.xyz / 0.05).astype(int)
    free = np.all((at % 2 == 0) & (at > 0) & (at < n), axis=1)
    mesh.dirichlet[:] = np.where(free, 0, 1)
    rho = _charge(mesh, 9)
    for precision, rtol in ((0, 1e-13), (1, 1e-12)):
        rc_j, phi_j, E_j, _, _, _ = _solve(mesh, precision, False, rtol, rho)
        rc_m, phi_m, E_m, it_m, rel_m, levels = _solve(mesh, precision, True, rtol, rho)
        assert [lv[0] for lv in levels] == [11**3, 11**3, 5**3] and free.sum() == 11**3
        assert rc_j == 0 and rc_m == 0 and rel_m <= rtol
        assert rel_err(phi_m, phi_j) < 1e-11 and rel_err(E_m, E_j) < 1e-9
