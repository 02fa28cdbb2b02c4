"""Where the runtime refuses a cooperative launch, every solve runs as launches instead.  Jacobi-CG sums in
the same order either way and gives the same bits; the multigrid solve agrees to its tolerance."""
import numpy as np
import pytest

import oracle as O
from conftest import rel_err
from faults import faults
from pic_helpers import pcg_csr_on_device
from test_gpu_batch_bits import _equal, _scenario, _state
from test_gpu_multigrid import _charge, _solve
from test_gpu_pcg_group import _system

pytestmark = pytest.mark.gpu


def _both(f):
    """f's result with cooperative launches and without."""
    with faults() as lib:
        one = f(lib)
        lib.fault_launches(1, 0)
        launched = f(lib)
        assert lib.fault_calls() > 0
    return one, launched


@pytest.mark.parametrize("R", (200, 500, 5000, 90000, 151552))
def test_csr_solve(lib, R):
    ptr, col, val, diag, rows = _system(R, np.random.default_rng(R))
    b = np.random.default_rng(1).standard_normal(R)

    def f(lib):
        return [pcg_csr_on_device(e, ptr, col, val, diag, b, np.zeros(R), 1e-13, 500)
                for e in (lib.scdat_pcg_csr, lib.scdat_pcg_csr_noalloc)]

    for a, z in zip(*_both(f)):
        assert a[0] == z[0] == 0 and a[2] == z[2] and np.array_equal(a[1], z[1])


@pytest.mark.parametrize("cells", [(9, 8, 7), (30, 27, 33), (46, 45, 44)])
@pytest.mark.parametrize("precision,rtol", ((0, 1e-13), (1, 1e-12)))
def test_jacobi_field_solve(lib, cells, precision, rtol):
    mesh = O.kuhn_box(cells, 0.05, body=tuple((c // 3, c // 3 + 2) for c in cells), bias=-10.0)
    rho = _charge(mesh, 9)
    one, launched = _both(lambda lib: _solve(mesh, precision, False, rtol, rho))
    assert one[0] == launched[0] == 0 and one[3] == launched[3]
    assert np.array_equal(one[1], launched[1]) and np.array_equal(one[2], launched[2])


@pytest.mark.parametrize("cells", [(24, 16, 40), (64, 48, 32)])
@pytest.mark.parametrize("precision,rtol", ((0, 1e-13), (1, 1e-12)))
def test_multigrid_field_solve(lib, cells, precision, rtol):
    mesh = O.kuhn_box(cells, 0.05, body=tuple((c // 3, c // 3 + 3) for c in cells), bias=-10.0)
    rho = _charge(mesh, 9)
    one, launched = _both(lambda lib: _solve(mesh, precision, True, rtol, rho))
    assert one[0] == launched[0] == 0 and abs(one[3] - launched[3]) <= 2
    assert rel_err(one[1], launched[1]) < 1e-11 and rel_err(one[2], launched[2]) < 1e-9


def test_multigrid_with_eleven_rows_a_thread(lib):
    mesh = O.kuhn_box((112, 96, 80), 0.05, body=((40, 52), (30, 44), (20, 40)), bias=-10.0)
    rho = _charge(mesh, 9)
    one, launched = _both(lambda lib: _solve(mesh, 1, True, 1e-12, rho))
    assert one[0] == launched[0] == 0 and abs(one[3] - launched[3]) <= 2
    assert rel_err(one[1], launched[1]) < 1e-11 and rel_err(one[2], launched[2]) < 1e-9


@pytest.mark.parametrize("use_graph", (True, False))
@pytest.mark.parametrize("blocks,second", ((8, (40, 38, 39)), (2, (40, 38, 39)), (1, (40, 38, 39)), (1, (44, 42, 43))))
def test_batch(lib, use_graph, blocks, second):
    """With fewer field blocks a thread of the loops takes up to four rows, those of the one launch too."""
    from scdat_b200 import capi

    def f(lib):
        doms = [_scenario((37, 35, 36), 5, 1), _scenario(second, 6, 1), _scenario((12, 11, 10), 7, 2)]
        b = capi.Batch([d[0] for d in doms], use_graph=use_graph, field_blocks_per_sm=blocks)
        b.step(2)
        out = [_state(d) for d in doms]
        b.close()
        for d in doms:
            d[0].close()
        return out

    one, launched = _both(f)
    _equal(launched, one)
