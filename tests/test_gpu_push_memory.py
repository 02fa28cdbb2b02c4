"""The push's deferred lists where memory is short: the species take turns in one set of lists and the results
are the same bits; a batch of two-species contexts needs no lists of its own."""
import pytest

import oracle as O
from faults import faults
from pic_helpers import gpu_domain, gpu_load_particles
from test_gpu_batch_bits import _equal, _scenario, _state

pytestmark = pytest.mark.gpu
ENTRY = 24  # bytes of a list entry


def _run(precision, lib, steps=3):
    mesh = O.kuhn_box((8, 7, 9), 0.05, body=((2, 4), (2, 4), (3, 5)), bias=-15.0)
    sp = O.plasma_species(1e10, 1.0, 1.0, 0.05, 24)
    sp = [sp[0], sp[1], sp[0]]
    parts = O.seed_particles(mesh, sp, 24, 5)
    dom = gpu_domain(mesh, 2e-8, face_bc=(2, 2, 2, 2, 1, 1), precision=precision, sort_interval=2)
    gpu_load_particles(dom, sp, parts)
    for s in range(3):
        dom.set_elastic(s, 1e18, 1e-19, mode=2)
    dom.set_potential(mesh.phi_bc)
    used = lib.fault_used()
    dom.step(steps)
    out = _state((dom, 3, len(parts["tet"])))
    dom.close()
    return out, used, len(parts["tet"]) // 3


@pytest.mark.parametrize("precision", (0, 1))
def test_one_set_of_lists_where_two_do_not_fit(lib, precision):
    """Down to the memory that one set needs: the arrays without the second set, and the staging of an upload."""
    from scdat_b200 import capi

    with faults() as flib:
        free, used, n = _run(precision, flib)
        second = ENTRY * (n + n // 4 + 2 * 4096)
        for budget in (used + 80 * n, used - second + 6 * 8 * n + 4096):
            flib.fault_budget(budget)
            short, less, _ = _run(precision, flib)
            assert less <= used - second
            _equal([short], [free])
        flib.fault_budget(used // 2)  # and where not even that fits, an error
        with pytest.raises(capi.ScdatError):
            _run(precision, flib)


def test_the_second_set_is_given_back_to_a_later_call(lib):
    from scdat_b200 import capi

    out, used, levels = [], [], []
    with faults() as flib:
        for tight in (False, True):
            dom, sp, n = _scenario((16, 16, 16), 3, 12)
            if tight:
                flib.fault_budget(used[0] - ENTRY * n // 4)
            dom.set_preconditioner(capi.PRECOND_MULTIGRID)
            used.append(flib.fault_used())
            flib.fault_budget(0)
            dom.step(2)
            levels.append(dom.solver_levels())
            out.append(_state((dom, sp, n)))
            dom.close()
    assert used[1] < used[0] - ENTRY * n // 4 and levels[0] == levels[1] and len(levels[0]) > 1
    _equal([out[1]], [out[0]])


def test_a_batch_needs_no_lists_of_its_own(lib):
    from scdat_b200 import capi

    with faults() as flib:
        dom, _, n = _scenario((10, 9, 8), 3, 16)
        before = flib.fault_used()
        b = capi.Batch([dom])
        b.step(2)
        assert flib.fault_used() - before < ENTRY * n // 8
        b.close()
        dom.close()
