"""A batch whose contexts are changed between its steps."""
import numpy as np
import pytest

from faults import faults
from test_gpu_batch_bits import _equal, _scenario, _state

pytestmark = pytest.mark.gpu


def test_step_after_a_compaction_is_bitwise_the_settled_store_s(lib):
    """scdat_compact leaves the re-sort's gather to the next reader, here the batch's step, which has to
    wait for it; reading the particles first settles the store."""
    from scdat_b200 import capi

    out = []
    for settle in (False, True):
        doms = [_scenario((16, 15, 14), k, 16) for k in range(3)]
        b = capi.Batch([d[0] for d in doms])
        b.step(1)
        for _ in range(3):
            for dom, sp, _ in doms:
                dom.compact()
                if settle:
                    [dom.get_particles(s) for s in range(sp)]
            b.step(1)
        out.append([_state(d) for d in doms])
        b.close()
        for d in doms:
            d[0].close()
    _equal(out[0], out[1])


def test_a_larger_population_between_steps(lib):
    """A context of the batch gets four times the particles, which the null collision defers whole on
    their first push: the batch's lists grow with them.  Bitwise the context alone."""
    from scdat_b200 import capi

    out = []
    for batched in (False, True):
        dom, sp, _ = _scenario((10, 9, 8), 3, 2)
        b = capi.Batch([dom]) if batched else None
        step = b.step if batched else dom.step
        step(1)
        large, _, n = _scenario((10, 9, 8), 4, 16)
        for s in range(sp):
            p = large.get_particles(s)
            dom.set_particles(s, p["x"], p["v"], p["tet"], p["id"])
            dom.set_elastic(s, 1e18, 1e-19, mode=2)
        large.close()
        step(2)
        out.append(_state((dom, sp, n)))
        if b:
            b.close()
        dom.close()
    _equal([out[1]], [out[0]])


def test_a_wait_that_runs_out_in_an_earlier_step_is_reported(lib):
    """The first step's solve lacks a block, so the last scenario's others give up their wait (some
    seconds) and its potential is void; the second step's solve is whole.  The call has to fail, every
    context has to count both steps, and the batch stays failed."""
    from scdat_b200 import capi

    with faults() as flib:
        doms = [_scenario(c, 8, 2) for c in ((6, 6, 6), (7, 8, 6), (12, 11, 10))]
        b = capi.Batch([d[0] for d in doms], use_graph=False)
        flib.fault_launches(0, 1)
        with pytest.raises(capi.ScdatError, match="wait ran out"):
            b.step(2)
        assert flib.fault_calls() == 2
        assert [d[0].stats()["completed_steps"] for d in doms] == [2, 2, 2]
        with pytest.raises(capi.ScdatError, match="wait ran out"):
            b.step(1)
        # the others' particles are counted after the re-sort of step 2, and new ones are taken as given
        for dom, sp, n in doms[:2]:
            assert sum(len(dom.get_particles(s)["id"]) for s in range(sp)) <= n
        b.close()
        for d in doms:
            d[0].close()
