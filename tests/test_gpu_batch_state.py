"""A batch whose contexts are changed between its steps."""
import numpy as np
import pytest

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
