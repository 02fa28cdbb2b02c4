"""Passes 2 and 3 over lists around what one round of their warps takes (148 SMs: 592 blocks of 8
warps of 32 entries, FP64 296 blocks): one entry, a warp and one more, the last list taken in one
round, the first taken in chunks and capped.  No particle has a location hint, so pass 1 puts all of
them in the list; some need many sub-steps.  Particles do not meet, so each has the same bits in
every list it is part of; the longest list, in chunks, is compared with all others."""
import functools

import numpy as np
import pytest

import oracle as O
from pic_helpers import gpu_domain, gpu_state

pytestmark = pytest.mark.gpu
H, DT, LONGEST = 0.05, 2e-8, 592 * 256 + 1


@functools.lru_cache(maxsize=None)
def _population():
    mesh = O.kuhn_box((6, 7, 5), H, body=((2, 4), (2, 4), (1, 3)), bias=-25.0)
    sp = O.plasma_species(1e10, 1.0, 1.0, H, 400)
    parts = O.seed_particles(mesh, sp, 400, 5)
    rng = np.random.default_rng(3)
    idx = rng.permutation(len(parts["tet"]))[:LONGEST]
    assert len(idx) == LONGEST
    return mesh, sp, parts["x"][idx], parts["v"][idx] * np.exp(rng.uniform(-2, 5, LONGEST))[:, None]


def _push(precision, n, batch=False):
    from scdat_b200 import capi

    mesh, sp, x, v = _population()
    dom = gpu_domain(mesh, DT, face_bc=(2,) * 6, precision=precision)
    dom.set_species(sp)
    dom.set_electric_field(np.random.default_rng(1).standard_normal((mesh.N, 3)) * 10.0)
    dom.set_particles(0, x[:n], v[:n], np.full(n, -1, np.int32), np.arange(n, dtype=np.uint32))
    if batch:
        b = capi.Batch([dom])
        b.step(1)
        b.close()
    else:
        dom.push()
    out = gpu_state(dom, 1, n)
    substeps = dom.stats()["substeps"]
    dom.close()
    return out, substeps


@functools.lru_cache(maxsize=None)
def _longest(precision):
    return _push(precision, LONGEST)


@pytest.mark.parametrize("precision,batch", ((0, False), (1, False), (1, True)))
@pytest.mark.parametrize("n", (1, 33, 296 * 256, 296 * 256 + 1, 592 * 256, LONGEST))
def test_the_length_of_the_list_does_not_matter(lib, precision, batch, n):
    ref, substeps = _longest(precision)
    assert substeps > 3 * LONGEST and (ref["status"] == O.ACTIVE).any() and (ref["status"] != O.ACTIVE).any()
    got, s2 = _push(precision, n, batch)
    for k in ("x", "v", "tet", "status"):
        assert np.array_equal(got[k], ref[k][:n], equal_nan=k in "xv"), k
    if n == LONGEST:
        assert s2 == substeps
