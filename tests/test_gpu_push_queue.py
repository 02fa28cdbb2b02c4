"""Pass 1's walking form (particles that leave their tet wait in their warp's queue and walk 32 at a
time) against the stay-first form, whose leavers run the sub-step loop of the later passes, and
against a one-scenario batch: the same particles, charge, ledger and collisions to the bit, for
populations around a warp, a full queue and a run of chunks, with particles that stay, walk, cross the
box, hit the body, leave through every kind of face, start without a location hint or need many
sub-steps, and with every collision mode."""
import numpy as np
import pytest

import oracle as O
from pic_helpers import gpu_domain

pytestmark = pytest.mark.gpu
H, DT = 0.05, 2e-8


def _run(route, count, bc, mode, kernel):
    from scdat_b200 import capi

    mesh = O.kuhn_box((6, 7, 5), H, body=((2, 4), (2, 4), (1, 3)), bias=-25.0)
    sp = O.plasma_species(1e10, 1.0, 1.0, H, 40)
    parts = O.seed_particles(mesh, sp, 40, 5)
    dom = gpu_domain(mesh, DT, face_bc=(bc,) * 6, precision=1, pcg_rtol=1e-10, deposit_kernel=kernel)
    dom.set_species(sp)
    rng = np.random.default_rng(count)
    for s in range(len(sp)):
        idx = np.nonzero(parts["species"] == s)[0]
        idx = rng.permutation(idx)[:count]
        v = parts["v"][idx] * np.exp(rng.uniform(-6, 2, len(idx)))[:, None] * (1.0 if s == 0 else 40.0)
        tet = parts["tet"][idx].astype(np.int32)
        tet[::17] = -1
        dom.set_particles(s, parts["x"][idx], v, tet, np.arange(len(idx), dtype=np.uint32) + 7)
        if mode >= 0:
            dom.set_elastic(s, 4e20, 1e-19, mode=mode)
        dom.set_push_mode(s, capi.PUSH_STAY_FIRST if route == "stay" else capi.PUSH_WALKING)
    dom.set_potential(mesh.phi_bc)
    dom.solve_field()
    b = capi.Batch([dom]) if route == "batch" else None
    (b or dom).step(2)
    out = [dom.get_particles(s) for s in range(len(sp))]
    fields = dom.fields()
    st = dom.stats()
    counts = {k: st[k] for k in ("substeps", "lost_events", "mcc_collisions", "active_particles", "total_energy")}
    led = dom.ledger()
    if b:
        b.close()
    dom.close()
    return out, fields, counts, led


@pytest.mark.parametrize("count", (1, 31, 33, 64, 95, 257, 3000))
@pytest.mark.parametrize("bc,mode,kernel", ((2, 2, 1), (1, 0, 0), (0, 1, 2), (2, -1, 1)))
def test_every_route_gives_the_same_bits(lib, count, bc, mode, kernel):
    ref, fields, counts, led = _run("walking", count, bc, mode, kernel)
    assert counts["substeps"] > 0
    if count >= 257:
        assert counts["lost_events"] > 0 and (mode < 0) == (counts["mcc_collisions"] == 0)
    for route in ("stay", "batch"):
        got, f2, c2, l2 = _run(route, count, bc, mode, kernel)
        assert c2 == counts, route
        assert np.array_equal(l2, led), route
        assert all(np.array_equal(a, b) for a, b in zip(f2, fields)), route
        for g, r in zip(got, ref):
            assert all(np.array_equal(g[k], r[k]) for k in ("x", "v", "tet", "status", "id")), route
