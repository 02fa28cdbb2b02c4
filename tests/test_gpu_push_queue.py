"""Pass 1's walking form (particles that leave their tet wait in their warp's queue and walk 32 at a
time) against the stay-first form, whose leavers run the sub-step loop of the later passes, and
against a one-scenario batch: the same particles, charge, ledger and collisions to the bit, for
populations around a warp, a full queue and a run of chunks, with particles that stay, walk, cross the
box, hit the body, leave through every kind of face, start without a location hint or need many
sub-steps, and with every collision mode."""
import numpy as np
import pytest

import oracle as O
from conftest import rel_err
from pic_helpers import gpu_domain, gpu_load_particles, gpu_state, oracle_cycle

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


@pytest.mark.parametrize("count", (1, 31, 33, 64, 95, 257, 3000))
@pytest.mark.parametrize("bc,kernel,nseg", ((2, 1, 10), (1, 0, 10), (0, 2, 3), (1, 1, 1), (2, 1, 37)))
def test_fp64_pass_1_against_the_oracle(lib, count, bc, kernel, nseg):
    """The FP64 form's pass 1 has the same queue; its oracle is the reference's push restated.  The
    bar is the parity tests': 1e-12 relative, the discrete outcomes exact.  The closed-form segment
    cloud is checked with one, few and many sample points."""
    o = O.Oracle(fast_locate=True)
    mesh = O.kuhn_box((6, 7, 5), H, body=((2, 4), (2, 4), (1, 3)), bias=-25.0)
    sp = O.plasma_species(1e10, 1.0, 1.0, H, 40)
    parts = O.seed_particles(mesh, sp, 40, 5)
    rng = np.random.default_rng(count)
    idx = rng.permutation(len(parts["tet"]))[:count]
    parts = {k: (v[idx] if isinstance(v, np.ndarray) and len(v) == len(parts["tet"]) else v) for k, v in parts.items()}
    m = len(parts["tet"])
    parts["id"] = np.arange(m).astype(parts["id"].dtype)
    parts["v"] = parts["v"] * np.exp(rng.uniform(-6, 2, m))[:, None] * np.where(parts["species"] == 0, 1.0, 40.0)[:, None]
    parts["tet"] = np.where(rng.random(m) < 0.06, -1, parts["tet"]).astype(np.int32)
    E = rng.standard_normal((mesh.N, 3)) * 30.0
    out = o.push(mesh, E, parts, sp, DT, nseg=nseg, kernel=kernel)
    L = mesh.xyz.max(axis=0) - mesh.xyz.min(axis=0)
    ref = o.boundary(mesh, out, parts, sp, (bc,) * 6, period=tuple(L) if bc == 2 else (0.0,) * 3, body_tally=True)
    dom = gpu_domain(mesh, DT, face_bc=(bc,) * 6, deposit_kernel=kernel, deposit_segments=nseg)
    gpu_load_particles(dom, sp, parts)
    dom.set_electric_field(E)
    dom.push()
    got = gpu_state(dom, len(sp), m)
    rho, led, st = dom.fields()[0], dom.ledger(), dom.stats()
    dom.close()
    assert st["substeps"] == out["substeps"]
    assert np.array_equal(got["status"], ref["status"])
    act = ref["status"] == O.ACTIVE
    if act.any():
        assert rel_err(got["x"][act], ref["x"][act]) < 1e-12 and rel_err(got["v"][act], ref["v"][act]) < 1e-12
        assert np.array_equal(got["tet"][act], ref["tet"][act])
    assert rel_err(rho, out["rho"]) < 1e-12
    assert np.array_equal(led[:, 4:6], ref["ledger"][:, 4:6])
