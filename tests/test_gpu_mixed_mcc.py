"""The precision form's null collisions over several steps against the oracle's FP64 run in the reference's
order, on the same Philox streams: the same collisions, survivors and ledger counts; states and fields to
the precision form's error budget of 1e-5.  A decision differs only where a random number lies within
FP32 rounding (1e-7) of its threshold: 1e-3 of a chance in these 3000 draws."""
import numpy as np
import pytest

import oracle as O
from conftest import rel_err
from pic_helpers import gpu_domain, gpu_load_particles, gpu_state, oracle_mcc_run

pytestmark = pytest.mark.gpu


def test_null_collisions_match_the_oracle(lib, orc):
    mesh = O.kuhn_box((4, 4, 4), 0.05)
    sp = O.plasma_species(1e10, 1.0, 1.0, 0.05, 6)
    parts = O.seed_particles(mesh, sp, 6, 33)
    dt, n_t, sigma, seed, nsteps, face_bc = 2e-8, 4e20, 1e-19, 777, 4, (1,) * 6
    ref = oracle_mcc_run(orc, mesh, sp, parts, nsteps, dt, face_bc, n_t, sigma, seed, mode=2)
    dom = gpu_domain(mesh, dt, face_bc=face_bc, precision=1, pcg_rtol=1e-10, pcg_max_iter=20000, body_tally=False, seed=seed)
    gpu_load_particles(dom, sp, parts)
    for s in range(len(sp)):
        dom.set_elastic(s, n_t, sigma, mode=2)
    dom.set_potential(mesh.phi_bc)
    dom.step(nsteps)
    st = gpu_state(dom, len(sp), len(parts["tet"]))
    stats, led = dom.stats(), dom.ledger()
    _, phi, _ = dom.fields()
    dom.close()
    assert stats["mcc_collisions"] == ref["hits"] and ref["hits"] > 100
    ids = ref["parts"]["id"]
    assert np.array_equal(np.sort(np.nonzero(st["status"] == O.ACTIVE)[0]), np.sort(ids))
    assert np.array_equal(led[:6, 4:6], ref["ledger"][:6, 4:6])
    assert np.abs(st["x"][ids] - ref["parts"]["x"]).max() <= 1e-5 * np.abs(ref["parts"]["x"]).max()
    assert rel_err(st["v"][ids], ref["parts"]["v"]) < 1e-5
    assert rel_err(phi, ref["phi"]) < 1e-5
