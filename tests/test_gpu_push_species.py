"""A push zeroes all it accumulates into in one launch and runs the species in two chains: with one to
five species of the same particles, an empty one among them, each gives the same charge, particles
and lists to the bit, push after push."""
import numpy as np
import pytest

import oracle as O
from pic_helpers import gpu_domain

pytestmark = pytest.mark.gpu
H, DT = 0.05, 2e-8


@pytest.mark.parametrize("precision", (0, 1))
@pytest.mark.parametrize("species", (1, 2, 3, 5))
def test_every_species_of_the_same_particles_gives_the_same(lib, precision, species):
    mesh = O.kuhn_box((6, 7, 5), H, body=((2, 4), (2, 4), (1, 3)), bias=-25.0)
    sp = O.plasma_species(1e10, 1.0, 1.0, H, 40)
    parts = O.seed_particles(mesh, sp, 40, 5)
    idx = np.nonzero(parts["species"] == 0)[0][:3000]
    tet = parts["tet"][idx].astype(np.int32)
    tet[::9] = -1
    dom = gpu_domain(mesh, DT, face_bc=(2,) * 6, precision=precision)
    dom.set_species([sp[0]] * species)
    dom.set_electric_field(np.random.default_rng(1).standard_normal((mesh.N, 3)) * 10.0)
    empty = 2 if species == 5 else -1
    for s in range(species):
        if s != empty:
            dom.set_particles(s, parts["x"][idx], 3.0 * parts["v"][idx], tet, np.arange(len(idx), dtype=np.uint32))
    charges = []
    for k in range(3):
        dom.push()
        q = [dom.species_charge(s) for s in range(species)]
        got = [dom.get_particles(s) for s in range(species)]
        assert np.abs(q[0]).sum() > 0
        for s in range(species):
            assert np.array_equal(q[s], np.zeros(mesh.N) if s == empty else q[0]), (k, s)
            if s != empty:
                assert all(np.array_equal(got[s][c], got[0][c]) for c in ("x", "v", "tet", "status", "id")), (k, s)
        charges.append(q[0])
    assert not np.array_equal(charges[0], charges[2])
    dom.close()
