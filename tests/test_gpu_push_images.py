"""Periodic images against the oracle: particles that leave a periodic box far from where they
re-enter it, with images in tet interiors, on shared faces, edges and vertices (where the search
order decides) and in the body hole, for populations around the sizes of a warp, a block and a run
of chunks.  Cell edge, time step and displacements are dyadic, so positions are exact and every
outcome has to be the oracle's: the same tet, the same status, the same position to the bit."""
import numpy as np
import pytest

import oracle as O
from pic_helpers import gpu_domain, gpu_load_particles, gpu_state, oracle_cycle

pytestmark = pytest.mark.gpu
H, DT = 2.0 ** -4, 2.0 ** -20


@pytest.mark.parametrize("neighbors", (True, False))
@pytest.mark.parametrize("count", (1, 31, 33, 257, 5000))
def test_images_land_where_the_oracle_puts_them(lib, count, neighbors):
    o = O.Oracle(fast_locate=True)
    n = (6, 5, 8)
    mesh = O.kuhn_box(n, H, body=((2, 4), (2, 3), (3, 5)))
    sp = O.plasma_species(1e10, 1.0, 1.0, H, 2)
    parts = O.seed_particles(mesh, sp, 1 + count // 100, 77)
    rng = np.random.default_rng(count)
    idx = rng.permutation(len(parts["tet"]))[:count]
    parts = {k: (v[idx] if isinstance(v, np.ndarray) and len(v) == len(parts["tet"]) else v) for k, v in parts.items()}
    m = len(parts["tet"])
    parts["id"] = np.arange(m).astype(parts["id"].dtype)
    parts["x"] = np.round(parts["x"] / H * 64) * H / 64 + H / 256  # dyadic, still near the seeded tet
    parts["tet"] = np.array([o.locate(mesh, p) for p in parts["x"]], np.int32)
    L = np.array(n) * H
    fine = rng.integers(0, 2 * np.array(n) * 4, (m, 3)) / 8.0  # eighths of a cell: ties among them
    fine[::2] = np.round(fine[::2] * 2) / 2                    # half of them on vertices and edge midpoints
    wraps = rng.integers(-2, 3, (m, 3))
    wraps[np.all(wraps == 0, axis=1), 0] = 1
    target = fine * H + wraps * L
    parts["v"] = (target - parts["x"]) / DT
    ref = oracle_cycle(o, mesh, sp, parts, 1, DT, (2,) * 6, np.zeros(mesh.N), neighbors=neighbors, body_tally=True)
    dom = gpu_domain(mesh, DT, face_bc=(2,) * 6, neighbors=neighbors)
    gpu_load_particles(dom, sp, parts)
    dom.set_potential(np.zeros(mesh.N))
    dom.push()
    got = gpu_state(dom, len(sp), m)
    led = dom.ledger()
    dom.close()
    assert np.array_equal(got["status"], ref["status"])
    act = ref["status"] == O.ACTIVE
    assert count < 100 or (act.any() and (~act).any())
    assert np.array_equal(got["x"][act], ref["x"][act])
    assert np.array_equal(got["tet"][act], ref["tet"][act])
    assert np.array_equal(led[:, 4:6], ref["ledger"][:, 4:6])
