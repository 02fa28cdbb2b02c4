"""The one-launch field solve gives the bits of the launched form: every dot product is summed in the
same order, whatever the launch shape.  A batch of more scenarios than SMs takes the launched loops (one
launch per kernel); the same scenario alone, and in a batch that fits the SMs, takes one launch.  The
steps' charge, potential, field, ledger and particles have to be equal, bit for bit."""
import numpy as np
import pytest

import oracle as O
from pic_helpers import gpu_domain, gpu_load_particles, gpu_state

pytestmark = pytest.mark.gpu
SM = 148


def _scenario(cells, seed, ppc=2, body=True):
    h = 0.05
    box = tuple((c // 3, c // 3 + max(1, c // 4)) for c in cells) if body else None
    mesh = O.kuhn_box(cells, h, body=box, bias=-15.0 if body else 0.0)
    sp = O.plasma_species(1e10, 1.0, 1.0, h, ppc)
    parts = O.seed_particles(mesh, sp, ppc, seed)
    dom = gpu_domain(mesh, 2e-8, face_bc=(2, 2, 2, 2, 1, 1), precision=1, pcg_rtol=1e-10, sort_interval=2)
    gpu_load_particles(dom, sp, parts)
    dom.set_potential(mesh.phi_bc)
    return dom, len(sp), len(parts["tet"])


def _state(s):
    dom, sp, n = s
    rho, phi, E = dom.fields()
    return dict(rho=rho, phi=phi, E=E, ledger=dom.ledger(), **gpu_state(dom, sp, n))


def _alone(args, steps):
    out = []
    for a in args:
        s = _scenario(*a)
        s[0].step(steps)
        out.append(_state(s))
        s[0].close()
    return out


def _batched(args, steps, extra=0, **kw):
    from scdat_b200 import capi

    doms = [_scenario(*a) for a in args] + [_scenario((2, 2, 2), 100 + k, 1, False) for k in range(extra)]
    b = capi.Batch([d[0] for d in doms], **kw)
    try:
        b.step(steps)
        return [_state(s) for s in doms[: len(args)]]
    finally:
        b.close()
        for d in doms:
            d[0].close()


def _equal(got, want):
    for g, w in zip(got, want):
        for key, v in w.items():
            assert np.array_equal(np.nan_to_num(g[key]), np.nan_to_num(v)), key


# rows: under a block of 256, up to 512 (one block, two virtual ones), several blocks
SMALL = [((6, 7, 6), 1), ((8, 8, 9), 2), ((13, 9, 10), 3), ((17, 12, 11), 4)]


@pytest.mark.parametrize("use_graph", (True, False))
def test_launched_loops_and_one_launch_give_the_same_bits(lib, use_graph):
    alone = _alone(SMALL, 3)
    _equal(_batched(SMALL, 3, use_graph=use_graph), alone)
    _equal(_batched(SMALL, 3, extra=SM, use_graph=use_graph), alone)


@pytest.mark.parametrize("cells", [((40, 40, 40), (35, 37, 36)), ((40, 40, 40),) * 3, ((44, 42, 40),) * 3 + ((30, 30, 30),)])
def test_several_rows_a_thread_give_the_bits_of_one(lib, cells):
    """Two, three and four rows a thread in the batch, one in each scenario's own solve."""
    args = [(c, 10 + k, 1) for k, c in enumerate(cells)]
    _equal(_batched(args, 2), _alone(args, 2))
