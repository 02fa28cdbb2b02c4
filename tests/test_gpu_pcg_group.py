"""The one-launch Jacobi-CG at the edges of its launch shapes: one row, a block's rows and one more (256 or 512),
one block per SM (148 x 256, 148 x 512) and one row more, two to four rows a thread, its largest
system and the first of the two-launch form; rows without entries and rows longer than the part of
the matrix that shared memory keeps.  Oracle: the solution the right-hand side was made from, in
FP64 on the host.  The matrices are diagonally dominant (Gershgorin: condition number under 4), so
a relative residual of 1e-13 bounds the relative error by 4e-13."""
import numpy as np
import pytest

from pic_helpers import pcg_csr_on_device

pytestmark = pytest.mark.gpu
SM = 148


def _system(R, rng):
    """Symmetric CSR: a chain, long-range pairs, one hub with up to 40 neighbours, some empty rows."""
    i = np.arange(R - 1)
    keep = rng.random(R - 1) < 0.8
    pairs = [np.stack([i[keep], i[keep] + 1], 1)]
    for off in (7, 61, 1021):
        if R > off:
            k = np.arange(0, R - off, 3)
            pairs.append(np.stack([k, k + off], 1))
    if R > 64:
        pairs.append(np.stack([np.full(40, R // 2), rng.permutation(np.setdiff1d(np.arange(R)[:4096], [R // 2]))[:40]], 1))
    p = np.unique(np.sort(np.concatenate(pairs), axis=1), axis=0) if R > 1 else np.zeros((0, 2), int)
    w = -rng.random(len(p))
    rows, cols, vals = np.concatenate([p[:, 0], p[:, 1]]), np.concatenate([p[:, 1], p[:, 0]]), np.concatenate([w, w])
    order = np.lexsort((cols, rows))
    rows, cols, vals = rows[order], cols[order], vals[order]
    ptr = np.zeros(R + 1, np.int64)
    np.add.at(ptr, rows + 1, 1)
    diag = 1.0 + 2.0 * np.bincount(rows, -vals, R)
    return np.cumsum(ptr).astype(np.int32), cols.astype(np.int32), vals, diag, rows


@pytest.mark.parametrize("R", (1, 2, 255, 256, 257, 512, 513, 4097, SM * 256, SM * 256 + 1, SM * 512 + 1, SM * 1024 + 1,
                               SM * 1536 + 1, SM * 2048, SM * 2048 + 1))
def test_solution_at_the_edges_of_the_launch_shapes(lib, R):
    rng = np.random.default_rng(R)
    ptr, col, val, diag, rows = _system(R, rng)
    x = rng.standard_normal(R)
    b = diag * x + np.bincount(rows, val * x[col], R)
    if len(col) == 0:
        col, val = np.zeros(1, np.int32), np.zeros(1)
    rc, got, it, rel = pcg_csr_on_device(lib.scdat_pcg_csr, ptr, col, val, diag, b, np.zeros(R), 1e-13, 500)
    assert rc == 0 and rel <= 1e-13 and it > 0
    assert np.linalg.norm(got - x) <= 4e-13 * np.linalg.norm(x)
    if R <= 1 << 18:
        rc, again, it2, _ = pcg_csr_on_device(lib.scdat_pcg_csr_noalloc, ptr, col, val, diag, b, np.zeros(R), 1e-13, 500)
        assert rc == 0 and it2 == it and np.array_equal(again, got)
    rc, _, it3, rel3 = pcg_csr_on_device(lib.scdat_pcg_csr, ptr, col, val, diag, b, np.zeros(R), 1e-13, 1)
    assert it3 == 1 and (rc == -5) == (rel3 > 1e-13)
