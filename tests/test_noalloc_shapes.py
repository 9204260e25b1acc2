"""The allocation-free CG (lpmgpu_cg_bsr_noalloc) on block-CSR systems of other shapes than a lattice's.

Rows of one block, rows around the widths that a warp takes at once (8 and 32 blocks in 2D, 3 and 12 in
3D), one row, and row counts around a block's 32 rows.  The oracle is numpy's dense solve.  The CG stops
at a residual of 1e-13 of b, so its solution is off by at most the condition number (below 1e3 here, by
the diagonal's dominance) times that; the bar is 1e-9."""
import ctypes as C

import numpy as np
import pytest

from _util import LPM, rel

pytestmark = pytest.mark.gpu


def _system(dim, n, width, seed):
    """A symmetric block matrix with up to about `width` blocks a row, diagonally dominant."""
    rng = np.random.default_rng(seed)
    A = np.zeros((n, n, dim, dim))
    for i in range(n):
        for j in rng.choice(n, size=min(n, max(1, width // 2)), replace=False):
            b = rng.standard_normal((dim, dim))
            A[i, j] += b
            A[j, i] += b.T
    full = A.transpose(0, 2, 1, 3).reshape(n * dim, n * dim)
    full += np.diag(np.abs(full).sum(1) * 1.05 + 1.0)
    A = full.reshape(n, dim, n, dim).transpose(0, 2, 1, 3)
    has = np.abs(A).sum((2, 3)) > 0
    rowptr = np.concatenate([[0], np.cumsum(has.sum(1))]).astype(np.int32)
    col = np.concatenate([np.nonzero(h)[0] for h in has]).astype(np.int32)
    val = A[has]
    return full, rowptr, col, np.ascontiguousarray(val.reshape(-1)), rng.standard_normal(n * dim)


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n,width", [(1, 1), (31, 1), (32, 3), (33, 9), (64, 26), (65, 50), (300, 70), (500, 300)])
def test_shapes(dim, n, width):
    import torch
    full, rowptr, col, val, b = _system(dim, n, width, 7 * n + dim)
    d = [torch.from_numpy(a).cuda() for a in (rowptr, col, val, b)]
    x = torch.full((n * dim,), 3.0, dtype=torch.float64, device="cuda")
    it = C.c_int64(-1)
    status = LPM.lib().lpmgpu_cg_bsr_noalloc(dim, n, *[C.c_void_p(a.data_ptr()) for a in (*d, x)], 1e-26, 0.0, 10000,
                                             None, C.byref(it))
    assert status == LPM.OK and it.value > 0
    assert rel(x.cpu().numpy(), np.linalg.solve(full, b)) <= 1e-9
