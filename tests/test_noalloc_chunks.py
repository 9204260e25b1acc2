"""The 3D allocation-free CG on systems too large for one cluster (lpm-cpp_b200/csrc/cg.cu:
k_cg_bsr_chunks), which takes a row 32 blocks at a time and copies values 16 bytes at a time.

Rows of one block, around one and two chunks (31, 33, 63 and 65 blocks inside the band, all lengths below
near its ends and where pairs are left out), with the values' address a multiple of 16 or of 8 bytes only.
The oracle is the residual b - A x in numpy: the CG stops at 1e-13 of b, and its recursion stays within a
few hundred roundings of the true residual, so the bar is 1e-12."""
import ctypes as C

import numpy as np
import pytest

from _util import LPM

pytestmark = pytest.mark.gpu


def _band(n, half, seed):
    """Upper pairs (i, j, block) of a symmetric band matrix of 2 half + 1 blocks a row, one in 20 left out."""
    rng = np.random.default_rng(seed)
    i = np.repeat(np.arange(n), half)
    j = i + np.tile(np.arange(1, half + 1), n)
    keep = (j < n) & (rng.random(len(i)) > 0.05)
    i, j = i[keep], j[keep]
    up = rng.standard_normal((len(i), 3, 3))
    diag = np.zeros((n, 3))
    np.add.at(diag, i, np.abs(up).sum(2))
    np.add.at(diag, j, np.abs(up).sum(1))
    d = np.zeros((n, 3, 3))
    d[:, [0, 1, 2], [0, 1, 2]] = diag * 1.05 + 1.0
    rows, cols = np.concatenate([i, j, np.arange(n)]), np.concatenate([j, i, np.arange(n)])
    val = np.concatenate([up, up.transpose(0, 2, 1), d])
    order = np.lexsort((cols, rows))
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32)
    return rowptr, cols[order].astype(np.int32), np.ascontiguousarray(val[order]), rows[order], rng.standard_normal(n * 3)


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("n,half", [(61001, 0), (2003, 15), (1901, 16), (1201, 31), (1103, 32)])
def test_chunked_rows(n, half, shift):
    import torch
    rowptr, col, val, rows, b = _band(n, half, n + shift)
    held = torch.zeros(val.size + 2, dtype=torch.float64, device="cuda")
    values = held[shift:shift + val.size]
    values.copy_(torch.from_numpy(val.reshape(-1)))
    d = [torch.from_numpy(a).cuda() for a in (rowptr, col)] + [values, torch.from_numpy(b).cuda()]
    x = torch.full((n * 3,), 3.0, dtype=torch.float64, device="cuda")
    it = C.c_int64(-1)
    status = LPM.lib().lpmgpu_cg_bsr_noalloc(3, n, *[C.c_void_p(a.data_ptr()) for a in (*d, x)], 1e-26, 0.0, 10000, None,
                                             C.byref(it))
    assert status == LPM.OK and it.value > 0
    xs = x.cpu().numpy().reshape(n, 3)
    ax = np.zeros((n, 3))
    np.add.at(ax, rows, np.einsum("kab,kb->ka", val, xs[col]))
    assert np.linalg.norm(ax.reshape(-1) - b) <= 1e-12 * np.linalg.norm(b)
