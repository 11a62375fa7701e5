"""The persistent solve at the row counts and block counts where it changes kernels or has its edges, against 64-bit
residuals."""
import numpy as np
import pytest
import torch

from luisacomputesimulator_b200.linear import ConjugateGradientSolver, make_bsr
from tests.gpu_util import dev, host

pytestmark = pytest.mark.gpu


def _band(n, reach, rng):
    """Symmetric diagonally dominant blocks between rows up to `reach` apart (in a cycle), as (D, rp, col, val)."""
    D = np.tile(np.eye(3), (n, 1, 1))
    reach = min(reach, (n - 1) // 2)
    rows, cols, vals = [], [], []
    i = np.arange(n)
    for d in range(1, reach + 1):
        u = rng.normal(size=(n, 3))
        u /= np.linalg.norm(u, axis=1, keepdims=True)
        H = 2.0 * u[:, :, None] * u[:, None, :] + 0.1 * np.eye(3)
        j = (i + d) % n
        np.add.at(D, i, H)
        np.add.at(D, j, H)
        rows += [i, j]
        cols += [j, i]
        vals += [-H, -H]
    if not rows:
        return D, np.zeros(n + 1, np.int64), np.zeros(0, np.int64), np.zeros((0, 3, 3))
    r, c, v = np.concatenate(rows), np.concatenate(cols), np.concatenate(vals)
    o = np.lexsort((c, r))
    return D, np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]), c[o], v[o]


def _f32(D, val):
    d = np.zeros((len(D), 3, 4), np.float32)
    d[:, :, :3] = D.transpose(0, 2, 1)
    return d, np.ascontiguousarray(val.transpose(0, 2, 1)).reshape(-1).astype(np.float32)


def _apply(D, rp, col, val, x):
    y = np.einsum("nij,nj->ni", D, x)
    if len(col):
        r = np.repeat(np.arange(len(D)), np.diff(rp))
        np.add.at(y, r, np.einsum("kij,kj->ki", val, x[col]))
    return y


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("n,reach,as_b", [
    (1, 0, False), (2, 0, False), (63, 6, False), (65, 6, True),   # less than a block, one row more; contacts alone
    (150, 20, False),                                              # 40 blocks a row: beyond the ones held in registers
    (9472, 3, False), (9473, 3, False),                            # 64 and 128 rows per block on 148 SMs
    (18944, 3, False), (18945, 3, False), (30001, 9, False),       # the largest system of one row per four lanes; beyond
    (20000, 60, False),                                            # 120 blocks a row
    (20000, 56, False), (20000, 64, False),                        # a matrix below and beyond three quarters of L2
])
def test_persistent_solve_at_the_edges(n, reach, as_b, fp64):
    rng = np.random.default_rng(n)
    D, rp, col, val = _band(n, reach, rng)
    diag, v32 = _f32(D, val)
    b = np.zeros((n, 4), np.float32)
    b[:, :3] = rng.normal(size=(n, 3))
    M = make_bsr(n, dev(rp.astype(np.int32)), dev(col.astype(np.int32)), dev(v32)) if len(col) else None
    x = torch.full((n, 4), 3.0, dtype=torch.float32, device="cuda")
    st = ConjugateGradientSolver(n).device_solve(dev(diag), None if as_b else M, M if as_b else None, dev(b), x, max_iter=300,
                                                 rel_tol=1e-5, abs_rz_tol=0.0, check_every=1, fp64_dots=fp64)
    assert st["status"] == 0
    got = host(x)[:, :3].astype(np.float64)
    res = np.linalg.norm(b[:, :3] - _apply(D, rp, col, val, got)) / np.linalg.norm(b[:, :3])
    # the recurrence stops at 1e-5; it leaves the true residual by a few roundings of A x per iteration, |A| |x| / |b|
    # being at most the condition number, here (1 + 4.2 * 2 * reach) / 1
    assert res <= 1e-5 + 4 * 2.0 ** -24 * np.sqrt(max(st["iterations"], 1)) * (1 + 8.4 * reach), (res, st)
