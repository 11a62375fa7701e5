"""Batched PCG at the row counts, block counts and alignments where its slices, chunks and copies have their edges,
against dense 64-bit solutions."""
import numpy as np
import pytest
import torch

from luisacomputesimulator_b200.linear import ConjugateGradientSolver, make_bsr, solve_batch
from tests.gpu_util import dev, host

pytestmark = pytest.mark.gpu


def _system(n, per_row, rng, long_row=False):
    """Diagonally dominant symmetric blocks; per_row off-diagonal blocks in expectation, some rows without any."""
    D = np.zeros((n, 3, 3))
    pairs = set()
    for i in range(n):
        for j in rng.integers(0, n, rng.integers(0, per_row + 1)):
            if i != j:
                pairs.add((min(i, j), max(i, j)))
        if long_row and n > 1 and i > 0:
            pairs.add((0, i))
    rows, cols, vals = [], [], []
    for i, j in sorted(pairs):
        u = rng.normal(size=3)
        u /= np.linalg.norm(u)
        H = np.outer(u, u) + 0.1 * np.eye(3)
        D[i] += H
        D[j] += H
        rows += [i, j]
        cols += [j, i]
        vals += [-H, -H]
    D += np.eye(3)
    order = np.lexsort((cols, rows)) if rows else np.zeros(0, int)
    rp = np.zeros(n + 1, np.int64)
    np.add.at(rp, np.asarray(rows, int) + 1, 1)
    return (D, np.cumsum(rp), np.asarray(cols, int)[order], np.asarray(vals).reshape(-1, 3, 3)[order],
            rng.normal(size=(n, 3)))


def _dense(sys_):
    D, rp, col, val, _ = sys_
    n = D.shape[0]
    M = np.zeros((3 * n, 3 * n))
    for i in range(n):
        M[3 * i:3 * i + 3, 3 * i:3 * i + 3] = D[i]
        for k in range(rp[i], rp[i + 1]):
            M[3 * i:3 * i + 3, 3 * col[k]:3 * col[k] + 3] += val[k]
    return M


def _offset_copy(t, words):
    """The tensor at an address `words` 4-byte words past a 16-byte boundary."""
    buf = torch.zeros(t.numel() + 4, dtype=t.dtype, device="cuda")
    out = buf[words:words + t.numel()]
    out.copy_(t.reshape(-1))
    return out


@pytest.mark.parametrize("cluster", [0, 1, 4, 16])
@pytest.mark.parametrize("sizes,per_row,long_row,as_b,shift", [
    ([1, 31, 32, 33], 3, False, False, 0),         # parts of one slice; runs that end a matrix off a 16-byte boundary
    ([255, 256, 257, 513], 12, False, False, 0),   # edges of a chunk
    ([640, 1300], 12, True, False, 0),             # a row of many windows, cut between them
    ([700, 90], 9, False, False, 1),               # arrays off a 16-byte boundary: read directly
    ([600, 300], 9, True, True, 0),                # everything in the contact matrix, none in the other
])
def test_batched_solves_at_the_edges(sizes, per_row, long_row, as_b, shift, cluster):
    rng = np.random.default_rng(7 + len(sizes))
    systems = [_system(n, per_row, rng, long_row) for n in sizes]
    off = np.concatenate([[0], np.cumsum(sizes)])
    n = int(off[-1])
    diag = np.zeros((n, 3, 4), np.float32)
    diag[:, :, :3] = np.concatenate([s[0] for s in systems]).transpose(0, 2, 1)
    nnz = np.concatenate([[0], np.cumsum([len(s[2]) for s in systems])])
    rp = np.concatenate([s[1][:-1] + o for s, o in zip(systems, nnz)] + [nnz[-1:]]).astype(np.uint32)
    col = np.concatenate([s[2] + o for s, o in zip(systems, off)]).astype(np.uint32)
    val = np.concatenate([s[3] for s in systems]).transpose(0, 2, 1).reshape(-1).astype(np.float32)
    b = np.zeros((n, 4), np.float32)
    b[:, :3] = np.concatenate([s[4] for s in systems])
    d_col, d_val = dev(col.view(np.int32)), dev(val)
    if shift:
        d_col, d_val = _offset_copy(d_col, shift), _offset_copy(d_val, shift)
    M = make_bsr(n, dev(rp.view(np.int32)), d_col, d_val)
    x = torch.full((n, 4), 5.0, dtype=torch.float32, device="cuda")
    stats = torch.zeros((len(sizes), 4), dtype=torch.int32, device="cuda")
    solve_batch(ConjugateGradientSolver(n), dev(off.astype(np.int32)), dev(diag), None if as_b else M, M if as_b else None,
                dev(b), x, stats, max_iter=400, rel_tol=1e-6, abs_rz_tol=0.0, cluster=cluster)
    torch.cuda.synchronize()
    assert (host(stats)[:, 3] == 0).all()
    got = host(x)[:, :3].astype(np.float64)
    for s, lo, hi in zip(systems, off[:-1], off[1:]):
        Ms = _dense(s)
        want = np.linalg.solve(Ms, s[4].reshape(-1))
        err = np.linalg.norm(got[lo:hi].reshape(-1) - want) / np.linalg.norm(want)
        # |dx| / |x| <= cond(M) times the residual's 1e-6 and the 32-bit rounding of the blocks
        assert err <= np.linalg.cond(Ms) * (1e-6 + 2.0 ** -22), (err, lo, hi)


def _residual(sys_, x):
    D, rp, col, val, b = sys_
    r = b - np.einsum("nij,nj->ni", D, x)
    rows = np.repeat(np.arange(len(D)), np.diff(rp))
    np.add.at(r, rows, -np.einsum("kij,kj->ki", val, x[col]))
    return np.linalg.norm(r) / np.linalg.norm(b)


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("sizes,cluster", [
    ([600] + [20] * 148, 1), ([600] + [33] * 79, 2),  # more CTAs than SMs, the largest scene of two chunks a CTA and more
    ([4200, 40], 16),                                 # clusters of 16
    ([3000, 2100], 1),                                # eight chunks a CTA
])
def test_batched_solves_by_every_variant(sizes, cluster, fp64):
    """The staged solve by 8 warps (the first three) and by 16, against 64-bit residuals."""
    rng = np.random.default_rng(len(sizes))
    systems = [_system(n, 9, rng) for n in sizes]
    off = np.concatenate([[0], np.cumsum(sizes)])
    n = int(off[-1])
    diag = np.zeros((n, 3, 4), np.float32)
    diag[:, :, :3] = np.concatenate([s[0] for s in systems]).transpose(0, 2, 1)
    nnz = np.concatenate([[0], np.cumsum([len(s[2]) for s in systems])])
    rp = np.concatenate([s[1][:-1] + o for s, o in zip(systems, nnz)] + [nnz[-1:]]).astype(np.uint32)
    col = np.concatenate([s[2] + o for s, o in zip(systems, off)]).astype(np.uint32)
    val = np.concatenate([s[3] for s in systems]).transpose(0, 2, 1).reshape(-1).astype(np.float32)
    b = np.zeros((n, 4), np.float32)
    b[:, :3] = np.concatenate([s[4] for s in systems])
    M = make_bsr(n, dev(rp.view(np.int32)), dev(col.view(np.int32)), dev(val))
    x = torch.full((n, 4), 5.0, dtype=torch.float32, device="cuda")
    stats = torch.zeros((len(sizes), 4), dtype=torch.int32, device="cuda")
    solve_batch(ConjugateGradientSolver(n), dev(off.astype(np.int32)), dev(diag), M, None, dev(b), x, stats, max_iter=400,
                rel_tol=1e-5, abs_rz_tol=0.0, cluster=cluster, fp64_dots=fp64)
    torch.cuda.synchronize()
    st = host(stats)
    assert (st[:, 3] == 0).all()
    got = host(x)[:, :3].astype(np.float64)
    for s, lo, hi, iters in zip(systems, off[:-1], off[1:], st[:, 0]):
        # the recurrence stops at 1e-5 and leaves the true residual by a few roundings of A x an iteration; eigenvalues lie
        # between 1 and 1 + 2 * 1.1 for each block of a row
        cond = 1 + 2.2 * np.diff(s[1]).max()
        assert _residual(s, got[lo:hi]) <= 1e-5 + 4 * 2.0 ** -24 * np.sqrt(max(iters, 1)) * cond
