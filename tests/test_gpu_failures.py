"""Failure detection without a GPU fault: every failure is made on the host (a NaN written into the inputs, a tree
whose parent links were overwritten, a wait that no block satisfies) and each entry point must report it as a
status code, with the context still usable afterwards.

Reference behaviour restated: PCG stops on a NaN/Inf r.z (precond_cg.cpp:717-721), the Newton loop reports
a non-finite direction (newton_solver.cpp:3731-3737), fn_check_construction clears the healthy flag when a
child does not name its parent (lbvh.cpp:598-611, check_health lbvh.cpp:1033-1036), and waits are bounded
(wait_for_write, lbvh.cpp:62-82)."""
import numpy as np
import pytest
import torch

from luisacomputesimulator_b200 import _capi as A
from luisacomputesimulator_b200.collision import LBVH, ptr, stream
from luisacomputesimulator_b200.linear import ConjugateGradientSolver, make_bsr
from luisacomputesimulator_b200.newton import NewtonSolver
from oracle import oracle as O
from tests import scenarios as SC
from tests.gpu_util import dev, host
from tests.test_gpu_pcg import _dev_bsr, contact_system

pytestmark = pytest.mark.gpu


def _status_of(exc):
    return str(exc.value).split(":")[1].split()[0]


@pytest.mark.parametrize("mode", ["plain", "fused", "rows", "cg1"])
def test_pcg_reports_nan_right_hand_side(mode):
    sc, diag, Am, Bm, b = contact_system()
    n = sc.num_verts
    b = b.copy()
    saved = b[n // 3, 1]
    b[n // 3, 1] = np.nan
    solver = ConjugateGradientSolver(n)
    x = torch.zeros((n, 4), dtype=torch.float32, device="cuda")
    with pytest.raises(A.LcsError) as e:
        solver.device_solve(dev(diag), _dev_bsr(n, Am), _dev_bsr(n, Bm), dev(b), x, max_iter=100,
                            check_every=25 if mode == "plain" else 1, plain=mode == "plain", rows=mode == "rows",
                            single_reduction=mode == "cg1")
    assert _status_of(e) == "LCS_ERR_NAN"
    # the same solver with the finite right-hand side restored still solves
    b[n // 3, 1] = saved
    st = solver.device_solve(dev(diag), _dev_bsr(n, Am), _dev_bsr(n, Bm), dev(b), x, max_iter=500,
                             check_every=25 if mode == "plain" else 1, plain=mode == "plain", rows=mode == "rows",
                             single_reduction=mode == "cg1")
    assert st["status"] == 0 and st["rel_residual"] <= 1e-4


@pytest.mark.parametrize("plain", [False, True])
def test_newton_step_reports_a_nan_position(plain):
    """A NaN position uploaded from the host: the step returns LCS_ERR_NAN (the PCG's r.z is not finite) instead of
    applying a non-finite direction, and a later upload of a finite state steps normally."""
    sc, x = SC.cloth_touching_sphere(gap=5e-4, n=32)
    sc.x = x.copy()
    gpu = NewtonSolver(sc, plain=plain, single_reduction=not plain)
    st = gpu.step()
    assert st.status == 0
    good_x, good_v = gpu.positions(), gpu.velocities()
    bad = good_x.copy()
    bad[100, 1] = np.nan  # a free cloth vertex
    gpu.upload(bad, good_v)
    with pytest.raises(A.LcsError) as e:
        gpu.step()
    assert _status_of(e) == "LCS_ERR_NAN"
    gpu.upload(good_x, good_v)
    st = gpu.step()
    assert st.status == 0
    xn = gpu.positions()
    assert np.isfinite(xn).all()
    assert O.min_distance(sc, xn) > 0.0


def _face_tree():
    sc, x = SC.cloth_touching_sphere(gap=2e-3)
    xd = dev(x)
    t = LBVH(A.LCS_TREE_FACE, sc.faces.shape[0])
    t.reduce_face_tree_aabb(xd, dev(sc.faces))
    t.construct_tree()
    return t


def test_corrupted_parent_links_make_the_tree_unhealthy():
    t = _face_tree()
    assert t.check_health()
    data = t.device_data()
    parent = data["parent"]
    n = t.n
    saved = parent.clone()
    # leaf 7 (node n - 1 + 7) now names the root as its parent although the root's children are other nodes
    leaf = n - 1 + 7
    root_kids = data["children"][0].cpu().numpy()
    assert leaf not in root_kids
    parent[leaf] = 0
    torch.cuda.synchronize()
    t.check_construction()
    assert not t.check_health()
    # a swapped pair of inner-node parents is caught as well
    parent.copy_(saved)
    host_parent = saved.cpu().numpy()
    a = 1
    b = next(k for k in range(2, n - 1) if host_parent[k] != host_parent[a])
    pa, pb = int(host_parent[a]), int(host_parent[b])
    parent[a] = pb
    parent[b] = pa
    torch.cuda.synchronize()
    t.check_construction()
    assert not t.check_health()
    # restored links are healthy again, and so is a fresh build
    parent.copy_(saved)
    torch.cuda.synchronize()
    t.check_construction()
    assert t.check_health()
    t.construct_tree()
    assert t.check_health()


@pytest.mark.parametrize("which", [0, 1])
def test_bounded_waits_run_out_and_report_timeout(which):
    """The slice-resident solve's reduction barrier (0) and neighbour-flag wait (1) with one block that never
    arrives: every other block gives up after a short poll limit and the call returns LCS_ERR_TIMEOUT."""
    lib = A.load()
    s = stream()
    assert lib.lcs_debug_pcg_wait(which, -1, 8, 1 << 20, s) == 0  # all blocks take part: the waits complete
    rc = lib.lcs_debug_pcg_wait(which, 3, 8, 1 << 12, s)
    assert A.STATUS[rc] == "LCS_ERR_TIMEOUT", A.STATUS.get(rc, rc)
    assert "ran out" in lib.lcs_last_error().decode()
    # the context is still usable: the same probe completes, and a solve runs
    assert lib.lcs_debug_pcg_wait(which, -1, 8, 1 << 20, s) == 0
    sc, diag, Am, Bm, b = contact_system()
    n = sc.num_verts
    x = torch.zeros((n, 4), dtype=torch.float32, device="cuda")
    st = ConjugateGradientSolver(n).device_solve(dev(diag), _dev_bsr(n, Am), _dev_bsr(n, Bm), dev(b), x,
                                                 max_iter=500, check_every=1, single_reduction=True)
    assert st["status"] == 0 and st["rel_residual"] <= 1e-4


def test_wait_probe_rejects_bad_arguments():
    lib = A.load()
    s = stream()
    assert A.STATUS[lib.lcs_debug_pcg_wait(2, -1, 8, 16, s)] == "LCS_ERR_INVALID"
    assert A.STATUS[lib.lcs_debug_pcg_wait(0, -1, 64, 16, s)] == "LCS_ERR_INVALID"
    assert A.STATUS[lib.lcs_debug_pcg_wait(0, 9, 8, 16, s)] == "LCS_ERR_INVALID"
    assert A.STATUS[lib.lcs_debug_pcg_wait(0, -1, 8, 0, s)] == "LCS_ERR_INVALID"


def test_copies_that_do_not_arrive_run_out_and_leave_the_product_right():
    """The batched solve's copies of the matrix to shared memory, one of which never completes: the warp gives up after a
    short poll limit, looks at no stage again (its words could be any column) and reads the blocks directly, so the
    product is that of the completed copies bit for bit and the call returns LCS_ERR_TIMEOUT."""
    lib = A.load()
    n = 97
    rng = np.random.default_rng(3)
    rp = np.concatenate([[0], np.cumsum(rng.integers(0, 40, n))]).astype(np.int32)
    col = rng.integers(0, n, rp[-1]).astype(np.int32)
    val = rng.normal(size=9 * rp[-1]).astype(np.float32)
    x = rng.normal(size=(n, 4)).astype(np.float32)
    keep = [dev(rp), dev(col), dev(val), dev(x)]
    M = make_bsr(n, *keep[:3])
    got = {}
    for omit, limit, want in ((0, 1 << 20, "LCS_OK"), (1, 1 << 12, "LCS_ERR_TIMEOUT"), (0, 1 << 20, "LCS_OK")):
        y = torch.full((n, 4), 9.0, dtype=torch.float32, device="cuda")
        rc = lib.lcs_debug_pcg_copy_wait(M, ptr(keep[3]), ptr(y), omit, limit, stream())
        assert A.STATUS[rc] == want, (omit, rc)
        got[omit] = host(y)[:, :3]
    np.testing.assert_array_equal(got[1], got[0])
    r = np.repeat(np.arange(n), np.diff(rp))
    t = np.einsum("kcr,kc->kr", val.reshape(-1, 3, 3).astype(np.float64), x[col, :3].astype(np.float64))
    y64, mag = np.zeros((n, 3)), np.zeros((n, 3))
    np.add.at(y64, r, t)
    np.add.at(mag, r, np.einsum("kcr,kc->kr", np.abs(val.reshape(-1, 3, 3).astype(np.float64)), np.abs(x[col, :3])))
    # each of a lane's up to 10 blocks, the 4 lanes and the 3 columns round once: (10 + 2 + 3) 2^-24 of the magnitudes
    assert (np.abs(got[1] - y64) <= 15 * 2.0 ** -24 * mag).all()
    assert A.STATUS[lib.lcs_debug_pcg_copy_wait(M, ptr(keep[3]), ptr(y), 0, 0, stream())] == "LCS_ERR_INVALID"


def test_exchange_of_small_systems_carries_whole_doubles_and_its_wait_runs_out():
    """The grid-wide sums of the persistent solve's small systems: right to the last bits with every block, and a timeout,
    after a short poll limit, with one that never takes part."""
    lib = A.load()
    rng = np.random.default_rng(2)
    for blocks in (2, 3, 31, 32):
        v = rng.normal(size=(blocks, 2)) * 10.0 ** rng.integers(-6, 6, (blocks, 2))
        vd, sums = dev(v), torch.zeros(3, dtype=torch.float64, device="cuda")
        assert lib.lcs_debug_pcg_exchange(ptr(vd), ptr(sums), -1, blocks, 1 << 20, stream()) == 0
        want, mag = v.astype(np.longdouble).sum(0), np.abs(v).sum(0)
        # five additions of a warp's tree round once each
        for got, w, m in zip(host(sums), (want[0], want[1], want[1]), (mag[0], mag[1], mag[1])):
            assert abs(got - w) <= 5 * 2.0 ** -53 * m, (blocks, got, w)
        rc = lib.lcs_debug_pcg_exchange(ptr(vd), ptr(sums), blocks - 1, blocks, 1 << 12, stream())
        assert A.STATUS[rc] == "LCS_ERR_TIMEOUT"
    assert lib.lcs_debug_pcg_exchange(ptr(vd), ptr(sums), -1, 32, 1 << 20, stream()) == 0
    assert A.STATUS[lib.lcs_debug_pcg_exchange(ptr(vd), ptr(sums), 32, 32, 16, stream())] == "LCS_ERR_INVALID"
