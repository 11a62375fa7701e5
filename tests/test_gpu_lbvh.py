"""LBVH parity: the CUDA build / refit / traversal against the oracle, bit for bit.

Sizes: config 1 (6,658 verts), a folded cloth (self contact), and config 2's 88,800-vertex
tube at full size (177,000-face and 265,800-edge trees)."""
import numpy as np
import pytest
import torch

from luisacomputesimulator_b200 import _capi as A
from luisacomputesimulator_b200.collision import LBVH
from oracle import oracle as O
from tests import scenarios as SC
from tests.gpu_util import SceneOnDevice, counts, dev, host
from tests.test_oracle_deep_tree import _max_inner_depth

pytestmark = pytest.mark.gpu

KINDS = {"face": (O.TREE_FACE, "faces"), "edge": (O.TREE_EDGE, "edges")}


def _scene(name):
    if name == "cloth_sphere":
        return SC.cloth_touching_sphere(gap=5e-4)
    if name == "folded":
        return SC.folded_cloth(n=48, gap=4e-4)
    if name == "tube":
        return SC.twisted_tube_state(angle=1.2)
    if name == "tube_state":  # the benchmarked state: 56 steps of the run from rest
        sc, x, _, _ = SC.tube_state()
        return sc, x
    raise KeyError(name)


def _build_both(sc, x, kind_name):
    kind, attr = KINDS[kind_name]
    elems = getattr(sc, attr)
    t_o = O.lbvh_build(kind, x, elems, sc.num_verts)
    bvh = LBVH(kind, elems.shape[0])
    xd, ed = dev(x), dev(elems)
    if kind == O.TREE_FACE:
        bvh.reduce_face_tree_aabb(xd, ed)
    else:
        bvh.reduce_edge_tree_aabb(xd, ed)
    bvh.construct_tree()
    return t_o, bvh, xd, ed


@pytest.mark.parametrize("scene", ["cloth_sphere", "folded", "tube"])
@pytest.mark.parametrize("kind_name", ["face", "edge"])
def test_topology_bit_exact(scene, kind_name):
    sc, x = _scene(scene)
    t_o, bvh, _, _ = _build_both(sc, x, kind_name)
    assert bvh.check_health()
    e = bvh.export()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(host(e["global_aabb"]), np.concatenate([t_o.gmin, t_o.gmax]))
    np.testing.assert_array_equal(host(e["morton"], np.uint64), t_o.morton)
    np.testing.assert_array_equal(host(e["morton_sorted"], np.uint64), t_o.morton_sorted)
    np.testing.assert_array_equal(host(e["sorted_get_original"], np.uint32), t_o.sorted_get_original)
    np.testing.assert_array_equal(host(e["parent"], np.uint32), t_o.parent)
    np.testing.assert_array_equal(host(e["children"], np.uint32), t_o.children)
    np.testing.assert_array_equal(host(e["object_idx"], np.uint32), t_o.object_idx)


def _refit_both(kind, x, x1, elems, off):
    t_o = O.lbvh_build(kind, x, elems, x.shape[0])
    bvh = LBVH(kind, elems.shape[0])
    xd, ed = dev(x), dev(elems)
    if kind == O.TREE_FACE:
        bvh.reduce_face_tree_aabb(xd, ed)
    else:
        bvh.reduce_edge_tree_aabb(xd, ed)
    bvh.construct_tree()
    O.lbvh_refit(t_o, x, x1, elems, off)
    bvh.update_and_refit(dev(off), xd, dev(x1), ed)
    e = bvh.export()
    torch.cuda.synchronize()
    return t_o, host(e["node_aabb"])


@pytest.mark.parametrize("m", [2, 3, 40, 511, 512, 513, 1025, 1600])
def test_refit_bit_exact_across_chunk_sizes(m):
    """Trees of one, two and several 512-leaf refit chunks (the refit computes each inner box from its
    sorted leaf range, in one chunk or across chunks) against the oracle's bottom-up walk."""
    sc, x = _scene("folded")
    faces = np.ascontiguousarray(sc.faces[:m])
    x1 = SC.random_motion(x, 1e-3, seed=m)
    t_o, got = _refit_both(O.TREE_FACE, x, x1, faces, sc.offset + np.float32(1e-4))
    np.testing.assert_array_equal(got[:, 0:3], t_o.node_aabb[:, 0:3])
    np.testing.assert_array_equal(got[:, 4:7], t_o.node_aabb[:, 4:7])


def test_refit_signed_zero_ties_bit_exact():
    """Leaf boxes whose extremes tie at +0 and -0 (zero thickness, coordinates of both signs of zero): the
    reference's union `a < b ? a : b` keeps the later of two equal values, so the node boxes' zero signs
    depend on the order of the unions; compared as bit patterns."""
    rng = np.random.default_rng(3)
    g = 48
    ii, jj = np.meshgrid(np.arange(g), np.arange(g), indexing="ij")
    x = np.zeros((g * g, 4), np.float32)
    x[:, 0] = np.where(rng.random(g * g) < 0.5, np.float32(0.0), np.float32(-0.0))
    x[:, 1] = (ii.ravel() * 0.01).astype(np.float32)
    x[:, 2] = np.where(rng.random(g * g) < 0.5, np.float32(0.0), np.float32(-0.0))
    x[(jj.ravel() % 7) == 3, 2] = np.float32(0.01) * (jj.ravel()[(jj.ravel() % 7) == 3]).astype(np.float32)
    idx = (ii * g + jj)
    edges = np.concatenate([np.stack([idx[:, :-1].ravel(), idx[:, 1:].ravel()], 1),
                            np.stack([idx[:-1, :].ravel(), idx[1:, :].ravel()], 1)]).astype(np.uint32)
    off = np.zeros(g * g, np.float32)
    t_o, got = _refit_both(O.TREE_EDGE, x, x.copy(), edges, off)
    assert (np.signbit(t_o.node_aabb[:, 0:3]).any() and (~np.signbit(t_o.node_aabb[:, 0:3])).any())
    np.testing.assert_array_equal(got[:, 0:3].view(np.uint32), t_o.node_aabb[:, 0:3].view(np.uint32))
    np.testing.assert_array_equal(got[:, 4:7].view(np.uint32), t_o.node_aabb[:, 4:7].view(np.uint32))


@pytest.mark.parametrize("scene", ["cloth_sphere", "folded", "tube"])
@pytest.mark.parametrize("kind_name", ["face", "edge"])
@pytest.mark.parametrize("fused", [False, True])
def test_refit_bit_exact(scene, kind_name, fused):
    sc, x = _scene(scene)
    t_o, bvh, xd, ed = _build_both(sc, x, kind_name)
    x1 = SC.random_motion(x, 1e-3, seed=7)
    x1d = dev(x1)
    off = dev(sc.offset + np.float32(1e-4))
    O.lbvh_refit(t_o, x, x1, getattr(sc, KINDS[kind_name][1]), sc.offset + np.float32(1e-4))
    for _ in range(2):  # twice: a refit over its own previous output
        if fused:
            bvh.update_and_refit(off, xd, x1d, ed)
        else:
            bvh.update_leaves(off, xd, x1d, ed)
            bvh.refit()
    e = bvh.export()
    torch.cuda.synchronize()
    got = host(e["node_aabb"])
    np.testing.assert_array_equal(got[:, 0:3], t_o.node_aabb[:, 0:3])
    np.testing.assert_array_equal(got[:, 4:7], t_o.node_aabb[:, 4:7])


@pytest.mark.parametrize("scene", ["cloth_sphere", "folded", "tube", "tube_state"])
@pytest.mark.parametrize("swept", [False, True])
def test_candidate_sets_bit_exact(scene, swept):
    sc, x = _scene(scene)
    x1 = SC.random_motion(x, 2e-3, seed=11) if swept else x
    D = SceneOnDevice(sc)
    xd, x1d = dev(x), dev(x1)
    for kind_name in ("face", "edge"):
        t_o, bvh, _, ed = _build_both(sc, x, kind_name)
        elems = getattr(sc, KINDS[kind_name][1])
        O.lbvh_refit(t_o, x, x1, elems, sc.offset)
        bvh.update_and_refit(D.offset, xd, x1d, ed)
        cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
        if kind_name == "face":
            want, n_want = O.lbvh_query_vf(t_o, x, x1, sc.d_hat, sc.offset)
            pairs = torch.zeros((n_want + 64, 2), dtype=torch.int32, device="cuda")
            bvh.broad_phase_query_from_verts(xd, x1d, cnt, pairs, D.d_hat, D.offset)
        else:
            want, n_want = O.lbvh_query_ee(t_o, x, x1, sc.edges, sc.d_hat, sc.offset)
            pairs = torch.zeros((n_want + 64, 2), dtype=torch.int32, device="cuda")
            bvh.broad_phase_query_from_edges(xd, x1d, D.edges, cnt, pairs, D.d_hat, D.offset)
        n = int(counts(cnt)[0])
        assert n == n_want
        got = host(pairs, np.uint32)[:n]
        np.testing.assert_array_equal(SC.sorted_pairs(got), SC.sorted_pairs(want))


def test_update_and_refit_before_construct_is_refused():
    """Leaf order, slots and refit tables come from the build: before it, update / refit / query / export
    are refused (LCS_ERR_INVALID) instead of reading tables that hold no indices; after it they run."""
    sc, x = _scene("folded")
    faces = np.ascontiguousarray(sc.faces[:700])
    edges = np.ascontiguousarray(sc.edges[:900])
    bvh = LBVH(O.TREE_FACE, faces.shape[0])
    ebvh = LBVH(O.TREE_EDGE, edges.shape[0])
    xd, fd, edd, off, dh = dev(x), dev(faces), dev(edges), dev(sc.offset), dev(sc.d_hat)
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    pairs = torch.zeros((1024, 2), dtype=torch.int32, device="cuda")
    for call in (lambda: bvh.update_and_refit(off, xd, xd, fd), lambda: bvh.update_leaves(off, xd, xd, fd),
                 bvh.refit, bvh.export, lambda: bvh.broad_phase_query_from_verts(xd, xd, cnt, pairs, dh, off),
                 lambda: ebvh.broad_phase_query_from_edges(xd, xd, edd, cnt, pairs, dh, off),
                 lambda: ebvh.broad_phase_query_from_edges_sym(xd, xd, edd, cnt, pairs, float(sc.d_hat[0]))):
        with pytest.raises(A.LcsError, match="LCS_ERR_INVALID"):
            call()
    bvh.reduce_face_tree_aabb(xd, fd)
    bvh.construct_tree()
    bvh.update_and_refit(off, xd, xd, fd)
    bvh.broad_phase_query_from_verts(xd, xd, cnt, pairs, dh, off)
    torch.cuda.synchronize()
    assert bvh.check_health()


def test_query_overflow_counts_without_writing_past_capacity():
    sc, x = _scene("cloth_sphere")
    D = SceneOnDevice(sc)
    t_o, bvh, xd, ed = _build_both(sc, x, "edge")
    bvh.update_and_refit(D.offset, xd, xd, ed)
    O.lbvh_refit(t_o, x, x, sc.edges, sc.offset)
    want, n_want = O.lbvh_query_ee(t_o, x, x, sc.edges, sc.d_hat, sc.offset)
    cap = 1000
    guard = torch.full((cap + 16, 2), -7, dtype=torch.int32, device="cuda")
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    bvh.broad_phase_query_from_edges(xd, xd, D.edges, cnt, guard[:cap], D.d_hat, D.offset)
    n = int(counts(cnt)[0])
    assert n == n_want and n > cap
    g = host(guard)
    assert np.all(g[cap:] == -7)  # nothing past capacity
    full = {tuple(p) for p in SC.sorted_pairs(want).tolist()}
    assert all(tuple(p) in full for p in g[:cap].astype(np.int64).tolist())


def test_single_leaf_tree_and_empty_queries():
    # one face: the reference's root is the leaf itself and both child reads hit it
    x = np.array([[0, 0, 0, 0], [1, 0, 0, 0], [0, 1, 0, 0], [0.2, 0.2, 0.0005, 0]], np.float32)
    faces = np.array([[0, 1, 2, 0]], np.uint32)
    t_o = O.lbvh_build(O.TREE_FACE, x, faces, 4)
    thick = np.zeros(4, np.float32)
    dhat = np.full(4, 1e-3, np.float32)
    O.lbvh_refit(t_o, x, x, faces, thick)
    want, n_want = O.lbvh_query_vf(t_o, x, x, dhat, thick)
    bvh = LBVH(O.TREE_FACE, 1)
    xd, fd = dev(x), dev(faces)
    bvh.reduce_face_tree_aabb(xd, fd)
    bvh.construct_tree()
    bvh.update_and_refit(dev(thick), xd, xd, fd)
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    pairs = torch.zeros((16, 2), dtype=torch.int32, device="cuda")
    bvh.broad_phase_query_from_verts(xd, xd, cnt, pairs, dev(dhat), dev(thick))
    n = int(counts(cnt)[0])
    assert n == n_want
    np.testing.assert_array_equal(SC.sorted_pairs(host(pairs, np.uint32)[:n]), SC.sorted_pairs(want))


@pytest.mark.parametrize("scene", ["cloth_sphere", "folded"])
def test_filtered_swept_lists_equal_static_queries_on_the_sweep(scene):
    """The fused Newton loop takes its DCD candidates from the previous CCD lists: filtering the swept
    list (x0 -> x1) at any x = x0 + t (x1 - x0), 0 <= t <= 1, must give the static-box list at x."""
    import ctypes as C
    from luisacomputesimulator_b200 import _capi as A
    from luisacomputesimulator_b200.collision import ptr, stream
    sc, x0 = _scene(scene)
    x1 = SC.random_motion(x0, 2e-3, seed=3)
    xm = x0.copy()
    xm[:, :3] = x0[:, :3] + np.float32(0.37) * (x1[:, :3] - x0[:, :3])
    D = SceneOnDevice(sc)
    lib = A.load()
    for kind_name, is_ee in (("face", 0), ("edge", 1)):
        t_o, bvh, _, ed = _build_both(sc, x0, kind_name)
        elems = getattr(sc, KINDS[kind_name][1])
        bvh.update_and_refit(D.offset, dev(x0), dev(x1), ed)
        cap = 64 * max(sc.num_verts, elems.shape[0])
        swept = torch.zeros((cap, 2), dtype=torch.int32, device="cuda")
        cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
        if is_ee:
            bvh.broad_phase_query_from_edges(dev(x0), dev(x1), D.edges, cnt, swept, D.d_hat, D.offset)
        else:
            bvh.broad_phase_query_from_verts(dev(x0), dev(x1), cnt, swept, D.d_hat, D.offset)
        assert int(counts(cnt)[0]) <= cap  # the whole swept list was written
        out = torch.zeros((cap, 2), dtype=torch.int32, device="cuda")
        ocnt = torch.zeros(1, dtype=torch.int32, device="cuda")
        A.check(lib.lcs_candidates_filter(is_ee, ptr(swept), ptr(cnt), cap, ptr(dev(xm)), ptr(ed), ptr(D.d_hat),
                                          ptr(D.offset), ptr(out), cap, ptr(ocnt), stream()), "filter")
        O.lbvh_refit(t_o, xm, xm, elems, sc.offset)
        if is_ee:
            want, n_want = O.lbvh_query_ee(t_o, xm, xm, sc.edges, sc.d_hat, sc.offset)
        else:
            want, n_want = O.lbvh_query_vf(t_o, xm, xm, sc.d_hat, sc.offset)
        n = int(counts(ocnt)[0])
        assert n == n_want and n <= int(counts(cnt)[0])
        np.testing.assert_array_equal(SC.sorted_pairs(host(out, np.uint32)[:n]), SC.sorted_pairs(want))


@pytest.mark.parametrize("scene", ["cloth_sphere", "folded", "tube", "tube_state"])
@pytest.mark.parametrize("swept", [False, True])
def test_once_per_pair_ee_query_matches_the_reference_set(scene, swept):
    """lcs_bvh_query_ee_sym (each pair met once, from the lower Morton position) returns the oracle's
    EE set bit for bit on scenes with thickness 0 and one d_hat -- the Newton loop's configuration."""
    sc, x = _scene(scene)
    sc.offset = np.zeros_like(sc.offset)
    sc.d_hat = np.full_like(sc.d_hat, sc.d_hat[sc.edges[0, 0]])
    x1 = SC.random_motion(x, 2e-3, seed=13) if swept else x
    D = SceneOnDevice(sc)
    xd, x1d = dev(x), dev(x1)
    t_o, bvh, _, ed = _build_both(sc, x, "edge")
    O.lbvh_refit(t_o, x, x1, sc.edges, sc.offset)
    bvh.update_and_refit(D.offset, xd, x1d, ed)
    want, n_want = O.lbvh_query_ee(t_o, x, x1, sc.edges, sc.d_hat, sc.offset)
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    pairs = torch.zeros((n_want + 64, 2), dtype=torch.int32, device="cuda")
    bvh.broad_phase_query_from_edges_sym(xd, x1d, D.edges, cnt, pairs, float(sc.d_hat[0]))
    n = int(counts(cnt)[0])
    assert n == n_want
    np.testing.assert_array_equal(SC.sorted_pairs(host(pairs, np.uint32)[:n]), SC.sorted_pairs(want))


def test_once_per_pair_ee_query_on_boxes_at_the_threshold():
    """A grid whose edge boxes sit at distance d_hat from each other on every axis (spacing = edge length
    + d_hat, scaled so the sums round): the strict test decides at the last ulp, from either side."""
    rng = np.random.default_rng(5)
    n = 40
    d = np.float32(1e-3)
    seg = []
    for i in range(n):
        for j in range(n):
            p = np.array([i * 3e-3, j * 3e-3, 0.0], np.float32)
            seg.append((p, p + np.array([2e-3, 0, 0], np.float32)))
            seg.append((p + np.array([0, 1e-3, 0], np.float32),
                        p + np.array([0, 1e-3, 0], np.float32) + np.float32(1e-3) * rng.normal(size=3).astype(np.float32)))
    x = np.zeros((2 * len(seg), 4), np.float32)
    for k, (a, b) in enumerate(seg):
        x[2 * k, :3], x[2 * k + 1, :3] = a, b
    edges = np.arange(2 * len(seg), dtype=np.uint32).reshape(-1, 2)
    V = x.shape[0]
    dh, off = np.full(V, d, np.float32), np.zeros(V, np.float32)
    t_o = O.lbvh_build(O.TREE_EDGE, x, edges, V)
    O.lbvh_refit(t_o, x, x, edges, off)
    want, n_want = O.lbvh_query_ee(t_o, x, x, edges, dh, off)
    bvh = LBVH(O.TREE_EDGE, edges.shape[0])
    xd, ed = dev(x), dev(edges)
    bvh.reduce_edge_tree_aabb(xd, ed)
    bvh.construct_tree()
    bvh.update_and_refit(dev(off), xd, xd, ed)
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    pairs = torch.zeros((n_want + 64, 2), dtype=torch.int32, device="cuda")
    bvh.broad_phase_query_from_edges_sym(xd, xd, ed, cnt, pairs, float(d))
    m = int(counts(cnt)[0])
    assert m == n_want and n_want > 0
    np.testing.assert_array_equal(SC.sorted_pairs(host(pairs, np.uint32)[:m]), SC.sorted_pairs(want))


def _deep_tree(kind_name):
    x, el = SC.deep_tree_elements(kind_name)
    V = x.shape[0]
    kind = KINDS[kind_name][0]
    t_o = O.lbvh_build(kind, x, el, V)
    bvh = LBVH(kind, el.shape[0])
    xd, ed = dev(x), dev(el)
    if kind == O.TREE_FACE:
        bvh.reduce_face_tree_aabb(xd, ed)
    else:
        bvh.reduce_edge_tree_aabb(xd, ed)
    bvh.construct_tree()
    z = np.zeros(V, np.float32)
    O.lbvh_refit(t_o, x, x, el, z)
    bvh.update_and_refit(dev(z), xd, xd, ed)
    return x, el, t_o, bvh, xd, ed


def _brute_force_count(x, el, r, ee):
    """Size of the complete candidate set (strict box overlap, no early exit)."""
    m = 2 if ee else 3
    lo, hi = x[el[:, :m], :3].min(1), x[el[:, :m], :3].max(1)
    if ee:  # edge i's query box: its box widened by r of its first vertex; pairs i < j
        rq = r[el[:, 0]][:, None]
        qlo, qhi = lo - rq, hi + rq
    else:  # vertex v's query box: the point widened by r[v]
        qlo, qhi = x[:, :3] - r[:, None], x[:, :3] + r[:, None]
    ov = (lo[None] < qhi[:, None]).all(2) & (hi[None] > qlo[:, None]).all(2)
    if ee:
        i, j = np.nonzero(ov)
        return int((i < j).sum())
    return int(ov.sum())


@pytest.mark.parametrize("kind_name", ["face", "edge"])
def test_deep_tree_traversal_ends_early_like_the_reference(kind_name):
    """A tree with inner nodes at depth >= 32, where the reference's 32-entry stack fills: every query whose
    walk meets a full stack ends there, keeping only the pairs found before (lbvh.cpp:293-360).  Per-vertex
    query radii mix queries that end early with queries that finish.  The GPU sets equal the oracle's, which
    are smaller than the complete sets; the early exit is reported."""
    x, el, t_o, bvh, xd, ed = _deep_tree(kind_name)
    V = x.shape[0]
    r = np.random.default_rng(7).uniform(200.0, 800.0, V).astype(np.float32)
    z = np.zeros(V, np.float32)
    ee = kind_name == "edge"
    if ee:
        want, n_want = O.lbvh_query_ee(t_o, x, x, el, r, z)
    else:
        want, n_want = O.lbvh_query_vf(t_o, x, x, r, z)
    assert 0 < n_want < _brute_force_count(x, el, r, ee)  # the reference's early exit removed pairs
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    pairs = torch.zeros((n_want + 64, 2), dtype=torch.int32, device="cuda")
    if ee:
        bvh.broad_phase_query_from_edges(xd, xd, ed, cnt, pairs, dev(r), dev(z))
    else:
        bvh.broad_phase_query_from_verts(xd, xd, cnt, pairs, dev(r), dev(z))
    n = int(counts(cnt)[0])
    assert n == n_want
    np.testing.assert_array_equal(SC.sorted_pairs(host(pairs, np.uint32)[:n]), SC.sorted_pairs(want))


def test_deep_tree_once_per_pair_query_falls_back_to_the_reference_walk():
    """The once-per-pair EE form relies on the set being symmetric, which the reference's early exit breaks:
    on a deep tree lcs_bvh_query_ee_sym runs the reference's full EE walk and returns its set."""
    x, el, t_o, bvh, xd, ed = _deep_tree("edge")
    V = x.shape[0]
    z = np.zeros(V, np.float32)
    for rad in (300.0, 520.0, 600.0):
        r = np.full(V, rad, np.float32)
        want, n_want = O.lbvh_query_ee(t_o, x, x, el, r, z)
        cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
        pairs = torch.zeros((max(n_want, 1) + 64, 2), dtype=torch.int32, device="cuda")
        bvh.broad_phase_query_from_edges_sym(xd, xd, ed, cnt, pairs, rad)
        n = int(counts(cnt)[0])
        assert n == n_want, (rad, n, n_want)
        np.testing.assert_array_equal(SC.sorted_pairs(host(pairs, np.uint32)[:n]), SC.sorted_pairs(want))


def _sheet(side):
    i = np.arange(side)
    X, Z = np.meshgrid(i, i, indexing="ij")
    v = X * side + Z
    pair = lambda a, b: np.stack([a.ravel(), b.ravel()], 1)  # noqa: E731
    el = np.concatenate([pair(v[:-1], v[1:]), pair(v[:, :-1], v[:, 1:]), pair(v[:-1, :-1], v[1:, 1:])]).astype(np.uint32)
    x = np.zeros((side * side, 4), np.float32)
    x[:, 0], x[:, 2] = X.ravel() * 0.01, Z.ravel() * 0.01
    return x, el


def _deep_sheet(side):
    """A sheet, uneven by 2 mm, and a few edges beside it that give the tree one path of 32 levels."""
    x, el = _sheet(side)
    x[:, 1] = 2e-3 * np.random.default_rng(side).random(len(x))
    deep, deep_el = SC.deep_tree_elements("edge")
    return np.concatenate([deep / 256, x]), np.concatenate([deep_el, el + np.uint32(len(deep))])


@pytest.mark.parametrize("side,swept,foreign", [(40, False, False), (53, False, False), (53, True, False), (60, True, True),
                                                (150, True, False)])
def test_general_ee_query_once_per_pair_and_its_fallback(side, swept, foreign):
    """The general EE query of one sheet, with per-vertex thickness and d_hat that spread by 30: trees of fewer than 32
    levels and 131,072 edges, each edge walking for itself; `foreign` queries with other positions than the tree's."""
    i = np.arange(side)
    X, Z = np.meshgrid(i, i, indexing="ij")
    v = X * side + Z
    pair = lambda a, b: np.stack([a.ravel(), b.ravel()], 1)  # noqa: E731
    el = np.concatenate([pair(v[:-1], v[1:]), pair(v[:, :-1], v[:, 1:]), pair(v[:-1, :-1], v[1:, 1:])]).astype(np.uint32)
    rng = np.random.default_rng(side)
    n = side * side
    x = np.zeros((n, 4), np.float32)
    x[:, 0], x[:, 2] = X.ravel() * 0.01, Z.ravel() * 0.01
    x[:, 1] = 2e-3 * rng.random(n)
    x1 = x + (rng.normal(0, 3e-3, x.shape).astype(np.float32) if swept else 0)
    th = rng.uniform(0, 2e-3, n).astype(np.float32)
    dh = rng.uniform(1e-4, 3e-3, n).astype(np.float32)
    t_o = O.lbvh_build(O.TREE_EDGE, x, el, n)
    O.lbvh_refit(t_o, x, x1, el, th)
    bvh = LBVH(O.TREE_EDGE, el.shape[0])
    xd, x1d, ed = dev(x), dev(x1), dev(el)
    bvh.reduce_edge_tree_aabb(xd, ed)
    bvh.construct_tree()
    bvh.update_and_refit(dev(th), xd, x1d, ed)
    qx = x1 if foreign else x
    want, n_want = O.lbvh_query_ee(t_o, qx, x1, el, dh, th)
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    pairs = torch.zeros((n_want + 64, 2), dtype=torch.int32, device="cuda")
    bvh.broad_phase_query_from_edges(dev(qx), x1d, ed, cnt, pairs, dev(dh), dev(th))
    assert int(counts(cnt)[0]) == n_want > 0
    np.testing.assert_array_equal(SC.sorted_pairs(host(pairs, np.uint32)[:n_want]), SC.sorted_pairs(want))


@pytest.mark.parametrize("side,swept,foreign", [(209, True, False), (210, True, False), (210, False, False), (210, True, True)])
def test_general_ee_query_around_its_once_per_pair_size(side, swept, foreign):
    """The general EE query around the 131,072 edges from which it meets each pair once (side 210 has 131,530) on a tree of
    more than 32 levels (a few edges beside the sheet make one path of it that deep), with per-vertex thickness and d_hat;
    `foreign` queries with other positions than the tree's, which the full walk has to answer."""
    x, el = _deep_sheet(side)
    rng = np.random.default_rng(side)
    n = len(x)
    x1 = x + (rng.normal(0, 3e-3, x.shape).astype(np.float32) if swept else 0)
    th = rng.uniform(0, 2e-3, n).astype(np.float32)
    dh = rng.uniform(1e-3, 3e-3, n).astype(np.float32)
    t_o = O.lbvh_build(O.TREE_EDGE, x, el, n)
    assert _max_inner_depth(t_o) >= 32
    O.lbvh_refit(t_o, x, x1, el, th)
    bvh = LBVH(O.TREE_EDGE, el.shape[0])
    xd, x1d, ed = dev(x), dev(x1), dev(el)
    bvh.reduce_edge_tree_aabb(xd, ed)
    bvh.construct_tree()
    bvh.update_and_refit(dev(th), xd, x1d, ed)
    qx = x1 if foreign else x
    want, n_want = O.lbvh_query_ee(t_o, qx, x1, el, dh, th)
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    pairs = torch.zeros((n_want + 64, 2), dtype=torch.int32, device="cuda")
    bvh.broad_phase_query_from_edges(dev(qx), x1d, ed, cnt, pairs, dev(dh), dev(th))
    assert int(counts(cnt)[0]) == n_want > 0
    np.testing.assert_array_equal(SC.sorted_pairs(host(pairs, np.uint32)[:n_want]), SC.sorted_pairs(want))


@pytest.mark.parametrize("kind_name", ["face", "edge"])
@pytest.mark.parametrize("rad", [0.1, 300.0, 800.0])
def test_deep_tree_without_pending_nodes(kind_name, rad):
    """The deep tree mirrored: its longest path turns left throughout, so that the reference's stack never fills, at any
    radius, and the 4-wide walks serve a tree of more than 32 levels."""
    x, el = SC.deep_tree_elements(kind_name)
    x[:, :3] = np.float32(1024.0) - x[:, :3]
    V = x.shape[0]
    ee = kind_name == "edge"
    t_o = O.lbvh_build(KINDS[kind_name][0], x, el, V)
    z = np.zeros(V, np.float32)
    O.lbvh_refit(t_o, x, x, el, z)
    bvh = LBVH(KINDS[kind_name][0], el.shape[0])
    xd, ed = dev(x), dev(el)
    (bvh.reduce_edge_tree_aabb if ee else bvh.reduce_face_tree_aabb)(xd, ed)
    bvh.construct_tree()
    bvh.update_and_refit(dev(z), xd, xd, ed)
    r = np.full(V, rad, np.float32)
    want, n_want = (O.lbvh_query_ee(t_o, x, x, el, r, z) if ee else O.lbvh_query_vf(t_o, x, x, r, z))
    assert n_want == _brute_force_count(x, el, r, ee)  # no early exit
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    pairs = torch.zeros((n_want + 64, 2), dtype=torch.int32, device="cuda")
    if ee:
        bvh.broad_phase_query_from_edges_sym(xd, xd, ed, cnt, pairs, rad)
    else:
        bvh.broad_phase_query_from_verts(xd, xd, cnt, pairs, dev(r), dev(z))
    assert int(counts(cnt)[0]) == n_want
    np.testing.assert_array_equal(SC.sorted_pairs(host(pairs, np.uint32)[:n_want]), SC.sorted_pairs(want))


def _ee_query(bvh, x, el, want, n_want, dh, th=None):
    """The general query (dh an array) or the once-per-pair one (dh a number) of an edge tree against an expected set."""
    xd, ed = dev(x), dev(el)
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    pairs = torch.zeros((n_want + 64, 2), dtype=torch.int32, device="cuda")
    if np.ndim(dh):
        bvh.broad_phase_query_from_edges(xd, xd, ed, cnt, pairs, dev(dh), dev(th))
    else:
        bvh.broad_phase_query_from_edges_sym(xd, xd, ed, cnt, pairs, dh)
    assert int(counts(cnt)[0]) == n_want
    np.testing.assert_array_equal(SC.sorted_pairs(host(pairs, np.uint32)[:n_want]), SC.sorted_pairs(want))


def _edge_trees(x, el, th):
    t_o = O.lbvh_build(O.TREE_EDGE, x, el, x.shape[0])
    O.lbvh_refit(t_o, x, x, el, th)
    bvh = LBVH(O.TREE_EDGE, el.shape[0])
    xd, ed = dev(x), dev(el)
    bvh.reduce_edge_tree_aabb(xd, ed)
    bvh.construct_tree()
    bvh.update_and_refit(dev(th), xd, xd, ed)
    return t_o, bvh


@pytest.mark.parametrize("side,far", [(60, 0.05), (290, 10.3)])
def test_general_ee_query_with_one_far_reaching_edge(side, far):
    """One edge reaches fifty times and ten thousand times as far as the others.  It lies beside the sheet and meets a
    tenth of it, so that its own walk ends nowhere; looked at with its reach, the others' walks of 251,000 edges would end early."""
    x, el = _deep_sheet(side)
    away = np.zeros((2, 4), np.float32)
    away[:, 0], away[1, 2] = 0.001 * side - far, 0.01
    el = np.concatenate([el, np.array([[len(x), len(x) + 1]], np.uint32)])
    x = np.concatenate([x, away])
    dh, th = np.full(len(x), 1e-3, np.float32), np.random.default_rng(1).uniform(0, 1e-3, len(x)).astype(np.float32)
    dh[-2:] = far
    t_o, bvh = _edge_trees(x, el, th)
    want, n_want = O.lbvh_query_ee(t_o, x, x, el, dh, th)
    assert n_want > len(el)
    _ee_query(bvh, x, el, want, n_want, dh, th)


def _turning_tree(n, chain):
    """Edges whose tree turns right `chain` times past subtrees of four (all bits but one of the last `chain` of the code
    set) and then holds the others, of one code, split by their ids: up to chain + 14 right turns past inner nodes."""
    cells = []
    for k in range(chain):
        c = np.full(3, 1023.5)
        c[2 - k % 3] -= 2 ** (k // 3)
        cells += [[c - 0.25, c + 0.25]] * 4
    m = n - len(cells) - 1
    s = int(np.ceil(m ** (1 / 3)))
    g = np.stack(np.unravel_index(np.arange(m), (s, s, s)), 1) / s * 0.999 + 1023.0005
    top = np.stack([g, g + 1e-3], 1)
    top[-1, 1] = 1024.0
    pts = np.concatenate([[[np.zeros(3), np.ones(3)]], cells, top]).reshape(-1, 3)
    x = np.zeros((2 * n, 4), np.float32)
    x[:, :3] = pts
    return x, np.arange(2 * n, dtype=np.uint32).reshape(-1, 2)


@pytest.mark.parametrize("n", [65535, 66001, 131072])  # a thread per edge, a warp per 32, also in the general query
@pytest.mark.parametrize("chain", [30, 24])    # 44 turns at most; more nodes of 31 turns than are listed
@pytest.mark.parametrize("mode", ["once", "general", "far", "ends"])
def test_ee_queries_of_a_tree_with_many_turns(n, chain, mode):
    """`far`: the edge at the far corner reaches through three quarters of the scene, and meets nothing; the walks of the
    others would keep more than 64 nodes pending with its reach.  `ends`: eight edges reach so far that their stacks of 32
    fill, as the oracle's do."""
    x, el = _turning_tree(n, chain)
    z = np.zeros(len(x), np.float32)
    dh = np.full(len(x), 1e-3, np.float32)
    if mode == "far":
        dh[:2] = 768.0
    if mode == "ends":
        dh[2:18] = 1200.0
    t_o, bvh = _edge_trees(x, el, z)
    want, n_want = O.lbvh_query_ee(t_o, x, x, el, dh, z)
    if mode == "ends":
        assert n_want < 8 * (n - 9)  # their walks ended: alone they would meet every edge of a higher id
    else:
        assert n_want >= 6 * chain
    _ee_query(bvh, x, el, want, n_want, 1e-3 if mode == "once" else dh, z)


@pytest.mark.parametrize("side", [53, 210])
def test_queries_between_a_leaf_update_and_its_refit(side):
    """Leaf boxes written by themselves are what the queries of a tree of 32 levels meet, inner boxes being those of the
    refit before; after the refit all are new."""
    x, el = _deep_sheet(side)
    z = np.zeros(len(x), np.float32)
    dh = np.full(len(x), 2e-3, np.float32)
    t_o, bvh = _edge_trees(x, el, z)
    y = x + np.random.default_rng(1).normal(0, 4e-3, x.shape).astype(np.float32)
    O.lib().orc_lbvh_update_leaves(t_o.kind, O._p(t_o.sorted_get_original), t_o.n, O._p(z), O._p(y), O._p(y), O._p(el),
                                   O._p(t_o.node_aabb))
    bvh.update_leaves(dev(z), dev(y), dev(y), dev(el))
    want, n_want = O.lbvh_query_ee(t_o, y, y, el, dh, z)
    for d in (dh, 2e-3):
        _ee_query(bvh, y, el, want, n_want, d, z)
    O.lbvh_refit(t_o, y, y, el, z)
    bvh.refit()
    all_pairs, n_all = O.lbvh_query_ee(t_o, y, y, el, dh, z)
    assert n_all > n_want
    for d in (dh, 2e-3):
        _ee_query(bvh, y, el, all_pairs, n_all, d, z)


def _pairs_across(n_pairs, m):
    """Elements (m corners each) of one code whose neighbours by id lie at both sides of a gap: one long element in the gap,
    of the first id, meets every inner node above them and a leaf in fifty.  A mirrored deep tree beside them makes it a
    tree of more than 32 levels, on which no stack fills."""
    x, el = SC.deep_tree_elements("edge" if m == 2 else "face")
    x[:, :3] = np.float32(1024.0) - x[:, :3]
    corner = x[:, :3].max(1) <= 1  # the elements of the pairs' cell: thin, or they would meet all of them
    x[corner, :2] *= 0.01
    if (len(el) + 1) % 2:  # pairs start at an even id
        el = np.concatenate([el, el[-1:]])
    i = np.arange(n_pairs)
    p = np.zeros((1 + 2 * n_pairs, m, 3))
    p[:, :, 2] = 0.5
    p[0, 0, :2], p[0, 1:, :2] = [0.5, 0.05], [0.5, 0.95]
    p[1::2, :, 0], p[2::2, :, 0] = 0.1, np.where(i % 50 == 0, 0.5, 0.9)[:, None]
    p[1:, 1:, 0] += 1e-4
    p[1:, :, 1] = np.repeat(0.05 + 0.9 * i / n_pairs, 2)[:, None]
    new = np.arange(m * len(p), dtype=np.uint32).reshape(-1, m) + np.uint32(len(x))
    if m == 3:
        new = np.concatenate([new, np.zeros((len(new), 1), np.uint32)], 1)
    xn = np.zeros((m * len(p), 4), np.float32)
    xn[:, :3] = p.reshape(-1, 3)
    return np.concatenate([x, xn]), np.concatenate([el, new]), len(x)


@pytest.mark.parametrize("kind_name,n_pairs", [("face", 49900), ("face", 55000), ("edge", 49900), ("edge", 55000), ("edge", 70000)])
@pytest.mark.parametrize("once", [False, True])
def test_queries_of_more_than_a_hundred_thousand_nodes(kind_name, n_pairs, once):
    """The query of the long element pops more than 100,000 nodes (fewer with 49,900 pairs) and ends there, as the oracle's
    does, without the pairs it would meet after that."""
    ee = kind_name == "edge"
    if once and not ee:
        pytest.skip("vertices have no once-per-pair form")
    x, el, first = _pairs_across(n_pairs, 2 if ee else 3)
    kind = KINDS[kind_name][0]
    t_o = O.lbvh_build(kind, x, el, len(x))
    assert _max_inner_depth(t_o) >= 32
    z, r = np.zeros(len(x), np.float32), np.full(len(x), 1e-6, np.float32)
    O.lbvh_refit(t_o, x, x, el, z)
    bvh = LBVH(kind, el.shape[0])
    xd, ed = dev(x), dev(el)
    (bvh.reduce_edge_tree_aabb if ee else bvh.reduce_face_tree_aabb)(xd, ed)
    bvh.construct_tree()
    bvh.update_and_refit(dev(z), xd, xd, ed)
    x1 = x.copy()
    if not ee:
        x1[first, 1] = 0.95  # one vertex moves along the gap
    want, n_want = O.lbvh_query_ee(t_o, x, x, el, r, z) if ee else O.lbvh_query_vf(t_o, x, x1, r, z)
    met = int((want[:, 0] == (len(el) - 2 * n_pairs - 1 if ee else first)).sum())
    assert (met >= n_pairs // 50) == (n_pairs < 50000)
    if ee:
        _ee_query(bvh, x, el, want, n_want, 1e-6 if once else r, z)
        return
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    pairs = torch.zeros((n_want + 64, 2), dtype=torch.int32, device="cuda")
    bvh.broad_phase_query_from_verts(xd, dev(x1), cnt, pairs, dev(r), dev(z))
    assert int(counts(cnt)[0]) == n_want
    np.testing.assert_array_equal(SC.sorted_pairs(host(pairs, np.uint32)[:n_want]), SC.sorted_pairs(want))


def test_queries_of_small_scenes_take_two_launches():
    """The question whether a walk may end early and the walk itself, which holds both ways of walking."""
    lib = A.load()
    x, el = _sheet(30)
    th, dh = np.zeros(len(x), np.float32), np.full(len(x), 1e-3, np.float32)
    _, edges = _edge_trees(x, el, th)
    quads = el.reshape(-1, 2)[:400]
    fa = np.concatenate([quads, np.roll(quads, 1, 0)], 1).astype(np.uint32)
    faces = LBVH(O.TREE_FACE, len(fa))
    xd, fd, ed = dev(x), dev(fa), dev(el)
    faces.reduce_face_tree_aabb(xd, fd)
    faces.construct_tree()
    faces.update_and_refit(dev(th), xd, xd, fd)
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    pairs = torch.zeros((200000, 2), dtype=torch.int32, device="cuda")
    for query in (lambda: faces.broad_phase_query_from_verts(xd, xd, cnt, pairs, dev(dh), dev(th)),
                  lambda: edges.broad_phase_query_from_edges(xd, xd, ed, cnt, pairs, dev(dh), dev(th)),
                  lambda: edges.broad_phase_query_from_edges_sym(xd, xd, ed, cnt, pairs, 1e-3)):
        before = lib.lcs_launch_count()
        query()
        assert lib.lcs_launch_count() - before == 2


def test_small_trees_hold_little_memory():
    """A tree's memory goes by its leaves: 100 trees of 500 faces, 41 KB each for the boxes and topology and 34 KB for the
    parts where a walk may end early, fit 20 MB."""
    LBVH(O.TREE_FACE, 500)
    free = torch.cuda.mem_get_info()[0]
    trees = [LBVH(O.TREE_FACE, 500) for _ in range(100)]
    assert free - torch.cuda.mem_get_info()[0] <= 20 << 20
    del trees
