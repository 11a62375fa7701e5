"""Workloads of the contact-and-solve path, each through the entry points a simulation program calls.

Six kinds of work:

* ``contact``   one collision pass of a Newton iteration through LBVH and NarrowPhasesDetector: both trees built
                and refitted, candidates, barrier contacts, their gradient, diagonal and off-diagonal blocks applied to
                a vector, their energy, then the swept trees, candidates and the CCD step bound;
* ``pcg``       one solve through ConjugateGradientSolver (the persistent solve or the row-resident ones);
* ``pcg_batch`` many scenes' systems in one call (solve_batch);
* ``spmv``      one block matrix-vector product;
* ``elements``  the per-element cloth evaluators and the elastic energy of the C ABI;
* ``newton``    one time step of a draped cloth, of the twisted tube, or of a batch of drapes, host state in and out.

Geometry: grid sheets with the spacings of the repository's scenes (1 cm drapes, 2-3 mm tube), d_hat 1e-3 m, the
cloth material of scenes.py (mu = lambda = 80, bending 5e-3), time step 1/60 s.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from luisacomputesimulator_b200 import _capi as A
from luisacomputesimulator_b200 import scenes as S
from luisacomputesimulator_b200.collision import LBVH, NarrowPhasesDetector
from luisacomputesimulator_b200.linear import ConjugateGradientSolver, make_bsr, solve_batch, spmv
from luisacomputesimulator_b200.newton import NewtonBatch, NewtonSolver

D_HAT = 1e-3
F32, F64 = torch.float32, torch.float64


def listed():
    return [
        # two 50 x 50 sheets in contact: the collision pass of a garment-sized scene, bound by launches
        dict(name="contact_5k", kind="contact", side=50, thickness=0.0, sym=True, fp64=False),
        # 89,888 vertices, the size of the tube configuration
        dict(name="contact_90k", kind="contact", side=212, thickness=0.0, sym=True, fp64=False),
        # 401,408 vertices with a contact thickness: the general edge query, beyond what a scene of the tests holds
        dict(name="contact_400k", kind="contact", side=448, thickness=5e-4, sym=False, fp64=False),
        # the 64 x 64 cloth of the drop configuration, the solver's defaults
        dict(name="pcg_4k", kind="pcg", nx=64, nz=64, mode="default", fp64=False, contacts=True),
        # the tube's 300 x 296 grid, the solve the Newton loop runs
        dict(name="pcg_89k_single", kind="pcg", nx=300, nz=296, mode="single", fp64=False, contacts=True),
        # a ragged large system in the precision form, beyond one thread per row
        dict(name="pcg_401k_fp64", kind="pcg", nx=633, nz=634, mode="default", fp64=True, contacts=True),
        # 48 drape systems of 2,000 to 16,000 rows in one call
        dict(name="pcg_batch_48", kind="pcg_batch", scenes=48, v_min=2000, v_max=16000, fp64=False),
        # a product with a million rows (the line search and residual checks of a large scene)
        dict(name="spmv_1m", kind="spmv", nx=1000, nz=1001, contacts=True),
        # per-element gradients and Hessians of an 88,800-vertex cloth, as a host assembling its own matrix reads them
        dict(name="elements_89k", kind="elements", nx=300, nz=296),
        # one step of the drop configuration's cloth lying on the icosphere
        dict(name="newton_drape_6k", kind="newton", scene="drape", side=64, scenes=1, mode="single", fp64=False,
             line_search=False),
        # the benchmark's time step: the twisted tube after 56 steps
        dict(name="newton_tube_89k", kind="newton", scene="tube", side=0, scenes=1, mode="single", fp64=False,
             line_search=False),
        # a batch of sixteen drapes of about 4,000 vertices, as the serving loop steps them
        dict(name="newton_batch_16", kind="newton", scene="batch", side=64, scenes=16, mode="batch", fp64=False,
             line_search=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["contact", "contact", "pcg", "pcg", "pcg", "pcg_batch", "spmv", "elements", "newton", "newton"])
    if kind == "contact":
        th = rng.choice([0.0, 5e-4])
        return dict(kind=kind, side=_log(rng, 12, 440), thickness=th, sym=th == 0.0 and rng.random() < 0.5,
                    fp64=rng.random() < 0.2)
    if kind == "pcg":
        mode = rng.choice(["default", "default", "rows", "single"])
        hi = 600 if mode == "default" else 330
        return dict(kind=kind, nx=_log(rng, 10, hi), nz=_log(rng, 10, hi), mode=mode, fp64=rng.random() < 0.3,
                    contacts=rng.random() < 0.7)
    if kind == "pcg_batch":
        lo = _log(rng, 300, 4000)
        return dict(kind=kind, scenes=rng.randint(3, 48), v_min=lo, v_max=lo * rng.randint(1, 4), fp64=rng.random() < 0.3)
    if kind == "spmv":
        return dict(kind=kind, nx=_log(rng, 20, 1000), nz=_log(rng, 20, 1000), contacts=rng.random() < 0.7)
    if kind == "elements":
        return dict(kind=kind, nx=_log(rng, 12, 300), nz=_log(rng, 12, 296))
    if rng.random() < 0.35:
        return dict(kind=kind, scene="batch", side=rng.randint(20, 64), scenes=rng.randint(2, 16), mode="batch",
                    fp64=rng.random() < 0.2, line_search=False)
    mode = rng.choice(["rows", "single", "deterministic"])
    return dict(kind=kind, scene="drape", side=rng.randint(20, 110), scenes=1, mode=mode, fp64=rng.random() < 0.2,
                line_search=mode != "deterministic" and rng.random() < 0.2)


# ------------------------------------------------------------------------------------------ grids
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _rand(g, *shape, lo=-1.0, hi=1.0):
    return torch.rand(shape, generator=g, device="cuda", dtype=F64) * (hi - lo) + lo


@functools.lru_cache(maxsize=6)
def _grid(nx, nz):
    """Topology of an nx x nz vertex grid, quads split on the (i, j)-(i + 1, j + 1) diagonal: faces (F, 3), edges (E, 2)
    in lexicographic order, bending stencils (B, 4) = hinge and wings, as int64 CUDA tensors."""
    v = torch.arange(nx * nz, device="cuda").reshape(nx, nz)
    a, b, c, d = v[:-1, :-1], v[1:, :-1], v[1:, 1:], v[:-1, 1:]
    faces = torch.stack([torch.stack([a, b, c], -1), torch.stack([a, c, d], -1)], 2).reshape(-1, 3)
    pair = lambda p, q: torch.stack([p.reshape(-1), q.reshape(-1)], 1)  # noqa: E731
    edges = torch.cat([pair(v[:-1], v[1:]), pair(v[:, :-1], v[:, 1:]), pair(a, c)])
    edges = edges[torch.argsort(edges[:, 0] * (nx * nz) + edges[:, 1])]
    quad = lambda p, q, r, s: torch.stack([t.reshape(-1) for t in (p, q, r, s)], 1)  # noqa: E731
    bend = torch.cat([quad(a, c, b, d),                                                      # across the diagonals
                      quad(v[1:-1, :-1], v[1:-1, 1:], v[:-2, :-1], v[2:, 1:]),               # across (i, j)-(i, j + 1)
                      quad(v[:-1, 1:-1], v[1:, 1:-1], v[:-1, :-2], v[1:, 2:])])              # across (i, j)-(i + 1, j)
    return faces, edges, bend


def _i32(t):
    return t.to(torch.int32).contiguous()


def _pad4(t, dtype):
    out = torch.zeros((t.shape[0], 4), dtype=dtype, device="cuda")
    out[:, :3] = t.to(dtype)
    return out


# ---------------------------------------------------------------------------------------- contact
ANGLE = math.radians(20.0)  # between the two sheets, so that no edges of the two are parallel
SPACING = 2.5e-3


def _sheet_mesh(m):
    f, e, _ = _grid(m, m)
    n = m * m
    return torch.cat([f, f + n]), torch.cat([e, e + n]), n


def _sheets(case, seed):
    """Two m x m sheets, the upper one turned by ANGLE and lying over the lower one at a gap that goes below the contact
    distance in patches; and the end positions of a Newton direction of up to half a millimetre."""
    m, th = case["side"], case["thickness"]
    g = _gen(seed)
    i = (torch.arange(m, device="cuda", dtype=F64) - (m - 1) / 2) * SPACING
    X, Z = torch.meshgrid(i, i, indexing="ij")
    X, Z = X.reshape(-1), Z.reshape(-1)
    ph = _rand(g, 4, lo=0.0, hi=2 * math.pi)
    bump = lambda x, z: 1e-3 * torch.sin(63 * x + ph[0]) * torch.sin(63 * z + ph[1])  # noqa: E731
    lo = torch.stack([X, bump(X, Z), Z], 1)
    c, s = math.cos(ANGLE), math.sin(ANGLE)
    x, z = c * X - s * Z, s * X + c * Z
    t = 0.5 + 0.5 * torch.sin(90 * x + ph[2]) * torch.sin(90 * z + ph[3])
    up = torch.stack([x, bump(x, z) + th + D_HAT * (0.3 + 6.0 * t), z], 1)
    p = torch.cat([lo, up]) + _rand(g, 2 * m * m, 3) * 5e-5
    d = _rand(g, 2 * m * m, 3) * 1e-4
    d[m * m:, 1] -= 4e-4
    return _pad4(p, F32), _pad4(p + d, F32)


def _areas(x, faces, edges):
    """Face areas, and a third of the adjacent face areas per vertex and per edge (float32)."""
    p = x[:, :3].to(F64)
    fa = 0.5 * torch.linalg.cross(p[faces[:, 1]] - p[faces[:, 0]], p[faces[:, 2]] - p[faces[:, 0]]).norm(dim=1)
    va = torch.zeros(x.shape[0], dtype=F64, device="cuda").index_add_(0, faces.reshape(-1), (fa / 3).repeat_interleave(3))
    n = x.shape[0]
    key = edges[:, 0] * n + edges[:, 1]
    ea = torch.zeros(edges.shape[0], dtype=F64, device="cuda")
    for k in range(3):
        q = torch.stack([faces[:, k], faces[:, (k + 1) % 3]], 1)
        ea.index_add_(0, torch.searchsorted(key, q.min(1).values * n + q.max(1).values), fa / 3)
    return fa.to(F32), va.to(F32), ea.to(F32)


def _contact_inputs(case, seed):
    faces, edges, _ = _sheet_mesh(case["side"])
    x0, x1 = _sheets(case, seed)
    n = x0.shape[0]
    g = _gen(seed + 500009)
    fa, va, ea = _areas(x0, faces, edges)
    st = dict(x0=x0, x1=x1, faces64=faces, edges64=edges, fa=fa, va=va, ea=ea, kappa=1e7,
              d_hat=torch.full((n,), D_HAT, dtype=F32, device="cuda"),
              offset=torch.full((n,), 0.5 * case["thickness"], dtype=F32, device="cuda"),
              body=torch.full((n,), -1, dtype=torch.int32, device="cuda"))
    mass = 2.0 * va * 3600.0  # shell of 2 kg / m^2 over dt^2
    st["diag0"] = torch.zeros((n, 3, 4), dtype=F32, device="cuda")
    for k in range(3):
        st["diag0"][:, k, k] = mass
    st["b0"] = _pad4(_rand(g, n, 3) * 1e-2, F32)
    st["u"] = _pad4(_rand(g, n, 3), F32)
    return st


def _prepare_contact(case, seed):
    st = _contact_inputs(case, seed)
    n, ne = st["x0"].shape[0], st["edges64"].shape[0]
    st["faces"] = torch.zeros((st["faces64"].shape[0], 4), dtype=torch.int32, device="cuda")
    st["faces"][:, :3] = st["faces64"].to(torch.int32)
    st["edges"] = _i32(st["edges64"])
    st["ft"], st["et"] = LBVH(A.LCS_TREE_FACE, st["faces"].shape[0]), LBVH(A.LCS_TREE_EDGE, ne)
    st["det"] = NarrowPhasesDetector(n, ne)
    st["case"] = case
    st["b"], st["diag"] = torch.empty_like(st["b0"]), torch.empty_like(st["diag0"])
    while True:  # the lists at the size this scene needs, as a running program has them
        _run_contact(st)
        if not st["det"].resize_buffers():
            break
    return st


def _candidates(st, xa, xb):
    det, c = st["det"], st["case"]
    st["ft"].update_and_refit(st["offset"], xa, xb, st["faces"])
    st["et"].update_and_refit(st["offset"], xa, xb, st["edges"])
    st["ft"].broad_phase_query_from_verts(xa, xb, det.count_view(0), det.broad_phase_list_vf, st["d_hat"], st["offset"])
    if c["sym"]:
        st["et"].broad_phase_query_from_edges_sym(xa, xb, st["edges"], det.count_view(1), det.broad_phase_list_ee, D_HAT)
    else:
        st["et"].broad_phase_query_from_edges(xa, xb, st["edges"], det.count_view(1), det.broad_phase_list_ee,
                                              st["d_hat"], st["offset"])


def _run_contact(st):
    det, c, x0, x1 = st["det"], st["case"], st["x0"], st["x1"]
    st["ft"].reduce_face_tree_aabb(x0, st["faces"])
    st["et"].reduce_edge_tree_aabb(x0, st["edges"])
    st["ft"].construct_tree()
    st["et"].construct_tree()
    det.reset_broadphase_count()
    det.reset_narrowphase_count()
    det.reset_toi()
    det.reset_energy()
    _candidates(st, x0, x0)
    det.vf_dcd_query_repulsion(x0, st["faces"], st["body"], st["va"], st["fa"], st["d_hat"], st["offset"], st["kappa"])
    det.ee_dcd_query_repulsion(x0, st["edges"], st["body"], st["ea"], st["d_hat"], st["offset"], st["kappa"])
    counts = det.counts.clone()
    st["b"].copy_(st["b0"])
    st["diag"].copy_(st["diag0"])
    det.device_perPair_evaluate_gradient_hessian(st["b"], st["diag"])
    bsr, _ = det.device_assemble_contact_triplet()
    y = spmv(st["diag"], None, bsr, st["u"])
    det.compute_contact_energy(x0, st["d_hat"], st["offset"])
    det.reset_broadphase_count()
    _candidates(st, x0, x1)
    det.vf_ccd_query(x0, x1, st["faces"], st["body"], st["offset"], fp64=c["fp64"])
    det.ee_ccd_query(x0, x1, st["edges"], st["body"], st["offset"], fp64=c["fp64"])
    return dict(dcd_counts=counts, ccd_counts=det.counts, toi=det.toi, energy=det.energy, b=st["b"], diag=st["diag"], y=y)


def _near(rows, cols, m, reach):
    """Index pairs (query, cell) of the grid cells within `reach` of each query's cell."""
    off = torch.arange(-reach, reach + 1, device="cuda")
    R = (rows[:, None, None] + off[None, :, None]).expand(-1, len(off), len(off)).reshape(rows.shape[0], -1)
    Q = (cols[:, None, None] + off[None, None, :]).expand(-1, len(off), len(off)).reshape(rows.shape[0], -1)
    ok = (R >= 0) & (R < m - 1) & (Q >= 0) & (Q < m - 1)
    q = torch.arange(rows.shape[0], device="cuda")[:, None].expand_as(R)[ok]
    return q, R[ok], Q[ok]


def _dot(a, b):
    return (a * b).sum(-1)


def _on_edge(p, a, b):
    """Coefficients (1 - t, t) of p's projection on the line a b (not clamped)."""
    r = b - a
    t = _dot(r, p - a) / _dot(r, r)
    return 1 - t, t


def _closest_triangle(p, t0, t1, t2):
    r0, r1, w = t1 - t0, t2 - t0, p - t0
    a00, a01, a11, b0, b1 = _dot(r0, r0), _dot(r0, r1), _dot(r1, r1), _dot(r0, w), _dot(r1, w)
    det = a00 * a11 - a01 * a01
    s0, s1 = (a11 * b0 - a01 * b1) / det, (a00 * b1 - a01 * b0) / det
    c = torch.stack([1 - s0 - s1, s0, s1], 1)
    inside = ((c >= 0) & (c <= 1)).all(1)
    out = c.clone()
    done = inside
    for first, (k, a, b) in enumerate(((0, 1, 2), (1, 0, 2), (2, 0, 1))):
        sel = ~done & ((c[:, k] < 0) if first < 2 else torch.ones_like(done))
        e0, _ = _on_edge(p, (t0, t1, t2)[a], (t0, t1, t2)[b])
        e0 = e0.clamp(0, 1)
        z = torch.zeros_like(c)
        z[:, a], z[:, b] = e0, 1 - e0
        out = torch.where(sel[:, None], z, out)
        done = done | sel
    return out


def _closest_edges(a0, a1, b0, b1):
    r, s, w = a1 - a0, b1 - b0, b0 - a0
    rr, ss, rs = _dot(r, r), _dot(s, s), _dot(r, s)
    cr = torch.linalg.cross(r, s)
    par = _dot(cr, cr) / (rr * ss + 1e-8)
    det = rr * ss - rs * rs
    p, q = (ss * _dot(r, w) - rs * _dot(s, w)) / det, (rs * _dot(r, w) - rr * _dot(s, w)) / det
    c = torch.stack([1 - p, p, 1 - q, q], 1)
    inside = ((c >= 0) & (c <= 1)).all(1) & (par >= 1e-4)
    best, out = torch.full_like(p, math.inf), c.clone()
    one, zero = torch.ones_like(p), torch.zeros_like(p)
    for k in range(4):
        if k < 2:
            e0, e1 = _on_edge((a0, a1)[k], b0, b1)
            cand = torch.stack([one - k, zero + k, e0.clamp(0, 1), e1.clamp(0, 1)], 1)
        else:
            e0, e1 = _on_edge((b0, b1)[k - 2], a0, a1)
            cand = torch.stack([e0.clamp(0, 1), e1.clamp(0, 1), one - (k - 2), zero + (k - 2)], 1)
        d = cand[:, 0, None] * a0 + cand[:, 1, None] * a1 - cand[:, 2, None] * b0 - cand[:, 3, None] * b1
        d2 = _dot(d, d)
        take = ~inside & (d2 < best)
        best = torch.where(take, d2, best)
        out = torch.where(take[:, None], cand, out)
    return out


def _exact_contact(case, seed):
    """Every vertex-face and edge-edge pair of the two sheets from the cells under each query, in 64 bits.  (Pairs of one
    sheet never come within the contact distance: its altitudes are 1.7 mm.)"""
    st = _contact_inputs(case, seed)
    m, th = case["side"], case["thickness"]
    n = m * m
    x = st["x0"][:, :3].to(F64)
    f_all, e_all = st["faces64"], st["edges64"]
    nf, ne = f_all.shape[0] // 2, e_all.shape[0] // 2
    c, s = math.cos(ANGLE), math.sin(ANGLE)
    # cell of a point in the lower / upper sheet's own grid
    flat = lambda p, up: (c * p[:, 0] + s * p[:, 2], -s * p[:, 0] + c * p[:, 2]) if up else (p[:, 0], p[:, 2])  # noqa: E731
    cell = lambda p, up: [torch.floor(t / SPACING + (m - 1) / 2).to(torch.int64) for t in flat(p, up)]  # noqa: E731
    idx, wgt, area = [], [], []
    for up in (0, 1):  # vertices of one sheet against the faces of the other
        vq = torch.arange(n, device="cuda") + n * (1 - up)
        q, r, k = _near(*cell(x[vq], up), m, 1)
        for half in (0, 1):
            fid = 2 * (r * (m - 1) + k) + half + nf * up
            f, v = f_all[fid], vq[q]
            w = _closest_triangle(x[v], x[f[:, 0]], x[f[:, 1]], x[f[:, 2]])
            idx.append(torch.cat([v[:, None], f], 1))
            wgt.append(torch.cat([torch.ones_like(w[:, :1]), -w], 1))
            area.append(0.5 * (st["va"][v].to(F64) + st["fa"][fid].to(F64)))
            keep = ((wgt[-1][..., None] * x[idx[-1]]).sum(1).square().sum(-1)) < (th + D_HAT) ** 2
            idx[-1], wgt[-1], area[-1] = idx[-1][keep], wgt[-1][keep], area[-1][keep]
    # lower edges by lower vertex: those of the cells around each upper edge's midpoint
    lo_e, up_e = e_all[:ne], e_all[ne:]
    start = torch.searchsorted(lo_e[:, 0].contiguous(), torch.arange(n + 1, device="cuda"))
    q, r, k = _near(*cell(x[up_e].mean(1), 0), m + 1, 2)
    for slot in range(3):
        v = r * m + k
        ok = (r < m) & (k < m)
        v = torch.where(ok, v, torch.zeros_like(v))
        eid = start[v] + slot
        ok = ok & (eid < start[v + 1])
        l, rr = lo_e[eid[ok]], up_e[q[ok]]
        w = _closest_edges(x[l[:, 0]], x[l[:, 1]], x[rr[:, 0]], x[rr[:, 1]])
        w = torch.cat([w[:, :2], -w[:, 2:]], 1)
        i = torch.cat([l, rr], 1)
        keep = (w[..., None] * x[i]).sum(1).square().sum(-1) < (th + D_HAT) ** 2
        idx.append(i[keep])
        wgt.append(w[keep])
        area.append(0.5 * (st["ea"][eid[ok]][keep].to(F64) + st["ea"][ne:][q[ok]][keep].to(F64)))
    idx, w, stiff = torch.cat(idx), torch.cat(wgt), torch.cat(area) * st["kappa"]
    dh = float(np.float32(D_HAT))
    diff = (w[..., None] * x[idx]).sum(1)
    dist = diff.norm(dim=1)
    nrm, d = diff / dist[:, None], dist - float(2 * np.float32(0.5 * th))
    lg = torch.log(d / dh)
    k1 = -stiff * (dh - d) * (2 * lg - dh / d + 1)
    k2 = stiff * ((dh / d + 2) * (dh / d) - 2 * lg - 3)
    b = st["b0"].to(F64)
    b[:, :3] = b[:, :3].index_add(0, idx.reshape(-1), ((k1[:, None] * w)[..., None] * nrm[:, None]).reshape(-1, 3))
    nn = nrm[:, :, None] * nrm[:, None, :]
    diag = st["diag0"].to(F64)
    diag[:, :, :3] = diag[:, :, :3].index_add(0, idx.reshape(-1),
                                              ((k2[:, None] * w * w)[..., None, None] * nn[:, None]).reshape(-1, 3, 3))
    u = st["u"][:, :3].to(F64)
    along = _dot((w[..., None] * u[idx]).sum(1), nrm) * k2
    y = torch.zeros_like(b)
    for k in range(3):
        y[:, k] = st["diag0"][:, k, k].to(F64) * u[:, k]
    y[:, :3] = y[:, :3].index_add(0, idx.reshape(-1), ((along[:, None] * w)[..., None] * nrm[:, None]).reshape(-1, 3))
    energy = (-stiff * (d - dh) ** 2 * lg).sum().reshape(1)
    return dict(dcd_counts=None, ccd_counts=None, toi=None, energy=energy, b=b, diag=diag, y=y)


# ------------------------------------------------------------------------------------ linear systems
SPRING = ((1, 0), (0, 1), (1, 1))     # the grid's edges
BEND = ((1, -1), (2, 1), (1, 2))      # the wing pairs of its hinges


def _csr(n, rows, cols, blocks):
    order = torch.argsort(rows * n + cols, stable=True)
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    val = blocks[order].transpose(1, 2).reshape(-1, 9).to(F32).contiguous()  # column-major
    return rp, cols[order], val


def _system(nx, nz, contacts, g):
    """Diagonal blocks, the cloth's off-diagonal blocks and contact blocks of one sheet's Newton system (a sum of
    k (u . (xi - xj))^2 terms over edges and wing pairs, point-triangle contacts between far parts, and inertia)."""
    n = nx * nz
    v = torch.arange(n, device="cuda").reshape(nx, nz)
    D = torch.zeros((n, 3, 3), dtype=F64, device="cuda")
    D += torch.eye(3, device="cuda", dtype=F64) * (0.72 * (0.75 + 0.25 * _rand(g, n, 1, 1)))
    rows, cols, blocks = [], [], []
    for di, dj in SPRING + BEND:
        if nx <= di or nz <= abs(dj):
            continue
        p = v[:nx - di, -dj:] if dj < 0 else v[:nx - di, :nz - dj]
        q = v[di:, :nz + dj] if dj < 0 else v[di:, dj:]
        p, q = p.reshape(-1), q.reshape(-1)
        k = 12.0 if (di, dj) in SPRING else 1.0
        u = torch.tensor([di, 0.0, dj], device="cuda", dtype=F64) + 0.2 * _rand(g, p.shape[0], 3)
        u = u / u.norm(dim=1, keepdim=True)
        H = k * (u[:, :, None] * u[:, None, :]) + 0.05 * k * torch.eye(3, device="cuda", dtype=F64)
        D.index_add_(0, p, H)
        D.index_add_(0, q, H)
        rows += [p, q]
        cols += [q, p]
        blocks += [-H, -H]
    Am = _csr(n, torch.cat(rows), torch.cat(cols), torch.cat(blocks))
    if not contacts:
        return D, Am, None
    m = max(n // 24, 1)  # a patch of contacts: vertices of one region against triangles of another
    base = int(n // 5)
    p = base + torch.arange(m, device="cuda")
    t = (torch.arange(m, device="cuda") + n // 2 + nz // 2)
    idx = torch.stack([p, t, t + 1, t + nz], 1) % n
    bary = torch.rand((m, 3), generator=g, device="cuda", dtype=F64) + 0.05
    w = torch.cat([torch.ones((m, 1), device="cuda", dtype=F64), -bary / bary.sum(1, keepdim=True)], 1)
    nr = _rand(g, m, 3)
    nr = nr / nr.norm(dim=1, keepdim=True)
    nn = 40.0 * nr[:, :, None] * nr[:, None, :]
    rows, cols, blocks = [], [], []
    for i in range(4):
        D.index_add_(0, idx[:, i], (w[:, i] ** 2)[:, None, None] * nn)
        for j in range(4):
            if i != j:
                rows.append(idx[:, i])
                cols.append(idx[:, j])
                blocks.append((w[:, i] * w[:, j])[:, None, None] * nn)
    return D, Am, _csr(n, torch.cat(rows), torch.cat(cols), torch.cat(blocks))


def _diag4(D):
    out = torch.zeros((D.shape[0], 3, 4), dtype=F32, device="cuda")
    out[:, :, :3] = D.transpose(1, 2).to(F32)
    return out


def _matrices(case, seed):
    """(rows per scene, diag, A, B, right-hand side) of a linear case; A, B: (row_ptr, col, val) or None."""
    g = _gen(seed)
    if case["kind"] != "pcg_batch":
        D, Am, B = _system(case["nx"], case["nz"], case["contacts"], g)
        n = D.shape[0]
        return [n], _diag4(D), Am, B, _pad4(_rand(g, n, 3), F32)
    parts, sizes = [], []
    for k in range(case["scenes"]):  # sizes spread over the case's range
        f = ((k * 29) % case["scenes"] + 0.5) / case["scenes"]
        side = max(4, int(round(math.sqrt(case["v_min"] * (case["v_max"] / case["v_min"]) ** f))))
        parts.append(_system(side, side, True, g))
        sizes.append(side * side)
    off = np.concatenate([[0], np.cumsum(sizes)])

    def cat(k):
        nnz = np.concatenate([[0], np.cumsum([p[k][1].shape[0] for p in parts])])
        rp = torch.cat([p[k][0][:-1] + int(o) for p, o in zip(parts, nnz)] + [torch.tensor([int(nnz[-1])], device="cuda")])
        return rp, torch.cat([p[k][1] + int(o) for p, o in zip(parts, off)]), torch.cat([p[k][2] for p in parts])
    n = int(off[-1])
    return sizes, _diag4(torch.cat([p[0] for p in parts])), cat(1), cat(2), _pad4(_rand(g, n, 3), F32)


def _prepare_linear(case, seed):
    sizes, diag, Am, B, b = _matrices(case, seed)
    n = diag.shape[0]
    bsr = lambda M: None if M is None else make_bsr(n, _i32(M[0]), _i32(M[1]), M[2])  # noqa: E731
    st = dict(case=case, diag=diag, A=bsr(Am), B=bsr(B), b=b, x=torch.empty_like(b))
    if case["kind"] == "spmv":
        return st
    st["solver"] = ConjugateGradientSolver(n)
    if case["kind"] == "pcg_batch":
        st["offsets"] = torch.tensor(np.concatenate([[0], np.cumsum(sizes)]), dtype=torch.int32, device="cuda")
        st["stats"] = torch.zeros((len(sizes), 4), dtype=torch.int32, device="cuda")
    return st


def _run_linear(st):
    c = st["case"]
    if c["kind"] == "spmv":
        return spmv(st["diag"], st["A"], st["B"], st["b"], st["x"])
    if c["kind"] == "pcg_batch":
        solve_batch(st["solver"], st["offsets"], st["diag"], st["A"], st["B"], st["b"], st["x"], st["stats"],
                    check_every=25, fp64_dots=c["fp64"])
        return st["x"]
    r = st["solver"].device_solve(st["diag"], st["A"], st["B"], st["b"], st["x"], fp64_dots=c["fp64"],
                                  rows=c["mode"] == "rows", single_reduction=c["mode"] == "single")
    return dict(x=st["x"], iterations=r["iterations"])


def _exact_linear(case, seed):
    sizes, diag, Am, B, b = _matrices(case, seed)
    n = diag.shape[0]
    D = diag[:, :, :3].to(F64).transpose(1, 2)
    mats = []
    for M in (Am, B):
        if M is not None:
            r = torch.repeat_interleave(torch.arange(n, device="cuda"), M[0][1:] - M[0][:-1])
            mats.append((r, M[1], M[2].to(F64).reshape(-1, 3, 3).transpose(1, 2)))

    def mul(x):
        y = (D @ x[..., None])[..., 0]
        for r, c, v in mats:
            y.index_add_(0, r, (v @ x[c][..., None])[..., 0])
        return y
    pad = lambda t: torch.cat([t, torch.zeros_like(t[:, :1])], 1)  # noqa: E731
    rhs = b[:, :3].to(F64)
    if case["kind"] == "spmv":
        return pad(mul(rhs))
    sc = torch.repeat_interleave(torch.arange(len(sizes), device="cuda"), torch.tensor(sizes, device="cuda"))
    dots = lambda p, q: torch.zeros(len(sizes), dtype=F64, device="cuda").index_add_(0, sc, _dot(p, q))  # noqa: E731
    minv = torch.linalg.inv(D)
    x, r, p = torch.zeros_like(rhs), rhs.clone(), torch.zeros_like(rhs)
    rz0, on, r0 = None, torch.ones(len(sizes), dtype=torch.bool, device="cuda"), None
    for it in range(100):  # the solver's rule: |r| <= 1e-4 |r0| or r.z < 1e-10, looked at every 25 iterations
        z = (minv @ r[..., None])[..., 0]
        rz, rr = dots(r, z), dots(r, r).sqrt()
        r0 = rr if r0 is None else r0
        if it % 25 == 0:
            on = on & ~((rz < 1e-10) | (rr <= 1e-4 * r0))
        beta = torch.zeros_like(rz) if rz0 is None else torch.where(rz0 < 1e-10, 0.0, rz / rz0)
        p = z + beta[sc][:, None] * p
        q = mul(p)
        alpha = torch.where(on, rz / dots(p, q), 0.0)[sc][:, None]
        x, r, rz0 = x + alpha * p, r - alpha * q, rz
    return pad(x) if case["kind"] == "pcg_batch" else dict(x=pad(x), iterations=None)


# ----------------------------------------------------------------------------------------- elements
def _cloth(case, seed):
    """A jittered sheet with the rest shape of a flat one: positions and per-element rest data (float32)."""
    nx, nz = case["nx"], case["nz"]
    faces, edges, bend = _grid(nx, nz)
    g = _gen(seed)
    n, h = nx * nz, 2e-3
    v = torch.arange(n, device="cuda")
    rest = torch.zeros((n, 3), dtype=F64, device="cuda")
    rest[:, 0], rest[:, 2] = (v // nz) * h, (v % nz) * h
    p = rest + 0.15 * h * _rand(g, n, 3)
    a, b = rest[faces[:, 1]] - rest[faces[:, 0]], rest[faces[:, 2]] - rest[faces[:, 0]]
    a1 = a / a.norm(dim=1, keepdim=True)
    nrm = torch.linalg.cross(a, b)
    area = 0.5 * nrm.norm(dim=1)
    a2 = torch.linalg.cross(nrm, a)
    a2 = a2 / a2.norm(dim=1, keepdim=True)
    dm = torch.stack([torch.stack([_dot(a1, a), _dot(a1, b)], 1), torch.stack([_dot(a2, a), _dot(a2, b)], 1)], 1)
    inv = torch.linalg.inv(dm).transpose(1, 2).reshape(-1, 4)  # columns of Dm^-1
    e = rest[bend[:, 1]] - rest[bend[:, 0]]
    w0 = torch.linalg.cross(e, rest[bend[:, 2]] - rest[bend[:, 0]]).norm(dim=1)
    w1 = torch.linalg.cross(e, rest[bend[:, 3]] - rest[bend[:, 0]]).norm(dim=1)
    f32 = lambda t: t.to(F32).contiguous()  # noqa: E731
    return dict(x=_pad4(p, F32), xt=_pad4(p + 1e-4 * _rand(g, n, 3), F32), faces=faces, edges=edges, bend=bend,
                mass=f32(2.0 * h * h * (0.75 + 0.25 * _rand(g, n))), rest_len=f32((rest[edges[:, 0]] - rest[edges[:, 1]]).norm(dim=1)),
                k_spring=f32(80.0 * (1 + 0.2 * _rand(g, edges.shape[0]))), dm_inv=f32(inv), area=f32(area),
                mu_lambda=f32(80.0 * (1 + 0.2 * _rand(g, faces.shape[0], 2))), angle=f32(0.3 * _rand(g, bend.shape[0])),
                hbar=f32((w0 + w1) / 2 / (3 * e.norm(dim=1))), k_bend=f32(5e-3 * (1 + 0.2 * _rand(g, bend.shape[0]))))


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _prepare_elements(case, seed):
    st = _cloth(case, seed)
    st["faces4"] = torch.zeros((st["faces"].shape[0], 4), dtype=torch.int32, device="cuda")
    st["faces4"][:, :3] = st["faces"].to(torch.int32)
    st["edges"], st["bend"] = _i32(st["edges"]), _i32(st["bend"])
    ne, nf, nb = st["edges"].shape[0], st["faces4"].shape[0], st["bend"].shape[0]
    new = lambda *s: torch.zeros(s, dtype=F32, device="cuda")  # noqa: E731
    st["out"] = dict(spring_g=new(ne, 2, 4), spring_h=new(ne, 4, 3, 4), face_g=new(nf, 3, 4), face_h=new(nf, 9, 3, 4),
                     bend_g=new(nb, 4, 4), bend_h=new(nb, 16, 3, 4), energy=torch.zeros(4, dtype=F64, device="cuda"))
    m = A.ClothElements()
    m.n_verts, m.n_springs, m.n_stretch_faces, m.n_bending = st["x"].shape[0], ne, nf, nb
    for field, t in (("mass", "mass"), ("springs", "edges"), ("spring_rest_len", "rest_len"), ("spring_stiffness", "k_spring"),
                     ("stretch_faces", "faces4"), ("stretch_dm_inv", "dm_inv"), ("stretch_area", "area"),
                     ("stretch_mu_lambda", "mu_lambda"), ("bending_edges", "bend"), ("bending_rest_angle", "angle"),
                     ("bending_hbar", "hbar"), ("bending_stiffness", "k_bend")):
        setattr(m, field, _ptr(st[t]))
    m.bending_scaling = 1.0
    st["cloth"] = m
    return st


def _run_elements(st):
    lib, o, p = A.load(), st["out"], {k: _ptr(t) for k, t in st.items() if isinstance(t, torch.Tensor)}
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    A.check(lib.lcs_eval_springs(p["x"], p["edges"], p["rest_len"], p["k_spring"], st["edges"].shape[0],
                                 _ptr(o["spring_g"]), _ptr(o["spring_h"]), s), "lcs_eval_springs")
    A.check(lib.lcs_eval_stretch_faces(p["x"], p["faces4"], p["dm_inv"], p["area"], p["mu_lambda"], st["faces4"].shape[0],
                                       _ptr(o["face_g"]), _ptr(o["face_h"]), s), "lcs_eval_stretch_faces")
    A.check(lib.lcs_eval_bending(p["x"], p["bend"], p["angle"], p["hbar"], p["k_bend"], 1.0, st["bend"].shape[0],
                                 _ptr(o["bend_g"]), _ptr(o["bend_h"]), s), "lcs_eval_bending")
    A.check(lib.lcs_material_energy(C.byref(st["cloth"]), p["x"], p["xt"], 1.0 / 60.0, 1e9, _ptr(o["energy"]), s),
            "lcs_material_energy")
    return o


def _record(blocks):
    """(n, k, 3, 3) blocks as float3x3 records: three columns of four values each."""
    out = torch.zeros(blocks.shape[:2] + (3, 4), dtype=F64, device="cuda")
    out[..., :3] = blocks.transpose(2, 3)
    return out


def _rows4(g):
    return torch.cat([g, torch.zeros_like(g[..., :1])], -1)


def _outer(a, b):
    return a[:, :, None] * b[:, None, :]


def _exact_elements(case, seed):
    st = {k: (t.to(F64) if t.dtype == F32 else t) for k, t in _cloth(case, seed).items()}
    x, eye = st["x"][:, :3], torch.eye(3, dtype=F64, device="cuda")
    h2 = float(np.float32(1.0) / (np.float32(1.0 / 60.0) * np.float32(1.0 / 60.0)))
    dx = x - st["xt"][:, :3]
    energy = [(0.5 * h2 * _dot(dx, dx) * st["mass"]).sum()]
    # springs: gradient and Hessian with the compressive part of the geometric term dropped
    d = x[st["edges"][:, 0]] - x[st["edges"][:, 1]]
    l, L, k = d.norm(dim=1), st["rest_len"], st["k_spring"]
    g = (k * (l - L) / l)[:, None] * d
    uu = _outer(d, d) / (l * l)[:, None, None]
    H = k[:, None, None] * uu + (k * (1 - L / l).clamp(min=0))[:, None, None] * (eye - uu)
    out = dict(spring_g=_rows4(torch.stack([g, -g], 1)), spring_h=_record(torch.stack([H, H, -H, -H], 1)))
    energy.append((0.5 * k * (l - L) ** 2).sum())
    # Baraff-Witkin stretch and shear, Hessian in F projected to positive semi-definite
    f, dm, area, (mu, lam) = st["faces"], st["dm_inv"], st["area"], st["mu_lambda"].unbind(1)
    e1, e2 = x[f[:, 1]] - x[f[:, 0]], x[f[:, 2]] - x[f[:, 0]]
    Fu, Fv = e1 * dm[:, 0:1] + e2 * dm[:, 1:2], e1 * dm[:, 2:3] + e2 * dm[:, 3:4]
    su, sv, i6 = Fu.norm(dim=1), Fv.norm(dim=1), _dot(Fu, Fv)
    Pu = (mu * (su - 1) / su)[:, None] * Fu + (lam * i6)[:, None] * Fv
    Pv = (mu * (sv - 1) / sv)[:, None] * Fv + (lam * i6)[:, None] * Fu
    w = torch.stack([torch.stack([-(dm[:, 0] + dm[:, 1]), -(dm[:, 2] + dm[:, 3])], 1),
                     torch.stack([dm[:, 0], dm[:, 2]], 1), torch.stack([dm[:, 1], dm[:, 3]], 1)], 1)
    out["face_g"] = _rows4(area[:, None, None] * (w[:, :, 0:1] * Pu[:, None] + w[:, :, 1:2] * Pv[:, None]))
    i2 = su * su + sv * sv
    lam0 = 0.5 * (i2 + torch.sqrt(12 * i6 * i6 + i2 * i2))
    q = torch.cat([i6[:, None] * Fu + lam0[:, None] * Fv, i6[:, None] * Fv + lam0[:, None] * Fu], 1)
    q = q / q.norm(dim=1, keepdim=True)
    sg = torch.sign(i6)[:, None, None]
    T = 0.5 * torch.cat([torch.cat([eye.expand(len(f), 3, 3), sg * eye], 2), torch.cat([sg * eye, eye.expand(len(f), 3, 3)], 2)], 1)
    tq = (T @ q[..., None])[..., 0]
    H6 = lam[:, None, None] * (i6.abs()[:, None, None] * (T - _outer(tq, tq) / _dot(tq, tq)[:, None, None]) +
                               lam0[:, None, None] * _outer(q, q))
    for k, (F, s) in enumerate(((Fu, su), (Fv, sv))):
        u = F / s[:, None]
        B = mu[:, None, None] * ((1 - 1 / s).clamp(min=0)[:, None, None] * eye + (1 / s).clamp(max=1)[:, None, None] * _outer(u, u))
        H6[:, 3 * k:3 * k + 3, 3 * k:3 * k + 3] += B
    H4 = H6.reshape(-1, 2, 3, 2, 3)
    K = area[:, None, None, None, None] * torch.einsum("nac,ncrds,nbd->nabrs", w, H4, w)
    order = [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 0), (1, 2), (2, 0), (2, 1)]
    out["face_h"] = _record(torch.stack([K[:, a, b] for a, b in order], 1))
    energy.append((area * (0.5 * mu * ((su - 1) ** 2 + (sv - 1) ** 2) + 0.5 * lam * i6 * i6)).sum())
    # dihedral bending, Gauss-Newton Hessian
    p0, p1, p2, p3 = (x[st["bend"][:, k]] for k in range(4))
    cr = lambda a, b: torch.linalg.cross(a, b)  # noqa: E731
    e0 = p0 - p1
    m1, m2 = cr(e0, p2 - p1), cr(p3 - p1, e0)
    s1, s2, l = _dot(m1, m1), _dot(m2, m2), e0.norm(dim=1)
    n1, n2 = cr(p1 - p2, p0 - p2), cr(p0 - p3, p1 - p3)
    theta = torch.atan2(_dot(cr(n2, n1), p1 - p0) / l, _dot(n1, n2))
    g2, g3 = (-l / s1)[:, None] * m1, (-l / s2)[:, None] * m2
    a1, a2 = -_dot(e0, p2 - p0) / (l * s1), _dot(e0, p3 - p0) / (l * s2)
    b1, b2 = _dot(e0, p2 - p1) / (l * s1), _dot(e0, p3 - p1) / (l * s2)
    g1, g0 = a1[:, None] * m1 - a2[:, None] * m2, b1[:, None] * m1 + b2[:, None] * m2
    G = torch.stack([g0, g1, g2, g3], 1)
    k = st["k_bend"] * st["hbar"]
    out["bend_g"] = _rows4((k * (theta - st["angle"]))[:, None, None] * G)
    order = [(i, i) for i in range(4)] + [(i, j) for i in range(4) for j in range(4) if i != j]
    out["bend_h"] = _record(torch.stack([k[:, None, None] * _outer(G[:, i], G[:, j]) for i, j in order], 1))
    energy.append((0.5 * k * (theta - st["angle"]) ** 2).sum())
    out["energy"] = torch.stack(energy)
    return out


# ------------------------------------------------------------------------------------------- newton
RADIUS = 0.2


@functools.lru_cache(maxsize=40)
def _drape_scene(side, subdiv):
    """A side x side cloth (1 cm spacing, less where that would reach round the sphere) over a pinned icosphere."""
    return S.cloth_on_sphere(n=side, spacing=min(0.01, 0.5 / side), subdiv=subdiv, radius=RADIUS)


def _drape_state(sc, side, seed):
    """The cloth laid on the sphere along its geodesics, 0.4 to 0.9 d_hat away, moving down at a few cm/s."""
    rng = np.random.default_rng(int(seed) * 31 + side)
    n = side * side
    x, v = sc.x.copy(), np.zeros_like(sc.x)
    p = sc.x[:n].astype(np.float64)
    r = np.maximum(np.hypot(p[:, 0], p[:, 2]), 1e-9)
    R = RADIUS + D_HAT * rng.uniform(0.4, 0.9, n)
    x[:n, 0] = R * np.sin(r / RADIUS) * p[:, 0] / r
    x[:n, 2] = R * np.sin(r / RADIUS) * p[:, 2] / r
    x[:n, 1] = R * np.cos(r / RADIUS)
    v[:n, :3] = rng.normal(0.0, 0.01, (n, 3))
    v[:n, 1] -= 0.05
    return x, v


@functools.lru_cache(maxsize=1)
def _tube():
    """The 300 x 296 tube after 56 steps of its run (its two rings turned against each other, touching itself)."""
    z = np.load("tests/golden/tube88k_state.npz")
    sc = S.twisted_tube(300, 296)
    x, v = sc.x.copy(), np.zeros_like(sc.x)
    x[:, :3], v[:, :3] = z["x"], z["v"]
    return sc, x, v, int(z["frame"])


def _sides(case):
    return [max(16, case["side"] - 3 * (k % 5)) for k in range(case["scenes"])]


def _prepare_newton(case, seed):
    frame = 0
    opts = dict(fp64=case["fp64"])
    if case["scene"] == "tube":
        sc, x, v, frame = _tube()
        v = v.copy()  # the seed's share: velocities off by about a millimetre per second
        free = sc.pinned == 0
        v[free, :3] += np.random.default_rng(seed).normal(0.0, 1e-3, (int(free.sum()), 3)).astype(np.float32)
        solver = NewtonSolver(sc, single_reduction=True, **opts)
    elif case["scene"] == "drape":
        sc = _drape_scene(case["side"], 4)
        x, v = _drape_state(sc, case["side"], seed)
        solver = NewtonSolver(sc, single_reduction=case["mode"] == "single", deterministic=case["mode"] == "deterministic",
                              energy_linesearch=case["line_search"], **opts)
    else:
        scs = [_drape_scene(s, 3) for s in _sides(case)]
        states = [_drape_state(sc, s, seed + 101 * k) for k, (sc, s) in enumerate(zip(scs, _sides(case)))]
        x, v = (np.concatenate([s[k] for s in states]) for k in (0, 1))
        solver = NewtonBatch(scs, **opts)
    pin = lambda a: torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()  # noqa: E731
    return dict(case=case, solver=solver, frame=frame, x=pin(x), v=pin(v), xo=pin(x * 0), vo=pin(v * 0))


def _run_newton(st):
    """One time step from the host's positions and velocities (lcs_newton_set_frame, lcs_newton_step_host)."""
    h, lib = st["solver"].h, st["solver"].lib
    A.check(lib.lcs_newton_set_frame(h, st["frame"]), "lcs_newton_set_frame")
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    A.check(lib.lcs_newton_step_host(h, p(st["x"]), p(st["v"]), p(st["xo"]), p(st["vo"]), C.byref(st["solver"].stats)),
            "lcs_newton_step_host")
    return dict(x=st["xo"], v=st["vo"])


# ---------------------------------------------------------------------------------------- interface
def prepare(case, seed):
    if case["kind"] == "contact":
        return _prepare_contact(case, seed)
    if case["kind"] == "elements":
        return _prepare_elements(case, seed)
    if case["kind"] == "newton":
        return _prepare_newton(case, seed)
    return _prepare_linear(case, seed)


def run(state):
    if "det" in state:
        return _run_contact(state)
    if "cloth" in state:
        return _run_elements(state)
    if "frame" in state:
        return _run_newton(state)
    return _run_linear(state)


def exact(case, seed):
    """64-bit values.  Newton steps have none: their solves stop at 100 iterations, long before the digits settle."""
    if case["kind"] == "contact":
        return _exact_contact(case, seed)
    if case["kind"] == "elements":
        return _exact_elements(case, seed)
    if case["kind"] == "newton":
        return None
    return _exact_linear(case, seed)


def work(case):
    if case["kind"] == "contact":  # positions, elements and per-vertex data in, sorted trees' boxes, blocks and vectors out
        n = 2 * case["side"] ** 2
        f, e = 2 * n, 3 * n
        return {"bytes": n * (16 * 3 + 12 + 2 * 64 + 2 * 16) + f * (16 + 4 + 2 * 64) + e * (8 + 4 + 2 * 64), "flops": 600 * n}
    if case["kind"] == "elements":
        n = case["nx"] * case["nz"]
        return {"bytes": n * (36 + 3 * (16 + 224) + 2 * (44 + 480) + 3 * (28 + 832)), "flops": n * (3 * 60 + 2 * 900 + 3 * 400)}
    if case["kind"] == "newton":
        n = {"drape": case["side"] ** 2 + 2562, "tube": 88800, "batch": sum(s * s + 642 for s in _sides(case))}[case["scene"]]
        # mesh, material data and state once; two Newton iterations' solves of fifty iterations
        return {"bytes": n * (64 + 2 * 52 + 3 * 40 + 12 * 8), "flops": 2 * 50 * n * (13 * 18 + 40)}
    if case["kind"] == "pcg_batch":
        n = case["scenes"] * math.sqrt(case["v_min"] * case["v_max"])
        return {"bytes": n * (48 + 32 + 12 * 40 + 20), "flops": 50 * n * (13 * 18 + 40)}
    n = case["nx"] * case["nz"]
    nb = 12 + (0.5 if case["contacts"] else 0.0)
    return {"bytes": n * (48 + 32 + 4 + nb * 40), "flops": (1 if case["kind"] == "spmv" else 75) * n * ((nb + 1) * 18 + 40)}


def tolerance(case):
    """About four times what another summation order, another solver form or the 64-bit values show."""
    if case["kind"] == "contact":  # differences of nearby 32-bit positions against a gap of a few tenths of a millimetre
        return {"rel": 1e-4, "max": 5e-3}
    if case["kind"] == "elements":  # the dihedral angle's arc cosine: 4e-5 of the bending gradient
        return {"rel": 1.5e-4, "max": 2e-2}
    if case["kind"] == "spmv":
        return {"rel": 2e-6, "max": 1e-4}
    if case["kind"] == "newton":  # classic against single-reduction recurrences: 2.7e-4 of the velocities, 4e-3 of one
        return {"rel": 1e-3, "max": 2e-2}
    return {"rel": 4e-5, "max": 2e-3}
