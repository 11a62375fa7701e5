"""The per-element evaluators at element counts around their warp and block sizes (32 elements per warp, 128 per block),
against the oracle: springs and stretch faces bit for bit, bending Hessians within 2e-6 of the largest entry (the
dihedral angle's acosf differs between CUDA and glibc by an ulp or so), with the words behind the outputs untouched."""
import ctypes as C

import numpy as np
import pytest
import torch

from luisacomputesimulator_b200 import _capi as A
from luisacomputesimulator_b200 import scenes as S
from oracle import oracle as O
from tests.gpu_util import dev, host

pytestmark = pytest.mark.gpu


def _ptr(t):
    return C.c_void_p(t.data_ptr())


@pytest.fixture(scope="module")
def cloth():
    sc = S.twisted_tube(24, 20)
    x = sc.x.copy()
    x[:, :3] += np.random.default_rng(5).normal(0, 2e-3, (sc.num_verts, 3)).astype(np.float32)
    return sc, x, dev(x)


def _outputs(n, grads, blocks):
    guard = 64  # floats behind each output
    g = torch.full((n * grads * 4 + guard,), 7.0, dtype=torch.float32, device="cuda")
    h = torch.full((n * blocks * 12 + guard,), 7.0, dtype=torch.float32, device="cuda")
    return g, h, guard


def _read(t, guard, shape):
    a = host(t)
    assert np.all(a[-guard:] == 7.0)
    return a[:-guard].reshape(shape)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 127, 128, 129, 1000])
def test_evaluators_at_odd_counts(cloth, n):
    sc, x, xd = cloth
    lib = A.load()
    e, k = sc.edges[:n], np.full(n, sc.spring_k, np.float32)
    g, h, gu = _outputs(n, 2, 4)
    ed, rl, kd = dev(e), dev(sc.rest_len[:n]), dev(k)
    A.check(lib.lcs_eval_springs(_ptr(xd), _ptr(ed), _ptr(rl), _ptr(kd), n, _ptr(g), _ptr(h), None))
    wg, wh = O.eval_springs(x, e, sc.rest_len[:n], k)
    np.testing.assert_array_equal(_read(g, gu, wg.shape), wg)
    np.testing.assert_array_equal(_read(h, gu, wh.shape), wh)

    m = min(n, sc.stretch_faces.shape[0])
    f, dm, ar = sc.stretch_faces[:m], sc.stretch_dm_inv[:m], sc.stretch_area[:m]
    ml = np.tile(np.float32([sc.stretch_mu, sc.stretch_lambda]), (m, 1))
    g, h, gu = _outputs(m, 3, 9)
    keep = [dev(f), dev(dm), dev(ar), dev(ml)]
    A.check(lib.lcs_eval_stretch_faces(_ptr(xd), *[_ptr(t) for t in keep], m, _ptr(g), _ptr(h), None))
    wg, wh = O.eval_stretch_faces(x, f, dm, ar, ml)
    np.testing.assert_array_equal(_read(g, gu, wg.shape), wg)
    np.testing.assert_array_equal(_read(h, gu, wh.shape), wh)

    m = min(n, sc.bending.shape[0])
    st, ra, hb, kb = sc.bending[:m], sc.bending_rest_angle[:m], sc.bending_hbar[:m], np.full(m, sc.bending_k, np.float32)
    g, h, gu = _outputs(m, 4, 16)
    keep = [dev(st), dev(ra), dev(hb), dev(kb)]
    A.check(lib.lcs_eval_bending(_ptr(xd), *[_ptr(t) for t in keep], float(sc.bending_scaling), m, _ptr(g), _ptr(h), None))
    wg, wh = O.eval_bending(x, st, ra, hb, kb, sc.bending_scaling)
    np.testing.assert_allclose(_read(h, gu, wh.shape), wh, rtol=0, atol=2e-6 * np.abs(wh).max())
    # an acosf difference of d radians moves the gradient by d k |dtheta/dx|, with k |dtheta/dx_i| = sqrt(k trace H_ii)
    kg = np.sqrt((kb * np.float32(sc.bending_scaling) * hb).astype(np.float64)[:, None] *
                 np.einsum("sicc->si", wh[:, :4, :, :3].astype(np.float64))).max()
    np.testing.assert_allclose(_read(g, gu, wg.shape), wg, rtol=0, atol=2e-6 * np.abs(wg).max() + 1e-6 * kg)
