"""The coarsest inverse (panel-wise Gauss-Jordan) and its application, on dense
matrices that need row swaps, against numpy's FP64 solve."""
import numpy as np
import pytest

import homo3d_b200 as H
from tests.conftest import random_field, to_lib_field

pytestmark = pytest.mark.gpu


def _dense(st, dims):
    nx, ny, nz = dims
    nv = nx * ny * nz
    K = np.zeros((nv, 3, nv, 3))
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    v = (x + nx * (y + ny * z)).ravel()
    for d in range(27):
        dx, dy, dz = d % 3 - 1, d // 3 % 3 - 1, d // 9 - 1
        w = ((x + dx) % nx + nx * ((y + dy) % ny + ny * ((z + dz) % nz))).ravel()
        K[v, :, w, :] += st[v, d].reshape(nv, 3, 3)
    return K.reshape(3 * nv, 3 * nv)


# coarsest grids of 4^3 (192 unknowns: whole panels), 5^3 (375: a last panel of 7),
# 5 x 6 x 7 (630), 6 x 7 x 8 (1008: the widest one-row launch), 7^3 (1029: two rows per
# thread, a last panel of 5) and 8^3 (1536, the largest)
@pytest.mark.parametrize("reso,project", [(8, 0), (10, 1), ((9, 11, 13), 0), ((12, 14, 15), 1), (14, 0), (15, 0)])
def test_coarsest_inverse(torch_cuda, reso, project):
    hd = H.Homogenization(reso, coarse_mode=H.COARSE_PROJECT if project else H.COARSE_EXACT)
    L = hd.nlevels - 1
    g, dims, nv = hd.mg.grids[L], hd.dims[L], hd.nv(L)
    rng = np.random.default_rng(nv)
    g.set(H.FIELD_STENCIL, rng.uniform(-1, 1, (nv, 27, 9)))
    g.assembleHostMatrix()
    K = _dense(g.get(H.FIELD_STENCIL).astype(np.float64), dims)
    f = to_lib_field(random_field(nv, 3))
    g.set(H.FIELD_F, f)
    g.solveHostEquation()
    b = f.astype(np.float64)  # [6, nv, 3]
    if project:
        b -= b.mean(axis=1, keepdims=True)
    ref = np.linalg.solve(K, b.reshape(6, -1).T).T
    got = g.get(H.FIELD_U).reshape(6, -1)
    # FP32 results: half an ulp, and cond(K) times FP64 rounding
    tol = 6e-8 + 1e-15 * np.linalg.cond(K) * 3 * nv
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max()
    hd.close()


def test_singular_coarsest_matrix_is_refused(torch_cuda):
    hd = H.Homogenization(10)
    g = hd.mg.grids[-1]
    st = np.random.default_rng(0).uniform(-1, 1, (hd.nv(hd.nlevels - 1), 27, 9))
    st[:, :, [0, 3, 6]] = 0  # no row couples to the first component
    g.set(H.FIELD_STENCIL, st)
    with pytest.raises(H.H3DError) as e:
        g.assembleHostMatrix()
    assert e.value.code == H.H3D_ERR_SINGULAR
    hd.close()
