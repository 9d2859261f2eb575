"""The quotients of the level-0 Gauss-Seidel step are the FP32 divisions, to the last bit."""
import numpy as np
import pytest

import homo3d_b200 as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rho", [1.0, 0.3, 0.0217, 0.0])
@pytest.mark.parametrize("w", [1.0, 0.7])
def test_first_colour_from_zero_is_a_division(torch_cuda, rho, w):
    """from u = 0 on a uniform density, the vertices of the first colour (odd in x, y and
    z) become w f / k: their neighbours are 0 and the self block is diagonal"""
    n = 16
    hd = H.Homogenization(n)
    hd.update(torch_cuda.full((n ** 3,), rho, device="cuda"))
    f = np.random.default_rng(1).uniform(-1, 1, (6, n, n, n, 3)).astype(np.float32)
    hd.grid.set(H.FIELD_F, f.reshape(6, -1, 3))
    hd.grid.set(H.FIELD_U, np.zeros((6, n ** 3, 3), np.float32))
    hd.grid.gs_relaxation(w)
    u = hd.grid.get(H.FIELD_U).reshape(f.shape)[:, 1::2, 1::2, 1::2]
    f = f[:, 1::2, 1::2, 1::2]
    k = np.diag(hd.element_matrix())[21:].astype(np.float32) * (np.float32(8) * (np.float32(1e-9) + np.float32(rho)))
    assert k.dtype == np.float32 and np.array_equal(u, np.float32(w) * f / k)
    hd.close()
