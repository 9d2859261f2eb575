"""Element energies in mirror-parity coefficients against the dense FP64 element
matrix: three different axes, a last partial CTA, and a pitched output."""
import numpy as np
import pytest

import homo3d_b200 as H

pytestmark = pytest.mark.gpu


def _strains():
    x = np.zeros((6, 8, 3))
    for a in range(8):
        p = [a & 1, (a >> 1) & 1, a >> 2]
        for i in range(3):
            x[i, a, i] = p[i]
        x[3, a, 1], x[3, a, 2] = p[2] / 2, p[1] / 2
        x[4, a, 0], x[4, a, 2] = p[2] / 2, p[0] / 2
        x[5, a, 0], x[5, a, 1] = p[1] / 2, p[0] / 2
    return x.reshape(6, 24)


@pytest.mark.parametrize("reso,pad", [(8, 0), ((9, 13, 15), 0), ((9, 13, 15), 5)])
def test_sensitivity_matches_dense_element_matrix(torch_cuda, reso, pad):
    hd = H.Homogenization(reso, E=3.0, nu=0.2)
    nx, ny, nz = hd.dims[0]
    rng = np.random.default_rng(nx)
    chi = rng.standard_normal((6, nx * ny * nz, 3)).astype(np.float32)
    chi += 100.0  # a translation far above the differences
    hd.grid.set(H.FIELD_CHI, chi)
    dC = rng.standard_normal((6, 6)).astype(np.float32)
    pitch = nx + pad
    sens = torch_cuda.full((nz, ny, pitch), 7.0, dtype=torch_cuda.float32, device="cuda")
    hd.Sensitivity(dC, sens, pitch if pad else -1)
    c = chi.astype(np.float64).reshape(6, nz, ny, nx, 3)
    U = np.stack([np.roll(c, (-(a >> 2), -((a >> 1) & 1), -(a & 1)), (1, 2, 3)) for a in range(8)], axis=-2)
    W = _strains().reshape(6, 1, 1, 1, 24) - U.reshape(6, nz, ny, nx, 24)
    KW = W @ hd.element_matrix()
    ref = np.zeros((nz, ny, nx))
    for i in range(6):
        for j in range(i, 6):
            w = float(dC[i, j]) + (float(dC[j, i]) if i != j else 0.0)
            ref += w * (W[i] * KW[j]).sum(-1)
    ref /= nx * ny * nz
    got = sens.cpu().numpy().astype(np.float64)
    # FP32 sums of about 60 products: the bound of test_gpu_energy
    assert np.abs(got[:, :, :nx] - ref).max() < 1e-5 * np.abs(ref).max()
    if pad:
        assert np.all(got[:, :, nx:] == 0)
    hd.close()
