"""The level-0 sweep and residual on grids whose rows fill their CTAs differently,
in every launch shape, against the FP64 oracle."""
import numpy as np
import pytest

import homo3d_b200 as H
from oracle import oracle as O
from tests.conftest import from_lib_field, random_field, to_lib_field

pytestmark = pytest.mark.gpu


# rows of 5 vertex pairs (six rows of a CTA leave two threads idle, and the last CTA
# of a parity's 25 rows is partial), of 10 on three different axes, of 40 (three rows in
# 128 threads) and of 80 (two rows in 160 threads, the larger CTA)
@pytest.mark.parametrize("reso", [10, (17, 21, 29), (71, 90, 100), 144])
def test_sweep_and_residual(torch_cuda, reso):
    axes = (reso,) * 3 if isinstance(reso, int) else reso
    hd = H.Homogenization(axes)
    nv = hd.nv()
    rho = np.random.default_rng(7).uniform(1e-3, 1, nv).astype(np.float32)
    hd.update(torch_cuda.tensor(rho, device="cuda"))
    m = O.MG(axes)
    m.set_density(rho.astype(np.float64))
    u0, f0 = to_lib_field(random_field(nv, 1)), to_lib_field(random_field(nv, 2))
    u0[:, 0] = 5.0  # the stored value of the pinned origin counts as 0
    hd.grid.set(H.FIELD_F, f0)
    m.u()[:] = from_lib_field(u0)
    m.u()[0] = 0
    m.f()[:] = from_lib_field(f0)
    scale = np.abs(m.f()).max()
    m.residual(0)
    hd.grid.set(H.FIELD_U, u0)
    hd.grid.update_residual()
    r = from_lib_field(hd.grid.get(H.FIELD_R))
    # FP32 sums of 81 products: the bound of test_gpu_parity
    assert np.abs(r - m.r()).max() < 2e-5 * max(scale, np.abs(m.r()).max())
    assert np.all(r[0] == 0)
    m.gs(0, 0.9)
    first = None
    for shape in range(H.NUM_SHAPES):
        hd.set_tuning(0, shape)
        hd.grid.set(H.FIELD_U, u0)
        hd.grid.gs_relaxation(0.9)
        u = hd.grid.get(H.FIELD_U)
        if first is None:
            first = u
            assert np.abs(from_lib_field(u) - m.u()).max() < 2e-5 * np.abs(m.u()).max()
            assert np.all(u[:, 0] == 0)
        assert np.array_equal(u, first), shape
    hd.close()
