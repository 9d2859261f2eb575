"""The level-0 kernels on rows that need CTAs of 256 and 512 threads."""
import numpy as np
import pytest

import homo3d_b200 as H
from tests.conftest import smooth_density

pytestmark = pytest.mark.gpu

SLAB = 8  # the fields repeat every SLAB planes


def _element_products(torch, ke, rho, u):
    """sum over elements of rho_e Ke u_e and of the nodes' own 3x3 blocks; u [nz, ny, nx, 3], periodic"""
    ku, blk = torch.zeros_like(u), torch.zeros(u.shape + (3,), dtype=u.dtype, device=u.device)
    node = [((a >> 2) & 1, (a >> 1) & 1, a & 1) for a in range(8)]
    U = torch.stack([u.roll(tuple(-s for s in n), (0, 1, 2)) for n in node], dim=-2)
    W = (U.reshape(u.shape[:3] + (24,)) @ ke) * rho[..., None]
    for a, n in enumerate(node):
        ku += W[..., 3 * a:3 * a + 3].roll(n, (0, 1, 2))
        blk += (rho[..., None, None] * ke[3 * a:3 * a + 3, 3 * a:3 * a + 3]).roll(n, (0, 1, 2))
    return ku, blk


def test_rows_of_640_vertices(torch_cuda):
    """640 x 256 x 256, the smallest grid with rows above 512: residual and one sweep in
    every launch shape against plain FP64 torch, on a period of planes far from the
    pinned origin"""
    torch = torch_cuda
    nx, ny, nz = dims = (640, 256, 256)
    rng = np.random.default_rng(3)
    cell = (SLAB, ny, nx)
    rho = rng.uniform(1e-3, 1, cell).astype(np.float32)
    uf = rng.uniform(-1, 1, (2, 6) + cell + (3,)).astype(np.float32)
    reps = nz // SLAB
    hd = H.Homogenization(dims, precision=H.PREC_FP32)
    assert hd.dims[0] == dims
    hd.update(torch.tensor(rho, device="cuda").repeat(reps, 1, 1).reshape(-1))
    field = lambda a: np.tile(a, (1, reps, 1, 1, 1)).reshape(6, -1, 3)
    u0, f0 = field(uf[0]), field(uf[1])
    hd.grid.set(H.FIELD_F, f0)
    hd.grid.set(H.FIELD_U, u0)
    hd.grid.update_residual()
    lo = 2 * SLAB  # a sweep carries the origin's influence at most one vertex per colour
    slab = lambda fld: hd.grid.get(fld).reshape(6, nz, ny, nx, 3)[:, lo:lo + SLAB].astype(np.float64)
    ke = torch.tensor(hd.element_matrix().astype(np.float32).astype(np.float64), device="cuda")
    r = torch.tensor(rho, device="cuda").double() + 1e-9
    got, want, swept = slab(H.FIELD_R), [], []
    z, y, x = torch.meshgrid(*(torch.arange(n, device="cuda") for n in cell), indexing="ij")
    colour = (1 - x % 2) + 2 * (1 - y % 2) + 4 * (1 - z % 2)
    for c in range(6):
        u, f = (torch.tensor(uf[k, c], device="cuda").double() for k in range(2))
        ku, D = _element_products(torch, ke, r, u)
        want.append((f - ku).cpu().numpy())
        for k in range(8):
            e = f - _element_products(torch, ke, r, u)[0]
            d0 = e[..., 0] / D[..., 0, 0]
            d1 = (e[..., 1] - D[..., 1, 0] * d0) / D[..., 1, 1]
            d2 = (e[..., 2] - D[..., 2, 0] * d0 - D[..., 2, 1] * d1) / D[..., 2, 2]
            u = torch.where((colour == k)[..., None], u + torch.stack([d0, d1, d2], -1), u)
        swept.append(u.cpu().numpy())
    # FP32 sums of 81 products: the bound of test_gpu_parity
    want, swept = np.stack(want), np.stack(swept)
    assert np.abs(got - want).max() < 2e-5 * np.abs(want).max()
    first = None
    for shape in range(H.NUM_SHAPES):
        hd.set_tuning(0, shape)
        hd.grid.set(H.FIELD_U, u0)
        hd.grid.gs_relaxation(1.0)
        u = slab(H.FIELD_U)
        if first is None:
            first = u
            assert np.abs(u - swept).max() < 2e-5 * np.abs(swept).max()
        assert np.array_equal(u, first), shape
    hd.close()


def test_lockstep_rows_of_320_vertices(torch_cuda):
    """a lockstep batch whose longest row takes the 256-thread CTAs, for a short row too:
    the single solves' results to the last bit in both launch shapes"""
    torch = torch_cuda
    rhos = [torch.tensor(smooth_density(256, seed=1, vol=0.4).reshape(256, 256, 256)[:, :, :1]
                         .repeat(320, axis=2).astype(np.float32).ravel(), device="cuda"),
            torch.tensor(smooth_density(32, seed=2, vol=0.4).astype(np.float32), device="cuda")]
    homs = [H.Homogenization(n, precision=H.PREC_FP32) for n in ((320, 256, 256), 32)]
    assert homs[0].dims[0] == (320, 256, 256)
    C, st = [], []
    for hd, r in zip(homs, rhos):
        hd.update(r)
        C.append(hd.elasticMatrix(1e-2))
        st.append(hd.last_stats)
    with H.Lockstep(homs) as lk:
        for shape in (0, 1):
            lk.set_shapes(shape, 0)
            for hd in homs:
                hd.reset_solutions()
            L = lk.elasticMatrix(1e-2)
            for i, hd in enumerate(homs):
                assert np.array_equal(L[i], C[i]), (shape, i)
                assert hd.last_stats["vcycles"] == st[i]["vcycles"]
                assert hd.last_stats["rel_res"] == st[i]["rel_res"]
    for hd in homs:
        hd.close()
