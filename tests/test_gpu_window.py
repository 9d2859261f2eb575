"""The window sums (radial convolution, its adjoint and the sensitivity filter) at
window widths and grid sizes that reach every path, against plain torch in FP64."""
import math

import numpy as np
import pytest

import homo3d_b200 as H

pytestmark = pytest.mark.gpu


def _window(torch, v, radius, weight, periodic):
    h, n = int(radius + 0.5), v.shape
    total, norm = torch.zeros_like(v), torch.zeros_like(v)
    for oz in range(-h, h + 1):
        for oy in range(-h, h + 1):
            for ox in range(-h, h + 1):
                w = weight((ox * ox + oy * oy + oz * oz) / radius ** 2)
                o = (oz, oy, ox)
                if periodic:
                    total += w * v.roll(tuple(-a for a in o), (0, 1, 2))
                    norm += w
                elif all(abs(a) < n[i] for i, a in enumerate(o)):
                    dst = tuple(slice(max(0, -a), n[i] - max(0, a)) for i, a in enumerate(o))
                    src = tuple(slice(max(0, a), n[i] - max(0, -a)) for i, a in enumerate(o))
                    total[dst] += w * v[src]
                    norm[dst] += w
    return total, norm


def _cone(q):
    return max(0.0, 1 - math.sqrt(q))


def _spline(q):
    return 1 - 6 * q + 8 * q ** 1.5 - 3 * q * q if q < 1 else 0.0


# windows of 1, 3, 5, 7, 9 and 11 cells (the first and last run cell by cell), on a grid
# narrower than a block of threads and with a partial column of four cells (10), one with
# a partial block in x and y (40), and ones where few or no windows are whole (12)
@pytest.mark.parametrize("n,radius,periodic", [(10, 0.4, True), (10, 1.2, False), (10, 2.6, True), (40, 2.0, True),
                                               (40, 2.0, False), (20, 2.6, False), (20, 4.3, True), (12, 4.3, False),
                                               (20, 5.2, True), (12, 5.2, False)])
def test_window_sums(torch_cuda, n, radius, periodic):
    torch = torch_cuda
    hd = H.Homogenization(n)
    shape = tuple(reversed(hd.dims[0]))
    rng = np.random.default_rng(1)
    x = torch.tensor(rng.uniform(0.1, 1, shape).astype(np.float32), device="cuda")
    g = torch.tensor(rng.uniform(0.1, 1, shape).astype(np.float32), device="cuda")
    out, adj, sens = torch.empty_like(x), torch.empty_like(x), g.clone()
    total, norm = _window(torch, x.double(), radius, _spline, periodic)
    hd.conv_radial(x, out, radius, periodic)
    hd.conv_radial(g, adj, radius, periodic, adjoint=True)
    oc = H.OCOptimizer(x.numel(), handle=hd)
    oc.filterSens(sens, x, -1, hd.dims[0], radius, periodic)
    hd.sync()
    # FP32 sums of (2h + 1)^3 positive terms (the spline's weights are positive below 1)
    tol = 6e-8 * (2 * int(radius + 0.5) + 1) ** 1.5 + 4e-7

    def err(a, b):
        return float((a.double() - b).abs().max() / b.abs().max())

    assert err(out, total / norm) < tol
    assert err(adj, _window(torch, g.double() / norm, radius, _spline, periodic)[0]) < tol
    total, norm = _window(torch, (g.double() * x.double()), radius, _cone, periodic)
    assert err(sens, total / (norm * x.double())) < tol
    hd.close()
