"""Performance cases of the framework: what its users have it compute, through its public entry points.

listed() names them, draw() gives more of the same ranges, prepare() makes what a program has in hand
before the call (inputs on the GPU, the handle it keeps), run() is one pass, work() the bytes and
operations of a pass, tolerance() how far another correct implementation may be, and exact() the same
answer in 64 bits from plain torch.

kinds of case
  evaluate      one design evaluation: load the density, build the multigrid hierarchy, solve the six
                unit-strain cases from a zero start, reduce the 6x6 elastic matrix
  iterate       one iteration of a design loop: penalise, evaluate with the stored solutions as the
                starting guess, sensitivities, filter and optimality-criteria update
  batch         several designs solved together in lockstep
  sensitivity   gradients of two functions of the elastic matrix from stored solutions (objective and
                constraint, as a constrained design loop asks for)
  filter        the radial density filter and its adjoint (forward and backward of the density chain)
  mma           one design update by the method of moving asymptotes
  warmnet       one forward and backward pass of the warm-start network
"""
import math
import time

import numpy as np
import torch

import homo3d_b200 as H

E, NU = 10.0, 0.3
RHO_MIN, RHO_FLOOR = 1e-3, 1e-9
PRECISION = {"refine": H.PREC_REFINE, "fp32": H.PREC_FP32, "mixed": H.PREC_MIXED}
STENCIL = {"fp16": H.STENCIL_FP16, "fp32": H.STENCIL_FP32}


# ---- the cases ---------------------------------------------------------------------------------

def listed():
    return [
        # the headline: a fresh design at the largest everyday grid, solved tightly
        {"name": "evaluate_256", "kind": "evaluate", "nx": 256, "ny": 256, "nz": 256, "precision": "refine",
         "stencil": "fp16", "tol": 1e-5, "vol": 0.3},
        # the plain FP32 scheme at a middle size and its usual tolerance
        {"name": "evaluate_128_fp32", "kind": "evaluate", "nx": 128, "ny": 128, "nz": 128, "precision": "fp32",
         "stencil": "fp16", "tol": 1e-3, "vol": 0.4},
        # a ragged cell: three different axes, FP32 coarse stencils for a high-contrast design
        {"name": "evaluate_80x96x112", "kind": "evaluate", "nx": 71, "ny": 89, "nz": 101, "precision": "refine",
         "stencil": "fp32", "tol": 1e-4, "vol": 0.35},
        # the smallest call: launches and host round trips
        {"name": "evaluate_16", "kind": "evaluate", "nx": 16, "ny": 16, "nz": 16, "precision": "refine",
         "stencil": "fp16", "tol": 1e-2, "vol": 0.3},
        # a design loop at its usual size and tolerance, past its first iterations
        {"name": "iterate_128", "kind": "iterate", "n": 128, "tol": 1e-2, "vol": 0.3, "objective": "bulk",
         "radius": 2.0},
        # the same loop on a coarse preview grid
        {"name": "iterate_48", "kind": "iterate", "n": 48, "tol": 1e-2, "vol": 0.4, "objective": "shear",
         "radius": 1.5},
        # a sweep over designs of uneven sizes
        {"name": "batch_mixed_24", "kind": "batch", "sizes": "64x8,96x8,128x8", "tol": 1e-3, "vol": 0.3},
        # a sweep over many small designs
        {"name": "batch_32x48", "kind": "batch", "sizes": "32x48", "tol": 1e-3, "vol": 0.3},
        # gradients for a constrained design loop
        {"name": "sensitivity_160", "kind": "sensitivity", "n": 144, "vol": 0.3},
        # the density filter of the expression layer, both directions
        {"name": "filter_112", "kind": "filter", "n": 112, "radius": 2.5, "periodic": True},
        # a constrained design update
        {"name": "mma_96", "kind": "mma", "n": 96 ** 3, "m": 2},
        # training the warm-start network
        {"name": "warmnet_32", "kind": "warmnet", "n": 32, "batch": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["evaluate", "evaluate", "evaluate", "iterate", "iterate", "batch", "sensitivity", "filter",
                       "mma", "warmnet"])
    vol = round(rng.uniform(0.3, 0.5), 3)
    if kind == "evaluate":
        n = _log(rng, 9, 224)  # odd requests are rounded up by the library
        axes = [n, n, n]
        if rng.random() < 0.4:  # three axes of one octave
            low = 1 << (n.bit_length() - 1)
            axes = [rng.randint(low + 1, 2 * low - low // 8) for _ in range(3)]
        precision, tol = rng.choice([("refine", 1e-5), ("refine", 1e-2), ("mixed", 1e-4), ("fp32", 1e-2),
                                     ("fp32", 1e-3)])
        return {"kind": kind, "nx": axes[0], "ny": axes[1], "nz": axes[2], "precision": precision,
                "stencil": rng.choice(["fp16", "fp16", "fp32"]), "tol": tol, "vol": vol}
    if kind == "iterate":
        return {"kind": kind, "n": _log(rng, 17, 160), "tol": 1e-2, "vol": vol,
                "objective": rng.choice(["bulk", "shear"]), "radius": rng.choice([1.5, 2.0, 3.0])}
    if kind == "batch":
        return {"kind": kind, "sizes": "%dx%d,%dx%d" % (_log(rng, 12, 40), rng.randint(3, 20), _log(rng, 40, 112),
                                                         rng.randint(1, 6)), "tol": 1e-3, "vol": vol}
    if kind == "sensitivity":
        return {"kind": kind, "n": _log(rng, 17, 200), "vol": vol}
    if kind == "filter":
        return {"kind": kind, "n": _log(rng, 17, 200), "radius": round(rng.uniform(1.2, 4.0), 2),
                "periodic": rng.random() < 0.5}
    if kind == "mma":
        return {"kind": kind, "n": _log(rng, 5000, 3000000), "m": rng.choice([1, 2])}
    return {"kind": kind, "n": 8 * rng.randint(1, 6), "batch": rng.randint(1, 6)}


def _rounded(n):
    """the grid size the library rounds a requested size up to (4 to 8 cells on the coarsest grid)"""
    l2 = math.log2(n)
    lcl = max(math.floor(l2) - 2, 0)
    return math.ceil(2 ** (l2 - lcl)) * 2 ** lcl


def _asked(case):
    return [case[a] for a in ("nx", "ny", "nz")] if "nx" in case else [case["n"]] * 3


def _grid(case):
    return [_rounded(n) for n in _asked(case)]


def _designs(case):
    out = []
    for part in case["sizes"].split(","):
        n, count = part.split("x")
        out += [int(n)] * int(count)
    return out


# ---- inputs ------------------------------------------------------------------------------------

def _mirror_average(v):
    """average over the mirror images and, for cubes, the axis permutations"""
    for ax in range(3):
        v = 0.5 * (v + v.flip(ax))
    if v.shape[0] == v.shape[1] == v.shape[2]:
        v = sum(v.permute(p) for p in [(0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0)]) / 6
    return v


def _density(grid, seed, vol):
    """a smooth symmetric design in [1e-3, 1] of mean vol, FP32, x fastest: a random sum of the
    cosines of wave numbers 0..2 per axis, clamped and shifted to the volume"""
    rng = np.random.default_rng([int(seed), 1])
    a, phi = rng.uniform(-1, 1, (3, 3, 3)), rng.uniform(0, 2 * np.pi, (3, 3, 3))
    c = torch.tensor(a * np.exp(1j * phi), device="cuda")
    for n in reversed(grid):  # contract kz, ky, kx in turn
        k = torch.arange(3, device="cuda", dtype=torch.float64)
        x = (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) / n
        w = torch.exp(2j * np.pi * k[:, None] * x[None, :])
        c = torch.tensordot(c, w, dims=([0], [0]))
    v = _mirror_average((0.3 + 0.25 * c.real).clamp(RHO_MIN, 1.0))  # [z, y, x]
    lo, hi = -2.0, 2.0
    for _ in range(40):
        t = 0.5 * (lo + hi)
        if float((v + t).clamp(RHO_MIN, 1.0).mean()) < vol:
            lo = t
        else:
            hi = t
    return (v + t).clamp(RHO_MIN, 1.0).float().contiguous().reshape(-1)


def _weights(objective):
    """d objective / d C: minus the bulk or the shear modulus"""
    d = np.zeros((6, 6), np.float32)
    if objective == "bulk":
        d[[0, 1, 2], [0, 1, 2]] = -1.0 / 3.0
        d[0, 1] = d[0, 2] = d[1, 2] = -2.0 / 3.0
    else:
        d[[3, 4, 5], [3, 4, 5]] = -1.0 / 3.0
    return d


def _random(shape, seed, lo, hi):
    rng = np.random.default_rng([int(seed), 2])
    return torch.tensor(rng.uniform(lo, hi, shape).astype(np.float32), device="cuda")


def _mma_inputs(case, seed):
    n, m = case["n"], case["m"]
    w = _random((m + 2, n), seed, 0.0, 1.0)
    x = (0.2 + 0.2 * w[0]).contiguous()
    df = (-(0.2 + 0.8 * w[1]) / x ** 2).contiguous()
    dg = [((0.5 + w[2 + i]) * (1000.0 / n)).contiguous() for i in range(m)]
    g = torch.stack([(d.double() * (x.double() - 0.3)).sum() for d in dg]).float()
    return x, df, dg, g


CONV = [(1, 16, 0), (16, 32, 1), (32, 64, 2), (64, 64, 3), (64, 32, 2), (32, 16, 1), (16, 16, 0)]
OUT = 18


def _net_params(seed):
    """weights and biases of the network's layers in the order the library stores them"""
    rng = np.random.default_rng([int(seed), 3])
    parts = []
    for ci, co, _ in CONV:
        parts += [rng.standard_normal(co * ci * 27) * np.sqrt(2.0 / (27 * ci)), rng.standard_normal(co) * 0.05]
    parts += [rng.standard_normal(OUT * 16) * 0.25, rng.standard_normal(OUT) * 0.05]
    return np.concatenate(parts).astype(np.float32)


def _net_inputs(case, seed):
    r, b = case["n"], case["batch"]
    x = torch.stack([_density([r] * 3, seed * 100 + i, 0.3) for i in range(b)]) ** 3
    return x.contiguous(), _random((b, OUT, r ** 3), seed, -0.1, 0.1)


def _handle(case):
    # the coarsest solve that design loops take (for high-contrast designs)
    return H.Homogenization(tuple(_asked(case)), E, NU, H.COARSE_PROJECT, precision=PRECISION[case.get("precision", "refine")],
                            stencil=STENCIL[case.get("stencil", "fp16")])


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "evaluate":
        grid = _grid(case)
        s["hom"] = _handle(case)
        s["rho"] = _density(grid, seed, case["vol"]) ** 3
    elif kind == "iterate":
        s["hom"] = _handle(case)
        s["rho0"] = _density(_grid(case), seed, case["vol"])
        s["rho"], s["phys"], s["sens"] = (torch.empty_like(s["rho0"]) for _ in range(3))
        s["dC"] = _weights(case["objective"])
    elif kind == "batch":
        s["homs"] = [H.Homogenization(n, E, NU, H.COARSE_PROJECT, precision=H.PREC_FP32) for n in _designs(case)]
        s["rhos"] = [_density([_rounded(n)] * 3, seed * 100 + i, case["vol"]) ** 3
                     for i, n in enumerate(_designs(case))]
        s["lock"] = H.Lockstep(s["homs"])
    elif kind == "sensitivity":
        s["hom"] = _handle(case)
        rho = _density(_grid(case), seed, case["vol"]) ** 3
        s["hom"].update(rho)
        s["hom"].elasticMatrix(1e-5)
        s["out"] = [torch.empty_like(rho) for _ in range(2)]
        s["dC"] = [_weights("shear"), _weights("bulk")]
    elif kind == "filter":
        s["hom"] = _handle(case)
        s["rho"] = _density(_grid(case), seed, 0.3)
        s["grad"] = _random(s["rho"].numel(), seed, -1.0, 0.0)
        s["out"] = [torch.empty_like(s["rho"]) for _ in range(2)]
    elif kind == "mma":
        s["x0"], s["df"], s["dg"], s["g"] = _mma_inputs(case, seed)
        s["x"] = torch.empty_like(s["x0"])
        s["mma"] = H.MMAOptimizer(case["m"], case["n"], 1.0, 0.0, 1000.0, 1.0)
        s["mma"].setBound(0.001, 1.0)
    else:
        s["net"] = H.WarmNet(case["n"], case["batch"], 0)
        s["net"].set_params(_net_params(seed))
        s["x"], s["t"] = _net_inputs(case, seed)
    torch.cuda.synchronize()
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "evaluate":
        s["hom"].reset_solutions()  # a fresh design starts from zero
        s["hom"].update(s["rho"])
        return s["hom"].elasticMatrix(case["tol"])
    if kind == "iterate":
        s["rho"].copy_(s["rho0"])
        s["hom"].penalize(s["rho"], s["phys"], 3.0)
        s["hom"].update(s["phys"])
        C = s["hom"].elasticMatrix(case["tol"])
        s["hom"].design_step(s["dC"], s["rho"], s["sens"], case["vol"], 3.0, "reflect6", case["radius"])
        return {"C": C, "rho": s["rho"], "sens": s["sens"]}
    if kind == "batch":
        for h in s["homs"]:
            h.reset_solutions()
        H.batch_update(s["homs"], s["rhos"])
        return s["lock"].elasticMatrix(case["tol"])
    if kind == "sensitivity":
        for dC, out in zip(s["dC"], s["out"]):
            s["hom"].Sensitivity(dC, out)
        return s["out"]
    if kind == "filter":
        s["hom"].conv_radial(s["rho"], s["out"][0], case["radius"], case["periodic"])
        s["hom"].conv_radial(s["grad"], s["out"][1], case["radius"], case["periodic"], adjoint=True)
        s["hom"].sync()
        return s["out"]
    if kind == "mma":
        s["x"].copy_(s["x0"])
        s["mma"].update(1, s["x"], s["df"], s["g"], s["dg"])
        return s["x"]
    loss = s["net"].gradients(s["x"], s["t"])
    return {"loss": loss, "grads": s["net"].grads()}


# ---- what a pass cannot do without -------------------------------------------------------------

# A V(1,1) cycle passes over a level's fields three times (two sweeps and a residual), each reading u
# and f and writing one field of six cases x three components; the coarse levels also read their
# stencils.  One operator application costs 81 x 6 multiply-adds per vertex, on the fine level after
# the assembly of its 27 blocks.
def _vcycle(nv, stencil, tight):
    fields = 3 * 18 * (4 * 3) + 12
    coarse = 3 * 243 * (4 if stencil == "fp32" else 2) + 3 * 18 * (4 * 3)
    return nv * (fields + coarse / 7.0), 3 * 2 * nv * (576 + 81 * 18 / 3) * (1 + 1 / 7.0)


def _solve_work(nv, case):
    cycles = max(1, math.ceil(-math.log10(case["tol"]) * 1.8))
    b, f = _vcycle(nv, case.get("stencil", "fp16"), case["tol"])
    setup = nv * (4 + 243 * (4 if case.get("stencil") == "fp32" else 2) / 7.0)
    return cycles * b + setup + nv * 18 * 8, cycles * f + nv * 2 * 576 * 7


def work(case):
    kind = case["kind"]
    if kind == "evaluate":
        b, f = _solve_work(math.prod(_grid(case)), case)
        return {"bytes": b, "flops": f}
    if kind == "iterate":  # past the first pass: one V-cycle from the stored solutions
        nv = math.prod(_grid(case))
        b, f = _vcycle(nv, "fp16", case["tol"])
        taps = (2 * int(case["radius"] + 0.5) + 1) ** 3
        return {"bytes": b + nv * (2 * 18 * 8 + 243 * 2 / 7.0 + 4 * 8), "flops": f + nv * (2 * 2 * 576 * 6 + 4 * taps)}
    if kind == "batch":
        w = [_solve_work(_rounded(n) ** 3, case) for n in _designs(case)]
        return {"bytes": sum(b for b, _ in w), "flops": sum(f for _, f in w)}
    if kind == "sensitivity":
        nv = math.prod(_grid(case))
        return {"bytes": 2 * nv * (18 * 8 + 4), "flops": 2 * nv * (2 * 576 * 6 + 2 * 24 * 21)}
    if kind == "filter":
        nv = math.prod(_grid(case))
        taps = (2 * int(case["radius"] + 0.5) + 1) ** 3
        return {"bytes": 4 * 4 * nv, "flops": 2 * 2 * taps * nv}
    if kind == "mma":  # about 30 Newton steps over the point, the direction and the problem data
        n, m = case["n"], case["m"]
        return {"bytes": 30.0 * n * 8 * (3 * 2 + 2 * (m + 1) + 4), "flops": 30.0 * n * (60 + 30 * m)}
    r, b = case["n"], case["batch"]
    mac = sum(27 * ci * co * (r >> l) ** 3 for ci, co, l in CONV) + 16 * OUT * r ** 3
    act = sum((ci + co) * (r >> l) ** 3 for ci, co, l in CONV) + OUT * r ** 3
    return {"bytes": 3.0 * 4 * b * act, "flops": 3.0 * 2 * b * mac}


def tolerance(case):
    return TOLERANCE[case["kind"]](case)


# About four times the error measured against exact().
TOLERANCE = {
    # C is a quadratic form: 4e-7 from the FP32 element matrix, a solve at 1e-2 that stops a cycle
    # earlier or later adds the square of its residual
    "evaluate": lambda c: {"rel": max(2e-6, 1e-3 * c["tol"])},
    "batch": lambda c: {"rel": 4e-6},
    # sensitivities are linear in a solution of relative residual 1e-2: 7e-5 to 1e-2
    "iterate": lambda c: {"rel": 3e-2, "max": 0.9},
    # and here in one of relative residual 1e-5
    "sensitivity": lambda c: {"rel": 4e-5, "max": 5e-3},
    "filter": lambda c: {"rel": 2.5e-6},
    "mma": lambda c: {"rel": 2e-7, "max": 1e-5},
    "warmnet": lambda c: {"rel": 1.5e-5, "max": 1e-3},
}


# ---- the same answers in 64 bits ---------------------------------------------------------------

def _material():
    D = np.zeros((6, 6))
    s = E / ((1 + NU) * (1 - 2 * NU))
    D[:3, :3] = s * NU
    D[[0, 1, 2], [0, 1, 2]] = s * (1 - NU)
    D[[3, 4, 5], [3, 4, 5]] = s * (1 - 2 * NU) / 2
    return D


def _element_matrix():
    """trilinear unit-cube element, 2x2x2 Gauss points; node a at (a & 1, a >> 1 & 1, a >> 2)"""
    D, K = _material(), np.zeros((24, 24))
    p = 0.5 / math.sqrt(3.0)
    for g in range(8):
        q = [0.5 + p * (1 if (g >> i) & 1 else -1) for i in range(3)]
        B = np.zeros((6, 24))
        for a in range(8):
            bit = [(a >> i) & 1 for i in range(3)]
            val = [q[i] if bit[i] else 1 - q[i] for i in range(3)]
            d = [(1 if bit[i] else -1) * val[(i + 1) % 3] * val[(i + 2) % 3] for i in range(3)]
            for i in range(3):
                B[i, 3 * a + i] = d[i]
            B[3, 3 * a + 1], B[3, 3 * a + 2] = d[2], d[1]
            B[4, 3 * a], B[4, 3 * a + 2] = d[2], d[0]
            B[5, 3 * a], B[5, 3 * a + 1] = d[1], d[0]
        K += B.T @ D @ B / 8
    return K


def _unit_strains():
    """[24, 6]: node displacements of the six unit strains on one element"""
    x = np.zeros((24, 6))
    for a in range(8):
        p = [a & 1, (a >> 1) & 1, a >> 2]
        for i in range(3):
            x[3 * a + i, i] = p[i]
        x[3 * a + 1, 3], x[3 * a + 2, 3] = p[2] / 2, p[1] / 2
        x[3 * a, 4], x[3 * a + 2, 4] = p[2] / 2, p[0] / 2
        x[3 * a, 5], x[3 * a + 1, 5] = p[1] / 2, p[0] / 2
    return x


class _Cell:
    """the periodic cell problem of one design in 64 bits: displacements [3, 6, z, y, x]"""

    def __init__(self, rho, grid):
        self.shape = (grid[2], grid[1], grid[0])
        self.rho = rho.double().reshape(self.shape) + RHO_FLOOR
        self.K = torch.tensor(_element_matrix(), device="cuda")
        self.X = torch.tensor(_unit_strains(), device="cuda")

    def gather(self, u):
        return torch.stack([u.roll((-(a >> 2), -((a >> 1) & 1), -(a & 1)), (2, 3, 4)) for a in range(8)])

    def scatter(self, f):
        return sum(f[a].roll((a >> 2, (a >> 1) & 1, a & 1), (2, 3, 4)) for a in range(8))

    def apply(self, u):
        e = self.gather(u).reshape(24, -1)
        return self.scatter((self.K @ e).reshape((8, 3, 6) + self.shape) * self.rho)

    def load(self):
        g = (self.K @ self.X).reshape(8, 3, 6, 1, 1, 1) * self.rho
        return self.scatter(g)

    def solve(self, tol=1e-9, seconds=12.0):
        """conjugate gradients with the diagonal as preconditioner; None if out of time"""
        f = self.load()
        d = torch.diagonal(self.K).reshape(8, 3, 1, 1, 1, 1) * self.rho
        inv = 1.0 / self.scatter(d.expand((8, 3, 6) + self.shape))
        dot = lambda a, b: (a * b).sum(dim=(0, 2, 3, 4), keepdim=True)  # noqa: E731
        u, r = torch.zeros_like(f), f.clone()
        z = inv * r
        p, rz = z.clone(), dot(r, z)
        rz0, t0 = rz.clone(), time.monotonic()
        for it in range(100000):
            q = self.apply(p)
            a = rz / dot(p, q)
            u += a * p
            r -= a * q
            z = inv * r
            new = dot(r, z)
            p = z + (new / rz) * p
            rz = new
            if it % 20 == 19:
                if float((rz / rz0).max()) < tol * tol:
                    return u
                if time.monotonic() - t0 > seconds:
                    return None
        return None

    def energies(self, u):
        """[6, 6, z, y, x]: (x_i - u_i)^T K (x_j - u_j) per element"""
        w = (self.X.reshape(8, 3, 6, 1, 1, 1) - self.gather(u)).reshape((24, 6) + self.shape)
        out = torch.empty((6, 6) + self.shape, dtype=torch.float64, device="cuda")
        for j in range(6):
            k = torch.tensordot(self.K, w[:, j], dims=([1], [0]))
            for i in range(6):
                out[i, j] = (w[:, i] * k).sum(0)
        return out

    def matrix(self, u):
        return ((self.energies(u) * self.rho).sum(dim=(2, 3, 4)) / self.rho.numel()).cpu().numpy()

    def gradient(self, u, dC):
        w = np.zeros((6, 6))
        for i in range(6):
            for j in range(i, 6):
                w[i, j] = float(dC[i, j]) + (float(dC[j, i]) if i != j else 0.0)
        e = self.energies(u)
        return torch.tensordot(torch.tensor(w, device="cuda"), e, dims=([0, 1], [0, 1])) / self.rho.numel()


def _window(v, radius, weight, periodic, mode):
    """sum of weight(|o|) v[p + o] over the window, and of the weights"""
    h = int(radius + 0.5)
    total, norm = torch.zeros_like(v), torch.zeros_like(v)
    n = v.shape
    one = torch.ones_like(v)
    for oz in range(-h, h + 1):
        for oy in range(-h, h + 1):
            for ox in range(-h, h + 1):
                w = weight(math.sqrt(ox * ox + oy * oy + oz * oz) / radius)
                if w == 0.0:
                    continue
                o = (oz, oy, ox)
                if periodic:
                    total += w * v.roll(tuple(-a for a in o), (0, 1, 2))
                    norm += w
                    continue
                dst = tuple(slice(max(0, -a), n[i] - max(0, a)) for i, a in enumerate(o))
                src = tuple(slice(max(0, a), n[i] - max(0, -a)) for i, a in enumerate(o))
                total[dst] += w * v[src]
                norm[dst] += w * one[src]
    return total, norm


def _cone(q):
    return max(0.0, 1.0 - q)


def _spline(q):
    return 1 - 6 * q ** 2 + 8 * q ** 3 - 3 * q ** 4 if q < 1 else 0.0


def _oc(sens, rho, vol, step=0.05, damp=0.5):
    lo, hi = 0.0, float(sens.abs().max())
    for _ in range(20):
        g = 0.5 * (lo + hi)
        b = -sens / g
        b = torch.where(b < 0, torch.full_like(b, 0.01), b)
        new = (b ** damp * rho).clamp(min=rho - step, max=rho + step).clamp(RHO_MIN, 1.0)
        mean = float(new.mean())
        if mean < vol - 1e-4:
            hi = g
        elif mean > vol + 1e-4:
            lo = g
        else:
            break
    return new


def _exact_mma(case, seed):
    """the minimiser of the convex separable approximation, from its dual"""
    x, df, dg, g = _mma_inputs(case, seed)
    x, df, g = x.double(), df.double(), g.double()
    m = case["m"]
    dg = torch.stack(dg).double()
    lo, hi = 0.001, 1.0
    dx = hi - lo
    low, upp = x - 0.5 * dx, x + 0.5 * dx
    a = torch.maximum(low + 0.1 * (x - low), torch.full_like(x, lo))
    b = torch.minimum(upp - 0.1 * (upp - x), torch.full_like(x, hi))

    def pq(d):
        p, q = d.clamp(min=0), (-d).clamp(min=0)
        e = 1e-3 * (p + q) + 1e-5 / dx
        return (p + e) * (upp - x) ** 2, (q + e) * (x - low) ** 2

    p0, q0 = pq(df)
    P, Q = pq(dg)
    rhs = (P / (upp - x) + Q / (x - low)).sum(1) - g

    def point(lam):
        p = (p0 + (lam[:, None] * P).sum(0)).sqrt()
        q = (q0 + (lam[:, None] * Q).sum(0)).sqrt()
        return ((p * low + q * upp) / (p + q)).clamp(min=a, max=b)

    def slack(lam):
        v = point(lam)
        y = (lam - 1000.0).clamp(min=0)
        return (P / (upp - v) + Q / (v - low)).sum(1) - rhs - y

    lam = torch.zeros(m, dtype=torch.float64, device="cuda")

    def level(i):  # lam[i] at which constraint i is met, the later ones solved inside
        l, h = 0.0, 1e7
        for k in range(56):
            lam[i] = 0.0 if k == 0 else 0.5 * (l + h)
            if i + 1 < m:
                level(i + 1)
            s = float(slack(lam)[i])
            if k == 0 and s <= 0:
                return
            if s > 0:
                l = float(lam[i])
            elif k:
                h = float(lam[i])

    level(0)
    return point(lam)


def _exact_net(case, seed):
    r, b = case["n"], case["batch"]
    x, t = _net_inputs(case, seed)
    flat = torch.tensor(_net_params(seed), device="cuda", dtype=torch.float64, requires_grad=True)
    at = [0]

    def take(*shape):
        n = math.prod(shape)
        at[0] += n
        return flat[at[0] - n:at[0]].reshape(shape)

    layers = [(take(co, ci, 3, 3, 3), take(co)) for ci, co, _ in CONV]
    wo, bo = take(OUT, 16), take(OUT)
    F = torch.nn.functional

    def conv(v, i):
        w, bias = layers[i]
        v = F.pad(v, (1,) * 6, mode="circular")
        out = bias.reshape(1, -1, 1, 1, 1)
        n = v.shape[-1] - 2
        for k in range(27):
            dz, dy, dx = k // 9, k // 3 % 3, k % 3
            out = out + torch.einsum("oi,bizyx->bozyx", w[:, :, dz, dy, dx],
                                     v[:, :, dz:dz + n, dy:dy + n, dx:dx + n])
        return out.relu()

    def up(v):
        return v.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)

    a0 = conv(x.double().reshape(b, 1, r, r, r), 0)
    a1 = conv(F.avg_pool3d(a0, 2), 1)
    a2 = conv(F.avg_pool3d(a1, 2), 2)
    a3 = conv(F.avg_pool3d(a2, 2), 3)
    d2 = conv(up(a3) + a2, 4)
    d1 = conv(up(d2) + a1, 5)
    d0 = conv(up(d1) + a0, 6)
    y = torch.einsum("oc,bczyx->bozyx", wo, d0) + bo.reshape(1, -1, 1, 1, 1)
    loss = ((y.reshape(b, OUT, -1) - t.double()) ** 2).mean()
    loss.backward()
    return {"loss": float(loss), "grads": flat.grad.cpu().numpy()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "mma":
        return _exact_mma(case, seed)
    if kind == "warmnet":
        return _exact_net(case, seed)
    if kind == "filter":
        shape = tuple(reversed(_grid(case)))
        rho = _density(_grid(case), seed, 0.3).double().reshape(shape)
        grad = _random(rho.numel(), seed, -1.0, 0.0).double().reshape(shape)
        total, norm = _window(rho, case["radius"], _spline, case["periodic"], 0)
        back, _ = _window(grad / norm, case["radius"], _spline, case["periodic"], 0)
        return [(total / norm).reshape(-1), back.reshape(-1)]
    if kind == "batch":
        if max(_designs(case)) > 64:
            return None
        out = []
        for i, n in enumerate(_designs(case)):
            grid = [_rounded(n)] * 3
            cell = _Cell(_density(grid, seed * 100 + i, case["vol"]) ** 3, grid)
            u = cell.solve(1e-7, 18.0 / len(_designs(case)))
            if u is None:
                return None
            out.append(cell.matrix(u))
        return np.stack(out)
    grid = _grid(case)
    if math.prod(grid) > 130 ** 3:
        return None
    rho = _density(grid, seed, case["vol"])
    cell = _Cell(rho ** 3, grid)
    u = cell.solve()
    if u is None:
        return None
    if kind == "evaluate":
        return cell.matrix(u)
    if kind == "sensitivity":
        return [cell.gradient(u, _weights(o)).reshape(-1) for o in ("shear", "bulk")]
    r = rho.double().reshape(cell.shape)
    sens = _mirror_average(cell.gradient(u, _weights(case["objective"])) * 3.0 * r ** 2)
    total, norm = _window(sens * r, case["radius"], _cone, False, 0)
    sens = total / (norm * r)
    new = _mirror_average(_oc(sens, r, case["vol"]))
    return {"C": cell.matrix(u), "rho": new.reshape(-1), "sens": sens.reshape(-1)}
