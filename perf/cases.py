"""Work that a program using this framework has it do, as timing cases.

Every case goes through a public entry point of the package: the
``Molecule`` methods on numpy arrays (the drop-in API), the same on device
pointers, the cubic-grid evaluation, the autograd binding, the electrostatic
potential and the AO values.  Molecules, density matrices and point sets are
those of the repository's own generator (``chemtoolscuda_b200.synthetic``),
whose five configurations are also the benchmark's workloads; the density
matrix is drawn on the GPU.

``exact`` restates each output in 64-bit torch arithmetic without calling the
package's kernels.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import chemtoolscuda_b200 as ctc
from chemtoolscuda_b200 import autograd as ctc_autograd
from chemtoolscuda_b200 import synthetic as S

ALPHA = 0.5
ALL = "rho,grad,hess,lap,tau_pd,tau_alpha,rdg"
# atoms, box edge (bohr) and occupied columns of each configuration; other
# sizes keep the atom density
BASE = {"c1": (12, 8.0, 20), "c2": (200, 25.0, 400), "c3": (60, 16.0, 120),
        "c4": (1000, (1000 / 0.01) ** (1 / 3), 2500), "c5": (100, 18.0, 200)}


def listed() -> list[dict]:
    return [
        # the smallest call: the density at a few points of a small molecule (an
        # optimiser or a line scan calling in a loop), numpy in and out
        dict(name="host_density_200", kind="host", config="c1", natom=12, n=200, keys="rho", precision="fp64"),
        # density of a small molecule at scattered points already on the GPU (the
        # 12-atom workload of the benchmark)
        dict(name="points_density_100k", kind="points", config="c1", natom=12, n=100_000, keys="rho",
             precision="fp64"),
        # GGA ingredients of a medium molecule at scattered points, tensor cores
        dict(name="points_gga_400k_tc", kind="points", config="c3", natom=60, n=400_003, keys="rho,grad",
             precision="tc"),
        # every local descriptor on a cube of a large molecule (pure d and f): the
        # benchmark's main workload on an odd grid, and its FP64 form on a smaller one
        dict(name="cube_all_tc", kind="cube", config="c2", natom=200, nx=81, ny=77, nz=85, spacing=0.2, keys=ALL,
             precision="tc"),
        dict(name="cube_all_fp64", kind="cube", config="c2", natom=200, nx=45, ny=43, nz=47, spacing=0.2, keys=ALL,
             precision="fp64"),
        # the drop-in call on numpy arrays, all descriptors: large and on tensor
        # cores, medium in the default precision
        dict(name="host_all_300k_tc", kind="host", config="c2", natom=200, n=300_000, keys=ALL, precision="tc"),
        dict(name="host_all_20k", kind="host", config="c3", natom=60, n=20_011, keys=ALL, precision="fp64"),
        # one step of a density functional on an atom-centred grid: rho, grad rho,
        # the functional, and its gradients to D and the coordinates
        dict(name="train_gga", kind="train", config="c3", natom=60, nrad=40, ntheta=8, nphi=14),
        # a large sparse system (Cartesian up to g, D cut off beyond 12 bohr) on a
        # cube that covers it
        dict(name="sparse_cube_tc", kind="cube", config="c4", natom=640, nx=101, ny=98, nz=99, spacing=0.45,
             keys="rho,grad,lap", precision="tc"),
        # electrostatic potential on nested molecular surfaces of a 100-atom
        # molecule, and at few points of a small one (charge fitting), numpy arrays
        dict(name="esp_surface_100k", kind="esp", config="c5", natom=100, n=100_000),
        dict(name="esp_host_1500", kind="esp_host", config="c1", natom=12, n=1500),
        # AO values and gradients on a batch of grid points (a caller that forms its
        # own matrices)
        dict(name="ao_grad_30k", kind="ao", config="c3", natom=60, n=30_000, deriv=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["host", "points", "points", "cube", "cube", "train", "esp", "esp_host", "ao"])
    if kind in ("host", "points"):
        config = rng.choice(["c1", "c2", "c3"])
        natom = _log(rng, 6, {"c1": 24, "c2": 200, "c3": 90}[config])
        return dict(kind=kind, config=config, natom=natom, n=_log(rng, 100, 300_000 if natom > 60 else 500_000),
                    keys=rng.choice(["rho", "rho,grad", "grad", "lap", "tau_pd", "rho,tau_pd", ALL]),
                    precision=rng.choice(["fp64", "tc"]) if natom < 100 else "tc")
    if kind == "cube":
        config = rng.choice(["c1", "c2", "c4"])
        natom = _log(rng, 10, {"c1": 24, "c2": 200, "c4": 400}[config])
        edge = 80 if natom > 60 else 100
        return dict(kind=kind, config=config, natom=natom, nx=rng.randint(15, edge), ny=rng.randint(15, edge),
                    nz=rng.randint(15, edge), spacing=rng.choice([0.2, 0.25, 0.3]),
                    keys=rng.choice(["rho", "rho,grad,lap", ALL]),
                    precision=rng.choice(["fp64", "tc"]) if natom < 60 else "tc")
    if kind == "train":
        return dict(kind=kind, config=rng.choice(["c1", "c3", "c4"]), natom=_log(rng, 8, 60),
                    nrad=rng.randint(10, 40), ntheta=rng.randint(4, 8), nphi=rng.randint(6, 14))
    if kind == "esp":
        return dict(kind=kind, config=rng.choice(["c1", "c5"]), natom=_log(rng, 8, 90), n=_log(rng, 2000, 90_000))
    if kind == "esp_host":
        return dict(kind=kind, config="c1", natom=_log(rng, 6, 16), n=_log(rng, 100, 2500))
    return dict(kind=kind, config=rng.choice(["c1", "c2", "c3"]), natom=_log(rng, 6, 60), n=_log(rng, 300, 20_000),
                deriv=rng.choice([0, 1, 2]))


# ------------------------------------------------------------------ inputs
def _structure(case: dict) -> S.SyntheticMolecule:
    """Atoms and basis of a case's molecule: the same for every seed, D still empty."""
    config, natom = case["config"], case["natom"]
    natom0, box0, _ = BASE[config]
    g = np.random.default_rng(natom)
    coords = S._place_atoms(g, natom, box0 * (natom / natom0) ** (1 / 3), 1.8)
    numbers = g.choice(np.array([1, 6, 8]), size=natom)
    return S.SyntheticMolecule(coords=coords, numbers=numbers.astype(np.int32), charges=numbers.astype(np.float64),
                               shells=S.make_basis(g, coords, numbers, S.RECIPES[config]), D=None, name=config)


def _molecule(case: dict, seed: int) -> S.SyntheticMolecule:
    """The case's molecule with a density matrix 2 C C^T of its own for every seed
    (C orthonormal); zero beyond 12 bohr between centres in the sparse configuration."""
    mol = _structure(case)
    natom0, _, nocc0 = BASE[case["config"]]
    M = mol.nbasis
    g = torch.Generator(device="cuda").manual_seed(seed)
    C = torch.randn(M, max(1, min(M, nocc0 * case["natom"] // natom0)), dtype=torch.float64, device="cuda",
                    generator=g)
    C, _ = torch.linalg.qr(C)
    D = 2.0 * (C @ C.T)
    D = 0.5 * (D + D.T)
    if case["config"] == "c4":
        at = torch.as_tensor(np.repeat([s.atom for s in mol.shells], [S.nfunc(s.angmoms[0]) for s in mol.shells]),
                             device="cuda")
        xyz = torch.as_tensor(mol.coords, device="cuda")
        far = torch.cdist(xyz, xyz, compute_mode="donot_use_mm_for_euclid_dist") > 12.0
        D.masked_fill_(far[at][:, at], 0.0)
    mol.D = D.cpu().numpy()
    return mol


def _surface_points(mol, n: int, seed: int) -> torch.Tensor:
    """n points on nested surfaces at 1.4, 1.6, 1.8, 2.0 times the atoms' radii
    (2.3 bohr for H, 3.2 otherwise), those inside another atom's sphere removed."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    xyz = torch.as_tensor(mol.coords, device="cuda")
    rad = torch.as_tensor(np.where(mol.numbers == 1, 2.3, 3.2), device="cuda")
    found, have = [], 0
    while have < n:
        a = torch.randint(0, len(xyz), (2 * n,), device="cuda", generator=g)
        s = 1.4 + 0.2 * torch.randint(0, 4, (2 * n,), device="cuda", generator=g).double()
        v = torch.randn(2 * n, 3, device="cuda", dtype=torch.float64, generator=g)
        R = rad[a] * s
        p = xyz[a] + R[:, None] * v / v.norm(dim=1, keepdim=True)
        d = torch.cdist(p, xyz, compute_mode="donot_use_mm_for_euclid_dist")
        inside = d < rad[None, :] * s[:, None] - 1e-9
        inside[torch.arange(2 * n, device="cuda"), a] = False
        # the number of points of an atom's sphere follows its area
        keep = ~inside.any(dim=1) & (torch.rand(2 * n, device="cuda", generator=g) < (R / 6.4) ** 2)
        found.append(p[keep])
        have += int(keep.sum())
    return torch.cat(found)[:n].contiguous()


def _atom_grid(mol, nrad: int, ntheta: int, nphi: int):
    """Atom-centred product grid (Gauss-Chebyshev radial, Gauss-Legendre times
    uniform angular) with Becke partition weights; points and weights on the GPU."""
    i = np.arange(1, nrad + 1)
    x = np.cos(i * math.pi / (nrad + 1))
    r = (1 + x) / (1 - x)
    wr = math.pi / (nrad + 1) * np.sin(i * math.pi / (nrad + 1)) ** 2 / np.sqrt(1 - x ** 2) * 2 / (1 - x) ** 2 * r ** 2
    ct, wt = np.polynomial.legendre.leggauss(ntheta)
    ph = 2 * math.pi * (np.arange(nphi) + 0.5) / nphi
    st = np.sqrt(1 - ct ** 2)
    dirs = np.stack([np.outer(st, np.cos(ph)).ravel(), np.outer(st, np.sin(ph)).ravel(), np.repeat(ct, nphi)], 1)
    wang = np.repeat(wt, nphi) * (2 * math.pi / nphi)
    shell = torch.as_tensor((r[:, None, None] * dirs[None]).reshape(-1, 3), device="cuda")
    w0 = torch.as_tensor((wr[:, None] * wang[None]).ravel(), device="cuda")
    xyz = torch.as_tensor(mol.coords, device="cuda")
    A = len(xyz)
    pts = (xyz[:, None, :] + shell[None]).reshape(-1, 3).contiguous()
    owner = torch.arange(A, device="cuda").repeat_interleave(len(shell))
    d = torch.cdist(pts, xyz, compute_mode="donot_use_mm_for_euclid_dist")
    R = torch.cdist(xyz, xyz, compute_mode="donot_use_mm_for_euclid_dist")
    R.fill_diagonal_(1.0)
    P = torch.empty_like(d)
    for a in range(A):
        mu = (d[:, a:a + 1] - d) / R[a]
        for _ in range(3):
            mu = 1.5 * mu - 0.5 * mu ** 3
        f = 0.5 * (1.0 - mu)
        f[:, a] = 1.0
        P[:, a] = f.prod(dim=1)
    w = P.gather(1, owner[:, None])[:, 0] / P.sum(dim=1) * w0.repeat(A)
    return pts, w.contiguous()


def _inputs(case: dict, seed: int) -> dict:
    mol = _molecule(case, seed)
    kind = case["kind"]
    x = dict(mol=mol)
    if kind in ("host", "points", "ao", "esp_host"):
        g = np.random.default_rng(seed + 1)
        x["points"] = S.random_points(g, mol, case["n"])
    elif kind == "esp":
        x["points"] = _surface_points(mol, case["n"], seed + 1)
    elif kind == "cube":
        x["shape"] = (case["nx"], case["ny"], case["nz"])
        x["origin"], x["axes"] = S.cube_grid(mol, case["spacing"], x["shape"])
        x["origin"] = x["origin"] + np.random.default_rng(seed).uniform(-0.5, 0.5, 3) * case["spacing"]
    else:
        x["points"], x["weights"] = _atom_grid(mol, case["nrad"], case["ntheta"], case["nphi"])
    return x


def _npoints(case: dict) -> int:
    if case["kind"] == "cube":
        return case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "train":
        return case["natom"] * case["nrad"] * case["ntheta"] * case["nphi"]
    return case["n"]


SHAPE = {"grad": (3,), "hess": (3, 3)}


def prepare(case: dict, seed: int) -> dict:
    x = _inputs(case, seed)
    kind = case["kind"]
    s = dict(case=case, mol=ctc.molecule_from_synthetic(x["mol"]))
    s["mol"].basis_set_to_constant_memory(precision=case.get("precision", "fp64"))
    if kind in ("host", "esp_host"):
        s["points"] = x["points"]
    elif kind == "cube":
        s.update(shape=np.asarray(x["shape"], np.int32), origin=x["origin"], axes=x["axes"])
    else:
        s["points"] = torch.as_tensor(x["points"], device="cuda")
    if kind in ("points", "cube"):
        lead = x["shape"] if kind == "cube" else (case["n"],)
        s["out"] = {k: torch.empty(lead + SHAPE.get(k, ()), dtype=torch.float64, device="cuda")
                    for k in case["keys"].split(",")}
        s["ptrs"] = {k: t.data_ptr() for k, t in s["out"].items()}
    if kind == "esp":
        s["out"] = torch.empty(case["n"], dtype=torch.float64, device="cuda")
    if kind == "ao":
        nq = (1, 4, 10)[case["deriv"]]
        s["out"] = torch.empty(nq, case["n"], s["mol"].nbasis, dtype=torch.float64, device="cuda")
    if kind == "train":
        s["weights"] = x["weights"]
        s["D"] = torch.as_tensor(x["mol"].D, device="cuda").requires_grad_(True)
        s["coords"] = torch.as_tensor(x["mol"].coords).requires_grad_(True)
    return s


def run(s: dict):
    case, mol = s["case"], s["mol"]
    kind = case["kind"]
    if kind == "host":
        if case["keys"] == "rho":
            return {"rho": mol.compute_density(s["points"], precision=case["precision"])}
        return mol.compute_local_descriptors(s["points"], case["keys"].split(","), precision=case["precision"],
                                             alpha=ALPHA)
    if kind == "esp_host":
        return mol.compute_electrostatic_potential(s["points"])
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "points":
        mol.eval_local_device(s["points"].data_ptr(), case["n"], case["precision"], s["ptrs"], alpha=ALPHA,
                              stream=stream)
        return s["out"]
    if kind == "cube":
        mol.eval_cubic_device(s["origin"], s["axes"], s["shape"], case["precision"], s["ptrs"], alpha=ALPHA,
                              stream=stream)
        return s["out"]
    if kind == "esp":
        mol.eval_esp_device(s["points"].data_ptr(), case["n"], s["out"].data_ptr(), stream=stream)
        return s["out"]
    if kind == "ao":
        mol.eval_ao_device(s["points"].data_ptr(), case["n"], case["deriv"], s["out"].data_ptr(), stream=stream)
        return s["out"]
    s["D"].grad = s["coords"].grad = None
    rho, grad = ctc_autograd.density_and_gradient(mol, s["points"], s["D"], s["coords"])
    L = ctc_autograd.gga_functional(rho, grad, s["weights"])
    L.backward()
    return {"L": L.detach(), "rho": rho.detach(), "grad": grad.detach(), "dD": s["D"].grad, "dR": s["coords"].grad}


# ------------------------------------------------------------------ work
def _reach(mol):
    """Per segment: centre, number of functions, and the distance beyond which it is below 1e-18."""
    c, nf, r = [], [], []
    for sh in mol.shells:
        a = np.asarray(sh.exponents)
        for am, co in zip(sh.angmoms, np.asarray(sh.coeffs)):
            l = abs(am)
            k = np.abs(co) * (2 * a / math.pi) ** 0.75 * (4 * a) ** (l / 2)
            d = np.arange(0.1, 60.0, 0.1)
            f = (k[None] * np.exp(-a[None] * d[:, None] ** 2)).sum(1) * d ** l
            far = np.nonzero(f > 1e-18)[0]
            c.append(sh.center)
            nf.append(S.nfunc(am))
            r.append(d[far[-1]] if len(far) else 0.0)
    return np.asarray(c), np.asarray(nf), np.asarray(r)


def _shape_of(case):
    """Basis size, mean number of functions and of their products that reach a point, mean primitives."""
    mol = _structure(case)
    g = np.random.default_rng(0)
    if case["kind"] == "cube":
        o, ax = S.cube_grid(mol, case["spacing"], (case["nx"], case["ny"], case["nz"]))
        idx = g.integers(0, (case["nx"], case["ny"], case["nz"]), size=(400, 3))
        p = o + idx @ ax
    elif case["kind"] == "train":
        p = np.concatenate([mol.coords + g.standard_normal((case["natom"], 3)) * w for w in (0.3, 1.0, 2.0)])
    else:
        p = S.random_points(g, mol, 400)
    c, nf, r = _reach(mol)
    on = np.linalg.norm(p[:, None] - c[None], axis=-1) <= r[None]
    k = (on * nf[None]).sum(1).astype(float)
    prim = np.mean([len(s.exponents) for s in mol.shells])
    return mol.nbasis, k.mean(), (k * k).mean(), len(c), prim


def work(case: dict) -> dict:
    n, kind = _npoints(case), case["kind"]
    M, k1, k2, nseg, prim = _shape_of(case)
    if kind in ("host", "points", "cube"):
        keys = case["keys"].split(",")
        rows = 4 if set(keys) & {"hess", "lap", "tau_pd", "tau_alpha"} else 1
        nq = 10 if set(keys) & {"hess", "lap", "tau_alpha"} else (4 if rows == 4 or set(keys) & {"grad", "rdg"} else 1)
        width = sum({"grad": 3, "hess": 9}.get(k, 1) for k in keys)
        # contraction over the functions that reach the point, and forming those
        flops = n * (2.0 * rows * k2 + 2.0 * (16 if rows == 4 else nq) * k1 + nq * k1 * 8)
        return {"bytes": 8.0 * (n * (width + (0 if kind == "cube" else 3)) + M * M), "flops": flops}
    if kind == "train":
        fwd = n * (2.0 * k2 + 8.0 * k1 + 32.0 * k1)
        bwd = n * (2.0 * k2 + 2.0 * 4 * k2 + 60.0 * k1 + 80.0 * k1)
        return {"bytes": 8.0 * (n * (3 + 1 + 4) + 2 * M * M), "flops": fwd + bwd}
    if kind == "ao":
        nq = (1, 4, 10)[case["deriv"]]
        return {"bytes": 8.0 * (3 * n + nq * n * M), "flops": n * k1 * nq * 8.0}
    # one Hermite recursion per pair of primitives within reach of each other
    pairs = 0.5 * (nseg * prim) * (k1 / M * nseg * prim) * 0.15
    return {"bytes": 8.0 * (4 * n + M * M), "flops": n * pairs * 76.0}


# ------------------------------------------------------------------ exact values in 64 bits
CART = {0: [(0, 0, 0)], 1: [(1, 0, 0), (0, 1, 0), (0, 0, 1)],
        2: [(2, 0, 0), (0, 2, 0), (0, 0, 2), (1, 1, 0), (1, 0, 1), (0, 1, 1)],
        3: [(3, 0, 0), (0, 3, 0), (0, 0, 3), (1, 2, 0), (2, 1, 0), (2, 0, 1), (1, 0, 2), (0, 1, 2), (0, 2, 1),
            (1, 1, 1)],
        4: [(0, 0, 4), (0, 1, 3), (0, 2, 2), (0, 3, 1), (0, 4, 0), (1, 0, 3), (1, 1, 2), (1, 2, 1), (1, 3, 0),
            (2, 0, 2), (2, 1, 1), (2, 2, 0), (3, 0, 1), (3, 1, 0), (4, 0, 0)]}
_R3, _R15, _R6, _R10 = math.sqrt(3), math.sqrt(15), math.sqrt(1.5), math.sqrt(2.5)
# real solid harmonics, m = 0, 1, -1, 2, -2, ... (the generator has no pure g)
PURE = {2: [[(1.0, 0, 0, 2), (-0.5, 2, 0, 0), (-0.5, 0, 2, 0)], [(_R3, 1, 0, 1)], [(_R3, 0, 1, 1)],
            [(0.5 * _R3, 2, 0, 0), (-0.5 * _R3, 0, 2, 0)], [(_R3, 1, 1, 0)]],
        3: [[(1.0, 0, 0, 3), (-1.5, 2, 0, 1), (-1.5, 0, 2, 1)],
            [(2 * _R6, 1, 0, 2), (-0.5 * _R6, 3, 0, 0), (-0.5 * _R6, 1, 2, 0)],
            [(2 * _R6, 0, 1, 2), (-0.5 * _R6, 2, 1, 0), (-0.5 * _R6, 0, 3, 0)],
            [(0.5 * _R15, 2, 0, 1), (-0.5 * _R15, 0, 2, 1)], [(_R15, 1, 1, 1)],
            [(0.5 * _R10, 3, 0, 0), (-1.5 * _R10, 1, 2, 0)], [(1.5 * _R10, 2, 1, 0), (-0.5 * _R10, 0, 3, 0)]]}


def _odd(n):
    return math.prod(range(n, 0, -2)) if n > 0 else 1


def _components(am: int):
    """Terms (coefficient, a, b, c) of every function of a segment."""
    l = abs(am)
    if am >= 0:
        return [[(1 / math.sqrt(_odd(2 * a - 1) * _odd(2 * b - 1) * _odd(2 * c - 1)), a, b, c)] for a, b, c in CART[l]]
    return [[(t[0] / math.sqrt(_odd(2 * l - 1)), *t[1:]) for t in comp] for comp in PURE[l]]


class _Basis:
    """Segments grouped by angular momentum, primitives padded to equal length."""

    def __init__(self, mol, dev="cuda"):
        groups, ao = {}, 0
        for sh in mol.shells:
            a = np.asarray(sh.exponents)
            for am, co in zip(sh.angmoms, np.asarray(sh.coeffs)):
                k = co * (2 * a / math.pi) ** 0.75 * (4 * a) ** (abs(am) / 2)
                groups.setdefault(int(am), []).append((sh.center, sh.atom, a, k, ao))
                ao += S.nfunc(am)
        self.M, self.groups = ao, []
        self.atom = np.zeros(ao, np.int64)
        for am, gs in groups.items():
            K = max(len(g[2]) for g in gs)
            pad = lambda v, f: np.concatenate([v, np.full(K - len(v), f)])  # noqa: E731
            for g in gs:
                self.atom[g[4]:g[4] + S.nfunc(am)] = g[1]
            t = lambda v: torch.as_tensor(np.asarray(v), device=dev)  # noqa: E731
            self.groups.append(dict(am=am, c=t([g[0] for g in gs]), a=t([pad(g[2], 1.0) for g in gs]),
                                    k=t([pad(g[3], 0.0) for g in gs]), ao=t([g[4] for g in gs]),
                                    amin=t([g[2].min() for g in gs])))

    def aos(self, pts, deriv):
        """[q][n, m] AO values and derivatives of the functions that reach the
        points, and their indices."""
        lo, hi = pts.min(0).values, pts.max(0).values
        qs, index = [[] for _ in range((1, 4, 10)[deriv])], []
        for g in self.groups:
            gap = (lo - g["c"]).clamp(min=0) + (g["c"] - hi).clamp(min=0)
            on = torch.nonzero(g["amin"] * (gap * gap).sum(1) < 80.0)[:, 0]
            if not len(on):
                continue
            c, al, kf, ao = g["c"][on], g["a"][on], g["k"][on], g["ao"][on]
            x = pts[:, None, :] - c[None]
            r2 = (x * x).sum(-1)
            R = [0.0, 0.0, 0.0]
            for i in range(al.shape[1]):
                e = kf[:, i] * torch.exp(-al[:, i] * r2)
                for d in range(deriv + 1):
                    R[d] = R[d] + (-2 * al[:, i]) ** d * e
            pw = [[torch.ones_like(r2)] for _ in range(3)]
            for ax in range(3):
                for _ in range(abs(g["am"])):
                    pw[ax].append(pw[ax][-1] * x[..., ax])

            def mono(co, e):
                if min(e) < 0 or co == 0:
                    return 0.0
                return co * pw[0][e[0]] * pw[1][e[1]] * pw[2][e[2]]

            def poly(terms):
                v = 0.0
                for co, e in terms:
                    v = v + mono(co, e)
                return v

            def d_(terms, ax):
                return [(co * e[ax], tuple(v - (j == ax) for j, v in enumerate(e))) for co, e in terms]

            for j, comp in enumerate(_components(g["am"])):
                t0 = [(t[0], t[1:]) for t in comp]
                P = poly(t0)
                qs[0].append(P * R[0])
                if deriv >= 1:
                    P1 = [poly(d_(t0, k)) for k in range(3)]
                    for k in range(3):
                        qs[1 + k].append(P1[k] * R[0] + P * x[..., k] * R[1])
                if deriv >= 2:
                    q = 4
                    for k in range(3):
                        for m in range(k, 3):
                            v = poly(d_(d_(t0, k), m)) * R[0] + (P1[k] * x[..., m] + P1[m] * x[..., k]) * R[1]
                            if k == m:
                                v = v + P * R[1]
                            qs[q].append(v + P * x[..., k] * x[..., m] * R[2])
                            q += 1
                index.append(ao + j)
        if not index:
            return [torch.zeros(len(pts), 0, dtype=torch.float64, device=pts.device) for _ in qs], \
                torch.zeros(0, dtype=torch.int64, device=pts.device)
        return [torch.cat(q, 1) for q in qs], torch.cat(index)


def _descriptors(basis, D, pts, keys):
    out = {k: torch.empty((len(pts),) + SHAPE.get(k, ()), dtype=torch.float64, device=pts.device) for k in keys}
    second = bool(set(keys) & {"hess", "lap", "tau_alpha"})
    step = max(256, int(4e9 / (8 * 30 * basis.M)))
    for p0 in range(0, len(pts), step):
        A, ix = basis.aos(pts[p0:p0 + step], 2 if second else 1)
        Dm = D[ix][:, ix]
        G = [A[q] @ Dm for q in range(4)]
        rho = (G[0] * A[0]).sum(1)
        grad = torch.stack([2 * (G[0] * A[1 + k]).sum(1) for k in range(3)], 1)
        tau = 0.5 * sum((G[1 + k] * A[1 + k]).sum(1) for k in range(3))
        v = dict(rho=rho, grad=grad, tau_pd=tau)
        if second:
            H = torch.empty(len(rho), 3, 3, dtype=torch.float64, device=pts.device)
            q = 4
            for k in range(3):
                for m in range(k, 3):
                    H[:, k, m] = H[:, m, k] = 2 * ((G[1 + k] * A[1 + m]).sum(1) + (G[0] * A[q]).sum(1))
                    q += 1
            lap = H[:, 0, 0] + H[:, 1, 1] + H[:, 2, 2]
            d43 = rho.clamp(min=0) ** (4 / 3)
            v.update(hess=H, lap=lap, tau_alpha=tau + ALPHA * lap)
            big = d43 > 1e-20
            v["rdg"] = 0.5 / (3 * math.pi ** 2) ** (1 / 3) * torch.where(
                big, grad.norm(dim=1) / torch.where(big, d43, torch.ones_like(d43)), torch.full_like(d43, 1e-20))
        for k in keys:
            out[k][p0:p0 + step] = v[k]
    return out


def _exact_train(x):
    mol, pts = x["mol"], x["points"]
    basis = _Basis(mol)
    D = torch.as_tensor(mol.D, device="cuda")
    v = _descriptors(basis, D, pts, ["rho", "grad"])
    rho, grad = v["rho"].requires_grad_(True), v["grad"].requires_grad_(True)
    mask = rho > 1e-10
    r43 = torch.where(mask, rho, torch.ones_like(rho)) ** (4.0 / 3.0)
    f = -0.7386 * r43 + 0.0042 * (grad * grad).sum(-1) / r43
    L = (x["weights"] * torch.where(mask, f, torch.zeros_like(f))).sum()
    vr, vg = torch.autograd.grad(L, [rho, grad])
    dD = torch.zeros_like(D)
    dR = torch.zeros(len(mol.coords), 3, dtype=torch.float64, device="cuda")
    atom = torch.as_tensor(basis.atom, device="cuda")
    second = ((4, 5, 6), (5, 7, 8), (6, 8, 9))
    step = max(256, int(4e9 / (8 * 30 * basis.M)))
    for p0 in range(0, len(pts), step):
        A, ix = basis.aos(pts[p0:p0 + step], 2)
        r, g = vr[p0:p0 + step, None], vg[p0:p0 + step]
        W = r * A[0] + 2 * sum(g[:, k:k + 1] * A[1 + k] for k in range(3))
        X = A[0].T @ W
        dD[ix[:, None], ix[None]] += 0.5 * (X + X.T)
        Dm = D[ix][:, ix]
        G = [A[q] @ Dm for q in range(4)]
        for j in range(3):
            c = -2 * r * A[1 + j] * G[0]
            for k in range(3):
                c = c - 2 * g[:, k:k + 1] * (A[second[j][k]] * G[0] + A[1 + j] * G[1 + k])
            dR[:, j].index_add_(0, atom[ix], c.sum(0))
    return {"L": L.detach(), "rho": rho.detach(), "grad": grad.detach(), "dD": dD, "dR": dR.cpu()}


def _boys(nmax, T):
    """F_n(T), n = 0..nmax: series of F_nmax and downward recursion, asymptotic beyond 70."""
    Ts = T.clamp(max=70.0)
    term = torch.full_like(T, 1.0 / (2 * nmax + 1))
    total = term.clone()
    for i in range(1, 260):
        term = term * (2 * Ts / (2 * nmax + 2 * i + 1))
        total = total + term
    e = torch.exp(-Ts)
    F = [None] * (nmax + 1)
    F[nmax] = e * total
    for n in range(nmax, 0, -1):
        F[n - 1] = (2 * Ts * F[n] + e) / (2 * n - 1)
    far = 0.5 * torch.sqrt(math.pi / T.clamp(min=1.0))
    for n in range(nmax + 1):
        F[n] = torch.where(T > 70.0, far, F[n])
        far = far * (2 * n + 1) / (2 * T.clamp(min=1.0))
    return F


def _exact_esp(mol, pts):
    """Nuclear minus electronic potential by the McMurchie-Davidson scheme over all primitive pairs."""
    basis = _Basis(mol)
    D = torch.as_tensor(mol.D, device="cuda")
    xyz = torch.as_tensor(mol.coords, device="cuda")
    q = torch.as_tensor(mol.charges, device="cuda")
    V = (q / torch.cdist(pts, xyz, compute_mode="donot_use_mm_for_euclid_dist")).sum(1)
    gs = basis.groups
    for ia, A in enumerate(gs):
        for B in gs[ia:]:
            la, lb = abs(A["am"]), abs(B["am"])
            L = la + lb
            I, J = torch.meshgrid(torch.arange(len(A["ao"])), torch.arange(len(B["ao"])), indexing="ij")
            keep = (I <= J) if A is B else torch.ones_like(I, dtype=torch.bool)
            I, J = I[keep].cuda(), J[keep].cuda()
            fac = torch.where(I == J, 1.0, 2.0).double() if A is B else torch.full(I.shape, 2.0, device="cuda").double()
            KA, KB = A["a"].shape[1], B["a"].shape[1]
            I, J, fac = (v.repeat_interleave(KA * KB) for v in (I, J, fac))
            ka = torch.arange(KA, device="cuda").repeat_interleave(KB).repeat(len(I) // (KA * KB))
            kb = torch.arange(KB, device="cuda").repeat(len(I) // KB)
            a, b = A["a"][I, ka], B["a"][J, kb]
            cc = fac * A["k"][I, ka] * B["k"][J, kb]
            on = cc != 0
            I, J, a, b, cc = (v[on] for v in (I, J, a, b, cc))
            p = a + b
            RA, RB = A["c"][I], B["c"][J]
            P = (a[:, None] * RA + b[:, None] * RB) / p[:, None]
            E = []
            for d in range(3):
                X = RA[:, d] - RB[:, d]
                e = {(0, 0, 0): torch.exp(-a * b / p * X * X)}
                z = torch.zeros_like(a)
                get = lambda i, j, t: e.get((i, j, t), z)  # noqa: E731
                for i in range(la + 1):
                    for j in range(lb + 1):
                        for t in range(i + j + 1):
                            if i == j == 0:
                                continue
                            i1, j1, w = (i - 1, j, -b / p * X) if j == 0 else (i, j - 1, a / p * X)
                            e[(i, j, t)] = get(i1, j1, t - 1) / (2 * p) + w * get(i1, j1, t) + (t + 1) * get(i1, j1, t + 1)
                E.append(e)
            tuv = [(t, u, s - t - u) for s in range(L + 1) for t in range(s, -1, -1) for u in range(s - t, -1, -1)]
            h = {k: torch.zeros_like(a) for k in tuv}
            for i, ca in enumerate(_components(A["am"])):
                for j, cb in enumerate(_components(B["am"])):
                    d = D[A["ao"][I] + i, B["ao"][J] + j] * cc * 2 * math.pi / p
                    for (fa, *ea) in ca:
                        for (fb, *eb) in cb:
                            for t in range(ea[0] + eb[0] + 1):
                                for u in range(ea[1] + eb[1] + 1):
                                    for v in range(ea[2] + eb[2] + 1):
                                        h[(t, u, v)] += fa * fb * d * E[0][(ea[0], eb[0], t)] * \
                                            E[1][(ea[1], eb[1], u)] * E[2][(ea[2], eb[2], v)]
            step = max(1, int(2e7 / len(pts)))
            for k0 in range(0, len(a), step):
                pk, Pk = p[k0:k0 + step, None], P[k0:k0 + step]
                X = [Pk[:, None, d] - pts[None, :, d] for d in range(3)]
                F = _boys(L, pk * (X[0] ** 2 + X[1] ** 2 + X[2] ** 2))
                R = {(0, 0, 0): (-2 * pk) ** L * F[L]}
                for n in range(L - 1, -1, -1):
                    new = {(0, 0, 0): (-2 * pk) ** n * F[n]}
                    for key in tuv[1:]:
                        if sum(key) > L - n:
                            break
                        ax = next(d for d in range(3) if key[d])
                        lower = tuple(v - (d == ax) for d, v in enumerate(key))
                        v = X[ax] * R[lower]
                        if key[ax] > 1:
                            v = v + (key[ax] - 1) * R[tuple(w - 2 * (d == ax) for d, w in enumerate(key))]
                        new[key] = v
                    R = new
                for key in tuv:
                    V -= h[key][k0:k0 + step] @ R[key]
    return V


def exact(case: dict, seed: int):
    kind = case["kind"]
    # a full pair sum of a larger molecule takes minutes in plain torch
    if kind in ("esp", "esp_host") and _npoints(case) * case["natom"] ** 2 > 4e5:
        return None
    x = _inputs(case, seed)
    mol = x["mol"]
    if kind == "train":
        return _exact_train(x)
    if kind == "cube":
        pts = torch.as_tensor(S.cube_points(x["origin"], x["axes"], x["shape"]), device="cuda")
    else:
        pts = torch.as_tensor(x["points"], device="cuda")
    if kind in ("esp", "esp_host"):
        V = _exact_esp(mol, pts)
        return V.cpu().numpy() if kind == "esp_host" else V
    basis = _Basis(mol)
    if kind == "ao":
        out = torch.zeros((1, 4, 10)[case["deriv"]], len(pts), basis.M, dtype=torch.float64, device="cuda")
        for p0 in range(0, len(pts), 4096):
            A, ix = basis.aos(pts[p0:p0 + 4096], case["deriv"])
            for q, v in enumerate(A):
                out[q, p0:p0 + 4096, ix] = v
        return out
    v = _descriptors(basis, torch.as_tensor(mol.D, device="cuda"), pts, case["keys"].split(","))
    if kind == "cube":
        return {k: t.reshape(x["shape"] + SHAPE.get(k, ())) for k, t in v.items()}
    return {k: t.cpu().numpy() for k, t in v.items()} if kind == "host" else v
