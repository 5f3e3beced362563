"""The work that programs have this package do, as cases that can be timed.

Each case is one pass through the package's public entry points on a molecule that is already on the GPU: the
exchange-correlation energy and potential of classical functionals in the FP64 form (the default) and the mixed
form, the density features alone, ``predict`` as an SCF driver calls it, the DM21 network's training step and its
second-order step, the chi tensor of the exact-exchange terms and the AO tables.  Molecules are seeded: atoms in a
box that grows with their number, s/p/d Gaussians on the atoms, grid points in shells around each atom (stored atom by
atom, log-normal weights), and density matrices that are projectors on an eighth of the AOs.
"""
import math

import torch

import graddft_gb300 as G

F64 = torch.float64
DEV = "cuda"
CLIP = 1e-30
LAYERS, WIDTH = 6, 256  # DM21's network
PRIMS = {0: 4, 1: 3, 2: 2}  # contracted shells per atom (4s 3p 2d = 23 AOs)


def listed():
    return [
        # The smallest call: one light molecule of a training set; latency and launches are what it costs.
        {"name": "blyp_tiny", "op": "xc", "functional": "BLYP", "precision": "fp64", "n_ao": 24, "n_grid": 3600},
        # H2O in def2-TZVP on a level-2 grid: energy and Fock matrix, one SCF cycle of a driver.
        {"name": "water_predict", "op": "predict", "functional": "BLYP", "precision": "fp64", "n_ao": 43,
         "n_grid": 33842},
        # An ordinary molecule with a gradient-corrected functional.
        {"name": "b88_medium", "op": "xc", "functional": "B88", "precision": "fp64", "n_ao": 115, "n_grid": 65536},
        # The largest molecule of a training set in the default form.
        {"name": "blyp_large", "op": "xc", "functional": "BLYP", "precision": "fp64", "n_ao": 400, "n_grid": 150001},
        # Density, gradient, Laplacian and kinetic density for a program's own functional; odd sizes.
        {"name": "features", "op": "features", "functional": "", "precision": "fp64", "n_ao": 187, "n_grid": 100003},
        # The headline contraction (512 AOs, mixed form) on a quarter of its grid.
        {"name": "blyp_mixed", "op": "xc", "functional": "BLYP", "precision": "tf32x3", "n_ao": 512, "n_grid": 262144},
        # predict with DM21 and both exact-exchange Fock terms from chi.
        {"name": "dm21_predict", "op": "predict", "functional": "DM21", "precision": "fp64", "n_ao": 64,
         "n_grid": 16384},
        # A training step of the network (E, V and the parameter gradients) in the default form.
        {"name": "dm21_step", "op": "step", "functional": "DM21", "precision": "fp64", "n_ao": 115, "n_grid": 16400},
        # The same in the mixed form, 256 AOs on a quarter of the benchmark's grid.
        {"name": "dm21_step_mixed", "op": "step", "functional": "DM21", "precision": "tf32x3", "n_ao": 256,
         "n_grid": 131072},
        # A loss that reads V_xc, as the differentiable SCF loop's does: first and second-order pass.
        {"name": "dm21_second_order", "op": "second", "functional": "DM21", "precision": "fp64", "n_ao": 96,
         "n_grid": 8192},
        # chi for DM21's two omegas, made once per density matrix.
        {"name": "chi", "op": "chi", "functional": "", "precision": "fp64", "n_ao": 115, "n_grid": 8192},
        # AO values, gradients and second derivatives of contracted shells, made once per geometry.
        {"name": "ao_tables", "op": "ao", "functional": "", "precision": "fp64", "n_ao": 506, "n_grid": 20001},
    ]


# op: (n_ao range, n_grid range, forms, functionals, the most that n_grid * n_ao^p may be, p)
RANGES = {
    "xc": ((24, 400), (3600, 150000), ("fp64", "tf32x3"), ("LSDA", "B88", "BLYP"), 2e10, 2),
    "features": ((24, 400), (3600, 150000), ("fp64", "tf32x3"), ("",), 2e10, 2),
    "predict": ((24, 72), (3600, 40000), ("fp64",), ("BLYP", "DM21"), 2e6, 1),
    "step": ((24, 256), (3600, 32000), ("fp64", "tf32x3"), ("DM21",), 3e6, 1),
    "second": ((24, 128), (3600, 12000), ("fp64",), ("DM21",), 1e6, 1),
    "chi": ((23, 138), (3600, 12000), ("fp64",), ("",), 1e6, 1),
    "ao": ((46, 506), (3600, 65000), ("fp64",), ("",), 1.5e7, 1),
}


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["xc", "xc", "xc", "features", "predict", "step", "second", "chi", "ao"])
    aos, grid, forms, functionals, most, p = RANGES[op]
    n_ao, n_grid = size(*aos), size(*grid)
    if op in ("chi", "ao"):
        n_ao = max(1, n_ao // 23) * 23
    n_grid = max(grid[0], min(n_grid, int(most / n_ao ** p)))
    return {"op": op, "functional": rng.choice(functionals), "precision": rng.choice(forms), "n_ao": n_ao,
            "n_grid": n_grid}


# ------------------------------------------------------------------ seeded molecules
class Draws:
    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(int(seed))

    def uniform(self, lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(shape, dtype=F64, device=DEV, generator=self.g)

    def normal(self, *shape):
        return torch.randn(shape, dtype=F64, device=DEV, generator=self.g)

    def integers(self, n, *shape):
        return torch.randint(0, n, shape, device=DEV, generator=self.g)


def make_atoms(d, n_ao):
    n = max(1, n_ao // 20)
    return d.uniform(-0.5, 0.5, n, 3) * 4.5 * n ** (1 / 3)  # bohr


def make_grid(d, atoms, n_grid):
    """Points in shells around each atom, stored atom by atom."""
    owner = torch.arange(n_grid, device=DEV) * atoms.shape[0] // n_grid
    x = d.uniform(0.0, 1.0, n_grid)
    r = 0.02 + 7.0 * x ** 2
    u = d.normal(n_grid, 3)
    coords = atoms[owner] + r[:, None] * u / u.norm(dim=1, keepdim=True)
    weights = torch.exp(-6.0 + d.normal(n_grid)) * (0.05 + r ** 2 / 4.0)
    return coords, weights


def make_primitives(d, atoms, n_ao):
    """n_ao normalised s/p/d Gaussians N (c0 + b.x + x A x) exp(-alpha x^2) on the atoms."""
    centre = atoms[torch.arange(n_ao, device=DEV) * atoms.shape[0] // n_ao]
    alpha = torch.exp(d.uniform(math.log(0.1), math.log(50.0), n_ao))
    kind = d.integers(9, n_ao)  # s, px, py, pz, xy, yz, xz, x2-y2, 2z2-x2-y2
    kind = torch.where(d.uniform(0.0, 1.0, n_ao) < 0.25, torch.zeros_like(kind), kind)
    c0 = (kind == 0).to(F64)
    b = torch.stack([(kind == 1 + i).to(F64) for i in range(3)], 1)
    A = torch.zeros((n_ao, 3, 3), dtype=F64, device=DEV)
    for k, (i, j) in ((4, (0, 1)), (5, (1, 2)), (6, (0, 2))):
        A[kind == k, i, j] = A[kind == k, j, i] = 0.5
    A[kind == 7] = torch.diag(torch.tensor([1.0, -1.0, 0.0], dtype=F64, device=DEV))
    A[kind == 8] = torch.diag(torch.tensor([-1.0, -1.0, 2.0], dtype=F64, device=DEV))
    i0 = (math.pi / (2 * alpha)) ** 1.5
    norm = torch.where(kind == 0, i0 ** -0.5, torch.where(kind <= 3, torch.sqrt(4 * alpha / i0), 4 * alpha / i0 ** 0.5))
    norm = torch.where(kind == 7, norm / 2, torch.where(kind == 8, norm / math.sqrt(12.0), norm))
    return centre, c0, b, A, alpha[:, None], norm[:, None]


def tables(basis, coords):
    """phi (grid, ao), its gradient and its diagonal second derivatives (grid, ao, 3); the radial part of an AO is a
    sum of Gaussians, (ao, primitives)."""
    centre, c0, b, A, alpha, coef = basis
    x = coords[:, None, :] - centre[None]
    r2 = (x * x).sum(-1)
    g0 = torch.zeros_like(r2)
    g1, g2 = torch.zeros_like(r2), torch.zeros_like(r2)  # d/d(r2) once and twice
    for k in range(alpha.shape[1]):
        e = coef[:, k] * torch.exp(-alpha[:, k] * r2)
        g0 += e
        g1 -= alpha[:, k] * e
        g2 += alpha[:, k] ** 2 * e
    Ax = torch.einsum("aij,raj->rai", A, x)
    P = c0 + torch.einsum("ai,rai->ra", b, x) + (Ax * x).sum(-1)
    dP = b + 2 * Ax
    d2P = 2 * torch.diagonal(A, dim1=1, dim2=2)
    P, g0, g1, g2 = P[..., None], g0[..., None], g1[..., None], g2[..., None]
    return ((P * g0)[..., 0], dP * g0 + 2 * x * P * g1,
            d2P * g0 + 4 * x * dP * g1 + P * (2 * g1 + 4 * x * x * g2))


def make_rdm1(d, n_ao):
    n_occ = max(1, n_ao // 8)
    out = []
    for _ in range(2):
        q = torch.linalg.qr(d.normal(n_ao, n_ao))[0][:, :n_occ]
        out.append(q @ q.T)
    return torch.stack(out)


def make_molecule(case, seed):
    d = Draws(seed)
    n_ao, n_grid = case["n_ao"], case["n_grid"]
    atoms = make_atoms(d, n_ao)
    coords, weights = make_grid(d, atoms, n_grid)
    m = {"d": d, "coords": coords, "weights": weights, "basis": make_primitives(d, atoms, n_ao),
         "rdm1": make_rdm1(d, n_ao)}
    if case["op"] == "predict":
        h = d.normal(n_ao, n_ao)
        t = d.normal(2 * n_ao, n_ao, n_ao) / n_ao
        t = (t + t.transpose(1, 2)) / 2
        m |= {"h1e": (h + h.T) / 2, "rep": torch.einsum("pab,pcd->abcd", t, t), "enuc": 9.0}
    if case["functional"] == "DM21":
        m["params"] = make_params(d)
        m["spread"] = d.uniform(0.6, 1.0, 2, 2, n_grid)
    return m


def make_params(d):
    p = {}

    def dense(k, n_in, n_out):
        lim = math.sqrt(6.0 / (n_in + n_out))
        p["Dense_%d" % k] = {"kernel": d.uniform(-lim, lim, n_in, n_out), "bias": d.uniform(-0.1, 0.1, n_out)}

    dense(0, 11, WIDTH)
    for i in range(LAYERS):
        dense(i + 1, WIDTH, WIDTH)
        p["LayerNorm_%d" % i] = {"scale": d.uniform(0.9, 1.1, WIDTH), "bias": d.uniform(-0.1, 0.1, WIDTH)}
    dense(LAYERS + 1, WIDTH, 3)
    return {"params": p}


def make_chi(m, phi):
    """A stand-in for chi (grid, omega, spin, ao): two scaled and spread copies of phi D."""
    x = torch.einsum("ra,sab->rsb", phi, m["rdm1"])
    return torch.stack([k * (1.0 + 0.3 * m["spread"][w, 0][:, None, None]) * x for w, k in enumerate((1.0, 0.6))], 1)


def make_ehf(m, rho):
    """Exact-exchange energy densities (omega, spin, grid) of the size of the local exchange."""
    scale = torch.tensor([1.0, 0.7], dtype=F64, device=DEV)[:, None, None]
    return -0.5 * m["spread"] * scale * torch.clamp(rho.T, min=0.0) ** (4 / 3)


def make_shells(case, seed):
    """Contracted s/p/d shells on the atoms: (centre, l, exponents, coefficients, angular rows) each."""
    d = Draws(seed)
    atoms = make_atoms(d, case["n_ao"])[: case["n_ao"] // 23]
    coords, weights = make_grid(d, atoms, case["n_grid"])
    rows = {0: torch.ones((1, 1), dtype=F64), 1: torch.eye(3, dtype=F64),
            2: torch.tensor([[0, 1.0, 0, 0, 0, 0], [0, 0, 0, 0, 1.0, 0], [-0.5, 0, 0, -0.5, 0, 1.0], [0, 0, 1.0, 0, 0, 0],
                             [0.8, 0, 0, -0.8, 0, 0]], dtype=F64)}  # on xx, xy, xz, yy, yz, zz
    shells = []
    host = atoms.cpu()
    for a in range(atoms.shape[0]):
        for l, count in ((0, 4), (1, 3), (2, 2)):
            k = PRIMS[l]
            exps = torch.exp(d.uniform(math.log(0.15), math.log(30.0), count, k)).cpu()
            coefs = (d.uniform(0.2, 1.0, count, k).cpu() * exps ** (0.75 + 0.5 * l))
            for c in range(count):
                shells.append((host[a], l, exps[c], coefs[c], rows[l]))
    return {"d": d, "coords": coords, "weights": weights, "shells": shells, "rdm1": make_rdm1(d, case["n_ao"])}


def shell_tables(shells, coords):
    """The AO tables of the contracted shells, by the formula."""
    most = max(PRIMS.values())
    centre, c0, b, A, alpha, coef = [], [], [], [], [], []
    for at, l, exps, coefs, rows in shells:
        for row in rows:
            centre.append(at)
            c0.append(float(row[0]) if l == 0 else 0.0)
            b.append(row if l == 1 else torch.zeros(3, dtype=F64))
            q = torch.zeros((3, 3), dtype=F64)
            if l == 2:
                for v, (i, j) in zip(row, ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))):
                    q[i, j] += v / 2
                    q[j, i] += v / 2
            A.append(q)
            pad = most - exps.shape[0]
            alpha.append(torch.cat([exps, torch.ones(pad, dtype=F64)]))
            coef.append(torch.cat([coefs, torch.zeros(pad, dtype=F64)]))
    basis = [torch.stack(v).to(DEV) for v in (centre, b, A, alpha, coef)]
    return tables((basis[0], torch.tensor(c0, dtype=F64, device=DEV), *basis[1:]), coords)


# ------------------------------------------------------------------ the package's side
def functional_of(case):
    name = case["functional"]
    if name != "DM21":
        from graddft_gb300 import popular_functionals

        return getattr(popular_functionals, name) if name else None
    if case["op"] == "predict":  # with the exact-exchange terms from chi
        return G.DM21(precision=case["precision"])
    return G.DM21(densitygrads=None, coefficient_input_grads=None, precision=case["precision"])


def prepare(case, seed):
    if case["op"] in ("chi", "ao"):
        from graddft_gb300.basis import Shell

        m = make_shells(case, seed)
        basis = G.ShellBasis([Shell(c.numpy(), l, e.numpy(), k.numpy(), r.numpy()) for c, l, e, k, r in m["shells"]])
        s = {"op": case["op"], "basis": basis, "coords": m["coords"]}
        basis.device_desc(m["coords"].device)
        if case["op"] == "chi":
            s |= {"rdm1": m["rdm1"], "ao": G.eval_ao(basis, m["coords"], 0)}
        return s
    m = make_molecule(case, seed)
    n_ao, n_grid = case["n_ao"], case["n_grid"]
    phi = torch.empty((n_grid, n_ao), dtype=F64, device=DEV)
    g1 = torch.empty((n_grid, n_ao, 3), dtype=F64, device=DEV)
    g2 = torch.empty_like(g1)
    for at in range(0, n_grid, 16384):
        phi[at:at + 16384], g1[at:at + 16384], g2[at:at + 16384] = tables(m["basis"], m["coords"][at:at + 16384])
    more = {}
    if case["functional"] == "DM21":
        if case["op"] == "predict":
            more = {"chi": make_chi(m, phi), "omegas": torch.tensor([0.0, 0.4], dtype=F64)}
        else:
            rho = torch.stack([((phi @ D) * phi).sum(1) for D in m["rdm1"]], 1)
            more = {"ehf": make_ehf(m, rho)}
    mol = G.Molecule(grid=G.Grid(m["coords"], m["weights"]), atom_index=None, nuclear_pos=None, ao=phi, grad_ao=g1,
                     grad_n_ao={2: g2}, rdm1=m["rdm1"], nuclear_repulsion=m.get("enuc", 0.0), h1e=m.get("h1e"), vj=None,
                     mo_coeff=None, mo_occ=None, mo_energy=None, rep_tensor=m.get("rep"), precision=case["precision"],
                     **more)
    mol.resident()
    s = {"op": case["op"], "mol": mol, "functional": functional_of(case), "params": m.get("params")}
    if case["op"] == "predict":
        s["predict"] = G.energy_predictor(s["functional"])
    if case["op"] == "second":
        for leaves in s["params"]["params"].values():
            for t in leaves.values():
                t.requires_grad_(True)
        s["tangent"] = tangent(m)
    return s


def tangent(m):
    t = m["d"].normal(*m["rdm1"].shape)
    return (t + t.transpose(1, 2)) / 2


def leaves_of(params):
    return [t for k in sorted(params["params"]) for _, t in sorted(params["params"][k].items())]


def run(s):
    op = s["op"]
    if op == "ao":
        return G.eval_ao(s["basis"], s["coords"], 2)
    if op == "chi":
        return G.generate_chi_tensor(s["rdm1"], s["ao"], s["coords"], s["basis"], [0.0, 0.4], chunk_size=4096)
    mol, f = s["mol"], s["functional"]
    if op == "features":
        return mol.resident().density(mol.rdm1)
    if op == "xc":
        return f.xc_energy_and_grads(None, mol)
    if op == "predict":
        return s["predict"](s["params"], mol)
    if op == "step":
        e, v, grads = f.xc_energy_and_grads_params(s["params"], mol)
        return e, v, leaves_of(grads)
    e, v = f.xc_energy_and_potential(s["params"], mol)
    wanted = leaves_of(s["params"])
    return e.detach(), v.detach(), list(torch.autograd.grad(e + (v * s["tangent"]).sum(), wanted))


def work(case):
    n, N, op = case["n_ao"], case["n_grid"], case["op"]
    planes = 8.0 * N * n
    net = 2.0 * N * (11 * WIDTH + LAYERS * WIDTH * WIDTH + 3 * WIDTH)  # one pass forward
    gga = case["functional"] in ("LSDA", "B88")
    if op == "xc":  # both contractions, both spins; the kinetic planes only where the Laplacian is read
        return {"bytes": planes * (4 if gga else 5) + 32.0 * n * n, "flops": (8.0 if gga else 32.0) * N * n * n}
    if op == "features":
        return {"bytes": planes * 5 + 16.0 * n * n + 96.0 * N, "flops": 16.0 * N * n * n}
    if op == "predict":
        b, f = planes * 5 + 8.0 * n ** 4, 32.0 * N * n * n + 4.0 * n ** 4
        if case["functional"] == "DM21":  # plus chi once, the network and the three exchange contractions
            b, f = b + 4 * planes, f + 3 * net + 12.0 * N * n * n + 24.0 * N * n
        return {"bytes": b, "flops": f}
    if op == "step":
        return {"bytes": planes * 5 + 32.0 * n * n + 32.0 * N, "flops": 32.0 * N * n * n + 3 * net}
    if op == "second":
        return {"bytes": planes * 5 + 48.0 * n * n + 32.0 * N, "flops": 64.0 * N * n * n + 9 * net}
    if op == "chi":  # both omegas' integrals of each pair once, at one operation each, and the contraction
        return {"bytes": planes * 5, "flops": N * n * n * (1.0 * 2 + 8.0)}
    return {"bytes": planes * 7 + 24.0 * N, "flops": 60.0 * N * n}


# ------------------------------------------------------------------ the same in plain torch, 64 bits
def clipped(x):
    return torch.where(x.abs() > CLIP, x, torch.zeros((), dtype=F64, device=DEV))


def features_of(D, phi, g1, g2):
    X = torch.einsum("ra,sab->srb", phi, D)
    K = torch.stack([torch.einsum("ra,sab->srb", g1[..., j], D) for j in range(3)], -1)
    rho = (X * phi).sum(-1).T
    grad = 2 * torch.einsum("srb,rbj->rsj", X, g1)
    kin = (K * g1).sum((-1, -2)).T
    return rho, grad, 2 * kin + 2 * (X * g2.sum(-1)).sum(-1).T, 0.5 * kin


def e_lsda(rho):
    rho = torch.clamp(rho, min=CLIP)
    total = rho.sum(1)
    z = (rho[:, 0] - rho[:, 1]) / total
    f = ((1 - z) ** (4 / 3) + (1 + z) ** (4 / 3) - 2) / (2 * (2 ** (1 / 3) - 1))
    para, ferro = (-0.75 * (k / math.pi) ** (1 / 3) * total ** (4 / 3) for k in (3.0, 6.0))
    return para + (ferro - para) * f


def e_b88(rho, grad):
    beta = 0.0042
    rho = torch.clamp(rho, min=CLIP)
    g = torch.sqrt(torch.clamp((grad ** 2).sum(-1), min=CLIP))
    x = g / rho ** (4 / 3)
    return -(beta * g * x / (1 + 6 * beta * x * torch.asinh(x))).sum(1)


def e_lyp(rho, grad, lapl):
    a, b, c, d = 0.04918, 0.132, 0.2533, 0.349
    cf = 0.3 * (3 * math.pi ** 2) ** (2 / 3)
    zero = torch.zeros((), dtype=F64, device=DEV)
    rho = torch.clamp(rho, min=CLIP)
    total = rho.sum(1)
    t = (torch.where(rho > CLIP, (grad ** 2).sum(-1) / rho, zero) - lapl) / 8
    gamma = 2 * (1 - (rho ** 2).sum(1) / total ** 2)
    inner = (2 ** (2 / 3) * cf * (rho ** (8 / 3)).sum(1) - total * t.sum(1) + (rho * t).sum(1) / 9
             + (rho * lapl).sum(1) / 18)
    third = total ** (-1 / 3)
    return -a * gamma / (1 + d * third) * (total + 2 * b * total ** (-5 / 3) * inner * torch.exp(-c * third))


def e_dm21(rho):
    return -2 * math.pi * (3 / (4 * math.pi)) ** (4 / 3) * (torch.clamp(rho, min=CLIP) ** (4 / 3)).sum(1)


def inputs_of(rho, grad, tau, ehf):
    rho = torch.clamp(rho.abs(), min=CLIP) * torch.sign(rho)
    return torch.cat([rho, (grad.sum(1) ** 2).sum(-1, keepdim=True), (grad ** 2).sum(-1), tau, ehf[:, 0].T, ehf[:, 1].T], 1)


def network(params, x):
    p = params["params"]

    def dense(k, v):
        return v @ p["Dense_%d" % k]["kernel"] + p["Dense_%d" % k]["bias"]

    x = torch.tanh(dense(0, torch.log(x.abs() + 1e-4)))
    for i in range(LAYERS):
        x = dense(i + 1, x) + x
        mean = x.mean(-1, keepdim=True)
        var = torch.clamp((x * x).mean(-1, keepdim=True) - mean * mean, min=0.0)
        ln = p["LayerNorm_%d" % i]
        x = torch.nn.functional.elu((x - mean) * torch.rsqrt(var + 1e-6) * ln["scale"] + ln["bias"])
    return 2.0 * torch.sigmoid(dense(LAYERS + 1, x) / 2.0)


def energy_of(name, feats, weights, params=None, ehf=None, clip_local=True, inputs_ehf=None):
    rho, grad, lapl, tau = feats
    clip = clipped if clip_local else (lambda v: v)
    if name == "DM21":
        inputs_ehf = ehf if inputs_ehf is None else inputs_ehf
        e = torch.stack([clip(e_dm21(rho)), clip(ehf[0].sum(0)), clip(ehf[1].sum(0))], 1)
        e = (network(params, inputs_of(rho, grad, tau, inputs_ehf)) * e).sum(1)
    else:
        e = clipped(e_lsda(rho))
        if name in ("B88", "BLYP"):
            e = e + clipped(e_b88(rho, grad))
        if name == "BLYP":
            e = e + clipped(e_lyp(rho, grad, lapl))
    return (clipped(weights) * clipped(e)).sum()


def exact(case, seed):
    op, name = case["op"], case["functional"]
    if op == "chi":
        return None  # range-separated integrals of contracted shells have no short plain form
    if op == "ao":
        m = make_shells(case, seed)
        return shell_tables(m["shells"], m["coords"])
    if case["n_grid"] * case["n_ao"] ** 2 > 1e11:
        return None
    m = make_molecule(case, seed)
    D = m["rdm1"].clone().requires_grad_(True)
    params = m.get("params")
    wanted = [] if params is None else leaves_of(params)
    for t in wanted:
        t.requires_grad_(True)
    T = tangent(m) if op == "second" else None
    step = 1 << 12 if op == "second" else 1 << 14
    E, V, P, Q, feats_out, hf = 0.0, torch.zeros_like(m["rdm1"]), [torch.zeros_like(t) for t in wanted], None, [], 0.0
    Q = [torch.zeros_like(t) for t in wanted]
    for at in range(0, case["n_grid"], step):
        part = slice(at, at + step)
        phi, g1, g2 = tables(m["basis"], m["coords"][part])
        w = m["weights"][part]
        feats = features_of(D, phi, g1, g2)
        if op == "features":
            feats_out.append([t.detach() for t in feats])
            continue
        ehf = None
        if name == "DM21":
            mine = {**m, "spread": m["spread"][..., part]}
            if op == "predict":
                chi = make_chi(mine, phi)
                ehf = -0.5 * torch.einsum("rwsc,src->wsr", chi, torch.einsum("ra,sac->src", phi, m["rdm1"]))
            else:
                ehf = make_ehf(mine, feats[0].detach())
        e = energy_of(name, feats, w, params, ehf)
        E = E + e.detach()
        got = torch.autograd.grad(e, [D] + wanted, create_graph=op == "second")
        V += got[0].detach()
        for a, b in zip(P, got[1:]):
            a += b.detach()
        if op == "second":
            for a, b in zip(Q, torch.autograd.grad((got[0] * T).sum(), wanted, allow_unused=True)):
                if b is not None:
                    a += b
        if op == "predict" and name == "DM21":
            still = [t.detach() for t in feats]
            u = ehf.clone().requires_grad_(True)
            through = [torch.autograd.grad(energy_of(name, still, w, params, u, False, ehf), u)[0],
                       torch.autograd.grad(energy_of(name, still, w, params, ehf, False, u), u)[0]]
            hf = hf - 0.5 * torch.stack([torch.einsum("rwsb,wsr,ra->sab", chi, g, phi) for g in through])
    if op == "features":
        got = [torch.cat(v) for v in zip(*feats_out)]
        return {"rho": got[0], "grad_rho": got[1], "lapl": got[2], "tau": got[3]}
    if op == "xc":
        return E, V
    if op == "step":
        return E, V, P
    if op == "second":
        return E, V, [a + b for a, b in zip(P, Q)]
    total = m["rdm1"].sum(0)
    J = torch.einsum("abcd,cd->ab", m["rep"], total)
    E = E + m["enuc"] + (total * m["h1e"]).sum() + (total * J).sum() / 2
    F = clipped(m["h1e"] + J + V)
    F = clipped((F + F.transpose(1, 2)) / 2)
    if name == "DM21":
        for f in hf:
            F = clipped(F + f + f.transpose(1, 2))
    return E, F
