"""The work that users of this framework have it do, as measurable cases.

A case is one call (or the calls of one step) through the public entry points:
preparing a Hamiltonian from a cage, applying it on device or host vectors, the
device Lanczos loop alone and for a batch of problems, the reference driver's
loop body on host state, the Ritz-vector pass, and the Hellmann-Feynman
derivatives.  Grids are sinc-DVR grids over +-0.4 Angstrom, the cage is 20
SPC/E waters on a dodecahedron, the molecule is H2 (the values of the
repository's own configurations).

`exact` restates the whole path in plain FP64 torch: basis tables, Alavi SPC/E
potential, angular quadrature, kinetic contractions and the Lanczos recurrence.
"""
import importlib
import math

import numpy as np
import torch

bsl = importlib.import_module("boundstate-lanczos_gb300")

BOX = 0.08  # nm, the full width of every axis
MASS, ROT, CEILING = 2.01588, 0.709648713, 18.0  # amu, kJ/mol, kJ/mol
HBAR, COULOMB = 0.0635077857002, 138.9354846111096  # amu nm^2/ps; kJ/mol nm/e^2
LJ_A, LJ_B = 1.364e-06, 1.533e-3  # H2 centre - O Lennard-Jones (SPC/E)
Q_H, Q_CM, H_OFFSET = 0.4932, -0.9864, 0.03707  # Alavi H2: e, e, nm
BODY = np.array([[0.0, 0.0, 0.006461408220], [-8.164965810e-2, 0.0, -0.05127361870],
                 [8.164965810e-2, 0.0, -0.05127361870]])
Q_WATER = np.array([-0.8476, 0.4238, 0.4238])
SYM = {"All": 0, "Even": 1, "Odd": 2}


def _case(op, n, l_max, sym, nodes, precision, name=None, **more):
    """nodes: theta points and half of the phi points of the quadrature."""
    nx, ny, nz = (n, n, n) if isinstance(n, int) else n
    c = {"op": op, "nx": nx, "ny": ny, "nz": nz, "l_max": l_max, "sym": sym, "theta": nodes[0], "phi": nodes[1],
         "precision": precision}
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one H v of the 15^3 para problem on device vectors: the smallest call, all latency
        _case("hv", 15, 4, "Even", (12, 12), "fp64", "hv fp64 15^3 para"),
        # one FP64 H v on a box with three different edges, odd l <= 3
        _case("hv", (37, 29, 33), 3, "Odd", (12, 12), "fp64", "hv fp64 37x29x33 l3"),
        # one mixed-precision H v of the full-size ortho problem
        _case("hv", 54, 5, "Odd", (12, 12), "mixed", "hv mixed 54^3 ortho"),
        # the plugin interface's H v (host buffers, reference layout, FP64: the default precision)
        _case("hv_host", 27, 5, "Odd", (12, 12), "fp64", "hv host fp64 27^3 ortho"),
        # the full-size production run: Lanczos loop 1 on the device, mixed precision (one block of
        # iterations of the thousands that a run has: later coefficients depend on every rounding)
        _case("lanczos", 54, 5, "Odd", (12, 12), "mixed", "lanczos mixed 54^3 ortho", niter=32),
        # the same problem on the FP64 path
        _case("lanczos", 54, 5, "Odd", (12, 12), "fp64", "lanczos fp64 54^3 ortho", niter=16),
        # a small single problem, bound by latency and launches
        _case("lanczos", 15, 4, "Even", (12, 12), "mixed", "lanczos mixed 15^3 para", niter=96),
        # several cages in both symmetry blocks on grids of 27, 33 and 41 points, one batch
        _case("batch", 41, 5, "Odd", (12, 12), "mixed", "batch mixed 8 problems", niter=32, problems=8),
        # the reference driver's loop body on page-locked host state, full size
        _case("step", 54, 5, "Odd", (12, 12), "mixed", "step host mixed 54^3 ortho"),
        # eigenvectors: Lanczos loop 2 with 10 Ritz vectors
        _case("ritz", 27, 5, "Odd", (12, 12), "mixed", "ritz mixed 27^3 10 levels", niter=32, levels=10),
        # derivatives of 10 levels with respect to the cage
        _case("gradient", 21, 5, "Odd", (16, 16), "fp64", "gradient 21^3 10 levels", levels=10),
        # a new cage: HvPrep (potential, quadrature blocks) and the first H v
        _case("prep", 41, 5, "Odd", (30, 30), "mixed", "prep 41^3 30x60"),
    ]


BASES = ((5, "Odd"), (4, "Even"), (5, "Odd"), (4, "Even"), (3, "Odd"), (3, "All"), (2, "All"), (6, "Even"), (5, "All"))


def draw(rng):
    def edge(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(("hv", "hv", "hv_host", "lanczos", "lanczos", "batch", "step", "ritz", "gradient", "prep"))
    l_max, sym = rng.choice(BASES)
    precision = rng.choice(("fp64", "mixed", "mixed"))
    top = {"hv": 54, "hv_host": 40, "lanczos": 54, "batch": 41, "step": 48, "ritz": 27, "gradient": 21,
           "prep": 37}[op]
    if l_max == 5 and sym == "All":
        top = min(top, 33)  # 36 functions
    if sym == "Even" and l_max == 6:
        top = min(top, 41)
    low = 10
    a = edge(low, top)
    shape = rng.random()
    n = (a, a, a) if shape < 0.6 else (a, a, edge(low, top)) if shape < 0.85 else (a, edge(low, top), edge(low, top))
    nodes = (rng.randint(8, 12), rng.randint(8, 12))
    more = {}
    if op == "lanczos":
        size = n[0] * n[1] * n[2]
        more["niter"] = (rng.randint(24, 32) if size > 30000 else rng.randint(32, 96)) if precision == "mixed" else rng.randint(8, 16)
    elif op == "batch":
        l_max, sym, precision, n = 5, "Odd", "mixed", (a, a, a)
        more = {"niter": rng.randint(24, 32), "problems": rng.randint(2, 8)}
    elif op == "ritz":
        more = {"niter": rng.randint(24, 32), "levels": rng.randint(2, 10)}
    elif op == "gradient":
        more = {"levels": rng.randint(1, 10)}
    elif op == "prep":
        nodes = (rng.randint(10, 30), rng.randint(10, 30))
    return _case(op, n, l_max, sym, nodes, precision, **more)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _cage(seed, radius=3.95):
    """20 waters: centres of mass (Angstrom) on a dodecahedron, random ZYZ Euler angles."""
    g = (1.0 + math.sqrt(5.0)) / 2.0
    v = [(x, y, z) for x in (-1, 1) for y in (-1, 1) for z in (-1, 1)]
    for s in (-1, 1):
        for t in (-1, 1):
            v += [(0, s / g, t * g), (s / g, t * g, 0), (s * g, 0, t / g)]
    rng = np.random.default_rng([seed, 11])
    euler = np.stack([rng.uniform(0, 2 * math.pi, 20), rng.uniform(0, math.pi, 20), rng.uniform(0, 2 * math.pi, 20)], 1)
    return np.array(v, dtype=np.float64) * (radius / math.sqrt(3.0)), euler


def _problems(case, seed):
    """(case, cage seed, radius) of each problem of a batch: pairs of ortho and para blocks, uneven edges."""
    out = []
    for b in range(case["problems"]):
        l_max, sym = ((5, "Odd"), (4, "Even"))[b % 2]
        n = max(8, int(round(case["nx"] * (1.0, 33 / 41, 27 / 41)[(b * 2 + b // 2) % 3])))
        c = dict(case, op="lanczos", l_max=l_max, sym=sym, nx=n, ny=n, nz=n)
        out.append((c, 1000 * seed + b // 2, 3.85 + 0.02 * (b // 2 % 10)))
    return out


def _hamiltonian(case, cage, keep=False):
    p = bsl.HvParams()
    p.nx, p.ny, p.nz = p.pnx, p.pny, p.pnz = case["nx"], case["ny"], case["nz"]
    p.x_max = p.y_max = p.z_max = p.px_max = p.py_max = p.pz_max = BOX
    p.l_max, p.theta_points, p.phi_points, p.symmetry = case["l_max"], case["theta"], case["phi"], SYM[case["sym"]]
    p.total_mass, p.rotational_constant, p.ceiling_potential = MASS, ROT, CEILING
    return bsl.Hamiltonian.from_cage(p, cage[0], cage[1], precision=case["precision"], keep_potential_grid=keep)


def _sizes(case):
    n = case["nx"] * case["ny"] * case["nz"]
    nn = sum(2 * l + 1 for l in range(case["l_max"] + 1) if case["sym"] == "All" or l % 2 == (case["sym"] == "Odd"))
    return n, nn, (case["l_max"] + 1) ** 2


def _normal(seed, *shape):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    return torch.randn(*shape, dtype=torch.float64, device="cuda", generator=g)


def _host_vectors(case, seed):
    """A unit Lanczos vector and an r of the reference layout, on the host."""
    n, _, full = _sizes(case)
    v = _normal(seed, 2, n * full)
    return (v[0] / v[0].norm()).cpu(), (v[1] / v[1].norm()).cpu()


def _psi(case, seed):
    """Smooth bound-state-like vectors [level, basis] of the reference layout."""
    full = (case["l_max"] + 1) ** 2
    x, y, z = (torch.linspace(-2.5, 2.5, case[k], dtype=torch.float64, device="cuda") for k in ("nx", "ny", "nz"))
    r = torch.stack(torch.meshgrid(z, y, x, indexing="ij")).reshape(3, -1)
    lin = _normal(seed, case["levels"], full, 3)
    amp = _normal(seed + 1, case["levels"], full, 1)
    out = (amp + lin @ r) * torch.exp(-0.5 * (r * r).sum(0))
    return out.reshape(case["levels"], -1).cpu().numpy()


def prepare(case, seed):
    op = case["op"]
    if op == "batch":
        return {"op": op, "hs": [_hamiltonian(c, _cage(s, r)) for c, s, r in _problems(case, seed)],
                "niter": case["niter"]}
    cage = _cage(seed)
    state = {"op": op, "case": case, "cage": cage}
    n, nn, _ = _sizes(case)
    if op != "prep":
        state["h"] = _hamiltonian(case, cage, keep=op == "gradient")
    if op in ("hv", "prep"):
        state["v"] = _normal(seed, n * nn)
        state["u"] = torch.empty_like(state["v"])
    elif op == "hv_host":
        state["vec"], state["uec"] = (x.numpy() for x in _host_vectors(case, seed))
    elif op == "step":
        state["vec"], state["rvec"] = (x.pin_memory().numpy() for x in _host_vectors(case, seed))
    elif op == "ritz":
        state["rows"] = _rows(case, seed)
    elif op == "gradient":
        state["psi"] = _psi(case, seed)
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    op = state["op"]
    if op == "batch":
        return bsl.lanczos_batch(state["hs"], state["niter"])
    if op == "prep":
        h = _hamiltonian(state["case"], state["cage"])
        h.hv_device(state["v"].data_ptr(), state["u"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        h.close()
        return state["u"]
    h, case = state["h"], state["case"]
    if op == "hv":
        h.hv_device(state["v"].data_ptr(), state["u"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return state["u"]
    if op == "hv_host":
        h.hv(state["vec"], state["uec"])  # uec += H vec, as the reference driver's r
        return state["uec"]
    if op == "lanczos":
        return h.lanczos(case["niter"])
    if op == "step":
        return (state["vec"], state["rvec"]) + tuple(h.step_host(state["vec"], state["rvec"]))
    if op == "ritz":
        return h.ritz(case["niter"], state["rows"])
    return h.hf_gradient(state["psi"], 60)


def work(case):
    """Of one pass: the potential as the precision holds it (FP64 upper triangles; FP32
    spherical-harmonic coefficients where the basis has them, else FP32 triangles), each
    vector read and written once per iteration, and the contractions' operations."""
    if case["op"] == "batch":
        parts = [work(c) for c, _, _ in _problems(case, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n, nn, full = _sizes(case)
    dim, tri = n * nn, nn * (nn + 1) // 2
    per = {(5, "Odd"): 66, (4, "Even"): 45, (3, "Odd"): 28}.get((case["l_max"], case["sym"]), tri)
    blocks = n * (8 * tri if case["precision"] == "fp64" else 4 * per)
    flops = 2.0 * dim * (case["nx"] + case["ny"] + case["nz"]) + 2.0 * n * nn * nn + 2.0 * dim
    op = case["op"]
    if op == "hv":
        return {"bytes": blocks + 16.0 * dim, "flops": flops}
    if op == "hv_host":
        return {"bytes": blocks + 24.0 * dim, "flops": flops}
    if op == "lanczos":
        return {"bytes": case["niter"] * (blocks + 24.0 * dim), "flops": case["niter"] * (flops + 6.0 * dim)}
    if op == "step":
        return {"bytes": blocks + 32.0 * n * full, "flops": flops + 8.0 * n * full}
    if op == "ritz":
        lev = case["levels"]
        return {"bytes": case["niter"] * (blocks + 24.0 * dim) + 8.0 * lev * n * full,
                "flops": case["niter"] * (flops + (6.0 + 2.0 * lev) * dim)}
    nodes = 2 * case["theta"] * case["phi"]
    if op == "gradient":  # per node: density of every level; per node, site and H atom: distance and 4 sums a level
        lev = case["levels"]
        return {"bytes": 8.0 * lev * n * full + 8.0 * n * nodes,
                "flops": n * nodes * (2.0 * nn * lev + 60 * 2 * (10.0 + 8.0 * lev))}
    # prep: 60 sites and two H atoms per node (about 10 operations each), then the blocks by sums over phi and theta
    return {"bytes": n * (8.0 * tri + 4.0 * tri), "flops": n * nodes * 60 * 2 * 10.0 + n * nodes * 2.0 * (4 * case["l_max"] + 1)
            + n * tri * case["theta"] * 2.0 + flops}


# ---------------------------------------------------------------------------
# the same in plain FP64
# ---------------------------------------------------------------------------
def _kinetic(n):
    dx = BOX / (n - 1)
    d = torch.arange(n, device="cuda").reshape(-1, 1) - torch.arange(n, device="cuda").reshape(1, -1)
    d2 = (d * d).double()
    t = torch.where(d == 0, torch.full_like(d2, math.pi ** 2 / 3), 2.0 / d2.clamp(min=1.0))
    return t * (1.0 - 2.0 * (d.abs() % 2).double()) * (HBAR * HBAR / (2.0 * MASS * dx * dx))


def _functions(case):
    """(l, m) of the symmetry block and its indices in the full basis (m outer, l inner)."""
    lm = [(l, m) for m in range(-case["l_max"], case["l_max"] + 1) for l in range(abs(m), case["l_max"] + 1)]
    keep = [i for i, (l, _) in enumerate(lm) if case["sym"] == "All" or l % 2 == (case["sym"] == "Odd")]
    return [lm[i] for i in keep], keep


def _angles(case):
    """Node directions [C, 3] and the basis functions times sqrt(weight) there [nn, C]."""
    x, w = np.polynomial.legendre.leggauss(case["theta"])
    b = (2 * np.arange(1, case["phi"] + 1) - 1) * (math.pi / (2 * case["phi"]))
    phi = np.concatenate([b, 2 * math.pi - b])
    ct, ph = (a.reshape(-1) for a in np.meshgrid(x, phi, indexing="ij"))
    wt = np.repeat(w, len(phi)) * (math.pi / case["phi"])
    st = np.sqrt(1.0 - ct * ct)
    u = np.stack([st * np.cos(ph), st * np.sin(ph), ct], 1)
    L = case["l_max"]
    p = {(0, 0): np.ones_like(ct)}
    for m in range(L + 1):
        if m:
            p[m, m] = (2 * m - 1) * st * p[m - 1, m - 1]
        for l in range(m + 1, L + 1):
            p[l, m] = ((2 * l - 1) * ct * p[l - 1, m] - (l + m - 1) * p.get((l - 2, m), 0.0 * ct)) / (l - m)
    rows = []
    for l, m in _functions(case)[0]:
        k = abs(m)
        norm = (-1) ** k * math.sqrt((2 * l + 1) * math.factorial(l - k) / (2.0 * math.factorial(l + k)))
        trig = np.full_like(ph, 1 / math.sqrt(2)) if m == 0 else np.cos(m * ph) if m > 0 else np.sin(k * ph)
        rows.append(norm * p[l, k] * trig / math.sqrt(math.pi) * np.sqrt(wt))
    return torch.from_numpy(u).cuda(), torch.from_numpy(np.array(rows)).cuda()


def _sites(cage):
    xyz = []
    for cm, (a, b, c) in zip(*cage):
        ca, sa, cb, sb, cc, sc = math.cos(a), math.sin(a), math.cos(b), math.sin(b), math.cos(c), math.sin(c)
        rot = np.array([[ca * cb * cc - sa * sc, -ca * cb * sc - sa * cc, ca * sb],
                        [sa * cb * cc + ca * sc, -sa * cb * sc + ca * cc, sa * sb], [-sb * cc, sb * sc, cb]])
        xyz += [rot @ s + 0.1 * cm for s in BODY]
    return torch.from_numpy(np.array(xyz)).cuda(), torch.from_numpy(np.tile(Q_WATER, len(cage[0]))).cuda()


def _points(case):
    x, y, z = (torch.arange(case[k], dtype=torch.float64, device="cuda") * (BOX / (case[k] - 1)) - BOX / 2
               for k in ("nx", "ny", "nz"))
    zz, yy, xx = torch.meshgrid(z, y, x, indexing="ij")
    return torch.stack([xx.reshape(-1), yy.reshape(-1), zz.reshape(-1)], 1)


def _potential(pts, u, sites):
    """V [points, nodes] of the Alavi H2 among the sites, and the unclipped values."""
    xyz, q = sites
    r = (pts[:, None, :] - xyz[None]).norm(dim=2)
    v = (COULOMB * Q_CM * q / r).sum(1)
    o = r[:, ::3]
    v = (v + (LJ_A / o ** 12 - LJ_B / o ** 6).sum(1))[:, None].repeat(1, len(u))
    for sign in (1.0, -1.0):
        h = pts[:, None, :] + sign * H_OFFSET * u[None]
        for i in range(len(q)):
            d = h - xyz[i]
            v += COULOMB * Q_H * q[i] / (d * d).sum(2).sqrt()
    return v


class _Plain:
    """H of one problem in FP64: u = T v + B l(l+1) v + V v on [nn, points]."""

    def __init__(self, case, cage):
        self.case = case
        self.t = [_kinetic(case[k]) for k in ("nx", "ny", "nz")]
        self.n, self.nn, self.full = _sizes(case)
        lm, self.keep = _functions(case)
        self.rot = torch.tensor([ROT * l * (l + 1) for l, _ in lm], dtype=torch.float64, device="cuda")
        u, y = _angles(case)
        sites, pts = _sites(cage), _points(case)
        self.blocks = torch.empty(self.n, self.nn, self.nn, dtype=torch.float64, device="cuda")
        yy = (y[:, None] * y[None]).reshape(self.nn * self.nn, -1).T.contiguous()
        step = max(1, 24_000_000 // len(u))
        for i in range(0, self.n, step):
            v = _potential(pts[i:i + step], u, sites).clamp(max=CEILING)
            self.blocks[i:i + step] = (v @ yy).reshape(-1, self.nn, self.nn)

    def __call__(self, v):
        c = self.case
        w = v.reshape(self.nn, c["nz"], c["ny"], c["nx"])
        out = w @ self.t[0] + self.t[1] @ w
        out = out + (self.t[2] @ w.reshape(self.nn, c["nz"], -1)).reshape(out.shape)
        v = v.reshape(self.nn, self.n)
        out = out.reshape(self.nn, self.n) + self.rot[:, None] * v
        return (out + torch.bmm(self.blocks, v.T.contiguous()[:, :, None])[:, :, 0].T).reshape(-1)

    def lanczos(self, niter, vectors=None):
        """alpha, beta, beta^2 from the uniform start; the part outside the block is one more coordinate."""
        dim, size = self.n * self.nn, self.n * self.full
        v = torch.full((dim + 1,), 1 / math.sqrt(size), dtype=torch.float64, device="cuda")
        v[dim] = math.sqrt((size - dim) / size)
        r = torch.zeros_like(v)
        alpha, beta = torch.zeros(niter, dtype=torch.float64), torch.zeros(niter + 1, dtype=torch.float64)
        for j in range(niter):
            if vectors is not None:
                vectors(j, v)
            r[:dim] += self(v[:dim])
            a = v @ r
            r -= a * v
            b = r.norm()
            alpha[j], beta[j + 1] = a.item(), b.item()
            v, r = r / b, -b * v
        return alpha.numpy(), beta.numpy(), (beta * beta).numpy()

    def whole(self, packed):
        """The reference layout of a packed vector, zero outside the block."""
        out = torch.zeros(self.full, self.n, dtype=torch.float64, device="cuda")
        out[self.keep] = packed.reshape(self.nn, self.n)
        return out.reshape(-1)


def _rows(case, seed, plain=None):
    """The lowest eigenvectors of the T_m of the run, one per level."""
    a, b, _ = (plain or _Plain(case, _cage(seed))).lanczos(case["niter"])
    _, vec = np.linalg.eigh(np.diag(a) + np.diag(b[1:-1], 1) + np.diag(b[1:-1], -1))
    return np.ascontiguousarray(vec[:, :case["levels"]].T)


def _exact_gradient(case, cage, psi):
    n, nn, full = _sizes(case)
    xyz, q = _sites(cage)
    u, y = _angles(case)
    pts = _points(case)
    psi = torch.from_numpy(psi).cuda().reshape(len(psi), full, n)[:, _functions(case)[1]]
    psi = psi / psi.reshape(len(psi), -1).norm(dim=1)[:, None, None]
    dq = torch.zeros(len(psi), len(q), dtype=torch.float64, device="cuda")
    dr = torch.zeros(len(psi), len(q), 3, dtype=torch.float64, device="cuda")
    da = torch.zeros(len(psi), 2, dtype=torch.float64, device="cuda")
    oxygen = (torch.arange(len(q), device="cuda") % 3 == 0).double()
    step = max(1, 2_000_000 // len(u))
    for i in range(0, n, step):
        p = pts[i:i + step]
        inside = _potential(p, u, (xyz, q)) < CEILING
        om = torch.einsum("nsp,sc->npc", psi[:, :, i:i + step], y) ** 2 * inside
        d = p[:, None, :] - xyz[None]
        r = d.norm(dim=2)
        tot = om.sum(2)
        dq += COULOMB * Q_CM * (tot @ (1 / r))
        f = COULOMB * Q_CM * q / r ** 3 + oxygen * (12 * LJ_A / r ** 14 - 6 * LJ_B / r ** 8)
        dr += torch.einsum("np,pwk->nwk", tot, f[:, :, None] * d)
        da[:, 1] += COULOMB * (tot @ (1 / r)) @ q
        for sign in (1.0, -1.0):
            h = p[:, None, :] + sign * H_OFFSET * u[None]
            for w in range(len(q)):
                e = h - xyz[w]
                inv = 1 / (e * e).sum(2).sqrt()
                s = torch.einsum("npc,pc->n", om, inv)
                dq[:, w] += COULOMB * Q_H * s
                da[:, 0] += COULOMB * q[w] * s
                dr[:, w] += COULOMB * Q_H * q[w] * torch.einsum("npc,pck->nk", om, e * (inv ** 3)[:, :, None])
    return dq, dr, da


def exact(case, seed):
    op = case["op"]
    if op == "batch":
        return [_Plain(c, _cage(s, r)).lanczos(case["niter"]) for c, s, r in _problems(case, seed)]
    cage = _cage(seed)
    if op == "gradient":
        return _exact_gradient(case, cage, _psi(case, seed))
    h = _Plain(case, cage)
    dim, size = h.n * h.nn, h.n * h.full
    if op in ("hv", "prep"):
        return h(_normal(seed, dim))
    if op == "lanczos":
        return h.lanczos(case["niter"])
    if op == "ritz":
        rows = _rows(case, seed, h)  # the reference stops adding to a vector once its rows' squares reach 1
        rows = torch.from_numpy(np.where(np.cumsum(rows * rows, axis=1) < 1.0 - 1e-16, rows, 0.0)).cuda()
        out = torch.zeros(len(rows), dim + 1, dtype=torch.float64, device="cuda")

        def add(j, v):
            out.add_(rows[:, j:j + 1] * v[None])

        h.lanczos(case["niter"], add)
        masked = out[:, dim:] / math.sqrt(size - dim) if size > dim else out[:, dim:]
        whole = torch.zeros(len(rows), h.full, h.n, dtype=torch.float64, device="cuda") + masked[:, :, None]
        whole[:, h.keep] = out[:, :dim].reshape(len(rows), h.nn, h.n)
        return whole.reshape(len(rows), -1)
    v, r = (x.cuda() for x in _host_vectors(case, seed))
    r = r + h.whole(h(v.reshape(h.full, h.n)[h.keep].reshape(-1)))
    if op == "hv_host":
        return r
    a = v @ r
    r = r - a * v
    b = r.norm()
    return r / b, -b * v, a, b, b * b
