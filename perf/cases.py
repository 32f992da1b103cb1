"""Timing cases of the XC build: what an SCF program has pgxc do.

A case is one call of the public API on a seeded molecule (pgxc.cases builds the
geometry, the basis and the grid):

  "host"      Context.build: one SCF cycle with host C, occ and ham_xc_arr, the
              call that stands in for calc_xcks / calc_xcks_nl
  "device"    Context.build_device: the same with every operand on the GPU
  "gradient"  Context.xc_gradient: the post-SCF nuclear gradient
  "geometry"  a new geometry: a context on a grid built on the device, its
              Becke weights, and the first SCF cycle on it
  "set"       Batch.run: one SCF cycle of many small molecules at once

exact() restates the outputs in plain torch, FP64, without screening.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(ROOT, "paragauss-gpl_b200") not in sys.path:
    sys.path.insert(0, os.path.join(ROOT, "paragauss-gpl_b200"))

from pgxc import cases as M  # noqa: E402
from pgxc import lib as L  # noqa: E402

F8 = torch.float64


def _case(name, call, atoms, mix, xc, nrad, nang, precision="fp64", threshold=0.0, ispin=1, shells="spd", keep=False,
          molecules=1):
    c = dict(call=call, atoms=atoms, mix=mix, xc=xc, nrad=nrad, nang=nang, precision=precision, threshold=threshold,
             ispin=ispin, shells=shells, keep=keep, molecules=molecules)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # the smallest molecule through the drop-in call and its defaults: launches and latency
        _case("water-vwn-host", "host", 3, "water", "VWN", 50, 194),
        # the same size with the INT8 contractions and C resident on the GPU
        _case("water-pbe-int8", "device", 3, "water", "PBE", 50, 194, "mixed", 1e-10),
        # a small organic molecule, drop-in defaults, a grid size that leaves a ragged last tile
        _case("mol12-pbe-host", "host", 12, "CHO", "PBE", 53, 194),
        # an open shell of ordinary size with every operand on the GPU
        _case("mol25-pbe-open", "device", 25, "CHON", "PBE", 50, 194, "fp64", 1e-10, 2),
        # an LDA with the basis values kept across SCF cycles, INT8
        _case("mol31-vwn-int8-keep", "device", 31, "CHO", "VWN", 60, 302, "mixed", 1e-10, keep=True),
        # a meta-GGA: tau in the density and in the potential
        _case("mol20-tpss-host", "host", 20, "CHO", "TPSS", 50, 194, "fp64", 1e-10),
        # the 60-atom C/H cluster of the benchmark: INT8 on the GPU, and the drop-in call with its defaults
        _case("ch60-pbe-int8", "device", 60, "CH", "PBE", 75, 302, "mixed", 1e-10),
        _case("ch60-pbe-host", "host", 60, "CH", "PBE", 75, 302),
        # the largest: 200 atoms with f shells, one GPU's share of the 500-atom workload
        _case("chon200-pbe-int8", "device", 200, "CHON", "PBE", 75, 302, "mixed", 1e-10, shells="f"),
        # one SCF cycle of a set of small molecules of 3 to 40 atoms, VWN and PBE alternating
        _case("set32-int8", "set", 40, "CHO", "VWN+PBE", 75, 302, "mixed", 1e-10, molecules=32),
        # once per geometry, after the SCF
        _case("grad40-pbe", "gradient", 40, "CHO", "PBE", 50, 194, "fp64", 1e-10),
        # once per geometry, before the SCF
        _case("geom41-pbe", "geometry", 41, "CHO", "PBE", 50, 194),
    ]


def draw(rng):
    call = rng.choice(["host", "host", "device", "device", "device", "gradient", "geometry", "set"])
    nrad, nang = rng.randint(30, 75), rng.choice([50, 110, 146, 194, 302])
    mix = rng.choice(["CH", "CHO", "CHON"])

    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if call == "set":
        return _case(None, call, rng.randint(10, 40), "CHO", "VWN+PBE", 75, 302, "mixed", 1e-10,
                     molecules=rng.randint(4, 32))
    if call == "gradient":
        return _case(None, call, size(3, 40), mix, rng.choice(["VWN", "PBE", "revPBE"]), nrad,
                     rng.choice([50, 110, 146, 194]), "fp64", rng.choice([0.0, 1e-10]), rng.choice([1, 1, 2]))
    if call == "geometry":
        return _case(None, call, size(3, 60), mix, rng.choice(["VWN", "PBE"]), nrad, nang,
                     *rng.choice([("fp64", 0.0), ("mixed", 1e-10)]))
    precision, threshold = rng.choice([("fp64", 0.0), ("fp64", 1e-10), ("mixed", 1e-10), ("mixed", 0.0)])
    xc = rng.choice(["VWN", "PWLDA", "PBE", "PBE", "revPBE", "PBEsol"] + (["TPSS"] if precision == "fp64" else []))
    shells = rng.choice(["spd", "spd", "f"])
    atoms = size(3, 100 if precision == "mixed" and threshold > 0.0 else 60)
    return _case(None, call, atoms, mix, xc, nrad, nang, precision, threshold, rng.choice([1, 1, 2]), shells,
                 keep=rng.random() < 0.2)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _molecule(case, seed):
    """The pgxc.cases.Case of a case: geometry, basis, grid and orbitals."""
    n = case["atoms"]
    rng = np.random.default_rng(seed)
    if case["mix"] == "water":
        els, xyz = M.water()
    else:
        share = {"CH": (.5, .5), "CHO": (.4, .4, .2), "CHON": (.3, .45, .15, .1)}[case["mix"]]
        k = [int(round(s * n)) for s in share]
        k[1] += n - sum(k)
        els, xyz = M.random_cluster(rng, list(zip(case["mix"], k)), max(2.5, (n / 0.035) ** (1 / 3)), 1.0)
    c = M.build_case("case", els, xyz, seed=seed, exp_range=(0.05, 1e4), nrad=case["nrad"], nang=case["nang"],
                     functional=case["xc"], nocc=max(1, sum(M.Z_OF[e] for e in els) // 2),
                     shells=M.SHELLS_F if case["shells"] == "f" else None, ispin=1, orthonormalise=False)
    # orbitals: noise, orthonormalised in the overlap of a coarse quadrature where that is quick to make
    g = torch.Generator(device="cuda").manual_seed(seed)
    nocc = c.nocc = min(c.nocc, c.nbas)
    S = _coarse_overlap(c) if n <= 100 else torch.eye(c.nbas, dtype=F8, device="cuda") * c.nbas / nocc
    C = []
    for _ in range(case["ispin"]):
        X = torch.randn(c.nbas, nocc, dtype=F8, device="cuda", generator=g)
        C.append(torch.linalg.solve_triangular(torch.linalg.cholesky(X.T @ S @ X), X.T, upper=False).T)
    c.C = torch.stack(C, 2).cpu().numpy()
    c.ispin = case["ispin"]
    if c.ispin == 1:
        c.occ = np.full((nocc, 1), 2.0)
    else:
        beta = np.ones(nocc)
        beta[nocc - max(1, nocc // 8):] = 0.0
        c.occ = np.stack([np.ones(nocc), beta], axis=1)
    return c


def _molecules(case, seed):
    """A set: molecules of 3 to case["atoms"] atoms, sizes and grids spread evenly, VWN and PBE alternating."""
    k = case["molecules"]
    return [_molecule(dict(case, atoms=3 + (case["atoms"] - 3) * i // max(1, k - 1), xc=("VWN", "PBE")[i % 2],
                           nrad=50 + 7 * i % 26, nang=(194, 302)[i // 2 % 2]), seed + 1000 * i) for i in range(k)]


class _Batch(L.Batch):
    def __del__(self):
        self.close()


def _context(c, case, **kw):
    return L.Context(c, precision=case["precision"], weighted=False, screen_threshold=case["threshold"],
                     keep_orbitals=case["keep"], **kw)


def _device(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def prepare(case, seed):
    s = {"case": case}
    if case["call"] == "set":
        mols = _molecules(case, seed)
        # the contexts' own chunk buffers stay small: the set has its own
        s["ctx"] = [L.Context(m, precision=case["precision"], weighted=False, screen_threshold=case["threshold"],
                              max_chunk_points=4096) for m in mols]
        s["C"] = [_device(m.c_fortran()) for m in mols]
        s["occ"] = [_device(m.occ_fortran()) for m in mols]
        off = np.concatenate([[0], np.cumsum([m.xc_length for m in mols])])
        s["ham"] = torch.zeros(int(off[-1]), dtype=F8, device="cuda")
        s["sums"] = torch.zeros(len(mols), 2, dtype=F8, device="cuda")
        s["batch"] = _Batch(s["ctx"], [t.data_ptr() for t in s["C"]], [t.data_ptr() for t in s["occ"]],
                              [s["ham"].data_ptr() + 8 * int(o) for o in off[:-1]],
                              [s["sums"].data_ptr() + 16 * i for i in range(len(mols))])
        return s
    c = s["mol"] = _molecule(case, seed)
    s["C"], s["occ"] = c.c_fortran(), c.occ_fortran()
    if case["call"] != "geometry":
        s["ctx"] = _context(c, case)
    if case["call"] == "device":
        s["C"], s["occ"] = _device(s["C"]), _device(s["occ"])
        s["ham"] = torch.zeros(c.xc_length, dtype=F8, device="cuda")
        s["sums"] = torch.zeros(2, dtype=F8, device="cuda")
    return s


def run(s):
    call = s["case"]["call"]
    if call == "set":
        s["batch"].run()
        return {"ham": s["ham"], "sums": s["sums"]}
    if call == "device":
        s["ctx"].build_device(s["C"].data_ptr(), s["occ"].data_ptr(), s["ham"].data_ptr(), s["sums"].data_ptr())
        return {"ham": s["ham"], "sums": s["sums"]}
    if call == "host":
        ham, exc, nel = s["ctx"].build(s["C"], s["occ"])
        return {"ham": ham, "sums": np.array([exc, nel])}
    if call == "gradient":
        grad, exc = s["ctx"].xc_gradient(s["C"], s["occ"])
        return {"grad": grad, "exc": exc}
    with _context(s["mol"], s["case"], on_grid=True) as ctx:
        w = ctx.grid_weights()
        ham, exc, nel = ctx.build(s["C"], s["occ"])
    return {"ham": ham, "sums": np.array([exc, nel]), "weights": w}


# ---------------------------------------------------------------------------
# work: inputs read once, outputs written once, and the operations of the basis
# values and the two contractions over the functions that reach a point
# ---------------------------------------------------------------------------
def work(case):
    sets = case["call"] == "set"
    atoms = (3 + case["atoms"]) / 2 if sets else case["atoms"]
    nrad, nang = (62.5, 248) if sets else (case["nrad"], case["nang"])
    per = {"water": 28 / 3, "CH": 11.5, "CHO": 13.0, "CHON": 12.5}[case["mix"]]  # functions per atom
    nbas, npts = per * atoms, 0.86 * nrad * nang * atoms
    # functions reaching a 128-point neighbourhood: all of a small molecule's, a constant number of a large one's
    near = nbas / (1 + nbas / (510 if case["threshold"] == 0.0 or case["call"] == "gradient" else 241))
    xc, ispin = case["xc"], case["ispin"]
    sweeps = 4 if xc == "TPSS" else 1
    flops = npts * (60 * near + 2 * 2 * near * near * ispin * sweeps)
    nbytes = 8 * (ispin * nbas * (2 * atoms + nbas / 2) + 4 * npts)
    if case["call"] in ("gradient", "geometry"):
        flops += npts * 30 * 6.2 * atoms  # partition weights: the cell functions that matter at a point
    return {"bytes": nbytes * case["molecules"], "flops": flops * case["molecules"]}


# ---------------------------------------------------------------------------
# the same outputs in plain torch
# ---------------------------------------------------------------------------
def _basis_table(c):
    """Per l: atom of each primitive, exponents, norms, contraction matrix
    (primitive, radial function), atom and first function of each radial
    function and the stride between its independent functions."""
    out = {}
    eo = co = f = 0
    for s in range(len(c.shell_l)):
        l, a, ne, nc = (int(v[s]) for v in (c.shell_l, c.shell_atom, c.shell_nexp, c.shell_ncontr))
        t = out.setdefault(l, dict(pa=[], e=[], n=[], blocks=[], ra=[], f=[], st=[]))
        t["pa"] += [a] * ne
        t["e"].append(c.exponents[eo:eo + ne])
        t["n"].append(c.norms[eo:eo + ne])
        t["blocks"].append(torch.from_numpy(c.contractions[co:co + ne * nc].reshape(nc, ne).T.copy()))
        t["ra"] += [a] * nc
        t["f"] += range(f, f + nc)
        t["st"] += [nc] * nc
        eo, co, f = eo + ne, co + ne * nc, f + (2 * l + 1) * nc
    dev = dict(device="cuda")
    return {l: dict(pa=torch.tensor(t["pa"], **dev), e=torch.from_numpy(np.concatenate(t["e"])).cuda(),
                    n=torch.from_numpy(np.concatenate(t["n"])).cuda(),
                    c=torch.block_diag(*t["blocks"]).cuda(), ra=torch.tensor(t["ra"], **dev),
                    f=torch.tensor(t["f"], **dev), st=torch.tensor(t["st"], **dev)) for l, t in out.items()}


def _harmonics(l, x, y, z):
    """Racah-normalised real solid harmonics and their gradients, in the order
    0, then the cosine and sine forms of each m."""
    o, i = torch.zeros_like(x), torch.ones_like(x)
    if l == 0:
        return [(i, o, o, o)]
    if l == 1:
        return [(z, o, o, i), (x, i, o, o), (y, o, i, o)]
    if l == 2:
        k = math.sqrt(3.0)
        return [(z * z - (x * x + y * y) / 2, -x, -y, 2 * z), (k * x * z, k * z, o, k * x), (k * y * z, o, k * z, k * y),
                (k / 2 * (x * x - y * y), k * x, -k * y, o), (k * x * y, k * y, k * x, o)]
    a, b, d = math.sqrt(3 / 8), math.sqrt(15.0), math.sqrt(5 / 8)
    q = x * x + y * y
    return [(z * z * z - 1.5 * z * q, -3 * x * z, -3 * y * z, 3 * z * z - 1.5 * q),
            (a * x * (4 * z * z - q), a * (4 * z * z - 3 * x * x - y * y), -2 * a * x * y, 8 * a * x * z),
            (a * y * (4 * z * z - q), -2 * a * x * y, a * (4 * z * z - x * x - 3 * y * y), 8 * a * y * z),
            (b / 2 * z * (x * x - y * y), b * x * z, -b * y * z, b / 2 * (x * x - y * y)),
            (b * x * y * z, b * y * z, b * x * z, b * x * y),
            (d * x * (x * x - 3 * y * y), 3 * d * (x * x - y * y), -6 * d * x * y, o),
            (d * y * (3 * x * x - y * y), 6 * d * x * y, 3 * d * (x * x - y * y), o)]


def _basis(table, nbas, coords, p, grad):
    """(1 or 4, points, nbas): functions and their gradients."""
    rel = p[:, None, :] - coords[None, :, :]
    r2 = (rel * rel).sum(-1)
    cols, idx = [], []
    for l, t in table.items():
        ar2 = t["e"] * r2[:, t["pa"]]
        v = torch.where(ar2 < 50.0, t["n"] * torch.exp(-ar2), torch.zeros_like(ar2))
        R = v @ t["c"]
        dR = (v * (-2 * t["e"])) @ t["c"] if grad else None
        d = rel[:, t["ra"], :]
        x, y, z = d[..., 0], d[..., 1], d[..., 2]
        for i, (Y, gx, gy, gz) in enumerate(_harmonics(l, x, y, z)):
            cols.append([Y * R] + ([gx * R + Y * x * dR, gy * R + Y * y * dR, gz * R + Y * z * dR] if grad else []))
            idx.append(t["f"] + i * t["st"])
    order = torch.argsort(torch.cat(idx))
    return [torch.cat([c[k] for c in cols], 1)[:, order] for k in range(4 if grad else 1)]


def _becke(coords, p, owner):
    r = (p[:, None, :] - coords[None, :, :]).pow(2).sum(-1).sqrt()
    n = len(coords)
    eye = torch.eye(n, dtype=F8, device=p.device)
    R = ((coords[:, None] - coords[None, :]).pow(2).sum(-1) + eye).sqrt()
    P = []
    for a in range(n):
        mu = (r[:, a:a + 1] - r) / R[a]
        for _ in range(3):
            mu = mu * (3 - mu * mu) / 2
        s = (1 - mu) / 2
        P.append(torch.where(eye[a] > 0, torch.ones_like(s), s).prod(1))
    P = torch.stack(P, 1)
    return P.gather(1, owner[:, None])[:, 0] / P.sum(1)


def _pw92(n, z):
    def g(a, a1, b1, b2, b3, b4):
        q = rs.sqrt()
        return -2 * a * (1 + a1 * rs) * torch.log(1 + 1 / (2 * a * (b1 * q + b2 * rs + b3 * rs * q + b4 * rs * rs)))

    rs = (3 / (4 * math.pi)) ** (1 / 3) / n.pow(1 / 3)
    e0 = g(.031091, .21370, 7.5957, 3.5876, 1.6382, .49294)
    e1 = g(.015545, .20548, 14.1189, 6.1977, 3.3662, .62517)
    al = g(.016887, .11125, 10.357, 3.6231, .88026, .49671)
    cf = 1 / (2 ** (4 / 3) - 2)
    f = cf * ((1 + z).pow(4 / 3) + (1 - z).pow(4 / 3) - 2)
    return n * (e0 + (e1 - e0) * f * z ** 4 - al * f * (1 - z ** 4) / (8 / 9 * cf))


def _vwn5(n, z):
    def ec(a, b, c, x0):
        Q, X0, X = math.sqrt(4 * c - b * b), (x0 + b) * x0 + c, (x + b) * x + c
        F = torch.atan(Q / (2 * x + b))
        return a / 2 * (torch.log(x * x / X) + 2 * b / Q * F
                        - b * x0 / X0 * (torch.log((x - x0) ** 2 / X) + 2 * (b + 2 * x0) / Q * F))

    x = (3 / (4 * math.pi) / n).pow(1 / 6)
    p, f, a = (ec(.0621841, 3.72744, 12.9352, -.10498), ec(.0310907, 7.06042, 18.0578, -.32500),
               ec(-.0337740, 1.13107, 13.0045, -.0047584))
    ff = 0.5 / (2 ** (1 / 3) - 1)
    dd = 8 / 9 * ff
    fz = ff * ((1 + z).pow(4 / 3) + (1 - z).pow(4 / 3) - 2)
    return n * (p + a * fz / dd * (1 + (dd / a * (f - p) - 1) * z ** 4))


def _functional(xc, ra, rb, gaa, gbb, gab):
    """Energy per volume of the spin densities (LDA and PBE-form keywords)."""
    n, g = ra + rb, gaa + gbb + 2 * gab
    z = (ra - rb) / n

    def slater(r):
        return -0.75 * (3 / math.pi) ** (1 / 3) * r.pow(4 / 3)

    f = (slater(2 * ra) + slater(2 * rb)) / 2
    f = f + (_vwn5(n, z) if xc == "VWN" else _pw92(n, z))
    if xc in ("VWN", "PWLDA"):
        return f
    kappa = 1.245 if xc == "revPBE" else 0.804
    mu = 10 / 81 if xc == "PBEsol" else 0.066725 * math.pi ** 2 / 3
    beta, gam = (0.046 if xc == "PBEsol" else 0.066725), 0.03109069086965489503494086371

    def enhanced(r, gs):
        s2 = gs / (4 * (3 * math.pi ** 2) ** (2 / 3) * r.pow(8 / 3))
        return slater(r) * kappa * mu * s2 / (kappa + mu * s2)

    f = f + (enhanced(2 * ra, 4 * gaa) + enhanced(2 * rb, 4 * gbb)) / 2
    phi = (((1 + z) / 2).pow(2 / 3) + ((1 - z) / 2).pow(2 / 3)) / 2 ** (1 / 3)
    gp = gam * phi ** 3
    A = beta / gam / (torch.exp(-_pw92(n, z) / n / gp) - 1 + 1e-30)
    t2 = g / (phi ** 2 * n.pow(7 / 3) + 1e-30) * math.pi / (16 * (3 * math.pi ** 2) ** (1 / 3))
    return f + n * gp * torch.log(1 + beta / gam * t2 * (1 + A * t2) / (1 + A * t2 + (A * t2) ** 2))


def _density(B, P, gga):
    """rho and grad rho of a density matrix on the points of the basis values B."""
    X = B[0] @ P
    return (X * B[0]).sum(1), [2 * (X * B[1 + k]).sum(1) for k in range(3)] if gga else None


def _point_energy(xc, rho, gr):
    """f on points from per-spin rho and grad rho; 0 where the density vanishes."""
    if len(rho) == 1:
        rho, gr = [rho[0] / 2] * 2, None if gr is None else [[v / 2 for v in gr[0]]] * 2
    live = (rho[0] > 1e-25) & (rho[1] > 1e-25)
    r = [torch.where(live, v, torch.ones_like(v)) for v in rho]
    dot = [torch.zeros_like(r[0])] * 3
    if gr is not None:
        dot = [torch.where(live, sum(a * b for a, b in zip(gr[i], gr[j])), torch.zeros_like(r[0]))
               for i, j in ((0, 0), (1, 1), (0, 1))]
    return torch.where(live, _functional(xc, *r, *dot), torch.zeros_like(r[0]))


def _density_matrices(c):
    C, occ = torch.from_numpy(c.C).cuda(), torch.from_numpy(c.occ).cuda()
    return [(C[:, :, s] * occ[:, s]) @ C[:, :, s].T for s in range(c.ispin)]


def _exact_build(c, weights=False):
    gga, table, P = c.functional not in ("VWN", "PWLDA"), _basis_table(c), _density_matrices(c)
    xc = None if c.functional == "TPSS" else c.functional
    coords = _device(c.coords)
    V = [torch.zeros(c.nbas, c.nbas, dtype=F8, device="cuda") for _ in P]
    E = N = 0.0
    ws = []
    step = max(1024, min(1 << 16, int(1.2e8) // c.nbas))
    for lo in range(0, c.npts, step):
        p, own = _device(c.grid_xyz[lo:lo + step]), _device(c.point_atom[lo:lo + step]).long()
        ws.append(torch.cat([_becke(coords, p[i:i + 8192], own[i:i + 8192]) for i in range(0, len(p), 8192)])
                  * _device(c.grid_wraw[lo:lo + step]))
        w, B = ws[-1], _basis(table, c.nbas, coords, p, gga)
        rho, gr = zip(*[_density(B, Ps, gga) for Ps in P])
        N += float((w * sum(rho)).sum())
        if xc is None:
            continue
        var = [v.clamp_min(0.0).requires_grad_() for v in rho]
        gv = [[v.requires_grad_() for v in g] for g in gr] if gga else None
        with torch.enable_grad():
            f = (w * _point_energy(xc, var, gv)).sum()
            d = torch.autograd.grad(f, var + ([v for g in gv for v in g] if gga else []), allow_unused=True)
        E += float(f.detach())
        for s in range(c.ispin):
            Z = B[0] * (d[s][:, None] / 2)
            if gga:
                for k in range(3):
                    Z = Z + B[1 + k] * d[c.ispin + 3 * s + k][:, None]
            H = Z.T @ B[0]
            V[s] += H + H.T
    out = {"sums": [None, N] if xc is None else np.array([E, N]), "ham": None}
    if xc is not None:
        j, k = torch.tril_indices(c.nbas, c.nbas, device="cuda")
        out["ham"] = torch.stack([v[k, j] for v in V], 1).reshape(-1)
    if weights:
        out["weights"] = torch.cat(ws)
    return out


def _exact_gradient(c):
    gga, table, P = c.functional not in ("VWN", "PWLDA"), _basis_table(c), _density_matrices(c)
    coords = _device(c.coords).requires_grad_()
    off = _device(c.grid_xyz) - coords.detach()[_device(c.point_atom).long()]
    E = 0.0
    step = max(512, min(8192, int(4e6) // c.nbas))
    for lo in range(0, c.npts, step):
        own = _device(c.point_atom[lo:lo + step]).long()
        p = coords[own] + off[lo:lo + step]
        B = _basis(table, c.nbas, coords, p, gga)
        rho, gr = zip(*[_density(B, Ps, gga) for Ps in P])
        e = (_device(c.grid_wraw[lo:lo + step]) * _becke(coords, p, own)
             * _point_energy(c.functional, [v.clamp_min(0.0) for v in rho], gr if gga else None)).sum()
        e.backward()
        E += float(e.detach())
    return {"grad": coords.grad, "exc": E}


def _coarse_overlap(c):
    """The overlap matrix on a 20 x 50 quadrature of the molecule's atoms."""
    xyz, w, owner = M.G.atomic_grids(c.coords, c.Z, 20, 50)
    coords, table = _device(c.coords), _basis_table(c)
    S = torch.zeros(c.nbas, c.nbas, dtype=F8, device="cuda")
    for lo in range(0, len(w), 16384):
        p = _device(xyz[lo:lo + 16384])
        b = _basis(table, c.nbas, coords, p, False)[0]
        v = _becke(coords, p, _device(owner[lo:lo + 16384]).long()) * _device(w[lo:lo + 16384])
        S += b.T @ (b * v[:, None])
    return S


def exact(case, seed):
    if case["call"] == "set":
        out = [_exact_build(m) for m in _molecules(case, seed)]
        return {"ham": torch.cat([o["ham"] for o in out]), "sums": np.stack([o["sums"] for o in out])}
    c = _molecule(case, seed)
    if case["call"] == "gradient":
        return _exact_gradient(c)
    return _exact_build(c, case["call"] == "geometry")
