"""The calls that a user of the grid XC quadrature makes, at the sizes it is used at.

Every case goes through the public front end (`proteindf_b200.xc.XcEngine`, the C ABI of
include/pdfxc.h). A case names a molecule (seeded water cluster or peptide-like chain, cc-pVDZ), a grid
preset, a functional and a path; geometry and density come from the seed. `exact` restates the
quadrature in plain torch FP64 without AO screening.

Fields of a case
  kind       build (closed shell), uks (open shell), batch (several molecules in one build),
             backward (the adjoint with the Becke-weight derivative), weights (Becke partition)
  molecule   water | chain;  size: molecules of the cluster / atoms of the chain
  grid       SG1 | USER-75x302 | FINE | ULTRA_FINE;  partition: Becke | SSWeight
  host       density and Fock matrix on the host (the drop-in's call) or on the device
"""
import math

import numpy as np
import torch

from proteindf_b200 import basis, grids, systems
from proteindf_b200.xc import GGA, XcEngine

DEV = "cuda"
PRESETS = dict(grids.PRESETS, SG1=dict(nrad=50, nang=194, radial="EM", mapping="TA", pruning="SG1"))


def _case(name, kind, molecule, size, functional, precision, grid="USER-75x302", host=True, ao_cutoff=1e-14,
          partition="Becke", count=1):
    c = dict(kind=kind, molecule=molecule, size=size, functional=functional, precision=precision, grid=grid, host=host,
             ao_cutoff=ao_cutoff, partition=partition, count=count)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one water molecule on the small grid of the reference: the shortest call, latency and launches
        _case("water1-svwn", "build", "water", 1, "SVWN", "fp64", grid="SG1"),
        # the water cluster of the LDA configuration, the drop-in's host call
        _case("water8-svwn", "build", "water", 8, "SVWN", "fp64"),
        # a small molecule on the INT8 path with a device-resident density (a Fock build kept on the GPU)
        _case("chain30-pbe-int8", "build", "chain", 30, "PBE", "mixed", host=False),
        # the headline configuration, FP64 and INT8: one SCF iteration of a 100-atom chain
        _case("chain100-b3lyp", "build", "chain", 100, "B3LYP", "fp64", grid="ULTRA_FINE", host=False),
        _case("chain100-b3lyp-int8", "build", "chain", 100, "B3LYP", "mixed", grid="ULTRA_FINE", host=False),
        # a protein-sized chain with the large systems' settings (Stratmann-Scuseria weights, AO cut-off 1e-10)
        _case("chain500-b3lyp", "build", "chain", 500, "B3LYP", "fp64", host=False, ao_cutoff=1e-10,
              partition="SSWeight"),
        _case("chain500-b3lyp-int8", "build", "chain", 500, "B3LYP", "mixed", host=False, ao_cutoff=1e-10,
              partition="SSWeight"),
        # open shell (radicals, spin-polarised SCF), both paths, the drop-in's host call
        _case("chain43-blyp-uks", "uks", "chain", 43, "BLYP", "fp64"),
        _case("chain77-b3lyp-uks-int8", "uks", "chain", 77, "B3LYP", "mixed"),
        # the differentiation configuration: dExc/dP and the nuclear gradient of a 30-atom PBE chain
        _case("chain30-pbe-backward", "backward", "chain", 30, "PBE", "fp64"),
        # many molecules in one build
        _case("batch12-b3lyp-int8", "batch", "chain", 60, "B3LYP", "mixed", count=12),
        # the grid producer's Becke partition, once per geometry
        _case("becke100", "weights", "chain", 100, "-", "fp64"),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["build"] * 5 + ["uks", "uks", "batch", "backward", "weights"])
    fn = rng.choice(["SVWN", "HFB", "BLYP", "B3LYP", "B3LYP", "PBE"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "build":
        if rng.random() < 0.25:
            return _case("", kind, "water", rng.randint(1, 8), fn, prec, host=rng.random() < 0.5,
                         grid=rng.choice(["SG1", "USER-75x302", "FINE", "ULTRA_FINE"]))
        n = _spread(rng, 10, 450)
        grid = rng.choice(["SG1", "USER-75x302", "FINE"] + (["ULTRA_FINE"] if n <= 100 else []))
        large = n > 150
        return _case("", kind, "chain", n, fn, prec, grid=grid, host=n <= 250 and rng.random() < 0.5,
                     ao_cutoff=1e-10 if large else 1e-14, partition="SSWeight" if large else "Becke")
    if kind == "uks":
        return _case("", kind, "chain", _spread(rng, 10, 110), fn, prec, grid=rng.choice(["SG1", "USER-75x302"]))
    if kind == "batch":
        return _case("", kind, "chain", rng.randint(20, 70), fn, prec, count=rng.randint(2, 12))
    if kind == "backward":
        return _case("", kind, "chain", _spread(rng, 10, 60), fn, "fp64", grid=rng.choice(["SG1", "USER-75x302"]))
    return _case("", kind, "chain", _spread(rng, 10, 110), "-", "fp64")


# ---------------------------------------------------------------------------------------- inputs


def _geometry(molecule, size, seed):
    if molecule == "water":
        return systems.water_cluster(size, seed=seed)
    for k in range(20):  # a seed whose walk runs into itself gives way to the next
        try:
            return systems.peptide_chain(size, seed=seed + 7919 * k)
        except RuntimeError:
            continue
    raise RuntimeError("no chain")


def _molecules(case, seed):
    """The shell tables of the case's molecules (one, or the batch's, of sizes between 10 and `size`)."""
    sizes = [case["size"]]
    if case["count"] > 1:
        sizes = np.random.default_rng(case["count"]).integers(10, case["size"] + 1, case["count"]).tolist()
    out = []
    for k, n in enumerate(sizes):
        syms, xyz = _geometry(case["molecule"], n, seed + 101 * k)
        out.append(basis.ShellTable(syms, xyz, basis.load_basis("cc-pVDZ")))
    return out


def _density(sh, seed, share=0.4):
    """P_A = C C^T with `share` of the orbitals occupied, from a seeded normal draw (numpy, host)."""
    nocc = max(1, int(share * sh.nao))
    a = torch.from_numpy(np.random.default_rng(seed).standard_normal((sh.nao, nocc))).to(DEV)
    q, _ = torch.linalg.qr(a)
    return q @ q.T


def _radii(sh, case):
    tab = grids.SG1_RADIUS if case["grid"] == "SG1" else grids.BRAGG_SLATER
    return [tab[int(z)] for z in sh.atom_z], np.array([grids.BECKE_RADIUS[int(z)] for z in sh.atom_z])


def _engine(case, sh):
    eng = XcEngine(precision=case["precision"], ao_cutoff=case["ao_cutoff"])
    eng.set_system(sh)
    return eng


def _generate(eng, sh, case):
    ar, br = _radii(sh, case)
    eng.generate_grid(ar, partition=case["partition"], becke_radius=br, **PRESETS[case["grid"]])


def _moving_grid(sh, case):
    """Single-centre points, weights and owners of a grid that moves with its atoms."""
    if case["grid"] != "SG1":
        return grids.molecular_grid(sh.atom_xyz, sh.atom_z, **PRESETS[case["grid"]])
    p, w, a = [], [], []
    leb = grids.lebedev_table()
    for k, z in enumerate(sh.atom_z):
        R = grids.SG1_RADIUS[int(z)]
        reg = (0.25, 0.5, 1.0, 4.5) if z <= 2 else (0.1667, 0.5, 0.9, 3.5)
        for i in range(1, 51):
            r, wr = grids.radial_em(R, 50, i)
            if r > 30.0:
                continue
            q = r / R
            t = leb[6 if q < reg[0] else 38 if q < reg[1] else 86 if q < reg[2] else 194 if q < reg[3] else 86]
            p.append(t[:, :3] * r + sh.atom_xyz[k])
            w.append(t[:, 3] * wr)
            a.append(np.full(len(t), k, dtype=np.int32))
    return np.concatenate(p), np.concatenate(w), np.concatenate(a)


def prepare(case, seed):
    mols = _molecules(case, seed)
    sh = mols[0]
    s = dict(case=case, mols=mols)
    kind = case["kind"]
    if kind == "batch":
        parts = []
        for m in mols:
            e = _engine(dict(case, precision="fp64"), m)
            _generate(e, m, case)
            xyzw, atom = e.get_grid()
            e.close()
            parts.append((m, xyzw, atom))
        s["grids"] = [xyzw for _, xyzw, _ in parts]
        s["P"] = [_density(m, seed + 31 * k).cpu().numpy() for k, m in enumerate(mols)]
        s["eng"] = XcEngine(precision=case["precision"], ao_cutoff=case["ao_cutoff"])
        s["eng"].set_batch(parts)
        return s
    eng = s["eng"] = _engine(case, sh)
    if kind == "weights":
        s["points"], s["w"], s["owner"] = _moving_grid(sh, case)
        s["br"] = _radii(sh, case)[1]
        return s
    if kind == "backward":
        p, w, a = _moving_grid(sh, case)
        br = _radii(sh, case)[1]
        wt = eng.becke_weights(p, a, w, br)
        keep = np.abs(wt) > 1e-16
        s["xyzw"], s["w"], s["owner"], s["br"] = np.c_[p[keep], wt[keep]], w[keep], a[keep], br
        eng.set_grid(s["xyzw"], s["owner"])
        s["P"] = _density(sh, seed).cpu().numpy()
        return s
    _generate(eng, sh, case)
    P = _density(sh, seed)
    if kind == "uks":
        s["P"] = P.cpu().numpy()
        s["PB"] = _density(sh, seed + 1, share=0.37).cpu().numpy()
    elif case["host"]:
        s["P"] = P.cpu().numpy()
    else:
        s["P"], s["V"] = P, torch.empty_like(P)
        torch.cuda.synchronize()  # the engine works on a stream of its own
    return s


def run(s):
    c, eng = s["case"], s["eng"]
    fn, kind = c["functional"], c["kind"]
    if kind == "weights":
        return eng.becke_weights(s["points"], s["owner"], s["w"], s["br"])
    if kind == "backward":
        dP, go, gw, exc = eng.xc_backward(fn, s["P"], w_single=s["w"], becke_radius=s["br"])
        return {"dP": dP, "orbital": go, "weight": gw, "exc": np.array([exc])}
    if kind == "uks":
        exc, na, nb, FA, FB = eng.build_vxc_uks(fn, s["P"], s["PB"])
        return {"sums": np.array([exc, na, nb]), "FA": FA, "FB": FB}
    if kind == "batch":
        exc, nel, F = eng.build_vxc_batched(fn, s["P"])
        return {"exc": exc, "nel": nel, "F": F}
    if c["host"]:
        exc, nel, F = eng.build_vxc(fn, s["P"])
        return {"sums": np.array([exc, nel]), "F": F}
    exc, nel = eng.build_vxc_device(fn, s["P"].data_ptr(), s["V"].data_ptr())
    return {"sums": np.array([exc, nel]), "F": s["V"]}


# ---------------------------------------------------------------------------------------- work


def _cut_radius(L, e, c, cutoff):
    r = np.arange(0.01, 60.0, 0.01)
    g = np.maximum(r[:, None] ** L, (L * r[:, None] ** max(L - 1, 0) if L else 0.0) + 2.0 * e * r[:, None] ** (L + 1))
    hit = np.nonzero((np.abs(c) * np.exp(-e * r[:, None] ** 2) * g).sum(1) >= cutoff)[0]
    return r[hit[-1]] if len(hit) else 0.0


def _reach(sh, pts, cutoff):
    """Mean of the squared and of the plain number of AOs that reach the cut-off at a point."""
    n = np.zeros(len(pts))
    memo = {}
    for k in range(sh.nshell):
        p0, m, L = sh.shell_p0[k], sh.shell_nprim[k], int(sh.shell_l[k])
        e, c = sh.prim_exp[p0:p0 + m], sh.prim_coef[p0:p0 + m]
        key = (L, tuple(e), tuple(c))
        if key not in memo:
            memo[key] = _cut_radius(L, e, c, cutoff)
        d2 = ((pts - sh.atom_xyz[sh.shell_atom[k]]) ** 2).sum(1)
        n += (2 * L + 1) * (d2 <= memo[key] ** 2)
    return float((n * n).mean()), float(n.mean())


def work(case):
    """Bytes: the grid (x, y, z, w), the density in, Vxc out. Flops: the two contractions over the AOs that
    reach the cut-off at each point, 2 n^2 each (four of X, Y_k and one of dExc/dP for the adjoint);
    an LDA needs half of each (symmetric operands). Weights: 15 operations per atom pair and point."""
    mols = _molecules(case, 1)
    fl = by = 0.0
    gga = case["functional"] in GGA
    for sh in mols:
        p, w, a = _moving_grid(sh, case)
        if case["kind"] == "weights":
            by += 8.0 * 5 * len(p) + 4.0 * len(p)
            fl += 15.0 * len(p) * sh.natom ** 2
            continue
        # single-centre points that the partition leaves a weight at: nearly all but the far ones
        sel = np.random.default_rng(0).choice(len(p), min(1500, len(p)), replace=False)
        n2, n1 = _reach(sh, p[sel], case["ao_cutoff"])
        spins = 2 if case["kind"] == "uks" else 1
        per = 2.0 * n2 * (5 if gga else 2) if case["kind"] == "backward" else 4.0 * n2 * (1.0 if gga else 0.5) * spins
        fl += per * len(p)
        by += 32.0 * len(p) + 16.0 * sh.nao ** 2 * spins
    return {"bytes": by, "flops": fl}


def tolerance(case):
    """About four times what plain torch FP64 without screening differs by (5- to 100-atom chains, SVWN, B3LYP,
    PBE): FP64 4e-15 (largest element 3e-14), with the AO cut-off at 1e-10 4e-12 (1e-10), INT8 (31-bit
    operands) 3e-10 (9e-9), Becke weights 2e-15."""
    if case["kind"] == "weights":
        return {"rel": 1e-14, "max": 2e-13}
    if case["precision"] == "mixed":
        return {"rel": 1.2e-9, "max": 4e-8}
    if case["ao_cutoff"] > 1e-14:
        return {"rel": 2e-11, "max": 1e-9}
    return {"rel": 2e-14, "max": 2e-13}


# ---------------------------------------------------------------------------------------- exact


def _powd(x, p):
    return torch.pow(x, p)


def _slater(ra, rb):
    k = -(3.0 / 2.0) * (3.0 / (4.0 * math.pi)) ** (1.0 / 3.0)
    return k * (_powd(ra, 4 / 3) + _powd(rb, 4 / 3))


def _vwn(ra, rb, v3):
    """Vosko, Wilk, Nusair 1980: fit V, or III (the sets B3LYP uses)."""
    P, F = ((3.72744, 12.9352, -0.10498), (7.06042, 18.0578, -0.325))
    if v3:
        P, F = ((13.0720, 42.7198, -0.409286), (20.1231, 101.578, -0.743294))
    rho = ra + rb
    x = (3.0 / (4.0 * math.pi) / rho) ** (1.0 / 6.0)
    zeta = (ra - rb) / rho

    def eps(A, b, c, x0):
        X, X0, Q = x * x + b * x + c, x0 * x0 + b * x0 + c, math.sqrt(4 * c - b * b)
        at = torch.atan(Q / (2 * x + b))
        return A * (torch.log(x * x / X) + 2 * b / Q * at - b * x0 / X0 * (
            torch.log((x - x0) ** 2 / X) + 2 * (2 * x0 + b) / Q * at))

    ep, ef = eps(0.0310907, *P), eps(0.01554535, *F)
    ea = eps(-1.0 / (6.0 * math.pi ** 2), 1.13107, 13.0045, -0.0047584)
    g = 9.0 / 8.0 * ((1 + zeta) ** (4 / 3) + (1 - zeta) ** (4 / 3) - 2.0)
    h = 4.0 / (9.0 * (2.0 ** (1 / 3) - 1.0)) * (ef - ep) / ea - 1.0
    return rho * (ep + ea * g * (1.0 + h * zeta ** 4))


def _b88(r, gam, lda):
    r43 = _powd(r, 4 / 3)
    x = torch.sqrt(gam) / r43
    k = -(3.0 / 2.0) * (3.0 / (4.0 * math.pi)) ** (1.0 / 3.0) if lda else 0.0
    f = r43 * (k - 0.0042 * x * x / (1.0 + 6.0 * 0.0042 * x * torch.asinh(x)))
    # the path (as the reference) takes no potential where the density or its squared gradient is below 1e-16
    return torch.where((r > 1e-16) & (gam > 1e-16), f, f.detach())


def _lyp(ra, rb, gaa, gab, gbb):
    a, b, c, d = 0.04918, 0.132, 0.2533, 0.349
    rho, rab = ra + rb, ra * rb
    m13 = rho ** (-1 / 3)
    om = torch.exp(-c * m13) * rho ** (-11 / 3) / (1 + d * m13)
    de = c * m13 + d * m13 / (1 + d * m13)
    cf = 2.0 ** (11 / 3) * 0.3 * (3 * math.pi ** 2) ** (2 / 3)
    f = -4 * a / (1 + d * m13) * rab / rho - cf * a * b * om * rab * (ra ** (8 / 3) + rb ** (8 / 3))
    ab = -a * b * om
    f = f + ab * (rab / 9 * (1 - 3 * de - (de - 11) * ra / rho) - rb * rb) * gaa
    f = f + ab * (rab / 9 * (1 - 3 * de - (de - 11) * rb / rho) - ra * ra) * gbb
    return f + ab * (rab / 9 * (47 - 7 * de) - 4 / 3 * rho * rho) * gab


def _pbe(ra, rb, gaa, gab, gbb):
    beta, kappa = 0.06672455060314922, 0.804
    gamma = (1 - math.log(2.0)) / math.pi ** 2
    mu = beta * math.pi ** 2 / 3
    f = 0.0
    for r, gm in ((ra, gaa), (rb, gbb)):
        n = 2 * r
        s2 = gm / ((3 * math.pi ** 2 * n) ** (2 / 3) * n * n)
        f = f + 0.5 * -0.75 * (3 / math.pi) ** (1 / 3) * n ** (4 / 3) * (1 + kappa - kappa / (1 + mu * s2 / kappa))
    rho = ra + rb
    z = (ra - rb) / rho
    rs = (3 / (4 * math.pi) / rho) ** (1 / 3)

    def G(A, a1, b1, b2, b3, b4):
        q = torch.sqrt(rs)
        return -2 * A * (1 + a1 * rs) * torch.log(1 + 1 / (2 * A * (b1 * q + b2 * rs + b3 * rs * q + b4 * rs * rs)))

    e0, e1 = G(0.0310907, 0.21370, 7.5957, 3.5876, 1.6382, 0.49294), G(0.01554535, 0.20548, 14.1189, 6.1977, 3.3662, 0.62517)
    ac = -G(0.0168869, 0.11125, 10.357, 3.6231, 0.88026, 0.49671)
    gam = 2 ** (4 / 3) - 2
    fz = ((1 + z) ** (4 / 3) + (1 - z) ** (4 / 3) - 2) / gam
    ec = e0 + ac * fz * (1 - z ** 4) / (8 / (9 * gam)) + (e1 - e0) * fz * z ** 4
    ph = 0.5 * ((1 + z) ** (2 / 3) + (1 - z) ** (2 / 3))
    ks2 = 4 * (3 * math.pi ** 2 * rho) ** (1 / 3) / math.pi
    t2 = (gaa + 2 * gab + gbb) / (4 * ph * ph * ks2 * rho * rho)
    A = beta / gamma / (torch.exp(-ec / (gamma * ph ** 3)) - 1)
    H = gamma * ph ** 3 * torch.log(1 + beta / gamma * t2 * (1 + A * t2) / (1 + A * t2 + (A * t2) ** 2))
    return f + rho * (ec + H)


def _functional(fn, ra, rb, gaa, gab, gbb):
    if fn == "SVWN":
        return _slater(ra, rb) + _vwn(ra, rb, False)
    if fn == "HFB":
        return _b88(ra, gaa, True) + _b88(rb, gbb, True)
    if fn == "BLYP":
        return _b88(ra, gaa, True) + _b88(rb, gbb, True) + _lyp(ra, rb, gaa, gab, gbb)
    if fn == "PBE":
        return _pbe(ra, rb, gaa, gab, gbb)
    return (0.80 * _slater(ra, rb) + 0.72 * (_b88(ra, gaa, False) + _b88(rb, gbb, False)) + 0.19 * _vwn(ra, rb, True)
            + 0.81 * _lyp(ra, rb, gaa, gab, gbb))


class _Shells:
    """The basis by classes of equal shells: (L, exponents, coefficients, atoms, first AOs) on the device."""

    def __init__(self, sh):
        cls = {}
        for k in range(sh.nshell):
            p0, m = sh.shell_p0[k], sh.shell_nprim[k]
            key = (int(sh.shell_l[k]), tuple(sh.prim_exp[p0:p0 + m]), tuple(sh.prim_coef[p0:p0 + m]))
            cls.setdefault(key, []).append((int(sh.shell_atom[k]), int(sh.shell_ao0[k])))
        self.nao = sh.nao
        self.cls = [(L, e, c, torch.tensor([a for a, _ in v], device=DEV), torch.tensor([o for _, o in v], device=DEV))
                    for (L, e, c), v in cls.items()]
        order = [o0 + k for L, _, _, _, o in self.cls for o0 in o.tolist() for k in range(2 * L + 1)]
        self.perm = torch.argsort(torch.tensor(order, device=DEV))

    def ao(self, r, R, grad):
        """phi (m, n) and, for a GGA, its gradient (3, m, n) at the points r for atoms at R."""
        s3 = 1.0 / math.sqrt(3.0)
        vals, grs = [], [[], [], []]
        for L, e, c, atoms, _ in self.cls:
            q = r[:, None, :] - R[atoms][None]
            x, y, z = q.unbind(-1)
            r2 = (q * q).sum(-1)
            S0 = S1 = 0.0
            for al, cf in zip(e, c):  # primitives beyond alpha r^2 = 30 are left out, as the path defines
                t = torch.where(al * r2 <= 30.0, cf * torch.exp(-al * r2), torch.zeros_like(r2))
                S0, S1 = S0 + t, S1 + al * t
            o, i = torch.zeros_like(x), torch.ones_like(x)
            if L == 0:
                A, D = [i], [(o, o, o)]
            elif L == 1:
                A, D = [x, y, z], [(i, o, o), (o, i, o), (o, o, i)]
            else:
                A = [x * y, z * x, y * z, 0.5 * (x * x - y * y), s3 * (z * z - 0.5 * (x * x + y * y))]
                D = [(y, x, o), (z, o, x), (o, z, y), (x, -y, o), (-s3 * x, -s3 * y, 2 * s3 * z)]
            vals.append(torch.stack([a * S0 for a in A], -1).flatten(1))
            if grad:
                for k, u in enumerate((x, y, z)):
                    grs[k].append(torch.stack([d[k] * S0 - 2 * u * a * S1 for a, d in zip(A, D)], -1).flatten(1))
        phi = torch.cat(vals, 1)[:, self.perm]
        return phi, torch.stack([torch.cat(g, 1)[:, self.perm] for g in grs]) if grad else None


def _points(fn, rho, grad, w):
    """f and the derivatives w df/drho_s, w (2 df/dg_ss + df/dg_ab) at points of two spins' densities."""
    live = (w != 0) & ((rho[0] > 1e-16) | (rho[1] > 1e-16))
    leaf = [torch.where(live, r, torch.ones_like(r)).clamp(min=1e-30).detach().requires_grad_() for r in rho]
    g = [(grad[0] * grad[0]).sum(0), (grad[0] * grad[1]).sum(0), (grad[1] * grad[1]).sum(0)] if grad else [w * 0 + 1] * 3
    g = [torch.where(live, v, torch.ones_like(v)).detach() for v in g]
    g = [g[0].clamp(min=1e-32).requires_grad_(), g[1].requires_grad_(), g[2].clamp(min=1e-32).requires_grad_()]
    f = _functional(fn, *leaf, *g)
    d = torch.autograd.grad(f.sum(), leaf + g, allow_unused=True)
    d = [torch.zeros_like(w) if t is None else torch.where(live, t, torch.zeros_like(t)) for t in d]
    return torch.where(live, f, torch.zeros_like(f)).detach(), w * d[0], w * d[1], w * (2 * d[2] + d[3]), w * (2 * d[4] + d[3])


def _xc(fn, sh, xyzw, Ps):
    """Exc, electron counts and Vxc of the spins' densities Ps (one: closed shell)."""
    S, gga = _Shells(sh), fn in GGA
    R = torch.from_numpy(sh.atom_xyz).to(DEV)
    step = max(2000, int(1.5e9 / (8 * sh.nao * (14 if gga else 6))))
    exc, nel = 0.0, [0.0] * len(Ps)
    V = [torch.zeros(sh.nao, sh.nao, dtype=torch.float64, device=DEV) for _ in Ps]
    for i in range(0, len(xyzw), step):
        b = torch.from_numpy(np.ascontiguousarray(xyzw[i:i + step])).to(DEV)
        w = b[:, 3]
        phi, dphi = S.ao(b[:, :3], R, gga)
        rho, grad = [], []
        for P in Ps:
            X = phi @ P
            rho.append((phi * X).sum(1))
            if gga:
                grad.append(2 * (dphi * X).sum(2))
        k = [0, 0] if len(Ps) == 1 else [0, 1]
        f, va, vb, ca, cb = _points(fn, [rho[j] for j in k], [grad[j] for j in k] if gga else None, w)
        exc += float((w * f).sum())
        for j, (v, c) in enumerate([(va, ca), (vb, cb)][:len(Ps)]):
            Z = 0.5 * v[:, None] * phi
            if gga:
                Z = Z + (dphi * (c * grad[j])[:, :, None]).sum(0)
            W = phi.T @ Z
            V[j] += W + W.T
            nel[j] += float((w * rho[j]).sum())
    return exc, nel, V


def _becke(R, br, r, owner):
    """Becke's partition with the size adjustment: P_owner / sum_m P_m at the points r."""
    d = torch.linalg.norm(r[:, None] - R[None], dim=-1)
    n = len(R)
    eye = torch.eye(n, dtype=torch.bool, device=DEV)
    RR = torch.linalg.norm(R[:, None] - R[None] + eye[..., None], dim=-1)
    u = (br[:, None] - br[None]) / (br[:, None] + br[None])
    a = (u / (u * u - 1)).clamp(-0.5, 0.5)
    mu = (d[:, :, None] - d[:, None, :]) / RR
    nu = mu + a * (1 - mu * mu)
    for _ in range(3):
        nu = 0.5 * nu * (3 - nu * nu)
    s = torch.where(eye, torch.ones_like(nu), 0.5 * (1 - nu)).prod(2)
    return s.gather(1, owner[:, None])[:, 0] / s.sum(1)


def _backward(s, sh):
    fn = s["case"]["functional"]
    gga = fn in GGA
    P = torch.from_numpy(s["P"]).to(DEV)
    S = _Shells(sh)
    R0 = torch.from_numpy(sh.atom_xyz).to(DEV)
    br = torch.from_numpy(s["br"]).to(DEV)
    xyzw = torch.from_numpy(s["xyzw"]).to(DEV)
    own = torch.from_numpy(s["owner"]).to(DEV).long()
    ws = torch.from_numpy(s["w"]).to(DEV)
    exc, _, V = _xc(fn, sh, s["xyzw"], [P])
    go, gw = torch.zeros_like(R0), torch.zeros_like(R0)
    step = max(1000, int(1e9 / (8 * sh.nao * 60)))
    for i in range(0, len(xyzw), step):
        r0, w, o = xyzw[i:i + step, :3], xyzw[i:i + step, 3], own[i:i + step]
        R = R0.clone().requires_grad_()
        r = r0 - R0[o] + R[o]
        phi, dphi = S.ao(r, R, gga)
        X = phi @ P
        rho = (phi * X).sum(1)
        gr = [2 * (dphi * X).sum(2)] * 2 if gga else None
        f, va, vb, ca, cb = _points(fn, [rho.detach()] * 2, [g.detach() for g in gr] if gga else None, w)
        # dE = va drho_a + vb drho_b + c d(gamma)/... with both spins alike
        e = ((va + vb) * rho).sum()
        if gga:
            g = gr[0]
            e = e + ((ca + cb).detach() * 0.5 * (g * g).sum(0)).sum()
        go += torch.autograd.grad(e, R)[0]
        fs = (f * ws[i:i + step]).detach()
        for j in range(0, len(w), 4000):
            R = R0.clone().requires_grad_()
            oj = o[j:j + 4000]
            om = _becke(R, br, r0[j:j + 4000] - R0[oj] + R[oj], oj)
            gw += torch.autograd.grad((fs[j:j + 4000] * om).sum(), R)[0]
    return {"dP": V[0].cpu().numpy(), "orbital": go.cpu().numpy(), "weight": gw.cpu().numpy(), "exc": np.array([exc])}


def exact(case, seed):
    if case["kind"] not in ("weights",) and case["size"] > (60 if case["kind"] == "backward" else 150):
        return None  # over 20 seconds
    s = prepare(case, seed)
    sh, fn, kind = s["mols"][0], case["functional"], case["kind"]
    if kind == "weights":
        R, br = (torch.from_numpy(v).to(DEV) for v in (sh.atom_xyz, s["br"]))
        out = np.empty(len(s["w"]))
        step = max(500, int(2e8 / (8 * sh.natom ** 2)))
        for i in range(0, len(out), step):
            r, o = (torch.from_numpy(v[i:i + step]).to(DEV) for v in (s["points"], s["owner"]))
            out[i:i + step] = _becke(R, br, r, o.long()).cpu().numpy() * s["w"][i:i + step]
        return out
    if kind == "backward":
        return _backward(s, sh)
    if kind == "batch":
        r = [_xc(fn, m, g, [torch.from_numpy(P).to(DEV)]) for m, g, P in zip(s["mols"], s["grids"], s["P"])]
        return {"exc": np.array([e for e, _, _ in r]), "nel": np.array([n[0] for _, n, _ in r]),
                "F": [V[0].cpu().numpy() for _, _, V in r]}
    xyzw = s["eng"].get_grid()[0]
    if kind == "uks":
        exc, (na, nb), (FA, FB) = _xc(fn, sh, xyzw, [torch.from_numpy(s[k]).to(DEV) for k in ("P", "PB")])
        return {"sums": np.array([exc, na, nb]), "FA": FA.cpu().numpy(), "FB": FB.cpu().numpy()}
    P = torch.from_numpy(s["P"]).to(DEV) if case["host"] else s["P"]
    exc, nel, V = _xc(fn, sh, xyzw, [P])
    return {"sums": np.array([exc, nel[0]]), "F": V[0].cpu().numpy() if case["host"] else V[0]}
