"""Basis screening of the grid planner (host): a shell stays in a group's basis when its envelope
reaches 0.2 of the AO cut-off at the group's nearest point."""
from types import SimpleNamespace

import numpy as np
import pytest

from proteindf_b200 import basis, grids, systems, xc

CUT = 1e-10


def radius(L, e, c, cutoff):
    r = np.arange(60.0, 0.0, -0.01)[:, None]
    env = (np.abs(c) * np.exp(-e * r * r) * np.maximum(r ** L, L * r ** max(L - 1, 0) + 2 * e * r ** (L + 1))).sum(1)
    hit = np.nonzero(env >= cutoff)[0]
    return r[hit[0], 0] + 0.01 if len(hit) else 0.0


def shell_radii(sh, cutoff):
    memo, out = {}, []
    for k in range(sh.nshell):
        p0, m, L = sh.shell_p0[k], sh.shell_nprim[k], int(sh.shell_l[k])
        e, c = sh.prim_exp[p0:p0 + m], sh.prim_coef[p0:p0 + m]
        key = (L, tuple(e), tuple(c))
        if key not in memo:
            memo[key] = radius(L, e, c, cutoff)
        out.append(memo[key])
    return np.array(out)


def nearest(sh, pts):
    """Distance of each shell's atom to its nearest point."""
    return np.sqrt(((pts[:, None] - sh.atom_xyz[None]) ** 2).sum(2).min(0))[sh.shell_atom]


def sphere(sh, pts):
    """Distance of each shell's atom to the points' bounding sphere."""
    cen = pts.mean(0)
    rad = np.sqrt(((pts - cen) ** 2).sum(1).max())
    return (np.sqrt(((sh.atom_xyz - cen) ** 2).sum(1)) - rad)[sh.shell_atom]


def expected(sh, pts):
    return int(((2 * sh.shell_l + 1) * (nearest(sh, pts) <= shell_radii(sh, 0.2 * CUT))).sum())


def vxc_of(sh, keep, xyzw, PA):
    """The oracle's Vxc of the kept shells alone, in the whole basis."""
    from oracle import oracle
    n = 2 * sh.shell_l + 1
    aos = np.concatenate([np.arange(o, o + c) for o, c in zip(sh.shell_ao0[keep], n[keep])])
    sub = SimpleNamespace(shell_atom=sh.shell_atom[keep], shell_l=sh.shell_l[keep],
                          shell_ao0=(np.cumsum(n[keep]) - n[keep]).astype(np.int32),
                          shell_nprim=sh.shell_nprim[keep], shell_p0=sh.shell_p0[keep], prim_exp=sh.prim_exp,
                          prim_coef=sh.prim_coef, atom_xyz=sh.atom_xyz, nao=len(aos), nshell=int(keep.sum()))
    V = np.zeros((sh.nao, sh.nao))
    V[np.ix_(aos, aos)] = oracle.xc("B3LYP", sub, xyzw, PA[np.ix_(aos, aos)])["vxc"]
    return V


@pytest.mark.parametrize("npts,spread", [(1, 0.0), (2, 10.0), (37, 3.0), (128, 6.0)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_nearest_point_screening_equals_brute_force(npts, spread, precision):
    """One group of points (two half groups `spread` apart): the planned basis against a brute-force count."""
    syms, xyz = systems.peptide_chain(60, seed=4)
    sh = basis.ShellTable(syms, xyz, basis.load_basis("cc-pVDZ"))
    rng = np.random.default_rng(npts)
    for at in (3, 17, 40):
        pts = xyz[at] + rng.uniform(-0.5, 0.5, (npts, 3)) + spread * (np.arange(npts) % 2)[:, None] * [1.0, 0.0, 0.0]
        plan = xc.plan_grid(sh, np.c_[pts, np.ones(npts)], precision=precision, ao_cutoff=CUT)
        assert plan["nblocks"] == 1
        assert plan["mean_nb"] == expected(sh, pts)


@pytest.mark.parametrize("seed", [1, 2])
def test_error_at_a_loose_cutoff_is_below_the_bounding_spheres(seed):
    """Vxc over twelve groups of 128 neighbouring points of a molecular grid: what the planned bases leave
    out is less than what the cut-off at the groups' bounding spheres would (0.47 to 0.61 of it over chains
    of 40 to 150 atoms, cut-offs of 1e-8 to 1e-12)."""
    syms, xyz = systems.peptide_chain(60, seed=seed)
    sh = basis.ShellTable(syms, xyz, basis.load_basis("cc-pVDZ"))
    allp, w, _ = grids.molecular_grid(xyz, sh.atom_z, nrad=75, nang=302, radial="GC", mapping="TA", pruning=True)
    rng = np.random.default_rng(seed)
    c = np.linalg.qr(rng.standard_normal((sh.nao, int(0.4 * sh.nao))))[0]
    PA = c @ c.T
    r_near, r_sphere = shell_radii(sh, 0.2 * CUT), shell_radii(sh, CUT)
    every = np.ones(sh.nshell, bool)
    err = {"planned": 0.0, "sphere": 0.0}
    groups = 0
    while groups < 12:
        near = np.argsort(((allp - allp[rng.integers(len(allp))]) ** 2).sum(1))[:128]
        pts = allp[near]
        if ((pts.max(0) - pts.min(0)) ** 2).sum() > 140.0:  # the planner would cut the group
            continue
        groups += 1
        xyzw = np.c_[pts, np.full(128, 0.05)]
        keep = nearest(sh, pts) <= r_near
        plan = xc.plan_grid(sh, xyzw, ao_cutoff=CUT)
        assert plan["nblocks"] == 1 and plan["mean_nb"] == ((2 * sh.shell_l + 1) * keep).sum()
        full = vxc_of(sh, every, xyzw, PA)
        err["planned"] += ((vxc_of(sh, keep, xyzw, PA) - full) ** 2).sum()
        err["sphere"] += ((vxc_of(sh, sphere(sh, pts) <= r_sphere, xyzw, PA) - full) ** 2).sum()
    assert 0.0 < err["planned"] < err["sphere"]
