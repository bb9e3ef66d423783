"""Basis screening of the grid planner (host): a shell stays in a group's basis when its envelope
reaches the AO cut-off at the nearest point of the group's bounding sphere and 0.3 of the cut-off at the
group's own nearest point."""
import numpy as np
import pytest

from proteindf_b200 import basis, systems, xc

CUT = 1e-10


def radius(L, e, c, cutoff):
    r = np.arange(60.0, 0.0, -0.01)[:, None]
    env = (np.abs(c) * np.exp(-e * r * r) * np.maximum(r ** L, L * r ** max(L - 1, 0) + 2 * e * r ** (L + 1))).sum(1)
    hit = np.nonzero(env >= cutoff)[0]
    return r[hit[0], 0] + 0.01 if len(hit) else 0.0


def expected(sh, pts):
    cen = pts.mean(0)
    rad = np.sqrt(((pts - cen) ** 2).sum(1).max())
    nb = 0
    for k in range(sh.nshell):
        p0, m, L = sh.shell_p0[k], sh.shell_nprim[k], int(sh.shell_l[k])
        e, c = sh.prim_exp[p0:p0 + m], sh.prim_coef[p0:p0 + m]
        A = sh.atom_xyz[sh.shell_atom[k]]
        if np.linalg.norm(A - cen) - rad <= radius(L, e, c, CUT) and \
                np.sqrt(((pts - A) ** 2).sum(1).min()) <= radius(L, e, c, 0.3 * CUT):
            nb += 2 * L + 1
    return nb


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
