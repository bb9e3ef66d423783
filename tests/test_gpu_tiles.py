"""Contraction tiles at the sizes where they can go wrong: a block of exactly n screened AOs, with n
around the tiles' edges (rows of 8, pairs of 16, tiles of 64 and 128), against the CPU restatement."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# s functions of one exponent on n hydrogen atoms in a small cube: every block screens in all of them
S_BASIS = {"H": [{"shell": "s", "prims": [[0.6, 1.0]]}]}


def system(n, npts=300, seed=0):
    from proteindf_b200 import basis
    rng = np.random.default_rng(seed + n)
    sh = basis.ShellTable(["H"] * n, rng.uniform(0.0, 4.0, (n, 3)), S_BASIS)
    xyzw = np.c_[rng.uniform(-1.0, 5.0, (npts, 3)), rng.uniform(0.01, 0.1, npts)]
    c = rng.standard_normal((n, max(1, n // 3))) / np.sqrt(n)
    return sh, xyzw, c @ c.T


@pytest.mark.parametrize("n", [1, 7, 8, 9, 16, 17, 40, 63, 64, 65, 73, 127, 128, 129, 200])
@pytest.mark.parametrize("fn", ["SVWN", "B3LYP"])
def test_fp64_tiles_vs_oracle(n, fn):
    """FP64: sums of n products per point and of 300 points per element in another order, and the
    functional's own roundings: a few thousand roundings of 1.1e-16 of the largest element."""
    from oracle import oracle
    from proteindf_b200.xc import XcEngine
    sh, xyzw, PA = system(n)
    eng = XcEngine()
    eng.set_system(sh)
    eng.set_grid(xyzw)
    exc, nel, V = eng.build_vxc(fn, PA)
    ref = oracle.xc(fn, sh, xyzw, PA)
    eng.close()
    assert abs(exc - ref["exc"]) <= 1e-12 * abs(ref["exc"])
    assert abs(nel - ref["nelec_alpha"]) <= 1e-12 * abs(nel)
    assert np.abs(V - ref["vxc"]).max() <= 1e-12 * np.abs(ref["vxc"]).max()
