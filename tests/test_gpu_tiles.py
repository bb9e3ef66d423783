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


@pytest.mark.parametrize("n", [1, 16, 63, 64, 65, 127, 128, 129, 200])
@pytest.mark.parametrize("fn", ["SVWN", "B3LYP"])
def test_int8_tiles_vs_oracle(n, fn):
    """INT8: operands cut at 2^-31 of a row's largest element, sums of up to 300 such products of
    random sign: 2^-31 sqrt(300) = 8e-9 of the largest element, and the sum over the points less."""
    from oracle import oracle
    from proteindf_b200.xc import XcEngine
    sh, xyzw, PA = system(n)
    eng = XcEngine(precision="mixed")
    eng.set_system(sh)
    eng.set_grid(xyzw)
    exc, nel, V = eng.build_vxc(fn, PA)
    ref = oracle.xc(fn, sh, xyzw, PA)
    eng.close()
    assert abs(exc - ref["exc"]) <= 8e-9 * abs(ref["exc"])
    assert np.abs(V - ref["vxc"]).max() <= 8e-9 * np.abs(ref["vxc"]).max()


@pytest.mark.parametrize("n", [1, 8, 9, 63, 64, 65, 129])
@pytest.mark.parametrize("fn", ["SVWN", "PBE"])
def test_open_shell_and_adjoint_tiles(n, fn):
    """With equal spins the open-shell build is the closed-shell one, and the adjoint's dExc/dP is
    the forward Vxc (the same sums in another order), at the tiles' edges."""
    from proteindf_b200.xc import XcEngine
    sh, xyzw, PA = system(n)
    eng = XcEngine()
    eng.set_system(sh)
    eng.set_grid(xyzw, np.arange(len(xyzw)) % n)
    exc, nel, V = eng.build_vxc(fn, PA)
    eu, na, nb, FA, FB = eng.build_vxc_uks(fn, PA, PA)
    dP, go, gw, eb = eng.xc_backward(fn, PA, dexc=2.0)
    eng.close()
    top = np.abs(V).max()
    assert abs(eu - exc) <= 1e-12 * abs(exc) and abs(eb - exc) <= 1e-12 * abs(exc)
    assert abs(na - nel) <= 1e-12 * nel and abs(nb - nel) <= 1e-12 * nel
    assert np.abs(FA - V).max() <= 1e-12 * top and np.abs(FB - V).max() <= 1e-12 * top
    assert np.abs(dP - 2.0 * V).max() <= 2e-12 * top


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_open_shell_buffers_follow_the_grid(precision):
    """A larger grid and a larger system after an open-shell build: the second spin's buffers are
    sized for them (the result is that of a fresh context)."""
    from proteindf_b200.xc import XcEngine
    eng = XcEngine(precision=precision)
    for n, npts in ((9, 200), (9, 3000), (70, 3000)):
        sh, xyzw, PA = system(n, npts)
        PB = 0.8 * PA
        eng.set_system(sh)
        eng.set_grid(xyzw)
        got = eng.build_vxc_uks("BLYP", PA, PB)
        fresh = XcEngine(precision=precision)
        fresh.set_system(sh)
        fresh.set_grid(xyzw)
        want = fresh.build_vxc_uks("BLYP", PA, PB)
        fresh.close()
        assert abs(got[0] - want[0]) <= 1e-12 * abs(want[0])
        for k in (3, 4):
            assert np.abs(got[k] - want[k]).max() <= 1e-12 * np.abs(want[k]).max()
    eng.close()
