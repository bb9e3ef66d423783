"""Partition weights bit for bit against the CPU restatement: the forms of the Becke weights by atom count
(near to 480, a warp per point to 1600, a thread per point above), the parts of a long call, and where the
near form's filter, sums and tables can go wrong."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def chain(n, seed):
    from proteindf_b200 import basis, grids, systems
    syms, xyz = systems.peptide_chain(n, seed=seed)
    sh = basis.ShellTable(syms, xyz, basis.load_basis("cc-pVDZ"))
    return sh, np.array([grids.BECKE_RADIUS[int(z)] for z in sh.atom_z])


def weights(sh, brad, pts, owner, **kw):
    from proteindf_b200.xc import XcEngine
    eng = XcEngine()
    eng.set_system(sh)
    w = eng.becke_weights(pts, owner, np.ones(len(pts)), brad, **kw)
    eng.close()
    return w


def near_points(sh, n, seed, spread=1.5):
    """Points around seeded atoms, each with its atom as the owner."""
    rng = np.random.default_rng(seed)
    owner = rng.integers(0, sh.natom, n).astype(np.int32)
    return sh.atom_xyz[owner] + spread * rng.standard_normal((n, 3)), owner


@pytest.mark.parametrize("n", [30, 60])
@pytest.mark.parametrize("what", ["place", "radius"])
def test_non_finite_pair_constants_show_in_every_weight(n, what):
    """Two atoms in one place (1/R_mn infinite) or of radius zero (a_mn 0/0): P of the first is a NaN at
    every point, and so is every weight, however far the two are from the point."""
    from oracle import oracle
    from proteindf_b200 import basis
    sh, brad = chain(n, seed=11)
    if what == "place":
        xyz = sh.atom_xyz.copy()
        xyz[1] = xyz[0]
        sh = basis.ShellTable(sh.symbols, xyz, basis.load_basis("cc-pVDZ"))
    else:
        brad[:2] = 0.0
    pts, owner = near_points(sh, 500, seed=n)
    ref = oracle.becke(sh.atom_xyz, brad, pts, owner)
    assert np.isnan(ref).all()
    assert np.isnan(weights(sh, brad, pts, owner)).all()


@pytest.mark.parametrize("n", [40, 100])
def test_far_points_equal_oracle_bit_for_bit(n):
    """Points at 1e3 to 1e9 bohr and beyond the range of FP32, where FP32 no longer tells the atoms'
    distances apart: the filter must not drop an atom that carries the sum."""
    from oracle import oracle
    sh, brad = chain(n, seed=1)
    rng = np.random.default_rng(n)
    far = np.repeat([1e3, 1e5, 3e5, 1e6, 1e7, 2e7, 5e7, 1e8, 1e9, 1e12, 1e39], 60)
    u = rng.standard_normal((len(far), 3))
    pts = far[:, None] * u / np.linalg.norm(u, axis=1)[:, None]
    owner = rng.integers(0, n, len(far)).astype(np.int32)
    w = weights(sh, brad, pts, owner)
    ref = oracle.becke(sh.atom_xyz, brad, pts, owner)
    assert np.array_equal(w, ref, equal_nan=True)


def test_contexts_of_different_sizes_in_several_threads():
    """The near form's shared memory depends on the atom count, its limit is the function's for the whole
    process: contexts of 60 and of 400 atoms on four host threads must not lower it for one another."""
    import threading
    from proteindf_b200.xc import XcEngine
    work, bad = [], []
    for n in (400, 60, 400, 60):
        sh, brad = chain(n, seed=9)
        eng = XcEngine()
        eng.set_system(sh)
        pts, owner = near_points(sh, 1, seed=n)
        work.append((eng, brad, pts, owner, eng.becke_weights(pts, owner, np.ones(1), brad)))
    start = threading.Barrier(len(work))

    def calls(eng, brad, pts, owner, want):
        start.wait()
        try:
            for _ in range(700):
                if not np.array_equal(eng.becke_weights(pts, owner, np.ones(1), brad), want):
                    bad.append("weights")
        except RuntimeError as e:
            bad.append(str(e))

    threads = [threading.Thread(target=calls, args=w) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for w in work:
        w[0].close()
    assert not bad, bad[:3]


@pytest.mark.parametrize("n", [4, 16, 17, 480, 481, 500, 1600, 1601])
def test_forms_at_their_ends_equal_oracle_bit_for_bit(n):
    """Molecules below, at and above the 16 atoms of a near list, the last atom count of the near form, the
    first ones and the last of the warp form, the first of the form with a thread per point; 300 points, of
    which one is far outside."""
    from oracle import oracle
    sh, brad = chain(n, seed=3)
    pts, owner = near_points(sh, 300, seed=n)
    pts[7] += 400.0
    assert np.array_equal(weights(sh, brad, pts, owner), oracle.becke(sh.atom_xyz, brad, pts, owner))


@pytest.mark.parametrize("form,n", [("near", 20), ("near", 60), ("warp", 481), ("ss", 60)])
def test_parts_of_a_long_call_equal_short_calls(form, n):
    """More than 65,536 points go through the kernels in parts that share the pair tables of the first; every
    point's weight is that of a call of its own part."""
    from proteindf_b200.xc import XcEngine
    sh, brad = chain(n, seed=4)
    npts = 65536 * 2 + 77 if n < 100 else 65536 + 77
    pts, owner = near_points(sh, npts, seed=n)
    w = 1.0 + np.arange(npts) / npts
    eng = XcEngine()
    eng.set_system(sh)
    call = eng.ss_weights if form == "ss" else lambda p, o, v: eng.becke_weights(p, o, v, brad)
    whole = call(pts, owner, w)
    for i in range(0, npts, 30000):
        s = slice(i, i + 30000)
        assert np.array_equal(call(pts[s], owner[s], w[s]), whole[s])
    eng.close()


def lattice(k, seed=0):
    """k^3 hydrogen atoms on a shaken lattice of 1.4 bohr, radii of two kinds: most P_m count at most points."""
    from proteindf_b200 import basis
    rng = np.random.default_rng(seed + k)
    n = k ** 3
    xyz = 1.4 * np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)
    sh = basis.ShellTable(["H"] * n, xyz + rng.uniform(-0.2, 0.2, (n, 3)), {"H": [{"shell": "s", "prims": [[0.6, 1.0]]}]})
    return sh, np.where(np.arange(n) % 3 == 0, 0.35, 0.70)


@pytest.mark.parametrize("k", [3, 4, 5])
@pytest.mark.parametrize("spread", [0.7, 10.0, 100.0])
def test_many_kept_pairs_equal_oracle_bit_for_bit(k, spread):
    """125 atoms with points far outside keep 37 of them a point: more pairs than a CTA's 1,024 at once, so its
    points are summed in several runs of atoms. The last CTA has 13 points."""
    from oracle import oracle
    sh, brad = lattice(k)
    pts, owner = near_points(sh, 301, seed=k, spread=spread)
    assert np.array_equal(weights(sh, brad, pts, owner), oracle.becke(sh.atom_xyz, brad, pts, owner))


@pytest.mark.parametrize("share", ["2.8e-14", "1e-9", "1e-4"])
@pytest.mark.parametrize("k", [3, 5])
def test_second_sum_equals_oracle_bit_for_bit(k, share, monkeypatch):
    """A looser drop threshold leaves the sum's last bits open at nearly every point (297 to 301 of the 301); they
    are summed over all atoms, to the same bits."""
    from oracle import oracle
    monkeypatch.setenv("PDFXC_BECKE_SHARE", share)
    sh, brad = lattice(k)
    pts, owner = near_points(sh, 301, seed=k)
    assert np.array_equal(weights(sh, brad, pts, owner), oracle.becke(sh.atom_xyz, brad, pts, owner))
