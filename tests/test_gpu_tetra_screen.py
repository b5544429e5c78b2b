"""The screened tetrahedron sums: every kernel variant at its edges, and the leg symmetry they use."""
import numpy as np
import pytest

from oracle import driver as D
from spring_b200 import synthetic as S
from spring_b200.api import from_crystal


@pytest.mark.parametrize("mesh", [(3, 3, 3), (4, 4, 4), (5, 4, 3), (1, 2, 6)])
def test_partner_map_carries_the_tetrahedra_onto_themselves(mesh):
    """q1 -> grid(-q0 - q1) is an involution that permutes the tetrahedra as vertex sets: channel 3 of
    the sums equals channel 2, and channel 1 is symmetric in its legs."""
    n = np.array(mesh)
    q = np.stack(np.meshgrid(*[np.arange(m) for m in mesh], indexing="ij"), -1).reshape(-1, 3, order="F")
    q = np.array([[g % n[0], g // n[0] % n[1], g // (n[0] * n[1])] for g in range(n.prod())])
    cr = S.build("rocksalt2")
    tet = D.make_tetrahedron(mesh, cr.G)[2] - 1
    sets = sorted(tuple(sorted(t)) for t in tet)
    for q0 in q:
        p = (-(q0 + q)) % n
        p = p[:, 0] + n[0] * (p[:, 1] + n[1] * p[:, 2])
        assert np.array_equal(p[p], np.arange(n.prod()))
        assert sorted(tuple(sorted(p[t])) for t in tet) == sets


@pytest.mark.gpu
@pytest.mark.parametrize("cell,N,nT,pol", [
    ("rocksalt2", 3, 1, None),                               # 162 tetrahedra: a last group of two lanes
    ("rocksalt2", 4, 2, None),                               # two of three temperature columns
    ("rocksalt2", 4, 4, None),                               # four of nine
    ("rocksalt2", 5, 9, [[1, 6], [2, 6], [2, 6]]),           # equal leg windows that start above 1
    ("rocksalt2", 4, 3, [[2, 5], [1, 3], [1, 6]]),           # unequal leg windows: all three channels
    ("rocksalt2", 4, 1, [[6, 6], [4, 4], [5, 6]]),
    ("rocksalt8", 2, 3, None),                               # four passes over s0, four s2 blocks
    ("rocksalt8", 2, 1, [[5, 21], [3, 19], [3, 19]]),        # s0 and s2 blocks with tails
    ("rocksalt8", 2, 2, [[1, 7], [24, 24], [1, 13]]),
])
def test_screened_tetrahedron_sums_match_oracle(cell, N, nT, pol):
    cr = S.build(cell)
    temps = list(np.linspace(100.0, 900.0, nT))
    st = D.Setup(cr, (N, N, N), temps)
    ctx, _ = from_crystal(cr, (N, N, N), temps, phonons={"grid": st.ph, "irr": st.ph0})
    p = None if pol is None else np.array(pol, np.int32)
    lw, p3 = ctx.linewidth3(1, st.nq0, delta="tetra", pol3=p)
    for i0 in range(st.nq0):
        for it in range(nT):
            r = D.linewidth3_q0(st, i0, delta="tetra", it=it, pol=p)
            np.testing.assert_allclose(lw[it, i0], r["lw"], rtol=1e-9, atol=1e-14 * np.abs(lw).max())
        np.testing.assert_allclose(p3[i0], r["p3_q0"], rtol=1e-9, atol=1e-14 * np.abs(p3).max())
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("mesh,nT,pol", [
    ((3, 3, 3), 1, None),                                    # a last group of two lanes
    ((2, 5, 3), 9, None),
    ((3, 4, 2), 2, [[3, 5], [2, 4], [1, 6], [5, 6]]),
    ((4, 4, 4), 4, [[1, 6], [6, 6], [2, 2], [1, 6]]),
])
def test_screened_four_phonon_sums_match_oracle(mesh, nT, pol):
    cr = S.build("rocksalt2", fc4=True)
    temps = list(np.linspace(100.0, 900.0, nT))
    W = np.eye(3, dtype=np.int32)[None]
    st = D.Setup(cr, mesh, temps, W=W, Rxyz=np.eye(3)[None])
    ctx, _ = from_crystal(cr, mesh, temps, phonons={"grid": st.ph, "irr": st.ph0}, W=W, Rxyz=np.eye(3)[None],
                          with_fc4=True)
    p = None if pol is None else np.array(pol, np.int32)
    first = st.nq0 // 2
    rate = ctx.linewidth4(first, 3, delta="tetra", pol4=p)
    for k in range(3):
        for it in range(nT):
            ro, _ = D.lw4_tetra(st, first - 1 + k, it, pol=p)
            np.testing.assert_allclose(rate[it, k], ro, rtol=1e-9, atol=1e-12 * max(np.abs(ro).max(), 1e-30))
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("delta", ["tetra", "gauss"])
@pytest.mark.parametrize("cell,N,nT", [("rocksalt2", 3, 1), ("rocksalt2", 4, 11), ("rocksalt8", 2, 2)])
def test_isotope_rate_matches_oracle(cell, N, nT, delta):
    """Six and 24 branches (one and four passes over s0), a last group of two tetrahedra, and more
    temperatures than the 3-phonon sums take."""
    cr = S.build(cell)
    temps = list(np.linspace(100.0, 900.0, nT))
    st = D.Setup(cr, (N, N, N), temps)
    ctx, _ = from_crystal(cr, (N, N, N), temps, phonons={"grid": st.ph, "irr": st.ph0})
    g2 = np.linspace(1e-3, 3e-3, cr.nbasis)
    rate = ctx.linewidth_iso(1, st.nq0, g2, delta=delta, sigma=0.3767)
    for i0 in range(st.nq0):
        wi = D.iso_w(cr.nbasis, st.ph0["evec"][i0], st.ph0["omega"][i0], st.ph["evec"], g2)
        ref = (D.iso_lw_gauss(st.ph0["omega"][i0], st.ph["omega"], wi, 0.3767) if delta == "gauss"
               else D.iso_lw_tetra(st.ph0["omega"][i0], st.ph["omega"], wi, st.tetra))
        for it in range(nT):
            np.testing.assert_allclose(rate[it, i0], ref, rtol=1e-9, atol=1e-14 * max(1.0, np.abs(rate).max()))
    ctx.close()


def _uneven(cr, seed=5):
    """The crystal with force constants that are not symmetric in their two legs."""
    cr.fc3 = cr.fc3 + np.random.default_rng(seed).normal(0.0, 1.0, size=cr.fc3.shape)
    return cr


@pytest.mark.gpu
@pytest.mark.parametrize("cell,mesh,nT", [("rocksalt2", (3, 3, 3), 2), ("rocksalt2", (4, 4, 2), 1), ("rocksalt8", (2, 2, 2), 1)])
def test_tetrahedron_sums_of_unsymmetrised_fc3_match_oracle(cell, mesh, nT):
    """W of a pair of equal points is not symmetric in its branches then (2^3: every q0 has such points)."""
    cr = _uneven(S.build(cell))
    temps = list(np.linspace(100.0, 900.0, nT))
    st = D.Setup(cr, mesh, temps, W=np.eye(3, dtype=np.int32)[None], Rxyz=np.eye(3)[None])
    ctx, _ = from_crystal(cr, mesh, temps, phonons={"grid": st.ph, "irr": st.ph0}, W=st.W, Rxyz=st.Rxyz)
    lw, p3 = ctx.linewidth3(1, st.nq0, delta="tetra")
    for i0 in range(0, st.nq0, 3):
        for it in range(nT):
            r = D.linewidth3_q0(st, i0, delta="tetra", it=it)
            np.testing.assert_allclose(lw[it, i0], r["lw"], rtol=1e-9, atol=1e-14 * np.abs(lw).max())
        np.testing.assert_allclose(p3[i0], r["p3_q0"], rtol=1e-9, atol=1e-14 * np.abs(p3).max())
    ctx.close()


@pytest.mark.gpu
def test_four_phonon_sums_with_a_vanishing_occupation_match_oracle():
    """n(q0) near the smallest double: (1 + n1) / n0 by itself is beyond the largest."""
    cr = S.build("rocksalt2", fc4=True)
    mesh, temps = (3, 3, 2), [30.0]
    W = np.eye(3, dtype=np.int32)[None]
    st = D.Setup(cr, mesh, temps, W=W, Rxyz=np.eye(3)[None])
    st.ph0["nbe"][0][4] = 5e-309
    ctx, _ = from_crystal(cr, mesh, temps, phonons={"grid": st.ph, "irr": st.ph0}, W=W, Rxyz=np.eye(3)[None],
                          with_fc4=True)
    rate = ctx.linewidth4(5, 1, delta="tetra")
    ro, _ = D.lw4_tetra(st, 4)
    assert np.all(np.isfinite(ro)) and ro.max() > 1e250
    np.testing.assert_allclose(rate[0, 0], ro, rtol=1e-9, atol=1e-12 * np.abs(ro).max())
    ctx.close()
