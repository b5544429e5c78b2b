"""V3 of cells with 12 and more branches (FP64 matrix kernel) and of the small ones beside it: W against the
oracle for every count of neighbour types, and the Gaussian sums with windows (equal on both legs: the pair folding's) and more than nine temperatures."""
import numpy as np
import pytest

from oracle import driver as D
from spring_b200 import synthetic as S
from spring_b200.api import Batch, from_crystal

pytestmark = pytest.mark.gpu

BASES = {
    "nb3": [[0, 0, 0], [.5, .5, 0], [.5, 0, .5]],
    "nb4": [[0, 0, 0], [0, .5, .5], [.5, 0, .5], [.5, .5, 0]],                        # 13 slots, every type
    "nb5": [[0, 0, 0], [.5, .5, .5], [.5, .5, 0], [.5, 0, .5], [0, .5, .5]],
    "nb6": [[0, 0, 0], [.5, 0, 0], [0, .5, 0], [0, 0, .5], [.5, .5, 0], [.5, .5, .5]],
    "nb7": [[0, 0, 0], [.5, 0, 0], [0, .5, 0], [0, 0, .5], [.5, .5, 0], [.5, .5, .5], [0, .5, .5]],
}


def _cell(name):
    if name == "nb8":
        return S.build("rocksalt8")
    b = np.array(BASES[name], float)
    cr = S.Crystal(name, 4.0 * np.eye(3), b, np.ones(len(b), np.int32), np.linspace(20.0, 60.0, len(b)))
    S.make_fc2(cr)
    S.make_fc3(cr)
    return cr


@pytest.mark.parametrize("name,nT,pol", [
    ("nb3", 2, None), ("nb4", 1, None), ("nb5", 10, None), ("nb6", 3, [[2, 11], [4, 9], [4, 9]]),
    ("nb7", 2, [[9, 20], [5, 21], [5, 21]]), ("nb8", 9, None), ("nb8", 11, [[17, 24], [8, 16], [8, 16]]),
])
def test_v3_cells_match_oracle(name, nT, pol):
    cr = _cell(name)
    mesh = (3, 2, 1)                      # pairs with q1 = q2, Gamma legs and general ones
    temps = list(np.linspace(100.0, 900.0, nT))
    ident = np.eye(3, dtype=np.int32)[None]
    st = D.Setup(cr, mesh, temps, W=ident, Rxyz=np.eye(3)[None])
    ctx, _ = from_crystal(cr, mesh, temps, phonons={"grid": st.ph, "irr": st.ph0}, W=ident, Rxyz=np.eye(3)[None])
    p = None if pol is None else np.array(pol, np.int32)
    lw, p3 = ctx.linewidth3(1, st.nq0, "gauss", 1.5, pol3=p)
    for i0 in range(st.nq0):
        r = D.linewidth3_q0(st, i0, with_w=True)
        w = ctx.scatter_w3(i0 + 1)
        np.testing.assert_allclose(w, r["sctr"], rtol=1e-9, atol=1e-12 * r["sctr"].max())
        for it in range(nT):
            g = D.linewidth3_q0(st, i0, "gauss", 1.5, it=it, pol=p)
            np.testing.assert_allclose(lw[it, i0], g["lw"], rtol=1e-9, atol=1e-14 * np.abs(lw).max())
        np.testing.assert_allclose(p3[i0], g["p3_q0"], rtol=1e-9, atol=1e-14 * np.abs(p3).max())
    ctx.close()


def test_first_atom_without_fc3_neighbours_matches_oracle():
    """No FC3 on the first atom: its part of the intermediate sums is never formed, and what lies in its place in
    shared memory (here NaN, left there by a run with undefined eigenvectors) must not reach W."""
    cr = _cell("nb4")
    mesh, temps = (7, 3, 2), [300.0]              # about 900 pairs: every SM takes part
    ident = np.eye(3, dtype=np.int32)[None]
    kw = dict(W=ident, Rxyz=np.eye(3)[None])
    st = D.Setup(cr, mesh, temps, **kw)
    bad = dict(st.ph, evec=np.full_like(st.ph["evec"], np.nan))
    before, _ = from_crystal(cr, mesh, temps, phonons={"grid": bad, "irr": st.ph0}, **kw)
    cr.fc3_atm_num[0] = 0
    ctx, _ = from_crystal(cr, mesh, temps, phonons={"grid": st.ph, "irr": st.ph0}, **kw)
    for c in (before, ctx):                       # both prepared: nothing else runs between the two calls below
        c.linewidth3(1, st.nq0, "gauss", 1.5)
    before.linewidth3(1, st.nq0, "gauss", 1.5)
    lw, _ = ctx.linewidth3(1, st.nq0, "gauss", 1.5)
    assert np.all(np.isfinite(lw))
    for i0 in (0, 5, st.nq0 - 1):
        r = D.linewidth3_q0(st, i0, "gauss", 1.5, with_w=True)
        np.testing.assert_allclose(lw[0, i0], r["lw"], rtol=1e-9, atol=1e-14 * np.abs(lw).max())
        before.linewidth3(1, st.nq0, "gauss", 1.5)
        w = ctx.scatter_w3(i0 + 1)
        np.testing.assert_allclose(w, r["sctr"], rtol=1e-9, atol=1e-12 * r["sctr"].max())
    before.close()
    ctx.close()


def test_generic_option_reaches_the_any_cell_kernel():
    """SPRING_OPT_GENERIC_V3 on a cell that the matrix kernel takes: the other kernel's sums (the same W to rounding,
    not the same bits), per call and as items of a batch in every s0 block."""
    cr = S.build("rocksalt8")
    st = D.Setup(cr, (2, 2, 2), [300.0])
    ctx, _ = from_crystal(cr, (2, 2, 2), [300.0], phonons={"grid": st.ph, "irr": st.ph0})
    small, _ = from_crystal(S.build("rocksalt2"), (3, 3, 3), [300.0])
    w, (lw, p3) = ctx.scatter_w3(2), ctx.linewidth3(1, st.nq0, "gauss", 0.8)
    ctx.use_generic_v3(True)
    wg, (lg, pg) = ctx.scatter_w3(2), ctx.linewidth3(1, st.nq0, "gauss", 0.8)
    assert not np.array_equal(wg, w)
    np.testing.assert_allclose(wg, w, rtol=1e-9, atol=1e-12 * w.max())
    np.testing.assert_allclose(lg, lw, rtol=1e-9, atol=1e-14 * lw.max())
    ref = D.linewidth3_q0(st, 1, "gauss", 0.8, with_w=True)
    np.testing.assert_allclose(wg, ref["sctr"], rtol=1e-9, atol=1e-12 * w.max())
    np.testing.assert_allclose(lg[0, 1], ref["lw"], rtol=1e-9, atol=1e-14 * lw.max())
    b = Batch()
    b.add_linewidth3(small, 1, small.nq0, 0.8)
    k = b.add_linewidth3(ctx, 1, st.nq0, 0.8)
    for config in ((1, 0, 6, 1), (0, 1, 12, 4), (1, 2, 6, 16)):
        b.set_config(*config)
        n = ctx.kernel_launches()
        b.run()
        assert ctx.kernel_launches() == n                    # its pairs are items of the persistent kernel
        np.testing.assert_allclose(b.result(k)[0], lw, rtol=1e-9, atol=1e-14 * lw.max())
        np.testing.assert_allclose(b.result(k)[1], p3, rtol=1e-9, atol=1e-14 * p3.max())
    b.close()
    ctx.close()
    small.close()


def test_every_neighbour_type_at_24_branches_matches_oracle():
    """Eight neighbour types per atom: the matrix kernel's layout does not fit, and the any-cell kernel works in s0
    blocks."""
    cr = S.build("rocksalt8")
    cr.fc3_atm_indx = np.array([[[0, 0, 0, nu + 1] for nu in range(8)]] * 8, np.int32)
    cr.fc3_atm_indx[:, 1:, 0] = [[(mu + nu) % 3 - 1 for nu in range(1, 8)] for mu in range(8)]
    cr.fc3_atm_num = np.full(8, 8, np.int32)
    f = np.random.default_rng(3).normal(0.0, 2.0, size=(8, 8, 8, 3, 3, 3))
    cr.fc3 = np.ascontiguousarray(0.5 * (f + f.transpose(0, 2, 1, 3, 5, 4)))
    st = D.Setup(cr, (2, 2, 1), [300.0])
    ctx, _ = from_crystal(cr, (2, 2, 1), [300.0], phonons={"grid": st.ph, "irr": st.ph0})
    lw, p3 = ctx.linewidth3(1, st.nq0, "gauss", 1.5)
    for i0 in range(st.nq0):
        r = D.linewidth3_q0(st, i0, "gauss", 1.5, with_w=True)
        np.testing.assert_allclose(ctx.scatter_w3(i0 + 1), r["sctr"], rtol=1e-9, atol=1e-12 * r["sctr"].max())
        np.testing.assert_allclose(lw[0, i0], r["lw"], rtol=1e-9, atol=1e-14 * np.abs(lw).max())
        np.testing.assert_allclose(p3[i0], r["p3_q0"], rtol=1e-9, atol=1e-14 * np.abs(p3).max())
    ctx.close()
