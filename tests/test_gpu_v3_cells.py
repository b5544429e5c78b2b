"""V3 of cells with 12 and more branches (FP64 matrix kernel) and of the small ones beside it: W against the
oracle for every count of neighbour types, and the Gaussian sums with windows (equal on both legs: the pair folding's) and more than nine temperatures."""
import numpy as np
import pytest

from oracle import driver as D
from spring_b200 import synthetic as S
from spring_b200.api import from_crystal

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
