"""The two-atom V3 kernel at its edges: groups of four pairs that straddle q0 and end early, every split of the
seven slots over the two basis atoms, fewer slots than seven, windows, and each temperature variant."""
import numpy as np
import pytest

from oracle import driver as D
from spring_b200 import synthetic as S
from spring_b200.api import from_crystal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split,mesh,nT,pol", [
    (None, (3, 2, 1), 1, None),            # four pairs per q0 at most: groups straddle q0
    (None, (1, 1, 1), 2, None),            # one pair in all
    ((7, 0), (3, 2, 1), 3, None),          # one basis atom holds every slot
    ((4, 3), (2, 3, 2), 4, None),          # 16 + 12 + 12 + 9 slot pairs: a block that needs padding
    ((2, 5), (3, 3, 1), 9, [[2, 5], [1, 4], [1, 4]]),
    ("short", (3, 2, 2), 3, [[4, 6], [2, 6], [2, 6]]),   # five slots on one atom, none of the second on the other
])
def test_two_atom_v3_matches_oracle(split, mesh, nT, pol):
    cr = S.build("rocksalt2")
    if split == "short":
        cr.fc3_atm_num = np.array([5, 4], np.int32)
        cr.fc3_atm_indx = cr.fc3_atm_indx.copy()
        cr.fc3_atm_indx[1, :, 3] = 2
        cr.fc3 = cr.fc3.copy()
        for mu in range(2):
            cr.fc3[mu, cr.fc3_atm_num[mu]:] = 0.0
            cr.fc3[mu, :, cr.fc3_atm_num[mu]:] = 0.0
    elif split is not None:
        cr.fc3_atm_indx = cr.fc3_atm_indx.copy()
        for mu in range(2):               # interleaved, so that the slots have to be regrouped
            cr.fc3_atm_indx[mu, :, 3] = np.random.default_rng(mu).permutation([1] * split[0] + [2] * split[1])
    temps = list(np.linspace(100.0, 900.0, nT))
    ident = np.eye(3, dtype=np.int32)[None]
    st = D.Setup(cr, mesh, temps, W=ident, Rxyz=np.eye(3)[None])
    ctx, _ = from_crystal(cr, mesh, temps, phonons={"grid": st.ph, "irr": st.ph0}, W=ident, Rxyz=np.eye(3)[None])
    p = None if pol is None else np.array(pol, np.int32)
    ctx.prepare3()
    lw, p3 = ctx.linewidth3(1, st.nq0, "gauss", 1.5, pol3=p)      # the pair range read on the device
    part, _ = ctx.linewidth3(st.nq0, 1, "gauss", 1.5, pol3=p)
    np.testing.assert_allclose(part[:, 0], lw[:, -1], rtol=1e-12, atol=1e-14 * np.abs(lw).max())
    for i0 in range(st.nq0):
        r = D.linewidth3_q0(st, i0, with_w=True)
        w = ctx.scatter_w3(i0 + 1)
        np.testing.assert_allclose(w, r["sctr"], rtol=1e-9, atol=1e-12 * max(r["sctr"].max(), 1e-300))
        for it in range(nT):
            g = D.linewidth3_q0(st, i0, "gauss", 1.5, it=it, pol=p)
            np.testing.assert_allclose(lw[it, i0], g["lw"], rtol=1e-9, atol=1e-14 * np.abs(lw).max())
        np.testing.assert_allclose(p3[i0], g["p3_q0"], rtol=1e-9, atol=1e-14 * np.abs(p3).max())
    ctx.close()
