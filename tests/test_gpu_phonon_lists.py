"""Phonons by the length of the list of points (lanes per point of two-atom cells, parts of the dipole term) and by
the number of branches (odd, even, 24): the points two meshes share, and the oracle's frequencies."""
import numpy as np
import pytest

from oracle import driver as D
from spring_b200 import synthetic as S
from spring_b200.api import from_crystal

pytestmark = pytest.mark.gpu

IDENT = dict(W=np.eye(3, dtype=np.int32)[None], Rxyz=np.eye(3)[None])


def _grid(cr, m, **kw):
    ctx, _ = from_crystal(cr, (m,) * 3, [300.0, 500.0], with_fc3=False, **IDENT, **kw)
    ctx.compute_phonons([300.0, 500.0])
    g = ctx.get_phonons(0)
    q = ctx.make_mesh()[0]
    ctx.close()
    return g, q


@pytest.mark.parametrize("fine,coarse,polar", [(14, 7, False), (15, 5, False), (16, 8, True)])
def test_long_and_short_lists_agree(fine, coarse, polar):
    cr = S.build("rocksalt2")
    if polar:
        S.make_polar(cr)
    kw = dict(dipole=dict(rmesh=(3, 3, 3))) if polar else {}
    (a, qa), (b, qb) = _grid(cr, fine, **kw), _grid(cr, coarse, **kw)
    pos = {tuple(q): i for i, q in enumerate(qa.tolist())}
    la = [pos[tuple(q)] for q in (qb * (fine // coarse)).tolist() if tuple(q) in pos]
    lb = [i for i, q in enumerate((qb * (fine // coarse)).tolist()) if tuple(q) in pos]
    assert len(la) == coarse ** 3
    w2a, w2b = a["omega"][la] ** 2, b["omega"][lb] ** 2   # eigenvalues: error n eps |D|, 1e-14 relative to the top
    np.testing.assert_allclose(w2a, w2b, rtol=0, atol=1e-12 * w2b.max())


@pytest.mark.parametrize("nb", [1, 3, 4, 8])
def test_branches_match_oracle(nb):
    if nb == 8:
        cr = S.build("rocksalt8")
    else:
        pos = np.array([[0, 0, 0], [.5, .5, 0], [.5, 0, .5], [0, .5, .5]])[:nb]
        cr = S.Crystal("cell", 4.0 * np.eye(3), pos, (np.arange(nb) % 2 + 1).astype(np.int32),
                       np.linspace(20.0, 60.0, nb))
        S.make_fc2(cr)
        S.make_fc3(cr)
    st = D.Setup(cr, (3, 2, 2), [300.0], **IDENT)
    ctx, _ = from_crystal(cr, (3, 2, 2), [300.0], with_fc3=False, **IDENT)
    ctx.compute_phonons([300.0])
    g = ctx.get_phonons(0)
    ctx.close()
    w = np.asarray(st.ph["omega"]).reshape(g["omega"].shape)
    np.testing.assert_allclose(g["omega"] ** 2, w ** 2, rtol=0, atol=1e-12 * (w ** 2).max())
    n = g["omega"].shape[1]
    e = g["evec"].reshape(-1, n, n)                               # orthonormal to n eps per rotation round
    np.testing.assert_allclose(np.einsum("qsr,qtr->qst", e.conj(), e), np.broadcast_to(np.eye(n), e.shape), atol=1e-11)


@pytest.mark.parametrize("nb", [2, 5, 6, 7])
def test_branches_of_random_springs_match_oracle(nb):
    """The remaining branch counts, and a two-atom cell with more neighbours than its own kernel takes (54)."""
    rng = np.random.default_rng(nb)
    cells = [(x, y, z) for x in (-1, 0, 1) for y in (-1, 0, 1) for z in (-1, 0, 1)]
    cells = cells if nb == 2 else [(x, 0, 0) for x in (-1, 0, 1)]
    bond = {}
    for R in cells:
        for mu in range(nb):
            for nu in range(nb):
                if (nu, mu, tuple(-x for x in R)) in bond:
                    bond[mu, nu, R] = bond[nu, mu, tuple(-x for x in R)].T
                else:
                    f = rng.normal(0.0, 1.0, size=(3, 3))
                    bond[mu, nu, R] = f + f.T + 60.0 * np.eye(3) if mu == nu and R == (0, 0, 0) else f
    cr = S.Crystal("springs", 4.0 * np.eye(3), rng.random((nb, 3)), np.ones(nb, np.int32), np.linspace(20.0, 60.0, nb))
    cr.fc2_atm_num = np.full(nb, len(cells) * nb, np.int32)
    slots = [(R, nu) for R in cells for nu in range(nb)]
    cr.fc2_atm_indx = np.array([[[*R, nu + 1] for R, nu in slots]] * nb, np.int32)
    cr.fc2 = np.array([[bond[mu, nu, R] for R, nu in slots] for mu in range(nb)])[..., None]
    st = D.Setup(cr, (3, 2, 2), [300.0], **IDENT)
    ctx, _ = from_crystal(cr, (3, 2, 2), [300.0], with_fc3=False, **IDENT)
    ctx.compute_phonons([300.0])
    g = ctx.get_phonons(0)
    ctx.close()
    w = np.asarray(st.ph["omega"]).reshape(g["omega"].shape)
    assert w.min() > 0.0
    np.testing.assert_allclose(g["omega"] ** 2, w ** 2, rtol=0, atol=1e-12 * (w ** 2).max())
    e = g["evec"].reshape(-1, 3 * nb, 3 * nb)
    np.testing.assert_allclose(np.einsum("qsr,qtr->qst", e.conj(), e), np.broadcast_to(np.eye(3 * nb), e.shape), atol=1e-11)
