"""The stored tetrahedron operator of the iterative kappa: rows in segments, several batches of q0,
the form that is not stored, and cells with more than one pass over s0."""
import numpy as np
import pytest
import torch

from oracle import driver as D
from spring_b200 import _lib as L
from spring_b200 import synthetic as S
from spring_b200.api import from_crystal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cell,N,nT", [("rocksalt2", 3, 1), ("rocksalt2", 6, 2), ("rocksalt8", 3, 1)])
def test_kappa_iter_operator_matches_oracle(cell, N, nT):
    cr = S.build(cell)
    temps = [300.0, 700.0][:nT]
    st = D.Setup(cr, (N, N, N), temps)
    ctx, _ = from_crystal(cr, (N, N, N), temps, phonons={"grid": st.ph, "irr": st.ph0})
    out = ctx.kappa_iter(eps_k=1e-6)
    for it in range(nT):
        ref = D.bte_iter(st, it=it, eps_k=1e-6)
        scale = np.abs(ref["kappa_rta"]).max()
        np.testing.assert_allclose(out["kappa_rta"][it], ref["kappa_rta"], rtol=1e-9, atol=1e-9 * scale)
        assert abs(int(out["iters"][it]) - ref["iters"]) <= 1
        np.testing.assert_allclose(out["kappa"][it], ref["kappa"], rtol=1e-6, atol=1e-6 * np.abs(ref["kappa"]).max())
    ctx.close()


@pytest.mark.parametrize("N", [4, 9])
def test_kappa_iter_same_without_the_stored_operator(N):
    """9^3: several batches of q0, rows in several segments."""
    cr = S.build("rocksalt2")
    ctx, _ = from_crystal(cr, (N, N, N), [300.0, 700.0])
    a = ctx.kappa_iter(eps_k=1e-6, max_iter=12)
    again = ctx.kappa_iter(eps_k=1e-6, max_iter=12)          # the kept operator
    np.testing.assert_array_equal(again["kappa"], a["kappa"])
    ctx.set_option(L.SPRING_OPT_BTE_ENTRIES, 1000)
    b = ctx.kappa_iter(eps_k=1e-6, max_iter=12)
    assert np.array_equal(a["iters"], b["iters"])
    for key in ("kappa", "kappa_rta"):
        # the same terms in another order: rows of about 1e4 terms, FP64
        np.testing.assert_allclose(b[key], a[key], rtol=1e-10, atol=1e-10 * np.abs(a[key]).max())
    ctx.set_option(L.SPRING_OPT_BTE_ENTRIES, -1)
    one = ctx.kappa_iter(eps_k=1e-6, max_iter=0)             # a limit inside the first queued block
    assert np.all(one["iters"] == 1)
    np.testing.assert_allclose(one["kappa_rta"], a["kappa_rta"], rtol=1e-10, atol=1e-10 * np.abs(a["kappa_rta"]).max())
    ctx.close()


@pytest.mark.parametrize("N", [3, 7])
def test_kappa_iter_small_sets_without_the_stored_operator(N):
    """F in shared memory against the sums that are not stored."""
    cr = S.build("rocksalt2")
    ctx, _ = from_crystal(cr, (N, N, N), [300.0])
    a = ctx.kappa_iter(eps_k=1e-9, max_iter=5)
    ctx.set_option(L.SPRING_OPT_BTE_ENTRIES, 10)
    b = ctx.kappa_iter(eps_k=1e-9, max_iter=5)
    np.testing.assert_allclose(b["kappa"], a["kappa"], rtol=1e-10, atol=1e-10 * np.abs(a["kappa"]).max())
    ctx.close()


def test_kappa_iter_gauss_rebuilt_operator_gives_the_same_bits():
    """16^3: F (295 KB) does not fit shared memory, and the entries are appended in another order each time."""
    cr = S.build("rocksalt2")
    ctx, _ = from_crystal(cr, (16, 16, 16), [300.0])
    a = ctx.kappa_iter_gauss(0.7534, eps_k=1e-9, max_iter=3)
    ctx.compute_phonons([300.0])
    b = ctx.kappa_iter_gauss(0.7534, eps_k=1e-9, max_iter=3)
    assert a["entries"] == b["entries"] and a["iters"][0] == 4
    np.testing.assert_array_equal(b["kappa"], a["kappa"])
    ctx.close()


def test_kappa_iter_of_unsymmetrised_fc3_matches_oracle():
    """W of a pair of equal points is not symmetric in its branches then, and F does not vanish where q = -q."""
    cr = S.build("rocksalt2")
    cr.fc3 = cr.fc3 + np.random.default_rng(5).normal(0.0, 1.0, size=cr.fc3.shape)
    st = D.Setup(cr, (3, 3, 2), [300.0])
    ctx, _ = from_crystal(cr, (3, 3, 2), [300.0], phonons={"grid": st.ph, "irr": st.ph0})
    ref = D.bte_iter(st, eps_k=1e-6)
    for entries in (-1, 10):                                 # stored, and recomputed in every iteration
        ctx.set_option(L.SPRING_OPT_BTE_ENTRIES, entries)
        out = ctx.kappa_iter(eps_k=1e-6)
        np.testing.assert_allclose(out["kappa_rta"][0], ref["kappa_rta"], rtol=1e-9,
                                   atol=1e-9 * np.abs(ref["kappa_rta"]).max())
        np.testing.assert_allclose(out["kappa"][0], ref["kappa"], rtol=1e-6, atol=1e-6 * np.abs(ref["kappa"]).max())
    ctx.close()


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_kappa_iter_gives_a_large_operator_back_when_it_is_stale():
    """New phonons or FC3 make the stored operator useless: a large one does not keep its memory from later calls."""
    cr = S.build("rocksalt2")
    ctx, _ = from_crystal(cr, (12, 12, 12), [300.0])
    first = ctx.kappa_iter(eps_k=1e-3, max_iter=2)
    ctx.compute_phonons([300.0])
    base = _free()
    for stale in (lambda: ctx.compute_phonons([300.0]),
                  lambda: ctx.set_fc3(cr.fc3_atm_num, cr.fc3_atm_indx, cr.fc3)):
        again = ctx.kappa_iter(eps_k=1e-3, max_iter=2)
        held = base - _free()
        assert held > 128 << 20                              # the case is one: the operator is large
        stale()
        assert base - _free() < 16 << 20
        np.testing.assert_allclose(again["kappa"], first["kappa"], rtol=1e-10, atol=1e-10 * np.abs(first["kappa"]).max())
    ctx.close()
