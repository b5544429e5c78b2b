"""Performance cases of the phonon-scattering path, called as a user's program calls it.

Every case is one call (or the short sequence of calls of one run) of the public Python layer
(:class:`spring_b200.api.Context`) on a seeded rocksalt crystal of :mod:`spring_b200.synthetic`.
``prepare`` makes what a program has in hand before the call: the crystal and its force constants,
the context with its mesh, irreducible set and phonons, and the temperatures.  ``run`` is the call.
``exact`` gives the same results in 64 bits from plain numpy and torch.

Kinds of case:

* ``kappa``       one kappa.x run: phonons, 3-phonon linewidths, isotope rate, RTA kappa;
* ``lw3``         3-phonon linewidths of a block of irreducible q0 (phonons in hand);
* ``lw4``         4-phonon rates of a block of irreducible q0;
* ``iter``        one kappa_iter.x run: phonons, then the iterative kappa;
* ``path``        one LineWidth.x run: linewidths at off-grid points of a path;
* ``phonons``     harmonic phonons with the dipole-dipole term, and the kappa they give.
"""
import math

import numpy as np
import torch

from spring_b200 import synthetic as S
from spring_b200.api import from_crystal

SIGMA = 0.3767           # 2 cm^-1 in rad/ps, the Gaussian width of the benchmark workload
G2 = (1.0e-3, 1.0e-3)    # isotope mass variance per basis atom
IDENTITY = (np.eye(3, dtype=np.int32)[None], np.eye(3)[None])
_groups = {}


def _case(name, kind, cell, mesh, temps, **more):
    c = dict(name=name, kind=kind, cell=cell, n1=mesh[0], n2=mesh[1], n3=mesh[2], temps=temps, delta="gauss",
             precision="fp64", q0_first=1, n_q0=0, points=0, symmetry=True)
    c.update(more)
    return c


def listed():
    return [
        # a convergence test's first mesh: everything fits one wave, so launches and waits count
        _case("kappa_gauss_5", "kappa", 2, (5, 5, 5), 1),
        # the benchmark workload: 24^3, 100/300/700 K, tensor-core V3
        _case("kappa_gauss_bf16x3_24", "kappa", 2, (24, 24, 24), 3, precision="bf16x3"),
        # kappa.x with its own delta form, the linear tetrahedron
        _case("kappa_tetra_16", "kappa", 2, (16, 16, 16), 3, delta="tetra"),
        # FP64 linewidths over a temperature scan, the 20^3 member of the batched workload
        _case("lw3_gauss_20_9T", "lw3", 2, (20, 20, 20), 9),
        # a larger cell (8 atoms, 24 branches)
        _case("lw3_gauss_8atom_6", "lw3", 8, (6, 6, 6), 9),
        # one rank's block of q0 on an uneven mesh without rotations
        _case("lw3_tetra_8atom_654", "lw3", 8, (6, 5, 4), 3, delta="tetra", symmetry=False, q0_first=11, n_q0=8),
        # four-phonon rates, the reference's delta form (FP64), every irreducible q0
        _case("lw4_tetra_5", "lw4", 2, (5, 5, 5), 1, delta="tetra"),
        # four-phonon rates on the tensor cores, a block of q0 as a rank of a distributed run has
        _case("lw4_gauss_bf16x3_8", "lw4", 2, (8, 8, 8), 1, precision="bf16x3", q0_first=5, n_q0=6),
        # kappa_iter.x, tetrahedron form
        _case("iter_tetra_6", "iter", 2, (6, 6, 6), 2, delta="tetra"),
        # the iterative kappa with Gaussian deltas and the tensor-core operator
        _case("iter_gauss_bf16x3_12", "iter", 2, (12, 12, 12), 3, precision="bf16x3"),
        # LineWidth.x along a path
        _case("path_tetra_12", "path", 2, (12, 12, 12), 2, delta="tetra", points=24),
        # phonons of a polar crystal with a larger cell
        _case("phonons_polar_8atom_8", "phonons", 8, (8, 8, 8), 3),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _near(rng, m, lo):
    """A mesh around m, its sides different."""
    return tuple(max(lo, m - rng.randint(0, 2)) for _ in range(3))


def draw(rng):
    kind = rng.choice(("kappa", "kappa", "lw3", "lw3", "lw4", "iter", "path", "phonons"))
    temps = rng.randint(1, 9)
    if kind == "kappa":
        if rng.random() < 0.5:
            m = _log_int(rng, 4, 16)
            c = _case("", kind, 2, (m, m, m), min(temps, 3) if m > 12 else temps, delta="tetra")
        else:
            m = _log_int(rng, 4, 24)
            c = _case("", kind, 2, (m, m, m), temps, precision=rng.choice(("fp64", "bf16", "bf16x3")))
    elif kind == "lw3":
        cell, delta = rng.choice((2, 8)), rng.choice(("gauss", "tetra"))
        if cell == 8:
            mesh = _near(rng, rng.randint(4, 6), 2)
            block = rng.randint(1, 8)
        else:
            mesh = _near(rng, _log_int(rng, 4, 14), 2)
            block = rng.randint(1, 40)
        nq = mesh[0] * mesh[1] * mesh[2]
        block = min(block, nq)
        c = _case("", kind, cell, mesh, temps, delta=delta, symmetry=False, q0_first=rng.randint(1, nq - block + 1),
                  n_q0=block)
    elif kind == "lw4":
        if rng.random() < 0.5:
            c = _case("", kind, 2, tuple(rng.choice((3, 5)) for _ in range(3)), min(temps, 2), delta="tetra",
                      symmetry=False, q0_first=rng.randint(1, 20), n_q0=rng.randint(1, 6))
        else:
            m = rng.randint(4, 8)
            c = _case("", kind, 2, (m, m, m), temps, precision=rng.choice(("fp64", "bf16x3")),
                      q0_first=rng.randint(1, 3), n_q0=rng.randint(1, 5))
    elif kind == "iter":
        delta = rng.choice(("gauss", "tetra"))
        m = rng.randint(4, 6) if delta == "tetra" else rng.randint(8, 12)
        c = _case("", kind, 2, (m, m, m), rng.randint(1, 2), delta=delta,
                  precision="fp64" if delta == "tetra" else rng.choice(("fp64", "bf16x3")))
    elif kind == "path":
        m = rng.randint(6, 12)
        c = _case("", kind, 2, (m, m, m), temps, delta=rng.choice(("gauss", "tetra")), points=rng.randint(2, 24))
    else:
        m = rng.randint(3, 8)
        c = _case("", kind, rng.choice((2, 8)), (m, m, m), temps)
    del c["name"]
    return c


def _crystal(case, seed):
    cr = S.rocksalt_primitive() if case["cell"] == 2 else S.rocksalt_cubic()
    S.make_fc2(cr, seed=seed)
    if case["kind"] != "phonons":
        S.make_fc3(cr, seed=seed + 1000003)
    else:
        S.make_polar(cr)
    if case["kind"] == "lw4":
        S.make_fc4(cr, seed=seed + 2000003, iters=60)
    return cr


def _group(case):
    if not case["symmetry"]:
        return IDENTITY
    if case["cell"] not in _groups:
        _groups[case["cell"]] = S.point_group(S.rocksalt_primitive() if case["cell"] == 2 else S.rocksalt_cubic())
    return _groups[case["cell"]]


def _temps(case):
    return [100.0, 300.0, 700.0][: case["temps"]] if case["temps"] <= 3 else list(np.linspace(100.0, 900.0, case["temps"]))


def _path_points(case, cr, seed):
    """Points of a path through the zone in a direction of the seed's own, none of them on the grid."""
    d = np.random.default_rng(seed + 7).uniform(0.15, 0.45, 3)
    t = (np.arange(case["points"]) + 0.5) / case["points"]
    return t[:, None] * (cr.G @ d)[None, :]


def _lw_guess(case, nq0, seed):
    """Linewidths of a finished run (rad/ps), as a restart file gives them."""
    return np.random.default_rng(seed + 9).uniform(0.01, 0.5, (case["temps"], nq0, 3 * case["cell"]))


def _block(case, nq0):
    first = min(case["q0_first"], nq0)
    return first, min(case["n_q0"] or nq0, nq0 - first + 1)


def prepare(case, seed):
    cr = _crystal(case, seed)
    W, R = _group(case)
    temps = _temps(case)
    polar = dict(rmesh=(5, 5, 5)) if case["kind"] == "phonons" else None
    ctx, info = from_crystal(cr, (case["n1"], case["n2"], case["n3"]), temps, W=W, Rxyz=R,
                             with_fc3=case["kind"] != "phonons", with_fc4=case["kind"] == "lw4", dipole=polar)
    ctx.set_precision(case["precision"])
    st = dict(case=case, ctx=ctx, Rxyz=info["Rxyz"], temps=temps, q0=_block(case, ctx.nq0))
    if case["kind"] == "path":
        st["points"] = _path_points(case, cr, seed)
        st["zero_centred"] = np.ones(case["points"], np.int32)
    if case["kind"] == "phonons":
        st["lw"] = _lw_guess(case, ctx.nq0, seed)
    if case["kind"] in ("lw3", "kappa"):
        ctx.prepare3()
    ctx.synchronize()
    return st


def run(st):
    case, ctx = st["case"], st["ctx"]
    kind, delta = case["kind"], case["delta"]
    first, count = st["q0"]
    if kind == "kappa":
        ctx.compute_phonons(st["temps"])
        ctx.reset_linewidths()
        lw, p3 = ctx.linewidth3(1, ctx.nq0, delta, SIGMA)
        iso = ctx.linewidth_iso(1, ctx.nq0, G2, delta, SIGMA)
        return dict(lw=lw, p3=p3, iso=iso, kappa=ctx.kappa_rta(st["Rxyz"]))
    if kind == "lw3":
        lw, p3 = ctx.linewidth3(first, count, delta, SIGMA)
        return dict(lw=lw, p3=p3)
    if kind == "lw4":
        return dict(rate=ctx.linewidth4(first, count, delta, SIGMA))
    if kind == "iter":
        ctx.compute_phonons(st["temps"])
        r = ctx.kappa_iter(1e-6, 200) if delta == "tetra" else ctx.kappa_iter_gauss(2 * SIGMA, 1e-6, 200)
        return dict(kappa=r["kappa"], kappa_rta=r["kappa_rta"], iters=r["iters"])
    if kind == "path":
        lw, om = ctx.linewidth_path(st["points"], st["zero_centred"], delta, SIGMA)
        return dict(lw=lw, omega=om)
    ctx.compute_phonons(st["temps"])
    ctx.set_linewidths(st["lw"])
    ph = ctx.get_phonons(1)
    kap, mode = ctx.kappa_rta(symm=False, mode=True)
    return dict(omega=ph["omega"], vel=ph["grp_vel"], nbe=ph["nbe"], kappa=kap, mode=mode)


def _nq0(case, nq):
    return max(1, nq // 36) if case["symmetry"] else nq


def work(case):
    n, nT = 3 * case["cell"], case["temps"]
    nq = case["n1"] * case["n2"] * case["n3"]
    kind = case["kind"]
    v3 = 4 * 27 * case["cell"] * 49 + 24 * n ** 4 + 3 * n ** 3           # flops of one pair's matrix elements
    delta = n ** 3 * (20 if case["delta"] == "gauss" else 6 * 18 * 4)    # window tests of one grid point's triples
    modes = 8 * nq * n * (2 + nT) + 16 * nq * n * n                      # frequencies, occupations, eigenvectors
    eig = nq / 2 * 60 * n ** 3
    if kind in ("kappa", "lw3"):
        n0 = _nq0(case, nq) if kind == "kappa" or not case["n_q0"] else case["n_q0"]
        return dict(bytes=modes + 8 * n0 * n * nT, flops=n0 * nq * (v3 / 2 + delta) + (eig if kind == "kappa" else 0))
    if kind == "lw4":
        n0 = case["n_q0"] or _nq0(case, nq)
        v4 = 4 * 81 * case["cell"] * 343 + 32 * n ** 5
        return dict(bytes=modes + 8 * n0 * n * nT, flops=n0 * nq * nq * (v4 / 6 + n * delta))
    if kind == "iter":
        return dict(bytes=modes + 72 * nT, flops=nq / 2 * nq * (v3 / 2 + delta) + eig)
    if kind == "path":
        return dict(bytes=modes + 8 * case["points"] * n * nT, flops=case["points"] * nq * (v3 + 2 * delta + 60 * n ** 3))
    return dict(bytes=modes + 24 * nq * n, flops=eig + nq / 2 * 250 * case["cell"] ** 2 * 90)


# ---- the same results in 64 bits -----------------------------------------------------------------

PI = math.pi
W_THZ = math.sqrt(1.60217733 * 6.02214076 * 10.0) * 10.0
VG_MS = W_THZ * 100.0
BE = math.sqrt(1.60217733 * 6.02214076 * 10.0) * 6.582119569 * 100.0 / 8.617333262
SCTR3 = 1.054571817 * 1.60217733 ** 2 * 6.02214076 ** 3 * 1.0e6 * PI * 0.0625
SCTR4 = 0.125 * PI * (1.054571817 * 1.602176565) ** 2 * 6.022140857 ** 4 * 1.0e6
KW_MK = 1.054571817 ** 2 * 0.001 / 1.380649
E2_EVA = (1.602176634 * 2.99792458) ** 2 * 6.241509074460763 * 0.1
RS2PI = 0.3989422804014327


def _t(x):
    return torch.as_tensor(np.ascontiguousarray(x), device="cuda" if torch.cuda.is_available() else "cpu")


def _mesh(case, cr):
    """Grid addresses folded around zero (first index fastest) and their Cartesian vectors."""
    n = np.array([case["n1"], case["n2"], case["n3"]])
    g = np.arange(n.prod())
    v = np.stack([g % n[0], g // n[0] % n[1], g // (n[0] * n[1])], 1)
    v = np.where(v > n // 2, v - n, v)
    return v, (v / n) @ cr.G.T


def _index(case, v):
    n = (case["n1"], case["n2"], case["n3"])
    return v[..., 0] % n[0] + n[0] * (v[..., 1] % n[1] + n[1] * (v[..., 2] % n[2]))


def _irreducible(case, v):
    """(grid index of each irreducible point, slot of each grid point): smallest index of each orbit."""
    W = _group(case)[0].astype(np.int64)
    rep = np.min(np.stack([_index(case, v @ w) for w in W] + [np.arange(len(v))]), 0)
    irr = np.unique(rep)
    return irr, np.searchsorted(irr, rep)


def _tetrahedra(case):
    n = np.array([case["n1"], case["n2"], case["n3"]])
    g = np.arange(n.prod())
    base = np.stack([g % n[0], g // n[0] % n[1], g // (n[0] * n[1])], 1)
    box = np.array([[0, 0, 0], [1, 0, 0], [0, 0, 1], [0, 1, 1], [1, 0, 1], [1, 1, 1], [1, 1, 0], [0, 1, 0]])
    corner = _index(case, base[:, None, :] + box[None])
    six = np.array([[0, 1, 2, 3], [2, 3, 4, 1], [5, 3, 4, 1], [5, 3, 6, 1], [6, 3, 7, 1], [0, 3, 7, 1]])
    return corner[:, six].reshape(-1, 4)


def _ewald(cr, q):
    """The dipole-dipole matrix and its gradient (before the masses) at points q, without the constant part."""
    eps, eps_i, tau, Z = cr.eps, np.linalg.inv(cr.eps), cr.tau(), cr.zstar
    p = -math.log(1e-6)
    rc = cr.latvec @ np.array([5 // 2 + 1, 0.0, 0.0])
    D = math.sqrt(rc @ eps_i @ rc)
    lmb = math.sqrt(p) / D
    nk = math.ceil(2.0 * p / (D * math.sqrt(np.trace(eps) / 3.0)) / np.linalg.norm(cr.G[:, 0]))

    def points(cell, m):
        x = np.arange(m) - m // 2
        return np.stack(np.meshgrid(x, x, x, indexing="ij"), -1).reshape(-1, 3) @ cell.T

    R, Gp = points(cr.latvec, 5), points(cr.G, 2 * nk + 1)
    t = tau[:, None] - tau[None]
    dv = R[:, None, None] - t[None]
    zero = np.all(np.abs(dv) < 1e-8, -1)
    de = lmb * dv @ eps_i
    ld = np.sqrt(np.einsum("rmnk,rmnk->rmn", de, dv) * lmb) + zero
    erfc = torch.special.erfc(torch.as_tensor(ld)).numpy()
    pe = 2.0 / math.sqrt(PI) * np.exp(-ld * ld)
    h1 = (3.0 * erfc / ld ** 3 + pe * (3.0 / ld ** 2 + 2.0)) / ld ** 2
    h2 = erfc / ld ** 3 + pe / ld ** 2
    H = np.einsum("rmna,rmnb->rmnab", de, de) * h1[..., None, None] - eps_i * h2[..., None, None]
    H[zero] = 0.0
    H = _t(H * lmb ** 3 / math.sqrt(np.linalg.det(eps))).to(torch.complex128)
    ph = np.exp(1j * q @ R.T)
    real = [torch.einsum("qr,rmnab->qmnab", _t(ph), H)]
    real += [torch.einsum("qr,rmnab->qmnab", _t(1j * ph * R[:, k]), H) for k in range(3)]
    K = q[:, None] + Gp[None]
    kek = np.einsum("qgi,ij,qgj->qg", K, eps, K)
    none = kek < 1e-14
    kg = np.where(none, 0.0, np.exp(-kek / (4 * lmb ** 2)) / np.where(none, 1.0, kek))
    kp = np.where(none, 0.0, 1.0 / np.where(none, 1.0, kek)) + 0.25 / lmb ** 2
    eK = K @ (eps + eps.T)
    tp, Kt, kgt = _t(t), _t(K), _t(kg)
    kmn = kgt[:, :, None, None] * torch.exp(1j * torch.einsum("qgk,mnk->qgmn", Kt, tp))
    Kc = Kt.to(torch.complex128)
    rec = [torch.einsum("qgmn,qga,qgb->qmnab", kmn, Kc, Kc)]
    for k in range(3):
        f = kmn * (1j * tp[None, None, :, :, k] - _t(eK[..., k] * kp)[:, :, None, None])
        d = torch.einsum("qgmn,qga,qgb->qmnab", f, Kc, Kc)
        s = torch.einsum("qgmn,qgb->qmnb", kmn, Kc)
        d[:, :, :, k, :] += s
        d[:, :, :, :, k] += s
        rec.append(d)
    cc = _t(np.einsum("mn,ab->mnab", np.eye(cr.nbasis), eps_i * 4 * lmb ** 3 / (3 * math.sqrt(PI * np.linalg.det(eps)))))
    Zt = _t(Z).to(torch.complex128)
    out = []
    for k in range(4):
        c = rec[k] * (4 * PI / cr.vol) - real[k] - (cc if k == 0 else 0.0)
        out.append(torch.einsum("mia,qmnij,njb->qmnab", Zt, c, Zt))
    return torch.stack(out).cpu().numpy()


def _dipole(cr, q):
    """D_ew and dD_ew/dq at points q; the non-analytic term along the next point of the list at q = 0."""
    nb, n = cr.nbasis, cr.ndof
    rs = np.repeat(1.0 / np.sqrt(cr.mass), 3)
    self_term = _ewald(cr, np.zeros((1, 3)))[0, 0].sum(1)

    def dyn(p):
        c = _ewald(cr, p)
        for m in range(nb):
            c[0, :, m, m] -= self_term[m]
        return c.transpose(0, 1, 2, 4, 3, 5).reshape(4, len(p), n, n) * E2_EVA * rs[:, None] * rs[None]

    out = np.concatenate([dyn(q[i:i + 64]) for i in range(0, len(q), 64)], 1)
    for i in np.flatnonzero(np.all(np.abs(q) < 1e-8, 1)):
        qh = q[i + 1] - q[i] if i + 1 < len(q) else q[i] - q[i - 1]
        h = np.linalg.norm(qh) / 8.0
        z = np.einsum("k,mak->ma", qh, cr.zstar).reshape(n) * rs
        out[0, i] += np.outer(z, z) * 4 * PI * E2_EVA / (cr.vol * (qh @ cr.eps @ qh))
        d = dyn(np.concatenate([0.5 * h * np.eye(3), -0.5 * h * np.eye(3)]))[0]
        out[1:, i] = (d[:3] - d[3:]) / h
    return out


def _phonons(cr, q, temps, polar=False):
    """omega, 1/omega, e [q][s][row], nBE [T][q][s] and velocities at points q."""
    n, rs = cr.ndof, 1.0 / np.sqrt(cr.mass)
    D = np.zeros((4, len(q), n, n), complex)
    for mu in range(cr.nbasis):
        for N in range(cr.fc2_atm_num[mu]):
            R = cr.latvec @ cr.fc2_atm_indx[mu, N, :3]
            nu = cr.fc2_atm_indx[mu, N, 3] - 1
            x = np.exp(1j * q @ R)[:, None, None] * (cr.fc2[mu, N, :, :, 0] * rs[mu] * rs[nu])
            for k, f in enumerate((1.0, 1j * R[0], 1j * R[1], 1j * R[2])):
                D[k, :, 3 * mu:3 * mu + 3, 3 * nu:3 * nu + 3] += f * x
    if polar:
        D += _dipole(cr, q)
    lam, v = np.linalg.eigh(D[0], UPLO="U")
    w = np.sqrt(np.abs(lam)) * np.where((lam < 0) & (np.abs(lam) > 1e-8), -1.0, 1.0)
    gamma = np.all(np.abs(q) < 1e-8, 1)
    zero = gamma[:, None] & (np.arange(n) < 3)
    with np.errstate(all="ignore"):
        vel = np.stack([np.einsum("qis,qij,qjs->qs", v.conj(), D[k], v, optimize=True).real for k in (1, 2, 3)], -1)
        vel = np.where(zero[..., None], 0.0, vel / (2 * w[..., None]) * VG_MS)
        one = np.where(zero, 0.0, 1.0 / (w * W_THZ))
        nbe = np.stack([np.where(zero, 0.0, 1.0 / np.expm1(BE * np.abs(w) / T)) for T in temps])
    return dict(om=w * W_THZ, one=one, ev=v.transpose(0, 2, 1), nbe=nbe, vel=vel, gamma=gamma)


def _legs(cr, num, idx, q, ph):
    """u[q][mu][(N, beta)][s] = m^-1/2 e(nu beta, s) exp(i q R) of every neighbour slot."""
    na = idx.shape[1]
    R = idx[..., :3] @ cr.latvec.T
    nu = idx[..., 3] - 1
    on = np.arange(na)[None] < num[:, None]
    f = np.exp(1j * np.einsum("qk,mnk->qmn", q, R)) * on / np.sqrt(cr.mass[nu])
    e = ph["ev"].reshape(len(q), -1, cr.nbasis, 3)[:, :, nu]
    return _t(np.einsum("qmn,qsmnb->qmnbs", f, e).reshape(len(q), cr.nbasis, na * 3, -1))


class _Crystal3:
    """W3 of one q0 against a batch of (q1, q2)."""

    def __init__(self, cr, nq):
        self.cr, self.scale = cr, SCTR3 / nq
        na = cr.fc3.shape[1]
        self.f = _t(cr.fc3.transpose(0, 3, 1, 4, 2, 5).reshape(cr.nbasis, 9 * na, 3 * na)).to(torch.complex128)
        self.mu = 1.0 / np.sqrt(cr.mass)

    def w(self, e0, one0, zero0, u1, one1, zero1, u2, one2, zero2):
        nb, n, B = self.cr.nbasis, self.cr.ndof, len(u1)
        phi = torch.zeros((B, n, n * n), dtype=torch.complex128, device=u1.device)
        for m in range(nb):
            y = (self.f[m] @ u2[:, m]).reshape(B, 3, -1, n)
            z = (u1[:, None, m].transpose(2, 3) @ y).reshape(B, 3, n * n)
            phi += (_t(e0[:, 3 * m:3 * m + 3] * self.mu[m]) @ z)
        W = phi.reshape(B, n, n, n).abs() ** 2 * self.scale
        W *= one0[None, :, None, None] * one1[:, None, :, None] * one2[:, None, None, :]
        return W.masked_fill(zero0[None, :, None, None] | zero1[:, None, :, None] | zero2[:, None, None, :], 0.0)


def _corner_weights(x, M, strict):
    """g and I[4] (by vertex) of tetrahedra with vertex energies M[..., 4] at energy x; used[...]."""
    S_, p = torch.sort(M, dim=-1, stable=True)
    m0, m1, m2, m3 = S_.unbind(-1)
    if strict:
        c1, c2, c3 = (x > m0) & (x < m1), (x > m1) & (x < m2), (x > m2) & (x < m3)
    else:
        c1, c2, c3 = (x >= m0) & (x < m1), (x >= m1) & (x < m2), (x >= m2) & (x <= m3)
    f = lambda a, b: (x - b) / (a - b)  # noqa: E731
    g1 = 3 * (x - m0) ** 2 / ((m1 - m0) * (m2 - m0) * (m3 - m0))
    g2 = 3 / ((m1 - m2) * (m3 - m0)) * ((x - m0) * (x - m2) / (m2 - m0) - (x - m1) * (x - m3) / (m1 - m3))
    g3 = 3 * (x - m3) ** 2 / ((m3 - m0) * (m3 - m1) * (m3 - m2))
    d = g2 * (m3 - m0)
    i1 = (f(m0, m1) + f(m0, m2) + f(m0, m3), f(m1, m0), f(m2, m0), f(m3, m0))
    i2 = (f(m0, m3) + 3 * f(m0, m2) * f(m2, m0) * f(m1, m2) / d, f(m1, m2) + 3 * f(m1, m3) ** 2 * f(m2, m1) / d,
          f(m2, m1) + 3 * f(m2, m0) ** 2 * f(m1, m2) / d, f(m3, m0) + 3 * f(m3, m1) * f(m1, m3) * f(m2, m1) / d)
    i3 = (f(m0, m3), f(m1, m3), f(m2, m3), f(m3, m0) + f(m3, m1) + f(m3, m2))
    g = torch.where(c1, g1, torch.where(c2, g2, torch.where(c3, g3, torch.zeros_like(g1))))
    I = torch.stack([torch.where(c1, a, torch.where(c2, b, torch.where(c3, c, torch.zeros_like(g1)))) / 3
                     for a, b, c in zip(i1, i2, i3)], -1)
    return g, torch.empty_like(I).scatter_(-1, p.expand_as(I), I), c1 | c2 | c3


def _no_nan(x):
    return torch.where(torch.isnan(x), 0.0, x)


def _delta(d, sigma):
    return torch.exp(-0.5 * (d / sigma) ** 2) * (RS2PI / sigma)


class _Three:
    """The 3-phonon sums of one mesh: W3 of a q0 with every grid q1, and its delta sums."""

    def __init__(self, case, cr, temps):
        self.case, self.cr, self.temps = case, cr, temps
        self.v, self.q = _mesh(case, cr)
        self.nq = len(self.v)
        self.ph = _phonons(cr, self.q, temps)
        self.W = _Crystal3(cr, self.nq)
        self.u = _legs(cr, cr.fc3_atm_num, cr.fc3_atm_indx, self.q, self.ph)
        self.om, self.one, self.nbe = _t(self.ph["om"]), _t(self.ph["one"]), _t(self.ph["nbe"])
        self.zero = _t(self.ph["gamma"][:, None] & (np.arange(cr.ndof) < 3))
        self.tet = _t(_tetrahedra(case)) if case["delta"] == "tetra" else None

    def partner(self, g0):
        return _index(self.case, -(self.v[g0][None] + self.v))

    def w3(self, g0, part):
        step = max(1, (1 << 27) // (self.cr.ndof ** 3 * 16))
        p, out = _t(part), []
        for i in range(0, self.nq, step):
            s = slice(i, i + step)
            out.append(self.W.w(self.ph["ev"][g0], self.one[g0], self.zero[g0], self.u[s], self.one[s], self.zero[s],
                                self.u[p[s]], self.one[p[s]], self.zero[p[s]]))
        return torch.cat(out)

    def gauss(self, w0, W, om2, n2, zero2, sigma):
        """(lw [T][s0], phase space [s0])"""
        w0, w1, w2 = w0[None, :, None, None], self.om[:, None, :, None], om2[:, None, None, :]
        out = (self.zero[:, None, :, None] | zero2[:, None, None, :]).expand(-1, len(W[0]), -1, -1)
        e1 = _delta(w0 - w1 - w2, sigma).masked_fill(out, 0.0)
        e2 = _delta(w0 + w1 - w2, sigma).masked_fill(out, 0.0)
        e3 = _delta(w0 - w1 + w2, sigma).masked_fill(out, 0.0)
        lw = [((W * ((a[:, None, :, None] + b[:, None, None, :] + 1) * e1
                     + (a[:, None, :, None] - b[:, None, None, :]) * (e2 - e3))).sum((0, 2, 3)))
              for a, b in zip(self.nbe, n2)]
        return torch.stack(lw), (e1 + e2 + e3).sum((0, 2, 3))

    def tetra(self, w0, W, om2, n2, strict=False):
        nT, n = len(self.temps), self.cr.ndof
        lw = torch.zeros((nT, n), dtype=torch.float64, device=W.device)
        p3 = torch.zeros(n, dtype=torch.float64, device=W.device)
        step = max(1, (1 << 24) // n ** 3)
        for i in range(0, len(self.tet), step):
            t = self.tet[i:i + step]
            o1, o2 = self.om[t][:, None, :, :, None], om2[t][:, None, :, None, :]
            for M, sg, ch in ((o1 + o2, 1.0, 0), (o2 - o1, 1.0, 1), (o1 - o2, -1.0, 1)):
                M = M.permute(0, 1, 3, 4, 2)
                g, I, _ = _corner_weights(w0[None, :, None, None], M, strict)
                p3 += g.sum((0, 2, 3))
                I *= (g * (sg / 6))[..., None]
                for v in range(4):
                    Iw = I[..., v] * W[t[:, v]]
                    for T in range(nT):
                        a, b = self.nbe[T][t[:, v]][:, None, :, None], n2[T][t[:, v]][:, None, None, :]
                        lw[T] += (Iw * (a + b + 1 if ch == 0 else a - b)).sum((0, 2, 3))
        return lw, p3

    def linewidth(self, g0):
        part = self.partner(g0)
        W, p = self.w3(g0, part), _t(part)
        if self.case["delta"] == "tetra":
            return self.tetra(self.om[g0], W, self.om[p], self.nbe[:, p])
        return self.gauss(self.om[g0], W, self.om[p], self.nbe[:, p], self.zero[p], SIGMA)


def _isotope(th, g0):
    cr, n = th.cr, th.cr.ndof
    e = _t(th.ph["ev"]).reshape(th.nq, n, cr.nbasis, 3)
    d = torch.einsum("qsbc,tbc->qtsb", e.conj(), e[g0])
    w0 = th.om[g0]
    W = (d.abs() ** 2 @ _t(np.array(G2))) * PI * w0[None, :, None] ** 2 * 0.5 / th.nq  # [q1][s0][s1]
    if th.tet is None:
        return (W * _delta(w0[None, :, None] - th.om[:, None, :], SIGMA)).sum((0, 2))
    g, I, _ = _corner_weights(w0[None, :, None], th.om[th.tet][:, None].permute(0, 1, 3, 2), False)
    I, g = _no_nan(I), _no_nan(g)
    return sum((I[..., v] * g / 6 * W[th.tet[:, v]]).sum((0, 2)) for v in range(4))


def _kappa_sum(om, nbe, lw, vel, weight, T, vol, nq, skip):
    """[s][9] contributions to kappa at one temperature; weight: [q][s][3][3] of v (x) v."""
    pre = np.where(skip, 0.0, om ** 2 * nbe * (nbe + 1.0) * 0.5 / lw)
    return (pre[..., None, None] * weight).sum(0).reshape(-1, 9) * KW_MK / (T * T * vol) / nq


def _exact_kappa(case, cr, temps):
    th = _Three(case, cr, temps)
    irr, slot = _irreducible(case, th.v)
    mult = np.bincount(slot)
    lw, p3, iso = [], [], []
    for g0 in irr:
        a, b = th.linewidth(int(g0))
        lw.append(a)
        p3.append(b)
        iso.append(_isotope(th, int(g0)))
    lw = torch.stack(lw, 1).cpu().numpy()
    iso = np.repeat(torch.stack(iso).cpu().numpy()[None], len(temps), 0)
    R = _group(case)[1]
    vel = th.ph["vel"][irr]
    rv = np.einsum("rij,qsj->qsri", R, vel)
    vv = np.einsum("qsri,qsrj->qsij", rv, rv) / (len(R) // mult)[:, None, None, None]
    tot = lw + 0.5 * iso
    skip = th.ph["gamma"][irr][:, None] & (np.arange(cr.ndof) < 3)
    with np.errstate(all="ignore"):
        kap = [_kappa_sum(th.ph["om"][irr], th.ph["nbe"][T][irr], tot[T], vel, vv, temps[T], cr.vol, th.nq, skip).sum(0)
               for T in range(len(temps))]
    return dict(lw=lw, p3=torch.stack(p3).cpu().numpy(), iso=iso, kappa=np.stack(kap))


def _exact_lw3(case, cr, temps):
    th = _Three(case, cr, temps)
    irr, _ = _irreducible(case, th.v)
    first, count = _block(case, len(irr))
    r = [th.linewidth(int(g)) for g in irr[first - 1:first - 1 + count]]
    return dict(lw=torch.stack([x[0] for x in r], 1).cpu().numpy(), p3=torch.stack([x[1] for x in r]).cpu().numpy())


def _orderings(nq, g1, g2, g3):
    """Which of its set's orderings a cell (q1, q2) is: 0 the first in grid order, else 1.. as listed here."""
    per = np.array([[0, 1, 2], [0, 2, 1], [1, 0, 2], [1, 2, 0], [2, 0, 1], [2, 1, 0]])
    cell = np.stack([g1, g2, g3], 1)
    keys = np.stack([cell[:, p[0]] * nq + cell[:, p[1]] for p in per], 1)
    rep = np.take_along_axis(cell, per[np.argmin(keys, 1)], 1)
    typ = np.zeros(len(cell), int)
    for t in range(5, -1, -1):
        typ[np.all(rep[:, per[t]] == cell, 1)] = t
    return typ


def _at_vertices(x, tt, n, k):
    """Values x[q][s] at the vertices tt[t][4], as [t][s0 1][s1 1][s2][s3][4] with s at place k."""
    y = x[tt].transpose(1, 2)
    return y.reshape(len(tt), 1, 1, n if k == 1 else 1, n if k == 2 else 1, 4)


def _exact_lw4(case, cr, temps):
    v, q = _mesh(case, cr)
    nq, n, nT = len(v), cr.ndof, len(temps)
    irr, _ = _irreducible(case, v)
    first, count = _block(case, len(irr))
    ph = _phonons(cr, q, temps)
    u = _legs(cr, cr.fc4_atm_num, cr.fc4_atm_indx, q, ph)
    na = cr.fc4.shape[1]
    f = _t(cr.fc4.transpose(0, 4, 1, 5, 2, 6, 3, 7).reshape(2, -1, 3 * na)).to(torch.complex128)
    om, one, nbe = _t(ph["om"]), _t(ph["one"]), _t(ph["nbe"])
    tet = _t(_tetrahedra(case))
    zero = _t(ph["gamma"][:, None] & (np.arange(n) < 3))
    rate = torch.zeros((nT, count, n), dtype=torch.float64, device=om.device)
    shape = lambda x, k: x.reshape(x.shape[0], *[n if i == k else 1 for i in range(4)])  # noqa: E731
    y3 = torch.stack([f[m] @ u[:, m] for m in range(2)], 1).reshape(nq, 2, -1, 3 * na, n)  # [q3][mu][a N1b][N2c][s3]
    for k, g0 in enumerate(irr[first - 1:first - 1 + count]):
        s0 = 3 if ph["gamma"][g0] else 0
        e0 = ph["ev"][g0]
        for g1 in range(nq):
            g2 = np.arange(nq)
            g3 = _index(case, -(v[g0] + v[g1] + v))
            t3 = _t(g3)
            phi = torch.zeros((nq, n, n ** 3), dtype=torch.complex128, device=om.device)
            for m in range(2):
                z = u[:, None, m].transpose(2, 3) @ y3[t3, m]                        # [q][a N1b][s2][s3]
                z = u[g1, m].T @ z.reshape(nq, 3, 3 * na, n * n)                     # [q][a][s1][s2 s3]
                phi += _t(e0[:, 3 * m:3 * m + 3] / math.sqrt(cr.mass[m])) @ z.reshape(nq, 3, n ** 3)
            W = phi.reshape(nq, n, n, n, n).abs() ** 2 * (SCTR4 / nq / nq)
            W *= one[g0][None, :, None, None, None] * shape(one[g1][None], 1) * shape(one, 2) * shape(one[t3], 3)
            W = W.masked_fill(zero[g0][None, :, None, None, None] | shape(zero[g1][None], 1) | shape(zero, 2)
                              | shape(zero[t3], 3), 0.0)
            w1, w2, w3 = shape(om[g1][None], 1), shape(om, 2), shape(om[t3], 3)
            w0 = om[g0][None, :, None, None, None]
            fac = []
            for T in range(nT):
                a, b, c = shape(nbe[T][g1][None], 1), shape(nbe[T], 2), shape(nbe[T][t3], 3)
                n0 = nbe[T][g0][None, :, None, None, None]
                fac.append((a * b * c / n0 / 6, (1 + a) * b * c / n0 / 2, (1 + a) * (1 + b) * c / n0 / 2))
            if case["delta"] == "gauss":
                for ch, M in enumerate((w1 + w2 + w3, w2 + w3 - w1, w3 - w1 - w2)):
                    Wd = W * _delta(w0 - M, SIGMA)
                    for T in range(nT):
                        rate[T, k, s0:] += (Wd * fac[T][ch])[:, s0:].sum((0, 2, 3, 4))
                continue
            # the W of a cell is read through its set's first ordering with the two 3-cycles' branches turned
            typ = _t(_orderings(nq, np.full(nq, g1), g2, g3))
            for t, turn in ((3, (2, 0, 1)), (4, (1, 2, 0))):
                at = torch.nonzero(typ == t)[:, 0]
                # slot k of the cell's own W holds branch (s1, s2, s3)[turn[k]]
                inv = [turn.index(j) for j in range(3)]
                W[at] = W[at].permute(0, 1, 2 + inv[0], 2 + inv[1], 2 + inv[2])
            for i in range(0, len(tet), 4096):
                tt = tet[i:i + 4096]
                x2, x3 = _at_vertices(om, tt, n, 1), _at_vertices(om[t3], tt, n, 2)
                x1 = om[g1].reshape(1, 1, n, 1, 1, 1)
                for ch, M in enumerate((x1 + x2 + x3, x2 + x3 - x1, x3 - x1 - x2)):
                    g, I, used = _corner_weights(om[g0].reshape(1, n, 1, 1, 1), M, False)
                    gI = torch.where(used[..., None], _no_nan(I) * _no_nan(g)[..., None] / 6, 0.0)
                    for T in range(nT):
                        F = W * fac[T][ch]
                        s = sum((gI[..., c] * F[tt[:, c]]).sum((0, 2, 3, 4)) for c in range(4))
                        rate[T, k, s0:] += s[s0:]
    return dict(rate=rate.cpu().numpy())


def _exact_iter(case, cr, temps):
    th = _Three(case, cr, temps)
    nq, n = th.nq, cr.ndof
    neg = _index(case, -th.v)
    rep = np.minimum(np.arange(nq), neg)
    tr = np.unique(rep)
    slot, sign = np.searchsorted(tr, rep), np.where(rep == np.arange(nq), 1.0, -1.0)
    deg = np.bincount(slot)
    dev = th.om.device
    negt = _t(neg)
    ops = []  # per q0: (plus, minus) weights times 4 W at [q1][s0][s1][s2]
    for g0 in tr:
        part = th.partner(int(g0))
        p = _t(part)
        W = 4.0 * th.w3(int(g0), part)
        w0 = th.om[g0]
        if case["delta"] == "gauss":
            a, b, c = th.om[:, None, :, None], th.om[p][:, None, None, :], w0[None, :, None, None]
            cut = lambda d: torch.where((d / (2 * SIGMA)) ** 2 < 80.0, _delta(d, 2 * SIGMA), 0.0)  # noqa: E731
            ops.append((W * cut(c + a - b), 0.5 * W * cut(c - a - b)))
            continue
        PQ = [torch.zeros((nq, n, n, n), dtype=torch.float64, device=dev) for _ in range(2)]
        o1, o2 = th.om[th.tet][:, None, :, :, None], th.om[negt[p]][th.tet][:, None, :, None, :]
        o3 = th.om[negt[p[negt]]][th.tet][:, None, :, None, :]
        for ch, M in enumerate((o2 - o1, o1 + o3)):
            g, I, used = _corner_weights(w0[None, :, None, None], M.permute(0, 1, 3, 4, 2), True)
            used = used & ((I.sum(-1) - 1.0).abs() < 5.0e-5)
            for v in range(4):
                x = th.tet[:, v] if ch == 0 else negt[th.tet[:, v]]
                PQ[ch].index_add_(0, x, torch.where(used, g * I[..., v] * ((1.0 if ch == 0 else 0.5) / 6), 0.0))
        ops.append((PQ[0] * W, PQ[1] * W))
    om, nbe, vel = th.ph["om"][tr], th.ph["nbe"][:, tr], th.ph["vel"][tr]
    skip = th.ph["gamma"][tr][:, None] & (np.arange(n) < 3)
    kappa, rta, iters = [], [], []
    for T, temp in enumerate(temps):
        N = th.nbe[T]
        A = torch.zeros((len(tr) * n, nq * n), dtype=torch.float64, device=dev)
        inv_tau = torch.zeros((len(tr), n), dtype=torch.float64, device=dev)
        for i, g0 in enumerate(tr):
            p = _t(th.partner(int(g0)))
            a, b = N[:, None, :, None], N[p][:, None, None, :]
            c = (a - b) * ops[i][0] + (1.0 + a + b) * ops[i][1]
            inv_tau[i] = c.sum((0, 2, 3))
            at = A[i * n:(i + 1) * n].reshape(n, nq, n)
            at += c.sum(3).transpose(0, 1)
            at.index_add_(1, p, c.sum(2).transpose(0, 1))
        it = inv_tau.cpu().numpy()
        live = ~skip & (np.abs(it) > 5.0e-5)
        div = np.where(live, it, 1.0)[..., None]
        F0 = np.where(live[..., None], 1.054571817 / 1.380649 * om[..., None] * vel / (div * temp * temp), 0.0)
        pre = np.where(skip, 0.0, deg[:, None] * om * nbe[T] * (nbe[T] + 1.0)) * 1.054571817e-3 / (nq * cr.vol)

        def kap(F):
            return np.einsum("qs,qsi,qsj->ij", pre, vel, F).reshape(9)

        F, old, count = F0, kap(F0), 0
        rta.append(old)
        while True:
            count += 1
            grid = (sign[:, None, None] * F[slot]).reshape(nq * n, 3)
            F = F0 - (A @ _t(grid)).cpu().numpy().reshape(F.shape) / div
            new = kap(F)
            if np.abs(new - old).max() < 1e-6 or count > 200:
                break
            old = new
        kappa.append(new)
        iters.append(count)
    return dict(kappa=np.stack(kappa), kappa_rta=np.stack(rta), iters=np.array(iters, np.int32))


def _exact_path(case, cr, temps, seed):
    th = _Three(case, cr, temps)
    pts = _path_points(case, cr, seed)
    p0 = _phonons(cr, pts, temps)
    lw = []
    for i in range(len(pts)):
        q2 = -(pts[i][None] + th.q)
        p2 = _phonons(cr, q2, temps)
        none = torch.zeros((th.nq, cr.ndof), dtype=torch.bool, device=th.om.device)
        W = th.W.w(p0["ev"][i], _t(p0["one"][i]), none[0], th.u, th.one, th.zero,
                   _legs(cr, cr.fc3_atm_num, cr.fc3_atm_indx, q2, p2), _t(p2["one"]), none)
        w0, om2, n2 = _t(p0["om"][i]), _t(p2["om"]), _t(p2["nbe"])
        r = th.tetra(w0, W, om2, n2, True) if case["delta"] == "tetra" else th.gauss(w0, W, om2, n2, none, SIGMA)
        lw.append(r[0])
    return dict(lw=torch.stack(lw, 1).cpu().numpy(), omega=p0["om"])


def _exact_phonons(case, cr, temps, seed):
    v, q = _mesh(case, cr)
    irr, slot = _irreducible(case, v)
    ph = _phonons(cr, q, temps, True)
    p0 = _phonons(cr, q[irr], temps, True)
    lw = _lw_guess(case, len(irr), seed)
    vv = np.einsum("qsi,qsj->qsij", ph["vel"], ph["vel"])
    skip = ph["gamma"][:, None] & (np.arange(cr.ndof) < 3)
    with np.errstate(all="ignore"):
        mode = [_kappa_sum(ph["om"], ph["nbe"][T], lw[T][slot], ph["vel"], vv, temps[T], cr.vol, len(v), skip)
                for T in range(len(temps))]
    return dict(omega=p0["om"], vel=p0["vel"], nbe=p0["nbe"], kappa=np.stack(mode).sum(1), mode=np.stack(mode))


def exact(case, seed):
    cr, temps = _crystal(case, seed), _temps(case)
    kind = case["kind"]
    if kind == "kappa":
        return _exact_kappa(case, cr, temps)
    if kind == "lw3":
        return _exact_lw3(case, cr, temps)
    if kind == "lw4":
        return _exact_lw4(case, cr, temps)
    if kind == "iter":
        return _exact_iter(case, cr, temps)
    if kind == "path":
        return _exact_path(case, cr, temps, seed)
    return _exact_phonons(case, cr, temps, seed)
