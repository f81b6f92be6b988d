"""FP64 RI-MP2 through residue products (csrc/mgemm.cu, rimp2_mod.cu) against
the FP64 oracle.  Sizes sit at the edges of the amplitude tiles (32), the GEMM
tiles (128 x 256) and the k-steps (128); ``stats["tile_n"]`` tells the route
(256: residues, 64: DMMA).  Tolerance: the sums of the test run over at most
n = 5000 terms, |error| <= n 2^-53 |x| |y| in either order, 1e-12 of the
largest element (measured 3e-15); where large elements of one operand meet
small ones of the other, 2^-53 of sums of |x_k y_k| by row and by column."""
import numpy as np
import pytest

from oracle import rimp2 as orc
from oracle import synthetic

pytestmark = pytest.mark.gpu


def _check(got, ref):
    sc, g, go, gv = got
    e_os, e_ss, gamma, d_o, d_v = ref
    assert abs(sc.e_os - e_os) <= 1e-13 * abs(e_os)
    assert abs(sc.e_ss - e_ss) <= 1e-13 * abs(e_ss)
    for x, y in ((g, gamma), (go, d_o), (gv, d_v)):
        assert np.abs(x - y).max() <= 1e-12 * np.abs(y).max()


@pytest.mark.parametrize("naux,nocc,nvir", [(640, 10, 128), (1153, 16, 65), (257, 24, 127), (383, 9, 193)])
@pytest.mark.parametrize("chunks", [1, 3])
def test_gradient_matches_oracle(fc, monkeypatch, naux, nocc, nvir, chunks):
    from ferric_b200 import rimp2
    b, eo, ev = synthetic.rimp2_inputs(naux, nocc, nvir)
    cc = -(-nocc // chunks)  # a chunk's block takes 8 bytes an element and 16 of residues
    monkeypatch.setenv("FERRIC_CUDA_CHUNK_BYTES", str(24 * (cc * nvir) ** 2))
    st = {}
    got = rimp2.rimp2_energy_grad(b, eo, ev, stats=st)
    assert st["tile_n"] == 256 and st["main_launches"] == chunks * (chunks + 1) // 2
    _check(got, orc.energy_gamma_deps(b, eo, ev))


def test_gradient_rows_out_of_range(fc):
    """A column of B below the residues' range (or not finite) takes the DMMA form."""
    from ferric_b200 import rimp2
    b, eo, ev = synthetic.rimp2_inputs(640, 10, 128)
    b[:, 7] *= 1e-104
    st = {}
    got = rimp2.rimp2_energy_grad(b, eo, ev, stats=st)
    assert st["tile_n"] == 64
    _check(got, orc.energy_gamma_deps(b, eo, ev))
    b[3, 5] = np.nan
    sc, g, go, gv = rimp2.rimp2_energy_grad(b, eo, ev, stats=st)
    assert st["tile_n"] == 64 and np.isnan(sc.e_total) and np.isnan(g).any()
    b[3, 5] = np.inf
    sc, g, go, gv = rimp2.rimp2_energy_grad(b, eo, ev, stats=st)
    assert st["tile_n"] == 64 and not np.isfinite(sc.e_total)


@pytest.mark.parametrize("naux,nocc,nvir,kappa", [(640, 12, 129, None), (1153, 16, 65, 1.1), (700, 1, 1300, None)])
def test_energy_matches_oracle(fc, naux, nocc, nvir, kappa):
    from ferric_b200 import rimp2
    b, eo, ev = synthetic.rimp2_inputs(naux, nocc, nvir)
    ref = orc.spin_components(b, np.concatenate([eo, ev]), nocc, nvir, kappa=kappa)
    st = {}
    e_os, e_ss = rimp2.rimp2_energy(b, eo, ev, kappa=kappa, stats=st)
    assert st["tile_n"] == 256
    # E_ss is a difference of sums of the size of E_os
    assert abs(e_os - ref[0]) <= 1e-13 * abs(ref[0]) and abs(e_ss - ref[1]) <= 1e-13 * abs(ref[0])


@pytest.mark.parametrize("naux,na,nva,nb,nvb", [(640, 17, 129, 15, 131), (500, 40, 66, 1, 105)])
def test_ump2_matches_oracle(fc, naux, na, nva, nb, nvb):
    from ferric_b200 import rimp2
    ba, oa, va = synthetic.rimp2_inputs(naux, na, nva)
    bb, ob, vb = synthetic.rimp2_inputs(naux, nb, nvb, seed_b=5, seed_eps=50)
    st = {}
    got = rimp2.ump2_energy(ba, oa, va, bb, ob, vb, stats=st)
    assert st["tile_n"] == 256
    # the same-spin sum is half of one spin's closed-shell E_ss
    e_aa = 0.5 * orc.spin_components(ba, np.concatenate([oa, va]), na, nva)[1]
    e_bb = 0.5 * orc.spin_components(bb, np.concatenate([ob, vb]), nb, nvb)[1]
    g = (ba.T @ bb).reshape(na, nva, nb, nvb)
    d = oa[:, None, None, None] + ob[None, None, :, None] - va[None, :, None, None] - vb[None, None, None, :]
    e_ab = float((g * g / d).sum())
    for x, y in zip(got, (e_aa, e_bb, e_ab)):
        assert abs(x - y) <= 1e-13 * abs(e_ab)


@pytest.mark.parametrize("naux,nocc,nvir", [(640, 10, 129), (513, 33, 64)])
def test_densities_match_oracle(fc, naux, nocc, nvir):
    from ferric_b200 import rimp2
    b, eo, ev = synthetic.rimp2_inputs(naux, nocc, nvir)
    st = {}
    got = rimp2.rimp2_energy_grad_dens(b, eo, ev, stats=st)
    assert st["tile_n"] == 256
    _check(got[:4], orc.energy_gamma_deps(b, eo, ev))
    t2, _ = orc.t2_and_integrals(b, eo, ev)
    for x, y in zip(got[4:], orc.mp2_density(t2, nocc, nvir)):
        assert np.abs(x - y).max() <= 1e-12 * np.abs(y).max()


def _rand(seed, *shape):
    import torch
    return torch.randn(shape, generator=torch.Generator("cuda").manual_seed(seed), device="cuda", dtype=torch.float64)


def _close(x, y, tol=1e-13):
    assert float((x - y).abs().max()) <= tol * float(y.abs().max())


@pytest.mark.parametrize("n,naux,nocc", [(257, 640, 192), (513, 401, 77)])
def test_dfk_rank_update(fc, n, naux, nocc):
    """K = W W^T through residues, split over (Q, i); non-finite C takes the DMMA form."""
    import torch
    from ferric_b200.dfjk import DfJK
    b = _rand(1, naux, n, n) / n
    b = b + b.transpose(1, 2)
    c = torch.linalg.qr(_rand(2, n, nocc))[0].contiguous()
    torch.cuda.synchronize()
    w = (b @ c).permute(1, 0, 2).reshape(n, -1)
    jk = DfJK(b)
    st = {}
    j, k = jk.jk_from_occ(c, stats=st)
    assert st["tile_n"] == 256
    torch.cuda.synchronize()
    _close(k, w @ w.T)
    _close(j, torch.einsum("q,qmn->mn", torch.einsum("qmn,mn->q", b, c @ c.T), b))
    assert torch.equal(k, k.T)
    c[3, 2] = float("nan")
    torch.cuda.synchronize()
    k = jk.k_from_occ(c, stats=st)
    torch.cuda.synchronize()
    assert st["tile_n"] == 64 and bool(torch.isnan(k).all())
    jk.close()


@pytest.mark.parametrize("naux,n,nl,nr", [(640, 257, 17, 769), (1025, 256, 90, 64)])
def test_dressing(fc, naux, n, nl, nr):
    import torch
    from ferric_b200 import dress
    t = _rand(3, naux, n, n)
    t = t + t.transpose(1, 2)
    m, cl, cr = _rand(4, naux, naux), _rand(5, n, nl), _rand(6, n, nr)
    torch.cuda.synchronize()
    st = {}
    b = dress.mo_dress(t, m, cl, cr, stats=st)
    assert st["tile_n"] == 256
    ref = m @ (cl.T @ t @ cr).reshape(naux, nl * nr)
    _close(b, ref)
    m[5, 7] = float("inf")  # its row takes the DMMA form: not finite there, the others as before
    torch.cuda.synchronize()
    b = dress.mo_dress(t, m, cl, cr, stats=st)
    torch.cuda.synchronize()
    assert st["tile_n"] == 64 and not bool(torch.isfinite(b[5]).any())
    _close(torch.cat([b[:5], b[6:]]), torch.cat([ref[:5], ref[6:]]))


@pytest.mark.parametrize("naux,nov", [(513, 8193), (300, 66000)])
def test_response_2c(fc, naux, nov):
    """Few tiles over a long K (split), and a K past one range of exact sums."""
    import torch
    from ferric_b200 import rimp2
    x, b, v = _rand(7, naux, nov), _rand(8, naux, nov), _rand(9, naux, naux)
    torch.cuda.synchronize()
    st = {}
    y, g = rimp2.rimp2_response_2c(x, b, v, stats=st)
    assert st["launches"] > 3 and st["tile_n"] == 256
    yr = v.T @ x
    _close(y, yr)
    _close(g, -2.0 * (v.T @ b) @ yr.T)


def _rowwise(got, a, b, c=64.0):
    """Rows and columns of got = a b^T against 80-bit sums, each in its 2-norm: within c 2^-53 of the row (column)
    of |a| |b|^T, where FP64 sums of these lengths lie (their own bound is K 2^-53 of it, element by element)."""
    s = np.abs(a).max(axis=1, keepdims=True)  # (so that no square below underflows)
    ref = a.astype(np.longdouble) @ b.T.astype(np.longdouble)
    err = (np.abs(got - ref) / s).astype(np.float64)
    mag = np.abs(a / s) @ np.abs(b).T
    for ax in (0, 1):
        e, m = np.linalg.norm(err, axis=ax), np.linalg.norm(mag, axis=ax)
        assert (e <= c * 2.0 ** -53 * m).all(), (ax, float((e / (m + 1e-300)).max()))


def _graded(case, m, n, k):
    """Operands whose large elements meet small ones: opposite slopes, a triangle, rows of one slope and of the other,
    one row apart, a row whose squares underflow."""
    rng = np.random.default_rng(17)
    a, b = rng.standard_normal((m, k)), rng.standard_normal((n, k))
    q = np.arange(k)
    if case == "slopes":
        a *= np.exp(-q / 20.0)
        b *= np.exp((q - k) / 20.0)
    elif case == "triangle":  # the first rows of a factor meet the partner's smallest elements
        a = np.where(q[None, :] <= np.arange(m)[:, None], a, 0.0)
        b *= np.exp((q - k) * 30.0 / k)
    elif case == "row":
        a[3] *= np.exp(-q / 10.0)
        b[:, :200] *= 1e-9
    else:
        a[3] *= 1e-170
    return a, b


CASES = ["slopes", "triangle", "row", "underflow"]


@pytest.mark.parametrize("case", CASES)
def test_graded_dressing(fc, case):
    """B = M MO^T through a square dressing: t = MO tensor with unit orbitals, so the dressing is the product tested."""
    from ferric_b200 import dress
    naux, n, nl = 640, 256, 64
    m, mo = _graded(case, naux, nl * n, naux)
    t = np.zeros((naux, n, n))
    t[:, :nl] = mo.T.reshape(naux, nl, n)
    # (Q|lr) = sum C_left[mu, l] t[Q, nu, mu] C_right[nu, r]: the tensor need not be symmetric here
    cl, cr = np.eye(n)[:, :nl], np.eye(n)
    st = {}
    got = dress.mo_dress(np.ascontiguousarray(t.transpose(0, 2, 1)), m, np.ascontiguousarray(cl), cr, stats=st)
    assert st["tile_n"] == 64
    sel = np.r_[0:7, naux - 7:naux]
    _rowwise(got[sel], m[sel], mo)


def test_guard_passes_ordinary_slopes(fc):
    """Slopes of e^-6 over the row: 0.02 by the guard's measure, above its line, and the residues' error (2^-61 / 0.02
    of |a| |b|^T) is below a single FP64 rounding's."""
    from ferric_b200 import dress
    naux, n, nl = 640, 256, 64
    rng = np.random.default_rng(23)
    q = np.arange(naux) * 6.0 / naux
    m, mo = rng.standard_normal((naux, naux)) * np.exp(-q), rng.standard_normal((nl * n, naux)) * np.exp(q)
    t = np.zeros((naux, n, n))
    t[:, :, :nl] = mo.T.reshape(naux, nl, n).transpose(0, 2, 1)
    st = {}
    got = dress.mo_dress(t, m, np.ascontiguousarray(np.eye(n)[:, :nl]), np.eye(n), stats=st)
    assert st["tile_n"] == 256
    sel = np.r_[0:7, naux - 7:naux]
    _rowwise(got[sel], m[sel], mo, c=1.0)


@pytest.mark.parametrize("case", CASES)
def test_graded_response(fc, case):
    from ferric_b200 import rimp2
    naux, nov = 513, 4099
    v, x = _graded(case, naux, nov, naux)
    st = {}
    y, g = rimp2.rimp2_response_2c(np.ascontiguousarray(x.T), np.ascontiguousarray(x.T), np.ascontiguousarray(v.T),
                                   stats=st)
    assert st["tile_n"] == 64
    sel = np.r_[0:7, naux - 7:naux]
    _rowwise(y[sel], v[sel], x)


def test_graded_rank_update(fc):
    """K of orbitals whose W rows are a strong block and a weak one on other aux rows."""
    from ferric_b200.dfjk import DfJK
    n, naux, nocc = 257, 640, 192
    rng = np.random.default_rng(5)
    b = np.zeros((naux, n, n))
    b[:320, :128, :128] = rng.standard_normal((320, 128, 128))
    b[320:, 128:, 128:] = 1e-6 * rng.standard_normal((320, 129, 129))
    b[320:, :128, :128] = 1e-11 * rng.standard_normal((320, 128, 128))
    b = b + b.transpose(0, 2, 1)
    c = np.linalg.qr(rng.standard_normal((n, nocc)))[0]
    st = {}
    jk = DfJK(b)
    k = jk.k_from_occ(np.ascontiguousarray(c), stats=st)
    jk.close()
    assert st["tile_n"] == 64
    w = (b.reshape(-1, n) @ c).reshape(naux, n, nocc).transpose(1, 0, 2).reshape(n, -1)
    sel = np.r_[0:3, 126:131]
    _rowwise(k[sel], w[sel], w, c=256.0)  # W itself is rounded: 2^-53 sums of n terms


def test_graded_spins(fc):
    """Two spins on aux rows that hardly overlap: E_ab is a sum of graded products."""
    from ferric_b200 import rimp2
    naux, no, nv = 700, 12, 129
    a, b = _graded("slopes", no * nv, no * nv, naux)
    eo, ev = synthetic.rimp2_inputs(2, no, nv)[1:]
    a, b = np.ascontiguousarray(a.T), np.ascontiguousarray(b.T)
    e = rimp2.ump2_energy(a, eo, ev, b, eo, ev)
    g = (a.T @ b).reshape(no, nv, no, nv)  # every element within 700 2^-53 sum_k |a_k b_k|, like the call's
    d = eo[:, None, None, None] + eo[None, None, :, None] - ev[None, :, None, None] - ev[None, None, None, :]
    ref = float((g * g / d).sum())
    assert abs(e[2] - ref) <= 1e-12 * abs(ref)


def test_graded_adjoint(fc):
    """Amplitudes of two blocks of orbitals, each on its own aux rows: Gamma's rows are products of one block each."""
    from ferric_b200 import rimp2
    naux, no, nv = 700, 12, 129
    b, eo, ev = synthetic.rimp2_inputs(naux, no, nv)
    b[350:, :no * nv // 2] *= 1e-13
    b[:350, no * nv // 2:] *= 1e-13
    b[350:] *= 1e-9
    _, g, go, gv = rimp2.rimp2_energy_grad(b, eo, ev)
    gamma = orc.energy_gamma_deps(b, eo, ev)[2]
    t2, _ = orc.t2_and_integrals(b, eo, ev)
    t4 = t2.reshape(no, nv, no, nv)
    tt = np.abs(2 * t4 - t4.transpose(0, 3, 2, 1)).reshape(no * nv, -1)
    mag = 4 * np.abs(b) @ tt.T
    e = np.abs(g - gamma)
    for ax in (0, 1):
        assert (np.linalg.norm(e, axis=ax) <= 700 * 2.0 ** -53 * np.linalg.norm(mag, axis=ax)).all()
