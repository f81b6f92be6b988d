"""The work that is measured: what a quantum-chemistry program has this
framework do, from one water molecule to the largest published shapes.

Every case goes through the package's public Python entry points with its
inputs on the GPU.  Shapes are the repository's own: the golden molecules of
``tests/golden``, the alkane series of the batched benchmark (C_n: naux
84n+28, nocc 4n+1, nvir 20n+9) and the synthetic tensors of ``bench.py``, with
the same distributions.  FP64 is the entry points' default precision and
"mixed" the option that large runs take, so both appear.
"""
from __future__ import annotations

import math

import numpy as np
import torch

DEV = "cuda"
F64 = torch.float64
_stream = None


def _program_stream():
    """The one stream of its own that the program queues its calls on (the
    library orders its work with torch's on any stream but the default one)."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def listed():
    return [
        # The smallest call: RI-MP2 of one water molecule, cc-pVDZ (tests/golden/h2o_ccpvdz):
        # geometry scans and tests make thousands of these, and latency is all they cost.
        dict(name="energy_water_f64", kind="energy", naux=84, nocc=5, nvir=19, precision="f64", kappa=0.0),
        # One SCF iteration of the same molecule (139 JK-fitting functions): J and K through the builders.
        dict(name="scf_water_f64", kind="jk_apart", n=24, naux=139, nocc=5, precision="f64"),
        # A correlation energy in the mixed form at a middle size: n-dodecane, cc-pVDZ.
        dict(name="energy_dodecane_mixed", kind="energy", naux=1036, nocc=49, nvir=249, precision="mixed", kappa=0.0),
        # A radical's unrestricted energy, uneven spins, odd sizes.
        dict(name="ump2_radical_f64", kind="ump2", naux=531, nocc=25, nvir=131, nocc_b=24, nvir_b=132,
             precision="f64"),
        # Energy and adjoint of n-octane, the step of a geometry optimisation at an ordinary size.
        dict(name="grad_octane_f64", kind="grad", naux=700, nocc=33, nvir=169, precision="f64"),
        # The rest of that analytic gradient: densities, Lagrangian and the 3c/2c response products.
        dict(name="gradient_chain_octane_f64", kind="chain", naux=700, nocc=33, nvir=169, nbf=202),
        # Energy and adjoint at the C20H42 def2-TZVP shapes in the default precision.
        dict(name="grad_c20_f64", kind="grad", naux=2150, nocc=81, nvir=791, precision="f64"),
        # The largest: the benchmark's synthetic RI-MP2 energy and adjoint in the mixed form.
        dict(name="grad_large_mixed", kind="grad", naux=4800, nocc=120, nvir=1100, precision="mixed"),
        # An SCF iteration on the benchmark's synthetic tensor in the default precision (an SCF's last iterations).
        dict(name="jk_600_f64", kind="jk", n=600, naux=2400, nocc=60, precision="f64"),
        # An SCF iteration at the C20H42 def2-TZVP shapes in the mixed form (an SCF's first iterations).
        dict(name="jk_c20_mixed", kind="jk", n=872, naux=2256, nocc=81, precision="mixed"),
        # MO transform and metric dressing before a C20H42 def2-TZVP correlation energy.
        dict(name="dress_c20_f64", kind="dress", naux=2150, n=872, nocc=81, nvir=791, precision="f64"),
        # Many small molecules of uneven size in one captured graph: alkanes C1..C8, energies and gradients.
        dict(name="batch_alkanes_mixed", kind="batch", nmol=128, precision="mixed"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mo_sizes(rng, occ_lo, occ_hi, vir_hi, aux_hi):
    """Occupied, virtual and auxiliary counts in the proportions that the orbital and fitting sets of the
    listed molecules span (cc-pVDZ to def2-TZVP)."""
    nocc = _log(rng, occ_lo, occ_hi)
    nvir = min(vir_hi, max(9, int(nocc * rng.uniform(3.8, 9.8))))
    naux = min(aux_hi, int((nocc + nvir) * rng.uniform(2.4, 3.9)))
    return dict(naux=naux, nocc=nocc, nvir=nvir)


def draw(rng):
    kind = rng.choice(["energy", "energy", "ump2", "grad", "grad", "chain", "jk", "jk", "jk_apart", "dress", "batch"])
    precision = rng.choice(["f64", "mixed"])
    if kind == "energy":
        kappa = round(rng.uniform(0.8, 1.6), 2) if precision == "f64" and rng.random() < 0.3 else 0.0
        return dict(kind=kind, precision=precision, kappa=kappa, **_mo_sizes(rng, 4, 81, 791, 2400))
    if kind == "ump2":
        s = _mo_sizes(rng, 4, 49, 400, 1600)
        s["nocc_b"] = s["nocc"] - rng.randint(1, 3)
        s["nvir_b"] = s["nvir"] + s["nocc"] - s["nocc_b"]
        return dict(kind=kind, precision=precision, **s)
    if kind == "grad":
        big = precision == "mixed"
        return dict(kind=kind, precision=precision, **_mo_sizes(rng, 4, 100 if big else 81, 900 if big else 791, 2400))
    if kind == "chain":
        s = _mo_sizes(rng, 4, 41, 240, 900)
        return dict(kind=kind, nbf=s["nocc"] + s["nvir"], **s)
    if kind in ("jk", "jk_apart"):
        n = _log(rng, 20, 872 if kind == "jk" else 400)
        return dict(kind=kind, n=n, naux=min(2400, int(n * rng.uniform(2.6, 5.0))),
                    nocc=max(3, int(n * rng.uniform(0.07, 0.2))), precision=precision)
    if kind == "dress":
        s = _mo_sizes(rng, 5, 70, 650, 1900)
        return dict(kind=kind, n=s["nocc"] + s["nvir"], precision=precision, **s)
    return dict(kind=kind, nmol=_log(rng, 8, 128), precision="mixed")


# ------------------------------------------------------------------ inputs --

def _gen(seed, part):
    return torch.Generator(device=DEV).manual_seed(1000003 * (seed % (1 << 31)) + part)


def _b_ov(seed, part, naux, nov):
    """B_Q,ia ~ 0.02 N(0, 1) exp(-Q / decay), the benchmark's distribution."""
    b = torch.randn((naux, nov), generator=_gen(seed, part), device=DEV, dtype=F64)
    b *= 0.02 * torch.exp(-torch.arange(naux, device=DEV, dtype=F64) / (3000.0 * naux / 4800.0))[:, None]
    return b


def _eps(seed, part, nocc, nvir):
    u = torch.rand(nocc + nvir, generator=_gen(seed, part), device=DEV, dtype=F64)
    occ = torch.sort(-20.0 + 19.7 * u[:nocc])[0]
    vir = torch.sort(0.05 + 5.95 * u[nocc:])[0]
    return occ.contiguous(), vir.contiguous()


def _sym3(seed, part, naux, n, scale):
    """(Q|mu nu)-like tensor, symmetric in the pair, decaying off its diagonal."""
    g = _gen(seed, part)
    idx = torch.arange(n, device=DEV, dtype=F64)
    env = 0.05 * torch.exp(-(idx[:, None] - idx[None, :]).abs() / scale)
    b = torch.empty((naux, n, n), device=DEV, dtype=F64)
    for q in range(0, naux, 256):
        x = torch.randn((min(256, naux - q), n, n), generator=g, device=DEV, dtype=F64) * env
        b[q:q + x.shape[0]] = (x + x.transpose(1, 2)) / math.sqrt(2.0)
    return b


def _orbitals(seed, part, n, k):
    """k orthonormal columns."""
    q, _ = torch.linalg.qr(torch.randn((n, k), generator=_gen(seed, part), device=DEV, dtype=F64))
    return q.contiguous()


def _metric_factor(seed, part, naux):
    """A symmetric positive factor with a Coulomb metric's spread (condition about 1e3)."""
    q = _orbitals(seed, part, naux, naux)
    w = torch.logspace(-1.0, 2.0, naux, device=DEV, dtype=F64)
    return ((q * w) @ q.T).contiguous()


def _alkanes(seed, nmol):
    u = torch.rand(nmol, generator=torch.Generator().manual_seed(seed % (1 << 31)))
    # the sizes' mix is the same for every seed (the graph's shape), the order is the seed's
    sizes = [1 + k % 8 for k in range(nmol)]
    return [sizes[i] for i in torch.argsort(u).tolist()]


def _tensors(case, seed):
    """The case's inputs as tensors (what `exact` and `prepare` share)."""
    k = case["kind"]
    if k in ("energy", "grad"):
        return (_b_ov(seed, 1, case["naux"], case["nocc"] * case["nvir"]), *_eps(seed, 2, case["nocc"], case["nvir"]))
    if k == "ump2":
        return (_b_ov(seed, 1, case["naux"], case["nocc"] * case["nvir"]), *_eps(seed, 2, case["nocc"], case["nvir"]),
                _b_ov(seed, 3, case["naux"], case["nocc_b"] * case["nvir_b"]),
                *_eps(seed, 4, case["nocc_b"], case["nvir_b"]))
    if k == "chain":
        eo, ev = _eps(seed, 2, case["nocc"], case["nvir"])
        b_full = _sym3(seed, 1, case["naux"], case["nbf"], 50.0)
        b_ov = b_full[:, :case["nocc"], case["nocc"]:].reshape(case["naux"], -1).contiguous()
        c = _orbitals(seed, 3, case["nbf"], case["nbf"])
        return (b_ov, eo, ev, b_full, _metric_factor(seed, 4, case["naux"]),
                c[:, :case["nocc"]].contiguous(), c[:, case["nocc"]:].contiguous())
    if k in ("jk", "jk_apart"):
        b = _sym3(seed, 1, case["naux"], case["n"], 50.0)
        c = _orbitals(seed, 2, case["n"], case["nocc"])
        return b, c, (c @ c.T).contiguous()
    if k == "dress":
        t = _sym3(seed, 1, case["naux"], case["n"], 50.0)
        c = _orbitals(seed, 2, case["n"], case["n"])
        return (t, _metric_factor(seed, 3, case["naux"]), c[:, :case["nocc"]].contiguous(),
                c[:, case["nocc"]:case["nocc"] + case["nvir"]].contiguous())
    mols = []
    for m, c in enumerate(_alkanes(seed, case["nmol"])):
        naux, nocc, nvir = 84 * c + 28, 4 * c + 1, 20 * c + 9
        mols.append((_b_ov(seed, 10 + 2 * m, naux, nocc * nvir), *_eps(seed, 11 + 2 * m, nocc, nvir)))
    return mols


def prepare(case, seed):
    t = _tensors(case, seed)
    torch.cuda.synchronize()
    s = dict(case=case, t=t)
    if case["kind"] in ("jk", "jk_apart"):
        from ferric_b200.dfjk import DfJK
        with torch.cuda.stream(_program_stream()):
            s["jk"] = DfJK(t[0], precision=case["precision"])  # the handle that an SCF keeps
        torch.cuda.synchronize()
        s["t"] = (None, t[1], t[2])
    elif case["kind"] == "batch":
        from ferric_b200.batch import Rimp2Batch
        s["batch"] = Rimp2Batch(t, grad=True, precision=case["precision"])  # the captured graph
    return s


# -------------------------------------------------------------- one pass --

def run(state):
    with torch.cuda.stream(_program_stream()):
        return _run(state)


def _run(state):
    from ferric_b200 import dress, rimp2
    case, t = state["case"], state["t"]
    kind = case["kind"]
    if kind == "energy":
        b, eo, ev = t
        return np.array(rimp2.rimp2_energy(b, eo, ev, kappa=case["kappa"] or None, precision=case["precision"]))
    if kind == "ump2":
        return np.array(rimp2.ump2_energy(*t, precision=case["precision"]))
    if kind == "grad":
        sc, gamma, d_o, d_v = rimp2.rimp2_energy_grad(*t, precision=case["precision"])
        return [np.array([sc.e_os, sc.e_ss]), gamma, d_o, d_v]
    if kind == "chain":
        b_ov, eo, ev, b_full, v, c_occ, c_vir = t
        x_ov, p_oo, p_vv, e = rimp2.ri_densities(b_ov, eo, ev)
        imat = rimp2.rimp2_imat(x_ov, b_full, case["nocc"], case["nvir"])
        y_ov, g2c = rimp2.rimp2_response_2c(x_ov, b_ov, v)
        g3c = rimp2.rimp2_response_3c(y_ov, c_occ, c_vir, 0, min(128, case["naux"]))  # one aux slab
        return [x_ov, p_oo, p_vv, np.array(e), imat, y_ov, g2c, g3c]
    if kind == "jk":
        return state["jk"].jk_from_occ(t[1])
    if kind == "jk_apart":
        return [state["jk"].j(t[2]), state["jk"].k_from_occ(t[1])]
    if kind == "dress":
        return dress.mo_dress(*t, precision=case["precision"])
    bt = state["batch"]
    bt.run(_program_stream())
    e_os, e_ss = bt.energies()
    # the flat gradient that an optimiser takes
    return [e_os, e_ss, torch.cat([g.reshape(-1) for g in bt.gamma]), torch.cat(bt.de_docc), torch.cat(bt.de_dvir)]


# ------------------------------------------------------------------ work --

def _mp2_flops(naux, nocc, nvir, grad):
    pairs = nocc * (nocc + 1) / 2
    return 2.0 * naux * nvir * nvir * pairs + (2.0 * naux * (nocc * nvir) ** 2 if grad else 0.0)


def work(case):
    k = case["kind"]
    if k == "energy":
        nov = case["nocc"] * case["nvir"]
        return dict(bytes=8.0 * case["naux"] * nov, flops=_mp2_flops(case["naux"], case["nocc"], case["nvir"], False))
    if k == "ump2":
        na, nb = case["nocc"] * case["nvir"], case["nocc_b"] * case["nvir_b"]
        fl = sum(_mp2_flops(case["naux"], o, v, False)
                 for o, v in ((case["nocc"], case["nvir"]), (case["nocc_b"], case["nvir_b"])))
        return dict(bytes=8.0 * case["naux"] * (na + nb), flops=fl + 2.0 * case["naux"] * na * nb)
    if k == "grad":
        nov = case["nocc"] * case["nvir"]
        return dict(bytes=16.0 * case["naux"] * nov, flops=_mp2_flops(case["naux"], case["nocc"], case["nvir"], True))
    if k == "chain":
        naux, no, nv, n = case["naux"], case["nocc"], case["nvir"], case["nbf"]
        nov, slab = no * nv, min(128, case["naux"])
        pairs = no * (no + 1) / 2
        fl = _mp2_flops(naux, no, nv, True) + 2.0 * nv * nv * pairs * (no + nv)
        fl += 4.0 * n * naux * nov + 6.0 * naux * naux * nov + 2.0 * slab * (nov * n + n * n * no)
        by = 8.0 * (3.0 * naux * nov + naux * n * n + 2.0 * naux * naux + no * no + nv * nv + 2.0 * n * n + slab * n * n)
        return dict(bytes=by, flops=fl)
    if k in ("jk", "jk_apart"):
        n, naux, no = case["n"], case["naux"], case["nocc"]
        one = 8.0 if case["precision"] == "f64" else 4.0
        return dict(bytes=one * naux * n * (n + 1) / 2 + 8.0 * (n * no + 2.0 * n * n),
                    flops=4.0 * naux * n * (n + 1) / 2 + 2.0 * naux * n * n * no + 1.0 * naux * no * n * (n + 1))
    if k == "dress":
        naux, n, no, nv = case["naux"], case["n"], case["nocc"], case["nvir"]
        return dict(bytes=8.0 * (naux * n * (n + 1) / 2 + naux * naux + n * (no + nv) + naux * no * nv),
                    flops=2.0 * naux * n * n * no + 2.0 * naux * no * n * nv + 2.0 * naux * naux * no * nv)
    by = fl = 0.0
    for j in range(case["nmol"]):
        c = 1 + j % 8
        naux, nocc, nvir = 84 * c + 28, 4 * c + 1, 20 * c + 9
        by += 16.0 * naux * nocc * nvir
        fl += _mp2_flops(naux, nocc, nvir, True)
    return dict(bytes=by, flops=fl)


def tolerance(case):
    # FP64: sums of up to 64000 terms in another order, 4e-15 measured.  Mixed: 23 to 31 bits of each
    # operand row and exact sums, 1e-6 measured (the dressing goes through the metric's factor).
    if case["kind"] == "chain" or case.get("precision") == "f64":
        return dict(rel=2e-14, max=2e-12)
    return dict(rel=2e-5 if case["kind"] == "dress" else 4e-6, max=1e-3)


# ---------------------------------------------------------- 64-bit answers --

def _pair_block(b, eo, ev, i):
    """(ia|jb) of one occupied i as (nvir, nocc, nvir), and its denominators."""
    nocc, nvir = eo.numel(), ev.numel()
    g = (b[:, i * nvir:(i + 1) * nvir].T @ b).view(nvir, nocc, nvir)
    d = eo[i] + eo[None, :, None] - ev[:, None, None] - ev[None, None, :]
    return g, d


def _mp2(b, eo, ev, kappa=0.0, grad=False):
    nocc, nvir = eo.numel(), ev.numel()
    e_os = torch.zeros((), device=DEV, dtype=F64)
    e_ss = torch.zeros((), device=DEV, dtype=F64)
    gamma = torch.empty_like(b) if grad else None
    d_o, d_v = torch.empty_like(eo), torch.zeros_like(ev)
    for i in range(nocc):
        g, d = _pair_block(b, eo, ev, i)
        gx = g.transpose(0, 2)  # (ib|ja)
        r = 1.0 / d
        if kappa:
            r = r * (1.0 - torch.exp(kappa * d)) ** 2
        e_os += (g * g * r).sum()
        e_ss += (g * (g - gx) * r).sum()
        if grad:
            tt = (2.0 * g - gx) * r
            gamma[:, i * nvir:(i + 1) * nvir] = 4.0 * (b @ tt.view(nvir, nocc * nvir).T)
            c = g * r * tt
            d_o[i] = -2.0 * c.sum()
            d_v += 2.0 * c.sum((1, 2))
    return e_os, e_ss, gamma, d_o, d_v


def exact(case, seed):
    kind = case["kind"]
    t = _tensors(case, seed)
    if kind == "energy":
        e_os, e_ss, _, _, _ = _mp2(*t, kappa=case["kappa"])
        return np.array([float(e_os), float(e_ss)])
    if kind == "grad":
        e_os, e_ss, gamma, d_o, d_v = _mp2(*t, grad=True)
        return [np.array([float(e_os), float(e_ss)]), gamma, d_o, d_v]
    if kind == "ump2":
        ba, oa, va, bb, ob, vb = t
        e_aa = 0.5 * float(_mp2(ba, oa, va)[1])
        e_bb = 0.5 * float(_mp2(bb, ob, vb)[1])
        e_ab, nva, nvb = 0.0, va.numel(), vb.numel()
        for i in range(oa.numel()):
            g = (ba[:, i * nva:(i + 1) * nva].T @ bb).view(nva, ob.numel(), nvb)
            d = oa[i] + ob[None, :, None] - va[:, None, None] - vb[None, None, :]
            e_ab += float((g * g / d).sum())
        return np.array([e_aa, e_bb, e_ab])
    if kind == "chain":
        b, eo, ev, b_full, v, c_occ, c_vir = t
        nocc, nvir = eo.numel(), ev.numel()
        e_os, e_ss, gamma, _, _ = _mp2(b, eo, ev, grad=True)
        t2 = torch.empty((nocc, nvir, nocc, nvir), device=DEV, dtype=F64)
        for i in range(nocc):
            g, d = _pair_block(b, eo, ev, i)
            t2[i] = g / d
        tt = 2.0 * t2 - t2.transpose(1, 3)
        p_oo = -(t2.reshape(nocc, -1) @ tt.reshape(nocc, -1).T)
        tv = t2.permute(1, 0, 2, 3).reshape(nvir, -1)
        p_vv = tv @ tt.permute(1, 0, 2, 3).reshape(nvir, -1).T
        x = gamma / 4.0
        x3 = x.view(-1, nocc, nvir)
        imat = torch.zeros_like(b_full[0])
        nt = nocc + nvir
        imat[:, :nocc] = -2.0 * torch.einsum("pia,pqa->qi", x3, b_full[:, :, nocc:nt])
        imat[:, nocc:nt] = -2.0 * torch.einsum("pia,pqi->qa", x3, b_full[:, :, :nocc])
        y = v.T @ x
        g2c = -2.0 * (v.T @ b) @ y.T
        slab = y[:min(128, y.shape[0])].view(-1, nocc, nvir)
        g3 = c_occ @ slab @ c_vir.T
        return [x, p_oo, p_vv, np.array(float(e_os + e_ss)), imat, y, g2c, 2.0 * (g3 + g3.transpose(1, 2))]
    if kind in ("jk", "jk_apart"):
        b, c, d = t
        dp = (b.reshape(b.shape[0], -1) @ d.reshape(-1))
        j = (dp @ b.reshape(b.shape[0], -1)).view_as(d)
        k = torch.zeros_like(d)
        for q in range(0, b.shape[0], 128):
            w = (b[q:q + 128] @ c).permute(1, 0, 2).reshape(d.shape[0], -1)
            k += w @ w.T
        return (j, k) if kind == "jk" else [j, k]
    if kind == "dress":
        e3, m, cl, cr = t
        mo = torch.empty((e3.shape[0], cl.shape[1] * cr.shape[1]), device=DEV, dtype=F64)
        for q in range(0, e3.shape[0], 128):
            mo[q:q + 128] = (cl.T @ e3[q:q + 128] @ cr).reshape(-1, mo.shape[1])
        return m @ mo
    out = [_mp2(*mol, grad=True) for mol in t]
    return [torch.stack([o[0] for o in out]), torch.stack([o[1] for o in out]),
            torch.cat([o[2].reshape(-1) for o in out]), torch.cat([o[3] for o in out]), torch.cat([o[4] for o in out])]
