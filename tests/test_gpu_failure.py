"""Failure detection without a GPU fault: a bounded wait that nothing will
end returns FC_ERR_TIMEOUT and leaves the context usable.

The MMA warps of the pair kernel and of the residue GEMM wait for each operand
stage with a limit
(FERRIC_CUDA_WAIT_MS, default 4 s); FERRIC_CUDA_TEST_DROP_LOAD=1 makes CTA 0's
producer issue no load for its first stage, so that wait runs out with
nothing in flight.  The other roles see the CTA's abort flag and leave their
loops; the producer waits (long limit) for every load it did issue, and TMEM
is released.  The call returns FC_ERR_TIMEOUT within the short limit, the
dispatcher declines to the CPU path on it, and the next call, without the
switch, gives the right energy."""
import ctypes
import time

import numpy as np
import pytest

from oracle import rimp2 as orc
from oracle import synthetic

pytestmark = pytest.mark.gpu


def test_pair_wait_runs_out_and_context_recovers(fc, monkeypatch):
    import ferric_b200._lib as L
    from ferric_b200 import rimp2
    b, eo, ev = synthetic.rimp2_inputs(200, 7, 65)
    ref = orc.spin_components(b, np.concatenate([eo, ev]), 7, 65)
    monkeypatch.setenv("FERRIC_CUDA_WAIT_MS", "50")
    monkeypatch.setenv("FERRIC_CUDA_TEST_DROP_LOAD", "1")
    for call in (lambda: rimp2.rimp2_energy(b, eo, ev, precision="mixed"),
                 lambda: rimp2.rimp2_energy_grad(b, eo, ev, precision="mixed")):
        t0 = time.perf_counter()
        with pytest.raises(L.FcError) as ei:
            call()
        assert ei.value.name == "FC_ERR_TIMEOUT"
        assert time.perf_counter() - t0 < 3.0      # the 50 ms limit ended it, not the 4 s default
    before = rimp2.STATS["cpu:FC_ERR_TIMEOUT"]
    assert rimp2.try_spin_components_on_device(b, np.concatenate([eo, ev]), 7, 65, mixed_ok=True) is None
    assert rimp2.STATS["cpu:FC_ERR_TIMEOUT"] == before + 1
    monkeypatch.delenv("FERRIC_CUDA_TEST_DROP_LOAD")
    for _ in range(2):
        e = rimp2.rimp2_energy(b, eo, ev, precision="mixed")
        assert abs(sum(e) - ref[2]) <= 2e-9 * abs(ref[2])
        sc, g, _, _ = rimp2.rimp2_energy_grad(b, eo, ev, precision="mixed")
        assert abs(sc.e_total - ref[2]) <= 2e-9 * abs(ref[2])


def test_residue_wait_runs_out_and_context_recovers(fc, monkeypatch):
    """The residue GEMM of every call that has one; a pinned Gamma is the caller's own again after the error."""
    import torch

    import ferric_b200._lib as L
    from ferric_b200 import dress, rimp2
    from ferric_b200.dfjk import DfJK
    b, eo, ev = synthetic.rimp2_inputs(1153, 16, 65)
    ref = orc.spin_components(b, np.concatenate([eo, ev]), 16, 65)
    gen = torch.Generator("cuda").manual_seed(3)

    def rand(*shape):
        return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64)

    t, m, cl, cr, x = rand(640, 257, 257), rand(640, 640), rand(257, 17), rand(257, 769), rand(640, 4099)
    t += t.transpose(1, 2).clone()
    c = torch.linalg.qr(rand(257, 192))[0].contiguous()
    torch.cuda.synchronize()
    jk = DfJK(t)
    gamma = torch.zeros(b.shape, dtype=torch.float64).pin_memory()
    d_o, d_v = np.zeros(16), np.zeros(65)

    def gradient(stats):  # into pinned memory, which takes Gamma's blocks while the call runs
        e, st = [ctypes.c_double(), ctypes.c_double()], L.FcStats()
        L.check(L.lib.fc_rimp2_energy_grad(
            L.ptr(b), 1153, 16, 65, L.ptr(eo), L.ptr(ev), 0, ctypes.byref(e[0]), ctypes.byref(e[1]), L.ptr(gamma),
            L.ptr(d_o), L.ptr(d_v), ctypes.byref(st)))
        stats.update(st.as_dict())
        return e[0].value, e[1].value

    calls = [lambda s: rimp2.rimp2_energy(b, eo, ev, stats=s),
             gradient,
             lambda s: jk.k_from_occ(c, stats=s),
             lambda s: dress.mo_dress(t, m, cl, cr, stats=s),
             lambda s: rimp2.rimp2_response_2c(x, x, m, stats=s)]
    good = [call({}) for call in calls]
    monkeypatch.setenv("FERRIC_CUDA_WAIT_MS", "50")
    monkeypatch.setenv("FERRIC_CUDA_TEST_DROP_LOAD", "1")
    for call in calls:
        t0 = time.perf_counter()
        with pytest.raises(L.FcError) as ei:
            call({})
        assert ei.value.name == "FC_ERR_TIMEOUT" and time.perf_counter() - t0 < 3.0
        gamma.fill_(7.0)
        torch.cuda.synchronize()
        assert bool((gamma == 7.0).all())
    monkeypatch.delenv("FERRIC_CUDA_TEST_DROP_LOAD")
    for call, old in zip(calls, good):
        st = {}
        new = call(st)
        assert st["tile_n"] == 256
        for p, q in zip(new if isinstance(new, tuple) else (new,), old if isinstance(old, tuple) else (old,)):
            assert torch.equal(p, q) if hasattr(p, "is_cuda") else p == q
    assert abs(calls[0]({})[0] - ref[0]) <= 1e-13 * abs(ref[0])
    jk.close()
