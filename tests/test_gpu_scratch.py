"""Scratch limits: a pool cap that leaves the FP64 calls what their DMMA forms take lets them run, whatever a faster
form would like to have, and memory that the library gives back on demand shrinks no later call."""
import contextlib

import numpy as np
import pytest

from oracle import rimp2 as orc
from oracle import synthetic

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def _cap(scratch):
    """At most `scratch` bytes beside what handles hold."""
    import ferric_b200._lib as L
    L.release_workspace()
    L.init(0, L.pool_used() + scratch)
    try:
        yield
    finally:
        L.init(0, 0)


def _dev(*arrays):
    import torch
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]


def _rand(seed, *shape):
    import torch
    return torch.randn(shape, generator=torch.Generator("cuda").manual_seed(seed), device="cuda", dtype=torch.float64)


def _close(x, y, tol=1e-12):  # sums of at most 50000 terms in another order
    assert float((x - y).abs().max()) <= tol * float(y.abs().max())


def test_energies_in_little_memory(fc):
    """16 bytes per pair tile are enough (the unrestricted form also lists its tiles): under a cap, and on a device
    that others have filled but for less than the integrals would take."""
    import torch
    from ferric_b200 import rimp2
    ins = _dev(*synthetic.rimp2_inputs(4, 24, 700))
    ref = rimp2.rimp2_energy(*ins), rimp2.ump2_energy(*ins, *ins)
    st = {}
    with _cap(2 << 20):
        got = rimp2.rimp2_energy(*ins, stats=st), rimp2.ump2_energy(*ins, *ins)
    assert st["tile_n"] == 64
    with _cap(1 << 40):
        torch.cuda.empty_cache()
        fill = torch.empty(torch.cuda.mem_get_info()[0] - (512 << 20), dtype=torch.uint8, device="cuda")
        full = rimp2.rimp2_energy(*ins, stats=st), rimp2.ump2_energy(*ins, *ins)
        del fill
        torch.cuda.empty_cache()
    assert st["tile_n"] == 64
    for one in (got, full):
        for x, y in zip(one[0] + one[1], ref[0] + ref[1]):
            assert abs(x - y) <= 1e-13 * abs(ref[0][0])


def test_gradients_under_cap(fc):
    """Two amplitude blocks and the pair tiles' partial sums; with densities the slabs of t and Tt besides."""
    from ferric_b200 import rimp2
    ins = _dev(*synthetic.rimp2_inputs(640, 12, 129))
    ref = rimp2.rimp2_energy_grad_dens(*ins)
    st = {}
    for call, scratch in ((rimp2.rimp2_energy_grad, 38723840), (rimp2.rimp2_energy_grad_dens, 77369600)):
        with _cap(scratch):
            got = call(*ins, stats=st)
        assert st["tile_n"] == 64
        assert abs(got[0].e_total - ref[0].e_total) <= 1e-13 * abs(ref[0].e_total)
        for x, y in zip(got[1:], ref[1:]):
            _close(x, y)
    small = _dev(*synthetic.rimp2_inputs(30, 40, 50))
    ref = rimp2.rimp2_energy_grad_dens(*small)
    with _cap(130380800):
        got = rimp2.rimp2_energy_grad_dens(*small)
    for x, y in zip(got[1:], ref[1:]):
        _close(x, y)


def test_products_under_cap(fc):
    import torch
    from ferric_b200 import dress, rimp2
    from ferric_b200.dfjk import DfJK
    # the fitted tensor C alone
    x, v = _rand(1, 513, 8193), _rand(2, 513, 513)
    torch.cuda.synchronize()
    ref = rimp2.rimp2_response_2c(x, x, v)
    with _cap(513 * 8193 * 8 + 512):
        got = rimp2.rimp2_response_2c(x, x, v)
    for a, b in zip(got, ref):
        _close(a, b)
    # gathered operands and 64 partial results
    b_ov, bf = _rand(3, 640, 12 * 129), _rand(4, 640, 141, 141)
    torch.cuda.synchronize()
    ref = rimp2.rimp2_imat(b_ov, bf, 12, 129)
    with _cap(108038400):
        _close(rimp2.rimp2_imat(b_ov, bf, 12, 129), ref)
    # C^T, W and 64 partial results of K
    n, naux, nocc = 257, 640, 192
    bb = _rand(5, naux, n, n)
    bb = bb + bb.transpose(1, 2)
    c = torch.linalg.qr(_rand(6, n, nocc))[0].contiguous()
    torch.cuda.synchronize()
    jk = DfJK(bb)
    ref = jk.k_from_occ(c)
    with _cap(8 * (nocc * n + n * naux * nocc + 64 * n * n) + 768):
        _close(jk.k_from_occ(c), ref)
    jk.close()
    # both transposed coefficients, the half transform, the MO tensor
    m, cl, cr = _rand(7, naux, naux), _rand(8, n, 17), _rand(9, n, 769)
    torch.cuda.synchronize()
    ref = dress.mo_dress(bb, m, cl, cr)
    with _cap(90919168):
        _close(dress.mo_dress(bb, m, cl, cr), ref)

def test_spare_memory_leaves_later_plans_alone(fc):
    """What an FP64 energy keeps for its next call is given back on demand: it takes no chunks from a later gradient."""
    import ferric_b200._lib as L
    from ferric_b200 import rimp2
    ins, small = _dev(*synthetic.rimp2_inputs(640, 24, 129)), _dev(*synthetic.rimp2_inputs(1200, 10, 105))

    def launches():
        st = {}
        rimp2.rimp2_energy_grad(*ins, precision="mixed", stats=st)
        return st["main_launches"]

    with _cap(1 << 40):
        assert launches() == 1  # its workspace is there
        held = L.pool_used()
        # the least that leaves all 24 orbitals in one chunk is less than that and what the energy keeps
        for mib in range(240, 640, 20):
            L.init(0, held + (mib << 20))
            if launches() == 1:
                break
        st = {}
        rimp2.rimp2_energy(*small, stats=st)
        assert st["tile_n"] == 256 and L.pool_used() > held + (20 << 20)
        assert launches() == 1


def test_release_workspace(fc):
    """What calls keep is freed on request, and the next call takes it again."""
    import ferric_b200
    from ferric_b200 import rimp2
    ins = _dev(*synthetic.rimp2_inputs(640, 24, 129))
    ferric_b200.release_workspace()
    held = ferric_b200.pool_used()
    e = rimp2.rimp2_energy(*ins)
    assert ferric_b200.pool_used() > held + (100 << 20)
    ferric_b200.release_workspace()
    assert ferric_b200.pool_used() == held and rimp2.rimp2_energy(*ins) == e
