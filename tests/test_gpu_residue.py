"""FP64 RI-MP2 through residue products (csrc/mgemm.cu, rimp2_mod.cu) against
the FP64 oracle.  Sizes sit at the edges of the amplitude tiles (64), the GEMM
tiles (128 x 256) and the k-steps (128); ``stats["tile_n"]`` tells the route
(256: residues, 64: DMMA).  Tolerance: the sums of the test run over at most
n = 5000 terms, |error| <= n 2^-53 |x| |y| in either order, 1e-12 of the
largest element (measured 3e-15)."""
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
    cc = -(-nocc // chunks)
    monkeypatch.setenv("FERRIC_CUDA_CHUNK_BYTES", str(23 * (cc * nvir) ** 2))
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
