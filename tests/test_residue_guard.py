"""The guard of FP64 residue products (ferric_b200/csrc/mgemm.cuh) restated on the CPU: its bound holds, ordinary
molecules' integrals pass it, and operands that would lose digits do not."""
import os

import numpy as np
import pytest

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")
LINE = 1.0 / 128


def _bounds(x, y):
    """Per row of x: the guard's lower bound of || |x_m| |y|^T ||_2 / (|x_m| |y|_F), and the thing itself."""
    nx, f = np.linalg.norm(x, axis=1), np.linalg.norm(y)
    a = np.abs(x) / nx[:, None]
    low = np.maximum(a @ np.abs(y).sum(0) / np.sqrt(len(y)), np.sqrt((a * a) @ (y * y).sum(0))) / f
    return low, np.linalg.norm(a @ np.abs(y).T, axis=1) / f


def _sides(x, y):
    (l0, t0), (l1, t1) = _bounds(x, y), _bounds(y, x)
    for low, true in ((l0, t0), (l1, t1)):
        assert (low <= true * (1 + 1e-12)).all()
    return min(l0.min(), l1.min())


@pytest.mark.parametrize("c", ["c1", "c2", "c3"])
def test_alkanes_pass(c):
    z = np.load(os.path.join(GOLDEN, "alkanes_c1_c3.npz"))
    b, eo, ev = z[c + "_b_ov"], z[c + "_eps_occ"], z[c + "_eps_vir"]
    g = (b.T @ b).reshape(len(eo), len(ev), len(eo), len(ev))
    d = eo[:, None, None, None] + eo[None, None, :, None] - ev[None, :, None, None] - ev[None, None, None, :]
    tt = ((2.0 * g - g.transpose(0, 3, 2, 1)) / d).reshape(b.shape[1], -1)
    assert _sides(b.T, b.T) > 4 * LINE and _sides(b, tt) > 2 * LINE


@pytest.mark.parametrize("f", ["h2o_ccpvdz", "h2o_augccpvdz", "ch4_ccpvdz"])
def test_small_molecules_pass(f):
    b = np.load(os.path.join(GOLDEN, f + ".npz"))["b_ov"]
    assert _sides(b.T, b.T) > 4 * LINE


def test_exchange_passes_and_opposite_slopes_do_not():
    z = np.load(os.path.join(GOLDEN, "h2o_ccpvdz.npz"))
    w = (z["b_jk"] @ z["c"][:, :int(z["nocc"])]).transpose(1, 0, 2).reshape(24, -1)
    assert _sides(w, w) > 2 * LINE
    rng = np.random.default_rng(1)
    q = np.arange(700)
    x, y = rng.standard_normal((50, 700)) * np.exp(-q / 20.0), rng.standard_normal((60, 700)) * np.exp((q - 700) / 20.0)
    assert _sides(x, y) < 1e-9
    # a triangular factor: its first row meets one, small, element of each partner
    assert _sides(np.tril(rng.standard_normal((700, 700))), y) < LINE
