"""The read-outs' load forms (csrc/vdiag.cuh): 16-byte loads where the level count
and the pointers allow, scalar ones otherwise, bands with and without gaps, and the
argmax that takes a root only where the square exceeds the running one.  Values
with many equal speeds, infinities and NaN against NumPy's argmax; means bit for
bit, sums to 1e-12 (a different summation tree)."""
import ctypes

import numpy as np
import pytest
import torch

from oraclev8_b200 import _lib as L
from oraclev8_b200 import diagnostics as D
from tests.gpu_helpers import dev

pytestmark = pytest.mark.gpu


class State:
    def __init__(self, u, v):
        self.u, self.v = u, v


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("shape", [(5, 3, 1), (6, 9, 7), (12, 10, 8), (33, 17, 40)])
@pytest.mark.parametrize("special", [None, np.inf, np.nan])
def test_speed_max_and_energy_match_numpy(shape, dtype, special):
    rng = np.random.default_rng(sum(shape))
    u, v = (np.round(rng.uniform(-3, 3, shape)) for _ in range(2))  # ties everywhere
    if special is not None:
        for _ in range(3):
            u[tuple(rng.integers(0, n) for n in shape)] = special
    st = State(dev(u, dtype), dev(v, dtype))
    nz = shape[2]
    masks = [np.ones(nz, bool), np.arange(nz) < max(1, nz // 2), np.arange(nz) % 2 == 0]
    for mask in masks:
        with np.errstate(invalid="ignore"):
            s = np.sqrt((u - 0.25) ** 2 + (v - 0.5) ** 2)
        flat = np.flatnonzero(np.broadcast_to(mask, shape))
        want = flat[int(np.argmax(s.ravel()[flat]))]
        val, idx = D._speed_max(st, mask, 0.25, 0.5)
        assert idx == want
        assert val == s.ravel()[want] or (np.isnan(val) and np.isnan(s.ravel()[want]))
    if special is None:
        ke = D.perturbation_ke(st, 0.25, 0.5)["pert_ke"]
        assert abs(ke - 0.5 * np.mean(s ** 2)) <= 1e-12 * ke


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("shape", [(7, 5, 3), (9, 8, 16), (16, 12, 45), (6, 6, 80)])
def test_band_means_match_numpy_bit_for_bit(shape, dtype):
    """Through the ring sums of one ring that holds every cell of one row: the
    band mean of each column is read back from a disk around its centre."""
    rng = np.random.default_rng(shape[2])
    u = rng.standard_normal(shape)
    st = State(dev(u, dtype), dev(-2.0 * u, dtype))
    uh = st.u.cpu().numpy().astype(np.float64)
    nx, ny, nz = shape
    w = D._workspace(st.u)
    for mask in (np.ones(nz, bool), np.arange(nz) >= nz // 3, np.arange(nz) % 3 != 1):
        keep, lev, n = D._levels(mask)
        want = uh[:, :, mask][:, :, 0].copy()
        for k in range(1, int(mask.sum())):
            want = want + uh[:, :, mask][:, :, k]
        want = want / mask.sum()
        for ix, iy in ((0, 0), (nx - 1, ny // 2), (nx // 2, ny - 1)):
            edges = np.array([0.0, 0.4])
            out = np.zeros(6)
            L.check(w.lib.oracle_b200_vdiag_rings(
                w.handle, ctypes.c_void_p(st.u.data_ptr()), ctypes.c_void_p(st.v.data_ptr()),
                L.OB_PREC_F64 if dtype == torch.float64 else L.OB_PREC_F32, lev, n, 1.0, 1.0,
                ix + 0.5, iy + 0.5, L.dptr(edges), 1, 0.3, L.dptr(out), D._stream(st.u)))
            assert out[0] == out[3] == 1.0
            assert out[1] == out[4] == want[ix, iy]
            assert out[2] == -2.0 * want[ix, iy]
