"""Read-outs of fields whose element count nears 2^31: an index that steps past the end by a
grid's stride must still be one."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("levels", [128, 129])
def test_speed_maximum_of_a_band_just_under_31_bits(levels):
    """4095 x 4097 columns: 128 levels of each are 2^31 - 128 values (a band of levels), 129 more
    than 32-bit indices take (every level)."""
    from oraclev8_b200 import diagnostics as D
    nx, ny, nz = 4095, 4097, 129
    n = nx * ny * nz
    if torch.cuda.mem_get_info()[0] < 2 * 4 * n + (4 << 30):
        pytest.skip("two fields of 8.7 GB do not fit")
    u = torch.zeros(nx, ny, nz, dtype=torch.float32, device="cuda")
    v = torch.zeros_like(u)
    u[nx - 1, ny - 1, levels - 1] = 3.0
    v[nx - 1, ny - 1, levels - 1] = 4.0
    v[17, 5, 100] = -4.5
    state, base = SimpleNamespace(u=u, v=v), SimpleNamespace(z=100.0 * np.arange(nz))
    d = D.low_level_vmax(state, base, 0.0, 0.0, 1.0, 1.0, z_top_m=100.0 * (levels - 1))
    assert d["vmax_lowlvl"] == 5.0 and d["z_vmax_m"] == 100.0 * (levels - 1)
    assert d["r_vmax_km"] == np.sqrt((nx - 0.5) ** 2 + (ny - 0.5) ** 2) / 1e3
    D._WORK.clear()  # its planes of doubles
    del u, v, state
    torch.cuda.empty_cache()
