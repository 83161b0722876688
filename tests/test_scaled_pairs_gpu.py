"""Screens with a factor each, in odd counts: the last transform of a call carries
one screen, and its second half has no entry in the factor table. Every form of the
column pass, each screen against the same draw without factors."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 100, 131, 192, 256, 512, 586, 1024])
@pytest.mark.parametrize("count,P", [(1, 0), (1, 3), (3, 3), (5, 16)])
def test_odd_counts_take_one_factor_a_screen(n, count, P):
    import torch

    from pyturb_gb300 import _lib
    from pyturb_gb300.backend import dptr, stream_handle, upload
    from pyturb_gb300.fourier import Grid, amplitude_table, subharmonic_tables

    dx = 0.02
    freqs, low = subharmonic_tables(n, dx, 0.15, 25.0, P)
    grid = Grid(n, dx, np.asarray(freqs) if P else np.zeros((0, 3)))
    amp = upload(np.asarray(amplitude_table(n, dx, 0.15, 25.0)))
    sh_amp = upload(np.asarray(low).reshape(P, 3, 3)) if P else None
    factors = torch.linspace(0.5, 2.0, count, device="cuda")   # the table ends with the last screen
    plain, scaled = (torch.empty((count, n, n), device="cuda") for _ in range(2))
    s, w = stream_handle(), (dptr(grid.work), grid.work_bytes)
    _lib.call("pt_generate", grid.handle, count, dptr(amp), dptr(sh_amp), None, None, 9, 4, 0, n, 1.5, 0,
              dptr(plain), *w, s)
    _lib.call("pt_generate_scaled", grid.handle, count, dptr(amp), dptr(sh_amp), 9, 4, 0, n, 1.5,
              dptr(factors), dptr(scaled), *w, s)
    # one rounding of the factor's product and one of the pixel's on each side
    torch.testing.assert_close(scaled, plain * factors[:, None, None], rtol=4 * 2.0 ** -24, atol=0.0)
