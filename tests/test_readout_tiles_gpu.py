"""Differentiable readout at the edges of its tiles and dispatch: widths around
the 64-column, 16- and 8-row warp blocks, pupils down to one pixel, every layer
count form, unit and cone magnifications below and above one."""

import numpy as np
import pytest

from oracle import readout_diff as rd
from test_readout_diff_gpu import make_case, rel, run_gpu

pytestmark = pytest.mark.gpu

# float32 sums of at most a few hundred products, each rounded at 2^-24, against
# float64; the position gradients subtract neighbouring samples of white noise
TOL, TOL_POS = 1e-5, 1e-4


@pytest.mark.parametrize("L,S,D,n,mags", [
    (1, 12, 1, 1, None), (2, 16, 2, 2, [1.0, 0.8]), (2, 20, 2, 7, [0.9, 1.0]),   # tiny pupils
    (1, 63, 1, 8, None), (2, 64, 2, 9, [1.0, 0.97]), (3, 65, 2, 62, [1.0, 0.5, 0.25]),
    (2, 127, 2, 30, [2.5, 4.0]), (2, 129, 2, 126, [1.0, 0.999]),
    (6, 70, 1, 64, None), (9, 81, 2, 63, [1.0] * 9), (10, 80, 2, 65, list(np.linspace(1.0, 0.7, 10))),
    (11, 72, 2, 40, list(np.linspace(1.0, 0.8, 11))),
], ids=lambda v: str(v) if not isinstance(v, list) else "lgs")
def test_tile_edges_match_oracle(L, S, D, n, mags):
    screens, w, pos0, mag, n, g = make_case(100 + S + n, 2, L, S, 2, D, n, mags)
    out, gs, gw, gp = run_gpu(screens, w, pos0, mag, n, g)
    assert rel(out, rd.layer_readout(screens.astype(np.float64), w.astype(np.float64), pos0, mag, n)) < TOL
    rgs, rgw, rgp = rd.layer_readout_vjp(screens, w.astype(np.float64), pos0, mag, n, g)
    assert rel(gs, rgs) < TOL
    assert rel(gw, rgw) < TOL_POS
    assert rel(gp, rgp) < TOL_POS
