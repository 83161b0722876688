"""Frames on either side of the bounds between the ways of forming them (phasor
tables, layer sums of one or four row pairs a thread, equally spaced runs), against
float64."""

import numpy as np
import pytest

from test_frame_rows_gpu import exact, rel

pytestmark = pytest.mark.gpu

TOL = 2e-6       # one rounded phasor a layer, and the transform
TOL_RUN = 4e-6   # a ratio applied up to 63 times from an exact anchor, and the transform


def layers_of(n, L, P, dx):
    from pyturb_gb300.backend import NoiseStream
    from pyturb_gb300.flow import SpectralLayers
    from pyturb_gb300.fourier import subharmonic_tables

    f = np.fft.fftfreq(n, d=dx)
    amp = np.broadcast_to((f[:, None] ** 2 + f[None] ** 2 + 0.01) ** (-0.9), (L, n, n)).copy()
    freqs, _ = subharmonic_tables(n, dx, 0.15, 25.0, P)
    return freqs, SpectralLayers(n, dx, freqs, amp, np.ones((P, L, 3, 3)) * amp.max(),
                                 [NoiseStream(s, None) for s in range(L)])


def check(n, L, P, F, uniform, tol):
    import torch

    dx = 0.05
    rng = np.random.default_rng(n + L + F)
    freqs, layers = layers_of(n, L, P, dx)
    S = torch.view_as_complex(layers.spectra).to(torch.complex128).cpu().numpy()
    c = torch.view_as_complex(layers.sh_coef).to(torch.complex128).cpu().numpy()[:P]
    sx, sy = rng.uniform(-30, 30, (2, 1 if uniform else F, L))
    if uniform:
        step = rng.uniform(-0.3, 0.3, (2, 1, L))
        sx, sy = sx + np.arange(F)[:, None] * step[0], sy + np.arange(F)[:, None] * step[1]
    got = layers.frames(sx, sy, 3, n - 7, 2.0).cpu()
    pick = np.unique(np.linspace(0, F - 1, 4).astype(int))
    want = 2.0 * exact(S, c, freqs, sx[pick], sy[pick], dx)[:, 3:n - 4, 3:n - 4]
    for q, f in enumerate(pick):
        assert rel(got[f], want[q]) < tol, f


@pytest.mark.parametrize("n,L,P,F", [
    (200, 9, 0, 29), (200, 9, 0, 30), (288, 3, 0, 14), (288, 3, 0, 15), (192, 2, 0, 18), (192, 2, 0, 19),
    (384, 2, 0, 1), (500, 2, 0, 4), (500, 2, 0, 5), (520, 2, 0, 1),           # no levels
    (150, 4, 3, 3), (150, 4, 3, 4), (150, 3, 3, 4), (91, 17, 1, 64), (255, 4, 2, 19), (192, 4, 3, 13), (192, 4, 3, 14),
    (288, 41, 1, 12), (288, 41, 1, 13), (320, 41, 1, 13), (289, 41, 1, 13),   # several launches of shifts
    (131, 5, 2, 3), (700, 2, 3, 2), (60, 1, 3, 1)])
def test_arbitrary_shifts(n, L, P, F):
    check(n, L, P, F, False, TOL)


@pytest.mark.parametrize("n,L,P,F", [
    (64, 9, 3, 11), (64, 9, 3, 12), (64, 3, 0, 23), (64, 3, 0, 24), (128, 4, 0, 31), (128, 4, 0, 32),
    (100, 3, 3, 23), (100, 3, 3, 24), (200, 5, 3, 7), (200, 5, 3, 8), (240, 3, 0, 10), (240, 3, 0, 11),
    (500, 2, 3, 3), (500, 2, 3, 4), (586, 2, 1, 3), (586, 2, 1, 4)])
def test_equally_spaced(n, L, P, F):
    check(n, L, P, F, True, TOL_RUN)
