"""Equally spaced frames on grids without a fused row kernel, against float64 sums:
odd and even sizes of each transform form, odd frame counts, runs that end in the
middle, every layer group, crops, and the frames one by one (the general path)."""

import numpy as np
import pytest

from test_frame_rows_gpu import exact, rel

pytestmark = pytest.mark.gpu

# a frame's ratio is rounded once (rms 7e-8 with its two factors) and applied up to 63
# times from an exact anchor: 63 / sqrt(3) * 7e-8 = 2.6e-6 over a run, and the transform
TOL = 4e-6


@pytest.mark.parametrize("n,L,F,P", [
    (8, 1, 2, 0), (12, 2, 3, 1), (64, 3, 9, 3), (32, 16, 65, 3), (128, 9, 64, 3), (100, 9, 64, 3),
    (129, 4, 37, 2), (278, 5, 16, 3), (331, 2, 5, 1), (384, 12, 3, 3), (500, 9, 41, 8),
    (586, 6, 7, 3), (640, 13, 40, 0), (1000, 3, 19, 3)])
def test_uniform_frames_match_float64(n, L, F, P):
    from pyturb_gb300.backend import NoiseStream
    from pyturb_gb300.flow import SpectralLayers
    from pyturb_gb300.fourier import subharmonic_tables

    dx = 0.05
    rng = np.random.default_rng(n + L)
    f = np.fft.fftfreq(n, d=dx)
    amp = np.broadcast_to((f[:, None] ** 2 + f[None] ** 2 + 0.01) ** (-0.9), (L, n, n)).copy()
    freqs, _ = subharmonic_tables(n, dx, 0.15, 25.0, P)
    layers = SpectralLayers(n, dx, freqs, amp, np.ones((P, L, 3, 3)) * amp.max(),
                            [NoiseStream(s, None) for s in range(L)])
    S = layers.spectra.double().cpu().numpy()
    S = S[..., 0] + 1j * S[..., 1]
    c = layers.sh_coef.double().cpu().numpy()
    c = (c[..., 0] + 1j * c[..., 1])[:P]
    s0, step = rng.uniform(-30, 30, (2, 1, L)), rng.uniform(-0.3, 0.3, (2, 1, L))
    sx, sy = s0 + np.arange(F)[:, None] * step
    crop = n // 8
    got = layers.frames(sx, sy, crop, n - 2 * crop, 2.0).cpu()
    want = 2.0 * exact(S, c, freqs, sx, sy, dx)[:, crop:n - crop, crop:n - crop]
    assert rel(got, want) < TOL
    assert rel(got[-1], want[-1]) < 2 * TOL
    one = layers.frames(sx[F - 1:], sy[F - 1:], crop, n - 2 * crop, 2.0).cpu()
    assert rel(got[-1], one[0].double().numpy()) < 2 * TOL
