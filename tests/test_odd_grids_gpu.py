"""Transforms and frames on grids that are not a power of two, at the edges of
each form: padded lengths 256 to 8192 of the prime-factor form, the prime radices,
3 x 2^k, against float64."""

import numpy as np
import pytest

from test_frame_rows_gpu import exact, rel

pytestmark = pytest.mark.gpu

TOL = 2e-6   # two length-M float32 transforms a line, M <= 8192, both passes


@pytest.mark.parametrize("n", [67, 128 + 6, 257, 262, 514, 1031, 1994, 2062,      # Bluestein
                               7, 11, 13, 77, 91, 121, 143, 169, 728, 1001,      # prime radices
                               15, 68])
def test_inverse_transform_matches_numpy(n):
    import torch

    from pyturb_gb300 import _lib
    from pyturb_gb300.backend import stream_handle
    from pyturb_gb300.fourier import Grid

    rng = np.random.default_rng(n)
    z = rng.standard_normal((2, n, n)) + 1j * rng.standard_normal((2, n, n))
    t = torch.from_numpy(np.stack([z.real, z.imag], -1).astype(np.float32)).cuda()
    z = t.cpu().numpy().astype(np.float64)
    g = Grid(n, 0.1, np.zeros((0, 3)))
    _lib.call("pt_ifft2", g.handle, t.data_ptr(), t.data_ptr(), 2, g.work.data_ptr(), g.work_bytes, stream_handle())
    want = np.fft.ifft2(z[..., 0] + 1j * z[..., 1]) * n * n
    assert rel(t.cpu(), np.stack([want.real, want.imag], -1)) < TOL


@pytest.mark.parametrize("n,L,F,P", [(67, 3, 1, 3), (134, 9, 5, 3), (134, 2, 3, 16), (257, 17, 6, 2), (586, 2, 2, 8),
                                     (1031, 1, 2, 0), (91, 4, 4, 3), (728, 3, 5, 3), (192, 3, 3, 3), (768, 2, 1, 8),
                                     (90, 129, 2, 1)])   # more layers than a launch's terms
def test_frames_match_float64(n, L, F, P):
    import torch

    from pyturb_gb300.backend import NoiseStream
    from pyturb_gb300.flow import SpectralLayers
    from pyturb_gb300.fourier import subharmonic_tables

    dx = 0.05
    rng = np.random.default_rng(n + L)
    f = np.fft.fftfreq(n, d=dx)
    k = min(L, 64)
    amp = np.broadcast_to((f[:, None] ** 2 + f[None] ** 2 + 0.01) ** (-0.9), (k, n, n)).copy()
    freqs, _ = subharmonic_tables(n, dx, 0.15, 25.0, P)
    layers = SpectralLayers(n, dx, freqs, amp, np.ones((P, k, 3, 3)) * amp.max(), [NoiseStream(s, None) for s in range(k)])
    if L > k:
        reps = -(-L // k)
        layers.spectra = layers.spectra.repeat(reps, 1, 1, 1)[:L].contiguous()
        layers.sh_coef = layers.sh_coef.repeat(1, reps, 1, 1, 1)[:, :L].contiguous()
        layers.L = L
        layers.grid.ensure_workspace(L)
    S = torch.view_as_complex(layers.spectra).to(torch.complex128).cpu().numpy()
    c = torch.view_as_complex(layers.sh_coef).to(torch.complex128).cpu().numpy()[:P]
    sx, sy = rng.uniform(-300, 300, (2, F, L))
    got = layers.frames(sx, sy, 3, n - 7, 2.0)
    want = 2.0 * exact(S, c, freqs, sx, sy, dx)[:, 3:n - 4, 3:n - 4]
    assert rel(got.cpu(), want) < TOL
    if L == F or L == 2:
        s1, s2 = rng.uniform(-300, 300, (2, L))
        got = layers.layer_screens(s1, s2)
        for l in range(L):
            assert rel(got[l].cpu(), exact(S[l:l + 1], c[:, l:l + 1], freqs, s1[l:l + 1, None], s2[l:l + 1, None], dx)[0]) < TOL
