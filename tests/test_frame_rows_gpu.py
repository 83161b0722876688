"""Frames at arbitrary shifts and the laser zoom at the edges of their dispatch:
register row kernel sizes and their neighbours, odd frame counts, shift tables
below and above one launch's parameters, per-layer mode, tiled zoom widths and
magnifications, against float64 sums of the same realisation."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# float32 transforms of unit-scale sums: a few roundings (6e-8) a stage, eleven stages at most
TOL = 1.5e-6


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


def exact(spectra, low, freqs, sx, sy, dx):
    """Frames (F, n, n) of the layer sum in float64 (the reference's -n/2 at Nyquist)."""
    n = spectra.shape[-1]
    f = np.fft.fftfreq(n, d=dx)
    x = (np.arange(n) - n / 2.0) * dx
    basis = np.exp(2j * np.pi * freqs[:, :, None] * x)
    out = []
    for a, b in zip(sx, sy):
        X = (spectra * np.exp(2j * np.pi * f * a[:, None])[:, :, None]
             * np.exp(2j * np.pi * f * b[:, None])[:, None, :]).sum(0)
        E = (np.exp(2j * np.pi * freqs[None] * a[:, None, None])[..., :, None]
             * np.exp(2j * np.pi * freqs[None] * b[:, None, None])[..., None, :])
        c = (low.transpose(1, 0, 2, 3) * E).sum(0)
        s = np.einsum("pij,pix,pjy->xy", c, basis, basis, optimize=True).real
        out.append(np.fft.ifft2(X).real * n * n + s - s.mean())
    return np.stack(out)


@pytest.mark.parametrize("n,L,F,P,per_layer", [
    (64, 3, 2, 3, False), (128, 2, 1, 16, False), (128, 5, 5, 3, True), (256, 9, 3, 3, False),
    (256, 21, 7, 2, False),       # 147 terms: the larger parameter block
    (512, 1, 1, 0, False), (512, 4, 3, 8, False), (1024, 2, 3, 3, False), (1024, 3, 3, 1, True),
    (2048, 1, 2, 3, False), (128, 90, 12, 1, False),   # several launches of whole pairs
    (128, 300, 2, 1, False),      # more layers than a launch's terms: the table kernels
    (96, 2, 3, 3, False)])
def test_frames_match_float64(n, L, F, P, per_layer):
    from pyturb_gb300.backend import NoiseStream
    from pyturb_gb300.flow import SpectralLayers
    from pyturb_gb300.fourier import subharmonic_tables

    dx = 0.05
    rng = np.random.default_rng(n + L)
    f = np.fft.fftfreq(n, d=dx)
    amp = np.broadcast_to((f[:, None] ** 2 + f[None] ** 2 + 0.01) ** (-0.9), (L, n, n)).copy()
    freqs, _ = subharmonic_tables(n, dx, 0.15, 25.0, P)
    low_amp = np.ones((P, L, 3, 3)) * amp.max()
    many = L > 64   # the fill takes 64 layers a call
    layers = SpectralLayers(n, dx, freqs, amp[:64], low_amp[:, :64], [NoiseStream(s, None) for s in range(min(L, 64))])
    if many:
        import torch

        reps = -(-L // 64)
        layers.spectra = layers.spectra.repeat(reps, 1, 1, 1)[:L].contiguous()
        layers.sh_coef = layers.sh_coef.repeat(1, reps, 1, 1, 1)[:, :L].contiguous()
        layers.L = L
        layers.grid.ensure_workspace(L)
    S = layers.spectra.double().cpu().numpy()
    S = S[..., 0] + 1j * S[..., 1]
    c = layers.sh_coef.double().cpu().numpy()
    c = (c[..., 0] + 1j * c[..., 1])[:P]
    if per_layer:
        sx, sy = rng.uniform(-300, 300, (2, L))
        got = layers.layer_screens(sx, sy)
        for l in range(L):
            want = exact(S[l:l + 1], c[:, l:l + 1], freqs, sx[l:l + 1, None], sy[l:l + 1, None], dx)[0]
            assert rel(got[l].cpu(), want) < TOL
        return
    sx, sy = rng.uniform(-300, 300, (2, F, L))
    crop = n // 8
    got = layers.frames(sx, sy, crop, n - 2 * crop, 2.0)
    want = 2.0 * exact(S, c, freqs, sx, sy, dx)[:, crop:n - crop, crop:n - crop]
    assert rel(got.cpu(), want) < TOL


@pytest.mark.parametrize("T", [1, 2, 4, 5, 6])
@pytest.mark.parametrize("n,ns,mag", [(16, 20, 0.9), (63, 80, 1.0), (65, 70, 0.25), (130, 200, 1.4), (1, 8, 0.5)])
def test_zoom_matches_float64(T, n, ns, mag):
    import torch

    from pyturb_gb300 import _lib
    from pyturb_gb300.backend import stream_handle

    rng = np.random.default_rng(T * n)
    L = 3
    screens = rng.standard_normal((L, ns, ns)).astype(np.float32)
    pos = (ns - 1) / 2 + (np.arange(n) - (n - 1) / 2) * mag * np.linspace(1, 0.7, L)[:, None]
    idx = np.clip(np.floor(pos).astype(int)[:, None] + np.arange(T)[:, None] - (T - 1) // 2, 0, ns - 1).astype(np.int32)
    w = rng.uniform(-1, 1, (L, T, n)).astype(np.float32)
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (idx, w, screens)]
    out = torch.empty((n, n), device="cuda")
    _lib.call("pt_lgs_zoom", L, ns, n, T, d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), 0.5,
              out.data_ptr(), stream_handle())
    want = 0.0
    for l in range(L):
        taken = screens[l].astype(np.float64)[idx[l][:, None, :, None], idx[l][None, :, None, :]]
        want = want + 0.5 * np.einsum("ai,bj,abij->ij", w[l].astype(np.float64), w[l].astype(np.float64), taken)
    assert rel(out.cpu(), want) < 1e-6   # at most 36 products a layer
