"""The pipelined column pass at its edges against float64: single images, odd
counts, more items than CTAs, no levels up to the most, crops, accumulation, and
the forms beside it (other sizes, levels, frequencies, a workspace at 8 bytes)."""

import numpy as np
import pytest

from test_frame_rows_gpu import rel

pytestmark = pytest.mark.gpu

TOL = 1.5e-6   # float32 transforms and low-order sums of unit-scale screens


@pytest.mark.parametrize("n,count,P,crop,sym,offset", [
    (256, 1, 0, 0, True, 0), (256, 3, 3, 0, True, 0), (256, 80, 16, 5, True, 0), (256, 3, 15, 0, True, 0),
    (512, 2, 3, 0, True, 0), (512, 41, 8, 7, True, 0), (512, 1, 9, 255, True, 0), (512, 2, 3, 0, True, 8),
    (1024, 1, 3, 0, True, 0), (1024, 9, 4, 100, True, 0), (1024, 2, 5, 0, True, 0),
    (512, 3, 2, 0, False, 0), (128, 5, 3, 1, True, 0), (2048, 2, 1, 0, True, 0)])
def test_generate_matches_float64(n, count, P, crop, sym, offset):
    import torch

    from pyturb_gb300 import _lib
    from pyturb_gb300.backend import stream_handle
    from pyturb_gb300.fourier import Grid

    rng = np.random.default_rng(n + count)
    dx, n_out, n_fft = 0.1, n - 2 * crop, (count + 1) // 2
    a = rng.uniform(0.2, 1.0, P) / (n * dx)
    freqs = np.stack([-a, np.zeros(P) if sym else 0.2 * a, a if sym else 1.3 * a], axis=1)
    g = Grid(n, dx, freqs)
    f = np.fft.fftfreq(n)
    amp = (0.01 * (f[:, None] ** 2 + f[None] ** 2 + 0.01) ** (-0.9)).astype(np.float32)
    amp /= np.sqrt((amp.astype(np.float64) ** 2).sum())
    sh_amp = rng.uniform(0.1, 1.0, (P, 9)).astype(np.float32)
    noise = rng.standard_normal((2, n_fft, n, n)).astype(np.float32)
    sh = rng.standard_normal((max(P, 1), 2, count, 9)).astype(np.float32)
    d = [torch.from_numpy(v).cuda() for v in (amp, sh_amp, noise, sh)]
    work = torch.empty(g.work_bytes + 16, dtype=torch.uint8, device="cuda")[offset:]
    out = torch.ones((count, n_out, n_out), device="cuda")
    _lib.call("pt_generate", g.handle, count, d[0].data_ptr(), d[1].data_ptr() if P else None, d[2].data_ptr(),
              d[3].data_ptr() if P else None, 0, 0, crop, n_out, 0.5, 1, out.data_ptr(), work.data_ptr(),
              g.work_bytes, stream_handle())
    z = torch.complex(d[2][0].double(), d[2][1].double()) * d[0].double()
    x = torch.fft.ifft2(z) * (n * n)
    want = torch.cat([x.real, x.imag])[:count]
    if P:
        grid = (np.arange(n) - n / 2.0) * dx
        basis = torch.from_numpy(np.exp(2j * np.pi * freqs[:, :, None] * grid)).cuda()
        coef = torch.complex(d[3][:, 0].double(), d[3][:, 1].double()) * d[1].double()[:, None]
        s = torch.einsum("pcij,pix,pjy->cxy", coef.reshape(P, count, 3, 3), basis, basis).real
        want = want + s - s.mean(dim=(1, 2), keepdim=True)
    want = 1.0 + 0.5 * want[:, crop:n - crop, crop:n - crop]
    assert rel(out.cpu(), want.cpu().numpy()) < TOL
