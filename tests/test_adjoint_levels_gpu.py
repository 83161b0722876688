"""Subharmonic adjoint kernels at their edges (column blocks, level passes,
other frequencies, chunks) against float64 sums of the same formulas."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-6   # float32 column sums of at most a few hundred terms, float64 beyond


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a) - b) / np.linalg.norm(b))


def basis(freqs, n, dx, crop, n_out):
    x = (np.arange(n) - n / 2.0) * dx
    full = np.exp(2j * np.pi * freqs[:, :, None] * x)
    return full[:, :, crop:crop + n_out], full.mean(-1)


@pytest.mark.parametrize("n,n_out,F,P,sym", [
    (2, 1, 1, 1, True), (130, 127, 3, 2, True), (128, 128, 2, 3, True), (160, 129, 2, 4, True),
    (300, 257, 1, 8, True), (64, 60, 2, 16, True), (96, 90, 2, 3, False)])
def test_projections_and_level_gradients(n, n_out, F, P, sym):
    import torch

    from pyturb_gb300 import _lib
    from pyturb_gb300.backend import stream_handle
    from pyturb_gb300.fourier import Grid

    rng = np.random.default_rng(n + P)
    dx, L, scale, crop = 0.1, 3, 0.7, (n - n_out) // 2
    a = rng.uniform(0.2, 1.0, P) / (n * dx)
    freqs = np.stack([-a, 0 * a if sym else 0.1 * a, a if sym else 1.5 * a], axis=1)
    grid = Grid(n, dx, freqs)
    g = rng.standard_normal((F, n_out, n_out)).astype(np.float32)
    dg = torch.from_numpy(g).cuda()
    proj = torch.empty((F, 18 * P + 1), dtype=torch.float64, device="cuda")
    s = stream_handle()
    _lib.call("pt_synth_adj_sh", grid.handle, F, crop, n_out, dg.data_ptr(), proj.data_ptr(), s)
    b, beta = basis(freqs, n, dx, crop, n_out)
    G = np.einsum("fxy,pix,pjy->fpij", g.astype(np.float64), b, b, optimize=True)
    got = proj.cpu().numpy()
    assert rel((got[:, 0:18 * P:2] + 1j * got[:, 1:18 * P:2]).reshape(G.shape), G) < TOL
    assert rel(got[:, 18 * P], g.astype(np.float64).sum((1, 2))) < TOL * n_out

    w = rng.uniform(0.5, 1.5, L).astype(np.float32)
    c = (rng.standard_normal((P, L, 3, 3)) + 1j * rng.standard_normal((P, L, 3, 3))).astype(np.complex64)
    sx, sy = rng.uniform(-50, 50, (2, F, L))
    part = rng.standard_normal((L, F, 3))
    gw = torch.full((L,), 2.0, dtype=torch.float64, device="cuda")
    gsh = torch.zeros((F + 1, L, 2), dtype=torch.float64, device="cuda")
    gc = torch.zeros((L, P, 3, 3, 2), dtype=torch.float64, device="cuda")
    d = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (w, c.view(np.float32), sx, sy, part)]
    nbytes = int(_lib.load().pt_synth_adj_levels_workspace_bytes(L, F, P))
    work = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    for accumulate in (0, 1):   # the second call adds the same chunk again
        _lib.call("pt_synth_adj_levels", grid.handle, L, F, 1, scale, d[0].data_ptr(), d[1].data_ptr(),
                  d[2].data_ptr(), d[3].data_ptr(), proj.data_ptr(), d[4].data_ptr(), accumulate,
                  gw.data_ptr(), gsh.data_ptr(), gc.data_ptr(), work.data_ptr(), nbytes, s)
    S = got[:, 18 * P]
    Q = np.float32(scale) * ((got[:, 0:18 * P:2] + 1j * got[:, 1:18 * P:2]).reshape(G.shape)
                             - (beta[:, :, None] * beta[:, None, :])[None] * S[:, None, None, None])
    E = (np.exp(2j * np.pi * sx[:, :, None, None] * freqs)[..., :, None]
         * np.exp(2j * np.pi * sy[:, :, None, None] * freqs)[..., None, :])
    EQ = E * Q[:, None]
    M = c.transpose(1, 0, 2, 3).astype(np.complex128)[None] * EQ
    im = (w[None, :, None, None, None] * M).imag
    assert rel(gw.cpu(), 2 * (M.real.sum((0, 2, 3, 4)) + part[..., 0].sum(1))) < 1e-9
    want = np.stack([-2 * np.pi * np.einsum("pi,flpij->fl", freqs, im),
                     -2 * np.pi * np.einsum("pj,flpij->fl", freqs, im)], -1) + part[..., 1:].transpose(1, 0, 2)
    assert rel(gsh.cpu()[1:], want) < 1e-9
    gc = gc.cpu().numpy()
    assert rel(gc[..., 0] + 1j * gc[..., 1], 2 * np.conj(w[:, None, None, None] * EQ.sum(0))) < 1e-9
