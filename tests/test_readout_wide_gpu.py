"""Differentiable readout of screens so large that a realisation's byte offsets pass
32 bits (in all layers together, or in one), on both sides of each bound, and of more
layers than one launch takes together."""

import numpy as np
import pytest

from oracle import readout_diff as rd
from test_readout_diff_gpu import make_case, rel, run_gpu

pytestmark = pytest.mark.gpu

# float32 sums of at most a few hundred products, each rounded at 2^-24, against
# float64; the position gradients subtract neighbouring samples of white noise
TOL, TOL_POS = 1e-5, 1e-4


@pytest.mark.parametrize("L,S,D,n,mags", [
    (12, 80, 1, 65, None), (13, 81, 2, 63, "half"), (16, 72, 2, 40, "last"), (17, 70, 1, 64, None),
    (20, 76, 2, 33, "first"), (21, 60, 2, 31, "half"), (31, 66, 2, 40, "last"), (32, 90, 2, 66, "half")])
def test_many_layers_match_oracle(L, S, D, n, mags):
    # cone magnifications in every layer, or only in the first or last of them, so that
    # launches of one image differ in their form
    lin = np.linspace(0.97, 0.8, L)
    one = {None: None, "half": lin, "first": np.where(np.arange(L) == 0, 0.9, 1.0),
           "last": np.where(np.arange(L) == L - 1, 0.9, 1.0)}[mags]
    screens, w, pos0, mag, n, g = make_case(L + n, 2, L, S, 2, D, n, one)
    out, gs, gw, gp = run_gpu(screens, w, pos0, mag, n, g)
    assert rel(out, rd.layer_readout(screens.astype(np.float64), w.astype(np.float64), pos0, mag, n)) < TOL
    rgs, rgw, rgp = rd.layer_readout_vjp(screens, w.astype(np.float64), pos0, mag, n, g)
    assert rel(gs, rgs) < TOL
    assert rel(gw, rgw) < TOL_POS
    assert rel(gp, rgp) < TOL_POS


def taps(p0, m, n, S):
    u = (p0 + m * np.arange(n)) % S
    i = np.floor(u).astype(np.int64)
    return i % S, (i + 1) % S, u - i


@pytest.mark.parametrize("L,S", [(3, 18918), (3, 18919), (2, 32767), (2, 32769)])
def test_wide_offsets_match_float64(L, S):
    import torch

    from pyturb_gb300.diff import layer_readout

    D, n = 2, 70
    torch.manual_seed(S)
    screens = torch.randn((1, L, S, S), device="cuda", requires_grad=True)
    w = torch.linspace(0.5, 1.5, L, device="cuda", requires_grad=True)
    mag = np.array([[1.0] * L, [0.9] * L])
    pos = np.array([[[S - 40.3137 - 5 * l, S - 20.7291 - 3 * l + 30 * d] for l in range(L)] for d in range(D)])[None]
    tp = torch.tensor(pos, device="cuda", requires_grad=True)
    out = layer_readout(screens, w, tp, mag, n)
    g = torch.randn(out.shape, device="cuda")
    gs, gw, gp = torch.autograd.grad(out, (screens, w, tp), g)
    g64 = g.double().cpu().numpy()
    w64 = w.detach().double().cpu().numpy()
    want, want_w, want_p = np.zeros((D, n, n)), np.zeros(L), np.zeros((D, L, 2))
    for l in range(L):
        block = {}
        for d in range(D):
            r0, r1, fr = taps(pos[0, d, l, 0], mag[d, l], n, S)
            c0, c1, fc = taps(pos[0, d, l, 1], mag[d, l], n, S)
            rows, cols = np.concatenate([r0, r1]), np.concatenate([c0, c1])
            t = torch.tensor
            v = screens.detach()[0, l][t(rows, device="cuda")][:, t(cols, device="cuda")].double().cpu().numpy()
            v = v.reshape(2, n, 2, n)
            a, b = fr[:, None], fc[None]
            val = (1 - a) * ((1 - b) * v[0, :, 0] + b * v[0, :, 1]) + a * ((1 - b) * v[1, :, 0] + b * v[1, :, 1])
            dr = (1 - b) * (v[1, :, 0] - v[0, :, 0]) + b * (v[1, :, 1] - v[0, :, 1])
            dc = (1 - a) * (v[0, :, 1] - v[0, :, 0]) + a * (v[1, :, 1] - v[1, :, 0])
            q = g64[0, 0, d]
            want[d] += w64[l] * val
            want_w[l] += (q * val).sum()
            want_p[d, l] = w64[l] * (q * dr).sum(), w64[l] * (q * dc).sum()
            for rr, wr in ((r0, 1 - a), (r1, a)):
                for cc, wc in ((c0, 1 - b), (c1, b)):
                    for y in range(n):
                        for x in range(n):
                            k = (rr[y], cc[x])
                            block[k] = block.get(k, 0.0) + w64[l] * q[y, x] * float(wr[y, 0] * wc[0, x])
        idx = np.array(list(block))
        got = gs[0, l][t(idx[:, 0], device="cuda"), t(idx[:, 1], device="cuda")].cpu().numpy()
        assert rel(got, np.array(list(block.values()))) < TOL
        assert int((gs[0, l] != 0).sum()) <= len(block)    # nothing anywhere else
    assert rel(out.detach()[0, 0].cpu(), want) < TOL
    assert rel(gw.cpu(), want_w) < TOL_POS
    assert rel(gp.cpu()[0], want_p) < TOL_POS


@pytest.mark.parametrize("n", range(1, 8))
@pytest.mark.parametrize("S,mags", [(31, [1.0, 0.9]), (29, [0.6, 1.0]), (40, [0.4, 0.25]), (66, [1.0, 2.5]), (130, [1.0, 1.0])])
def test_small_pupils_match_oracle(S, mags, n):
    screens, w, pos0, mag, n, g = make_case(S + n, 2, 2, S, 3, 2, n, mags)
    _, gs, gw, gp = run_gpu(screens, w, pos0, mag, n, g)
    rgs, rgw, rgp = rd.layer_readout_vjp(screens, w.astype(np.float64), pos0, mag, n, g)
    assert rel(gs, rgs) < TOL
    assert rel(gw, rgw) < TOL_POS
    assert rel(gp, rgp) < TOL_POS


@pytest.mark.parametrize("S", [300, 46400])   # 46400^2 is beyond a 32-bit pixel index
def test_tiny_pupil_on_a_wide_screen(S):
    import torch

    from pyturb_gb300.diff import layer_readout

    screens = torch.zeros((1, 1, S, S), device="cuda", requires_grad=True)
    w = torch.full((1,), 1.5, device="cuda")
    pos = torch.tensor([[[[S - 1.75, S - 2.5]]]], dtype=torch.float64, device="cuda")
    g = torch.arange(1.0, 5.0, device="cuda").reshape(1, 1, 1, 2, 2)
    out = layer_readout(screens, w, pos, np.ones((1, 1)), 2)
    (gs,) = torch.autograd.grad(out, screens, g)
    # samples at rows S - 1.75 and S - 0.75, columns S - 2.5 and S - 1.5 (all weights exact)
    want = np.zeros((3, 3))
    for y in range(2):
        for x in range(2):
            want[y:y + 2, x:x + 2] += 1.5 * float(g[0, 0, 0, y, x]) * np.outer([0.75, 0.25], [0.5, 0.5])
    rows, cols = torch.tensor([S - 2, S - 1, 0], device="cuda"), torch.tensor([S - 3, S - 2, S - 1], device="cuda")
    np.testing.assert_array_equal(gs[0, 0][rows][:, cols].cpu().numpy(), want.astype(np.float32))
    assert int((gs != 0).sum()) == 9
