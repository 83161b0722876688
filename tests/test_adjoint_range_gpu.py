"""Weight and shift gradients of the synthesis whose terms are large: sums that pass
the float32 range on the way, and single infinite terms."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def params(n, dx, w, S, Z, F):
    """pt_synth_adj_params (L, F, 3) with unit phasors."""
    import torch

    from pyturb_gb300 import _lib
    from pyturb_gb300.backend import stream_handle

    L = len(w)
    ph = np.zeros((L, F, 2, n, 2), np.float32)
    ph[..., 0] = 1.0
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (w, S.view(np.float32), Z.view(np.float32), ph)]
    out = torch.empty((L, F, 3), dtype=torch.float64, device="cuda")
    _lib.call("pt_synth_adj_params", n, dx, L, F, *(t.data_ptr() for t in d), out.data_ptr(), stream_handle())
    return out.cpu().numpy()


def frames(Z):
    """The two frames' gradient spectra of a transformed pair."""
    D = np.conj(Z.astype(np.complex128))
    mirror = np.conj(np.roll(D[::-1, ::-1], (1, 1), (0, 1)))
    return (D + mirror) / 2, (D - mirror) / 2j


@pytest.mark.parametrize("n,F", [(33, 2), (64, 1), (96, 4)])
def test_sums_beyond_float32_match_float64(n, F):
    # terms near 1e38 in the weight sums and 1e34 in the shift sums: a few of the former
    # leave the float32 range
    rng = np.random.default_rng(n)
    L, dx, pairs = 2, 0.1, (F + 1) // 2
    w = np.array([0.5, 1.5], np.float32)
    S = (1e19 * (rng.uniform(1, 2, (L, n, n)) + 1e-4j * rng.uniform(1, 2, (L, n, n)))).astype(np.complex64)
    A = 1e19 * rng.uniform(0.5, 1, (2, pairs, n, n))
    A = (A + np.roll(A[..., ::-1, ::-1], (1, 1), (-2, -1))) / 2     # each frame's gradient spectrum is real
    Z = (A[0] + 1j * A[1]).astype(np.complex64)
    k = np.fft.fftfreq(n, d=dx)
    got = params(n, dx, w, S, Z, F)
    for l in range(L):
        for f in range(F):
            q = np.conj(frames(Z[f // 2])[f % 2]) * S[l].astype(np.complex128)
            # every term is rounded a few times in float32; the sums are of one sign but
            # for the frequencies' own, so errors are compared with the terms' sizes
            assert abs(got[l, f, 0] - q.real.sum()) < 1e-6 * np.abs(q.real).sum()
            ramp = -2 * np.pi * w[l]
            for c, want in ((1, (k[:, None] * q.imag).sum()), (2, (k[None] * q.imag).sum())):
                assert abs(got[l, f, c] - ramp * want) < 1e-6 * abs(ramp) * np.abs(q.imag).sum() / (2 * dx)


def test_an_infinite_term_stays_infinite():
    n, dx = 16, 0.1
    w = np.array([2.0], np.float32)
    S, Z = np.zeros((1, n, n), np.complex64), np.zeros((1, n, n), np.complex64)
    S[0, 5, 3] = 1e19j
    Z[0, 5, 3] = Z[0, n - 5, n - 3] = 1e19   # frame 0: G = 1e19 there, so q = 1e38 i
    got = params(n, dx, w, S, Z, 1)[0, 0]
    assert got[0] == 0.0
    assert got[1] == -np.inf                  # 5 * 1e38 is beyond float32
    np.testing.assert_allclose(got[2], -2 * np.pi * 2.0 / (n * dx) * 3e38, rtol=1e-6)
