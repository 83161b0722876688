"""Inputs of the synthesis adjoint as a caller may give them: a scale that float32
does not hold, level coefficients that are a lazy conjugate."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def level_gradients(scale, conj=False, n=32, F=5, L=2, P=2):
    """Shift and level gradients of frames whose spectra are zero: the levels' alone."""
    import torch

    from pyturb_gb300.diff import spectral_synthesis
    from pyturb_gb300.fourier import Grid, subharmonic_tables

    rng = np.random.default_rng(1)
    freqs, _ = subharmonic_tables(n, 0.1, 0.15, 25.0, P)
    grid = Grid(n, 0.1, np.asarray(freqs))
    t = lambda a, d: torch.tensor(a, dtype=d, device="cuda", requires_grad=True)  # noqa: E731
    c = rng.standard_normal((P, L, 3, 3)) + 1j * rng.standard_normal((P, L, 3, 3))
    c = t(c.conj() if conj else c, torch.complex64)
    shifts = t(rng.uniform(-5, 5, (F, L, 2)), torch.float64)
    S = torch.zeros((L, n, n), dtype=torch.complex64, device="cuda")
    w = torch.ones(L, device="cuda")
    out = spectral_synthesis(S, w, shifts, grid, 2, n - 4, scale, c.conj() if conj else c, frames_per_chunk=3)
    g = torch.tensor(rng.standard_normal(out.shape), dtype=torch.float32, device="cuda")
    gsh, gc = torch.autograd.grad(out, (shifts, c), g)
    return gsh.cpu().numpy(), gc.cpu().numpy()


@pytest.mark.parametrize("scale", [1.0 + 2.0 ** -24, 0.7, 500.0 / (2 * np.pi), 2.0])
def test_level_gradients_take_the_scale_in_float64(scale):
    # the gradients are linear in the scale; each side rounds a few times in float64
    one, _ = level_gradients(1.0)
    got, _ = level_gradients(scale)
    np.testing.assert_allclose(got, scale * one, rtol=0, atol=1e-13 * np.abs(scale * one).max())


def test_conjugate_view_of_the_coefficients():
    shifts, coef = level_gradients(0.5)
    shifts_c, coef_c = level_gradients(0.5, conj=True)   # conj(conj(c)) as a view
    np.testing.assert_array_equal(shifts_c, shifts)
    np.testing.assert_array_equal(coef_c, coef.conj())
