"""Error growth along a run of equally spaced frames: the ratio that carries a layer
from frame to frame is one rounded phasor of the exact phase."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# A phase in turns rounds to float32 with 0.7e-8 rms, 4.2e-8 radians, and the phasor's
# components add 2.1e-8: 4.7e-8 a ratio, which fifteen steps carry to 7.0e-7. Fifteen
# rounded products add 1.2e-7, the transform 1.7e-7: 7.3e-7 in all on a white spectrum.
# (A ratio that is a product of two such phasors: 1.0e-6.)
TOL = 8.5e-7


@pytest.mark.parametrize("seed", range(4))
def test_last_frame_of_a_run(seed):
    import torch

    from pyturb_gb300.backend import NoiseStream
    from pyturb_gb300.flow import SpectralLayers

    n, dx, F = 1000, 0.02, 16    # the frames of one run at this size
    f = np.fft.fftfreq(n, d=dx)
    rng = np.random.default_rng(seed)
    layer = SpectralLayers(n, dx, np.zeros((0, 3)), np.ones((1, n, n)), np.zeros((0, 1, 3, 3)),
                           [NoiseStream(seed, None)])
    s0, step = rng.uniform(-30, 30, 2), rng.uniform(-0.3, 0.3, 2)
    s = s0 + np.arange(F)[:, None] * step
    got = layer.frames(s[:, :1], s[:, 1:], 0, n, 1.0)[-1].double()
    S = torch.view_as_complex(layer.spectra.double())[0]
    k = torch.tensor(f, device="cuda")
    px, py = (torch.exp(2j * np.pi * k * float(v)) for v in s[-1])
    want = torch.fft.ifft2(S * px[:, None] * py[None]).real * n * n
    assert float((got - want).norm() / want.norm()) < TOL
