"""One row step's error in the anchored modes: what rounding the new row once leaves,
and nothing that stays the same from step to step."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# Rounding a pixel x to float32 is off by 2^-24 |x| (ulp over sqrt(12), averaged over the
# mantissa: 2.4e-8 |x|), independently from pixel to pixel, and an orthonormal mode keeps
# that. The correction itself is off by a few rounding errors of a thousandth of it.
TOL = 4e-8
# the mean over 100 steps of independent errors is a tenth of that
TOL_MEAN = 8e-9


@pytest.mark.parametrize("W,S", [(364, 2), (728, 9)])
def test_anchored_modes_of_one_step(W, S):
    import torch
    from scipy.fft import dct

    from pyturb_gb300.backend import NoiseStream
    from pyturb_gb300.covariance import AnchorTables, build_operator
    from pyturb_gb300.extrude import RingExtruder
    from pyturb_gb300.fourier import PhaseScreen

    m, steps, dx = 2, 100, 1.0 / 128
    op = build_operator(W, m, dx, 25.0, want_float64=True)
    ring = RingExtruder(W, m, steps + m + 1, [], [0] * S, [1.0] * S,
                        [NoiseStream(50 + s, np.random.default_rng) for s in range(S)],
                        device_operator=op.M, anchor=AnchorTables([op], 32))
    source = PhaseScreen(n=1 << (W - 1).bit_length(), pixel_scale=dx, r0=1.0, L0=25.0, seed=3)
    for s in range(S):
        ring.seed_rows(s, source.generate()[:m, :W].contiguous())
    A = op.M64
    ring.extrude([steps] * S)
    rows = ring.buf.double()
    draws = [np.random.default_rng(50 + s) for s in range(S)]
    errors = []
    for k in range(steps):
        beta = torch.from_numpy(np.stack([q.standard_normal(W) for q in draws])).cuda().float().double()
        z = torch.cat([rows[:, k:k + m].reshape(S, -1), beta], 1)
        errors.append((rows[:, k + m] - z @ A.T).cpu().numpy())
    size = float(rows[:, m:].square().mean().sqrt())
    modes = dct(np.array(errors), type=2, norm="ortho", axis=2)[:, :, :32]
    assert np.sqrt((modes ** 2).mean()) < TOL * size
    assert np.sqrt((modes.mean(0) ** 2).mean()) < TOL_MEAN * size
