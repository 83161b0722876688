"""Row steps of few screens against a float64 recursion: widths around the CTA
count's multiples, every job-count form, mixed row counts and groups, with and
without the anchor."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# float32 dot products of K <= 2400 terms (rounding at most K 2^-24 of the
# absolute sum, in practice sqrt(K)) carried over four rows of a contracting recursion
TOL = 2e-6


def contraction(rng, G, W, m):
    A = rng.standard_normal((G, W, m * W)) * (0.5 / np.sqrt(m * W))
    B = rng.standard_normal((G, W, W)) / np.sqrt(W)
    return np.concatenate([A, B], axis=2).astype(np.float32)


@pytest.mark.parametrize("W,m,counts,groups,anchored", [
    (4, 1, [3], [0], False), (31, 2, [4, 2, 0], [0, 0, 0], False), (33, 2, [1, 4], [0, 1], True),
    (152, 2, [2] * 9, [0] * 9, True), (153, 3, [4, 1, 3, 0, 2], [1, 0, 1, 0, 1], True),
    (305, 2, [2, 3] * 5, [0] * 10, True), (457, 1, [1] * 16, [0] * 16, False),
    (760, 2, [2], [0], True), (761, 2, [3, 1], [0, 0], True),
    (200, 2, [2] * 17, [0] * 17, True),   # one job more than the row step takes: the tiled product
])
def test_rows_match_float64_recursion(W, m, counts, groups, anchored):
    import torch

    from pyturb_gb300.backend import NoiseStream
    from pyturb_gb300.covariance import AnchorTables, ExtrusionOperator
    from pyturb_gb300.extrude import RingExtruder

    rng = np.random.default_rng(W + m)
    S, G = len(counts), max(groups) + 1
    M = contraction(rng, G, W, m)
    dev = torch.from_numpy(M).cuda()
    anchor = None
    if anchored:
        anchor = AnchorTables([ExtrusionOperator(W, m, [], dev[g], dev[g].double()) for g in range(G)])
    bscale = list(rng.uniform(0.5, 2.0, S))
    cap = m + 3 if S < 9 else m + 9     # short rings wrap inside the run
    ring = RingExtruder(W, m, cap, [], groups, bscale,
                        [NoiseStream(50 + s, np.random.default_rng) for s in range(S)],
                        device_operator=dev, anchor=anchor)
    seeds = rng.standard_normal((S, m, W)).astype(np.float32)
    for s in range(S):
        ring.seed_rows(s, torch.from_numpy(seeds[s]).cuda())
    ring.extrude(counts)
    got = ring.buf.double().cpu().numpy()

    draws = [np.random.default_rng(50 + s) for s in range(S)]
    rows = [list(seeds[s].astype(np.float64)) for s in range(S)]
    for k in range(max(counts)):
        for s in range(S):
            if k < counts[s]:
                beta = draws[s].standard_normal(W) * np.float32(bscale[s])
                rows[s].append(M[groups[s]].astype(np.float64) @ np.concatenate(rows[s][-m:] + [beta]))
    for s in range(S):
        assert ring.top[s] == m + counts[s]
        for v in range(max(0, len(rows[s]) - cap), len(rows[s])):
            err = np.linalg.norm(got[s, v % cap] - rows[s][v]) / np.linalg.norm(rows[s][v])
            assert err < TOL, (s, v)
