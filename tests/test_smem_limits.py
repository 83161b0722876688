"""The dynamic shared-memory limit of a kernel is state that host threads and devices
share: one helper raises it, and no call lowers it under another."""

import re
import threading
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "pyturb_gb300" / "csrc"


def test_one_place_sets_the_limit_of_the_spectral_kernels():
    source = (CSRC / "spectral.cu").read_text()
    assert "cudaFuncSetAttribute" not in source
    assert re.search(r"allow_smem\(\(const void\*\)kernel, bytes, true, name\)", source)


def test_one_place_sets_the_limit():
    # a flag of the process behind such a call would skip the second device of a process
    users = [p.name for p in sorted(CSRC.glob("*.cu*")) if "cudaFuncSetAttribute" in p.read_text()]
    assert users == ["capi.cu"]
    helper = (CSRC / "capi.cu").read_text().split("int allow_smem(")[1].split("\n}\n")[0]
    assert "cudaFuncGetAttributes" in helper and not re.search(r"static (bool|int|size_t)", helper)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [512, 586])
def test_threads_of_different_levels_do_not_refuse_each_other(n):
    import torch

    from pyturb_gb300.fourier import PhaseScreen

    # the column pass needs more shared memory with eight levels than with none
    screens = [PhaseScreen(n=n, pixel_scale=0.02, r0=0.15, L0=25.0, subharmonics=p, seed=3) for p in (0, 8)]
    want = [s.generate(2).cpu().numpy() for s in screens]
    errors, streams = [], [torch.cuda.Stream() for _ in screens]
    start = threading.Barrier(len(screens))

    def draw(screen, stream):
        try:
            with torch.cuda.stream(stream):
                start.wait()
                for _ in range(600):
                    screen.generate(2)
        except Exception as e:   # noqa: BLE001 - reported below
            errors.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=draw, args=q) for q in zip(screens, streams)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors
    assert all(np.isfinite(w).all() for w in want)
