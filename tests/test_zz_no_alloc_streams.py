"""The allocation-free inverse FFT from several streams and threads: all calls share
one scratch image and one twiddle table on the device, and must follow one another."""

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [False, True])
def test_overlapping_calls_follow_one_another(threads):
    import torch

    from pyturb_gb300 import _lib

    sizes = (384, 512, 200, 1024)
    torch.manual_seed(0)
    inputs = [torch.randn((2, n, n, 2), device="cuda") for n in sizes]
    streams = [torch.cuda.Stream() for _ in sizes]
    calls = 40

    def run(k, outs, stream):
        for out in outs:
            _lib.call("pt_ifft2_noalloc", sizes[k], inputs[k].data_ptr(), out.data_ptr(), 2, stream)

    want = [torch.empty_like(x) for x in inputs]
    for k in range(len(sizes)):
        run(k, [want[k]], torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    for k, n in enumerate(sizes):
        exact = torch.fft.ifft2(torch.view_as_complex(inputs[k]).to(torch.complex128)) * n * n
        assert float((torch.view_as_complex(want[k]) - exact).norm() / exact.norm()) < 2e-6
    outs = [[torch.full_like(x, np.nan) for _ in range(calls)] for x in inputs]
    torch.cuda.synchronize()
    jobs = [(k, outs[k], streams[k].cuda_stream) for k in range(len(sizes))]
    if threads:
        workers = [threading.Thread(target=run, args=j) for j in jobs]
        for w in workers:
            w.start()
        for w in workers:
            w.join()
    else:
        for c in range(calls):
            for k, o, s in jobs:
                run(k, o[c:c + 1], s)
    torch.cuda.synchronize()
    for k in range(len(sizes)):
        for out in outs[k]:
            assert torch.equal(out, want[k])
