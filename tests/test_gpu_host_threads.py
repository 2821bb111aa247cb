"""Transforms of different bandwidths from several host threads at once: one kernel serves a range of sizes, each
with its own amount of shared memory, and a launch must not depend on what another thread launches
between its preparation and itself. Every call returns 0, and every result is the single-threaded one
bit for bit."""
import sys
import threading

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _in_threads(work):
    errors, gate = [], threading.Barrier(len(work))

    def run(fn):
        try:
            gate.wait()
            fn()
        except BaseException as e:   # reported by the main thread
            errors.append(e)

    old = sys.getswitchinterval()
    sys.setswitchinterval(1e-5)
    try:
        threads = [threading.Thread(target=run, args=(fn,)) for fn in work]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        sys.setswitchinterval(old)
    assert not errors, errors


# pairs that share a kernel: the DWT's matrix form up to B = 192, 256 and 512, its passes and those of the FFT
@pytest.mark.parametrize("bands", [(137, 166), (193, 251)])
def test_dwt_from_two_threads(lib, bands):
    from pfsoftlib_b200.shard import ShardPlan

    work, state = [], []
    for B in bands:
        g = torch.Generator(device="cuda")
        g.manual_seed(B)
        plan = ShardPlan(B, 64, 5)   # a 64th of the classes: short launches
        x = torch.randn((2 * B) ** 3, dtype=torch.complex128, device="cuda", generator=g)
        want = torch.empty(plan.coef_elems(), dtype=torch.complex128, device="cuda")
        plan.dwt_forward(x, want)
        back = torch.zeros_like(x)
        plan.dwt_inverse(want, back)
        got, gback = torch.empty_like(want), torch.zeros_like(x)
        stream = torch.cuda.Stream()
        state.append((want, got, back, gback))

        def loop(plan=plan, x=x, want=want, got=got, gback=gback, stream=stream):
            for i in range(1500):
                plan.dwt_forward(x, got, stream)
                plan.dwt_inverse(want, gback, stream)
                if i % 100 == 99:
                    stream.synchronize()

        work.append(loop)
    torch.cuda.synchronize()
    _in_threads(work)
    torch.cuda.synchronize()
    for want, got, back, gback in state:
        assert torch.equal(want, got) and torch.equal(back, gback)


def test_layers_from_two_threads(lib):
    """The two-stage, matrix and leftover passes at lengths with different amounts of shared memory."""
    work, state = [], []
    for lengths in ((448, 244, 1000), (544, 362, 648)):
        xs = []
        for n in lengths:
            g = torch.Generator(device="cuda")
            g.manual_seed(n)
            xs.append(torch.randn(3 * 8 * n, dtype=torch.complex128, device="cuda", generator=g))
        stream = torch.cuda.Stream()

        def once(stream, lengths=lengths, xs=xs):
            out = []
            for n, x in zip(lengths, xs):
                y = x.clone()
                assert lib.pfsoft_cuda_layer_wise_dft2(n, 8, 3, y.data_ptr(), 1.0, stream.cuda_stream) == 0, lib.pfsoft_last_error()
                out.append(y)
            return out

        want = once(torch.cuda.current_stream())

        def loop(once=once, want=want, stream=stream):
            with torch.cuda.stream(stream):
                for _ in range(600):
                    got = once(stream)
                    assert all(torch.equal(a, b) for a, b in zip(got, want))

        work.append(loop)
    torch.cuda.synchronize()
    _in_threads(work)


def test_transforms_from_two_threads(lib):
    """The host entry point, B = 137 beside B = 166."""
    from pfsoftlib_b200 import DSOFTFourierCoefficients, FourierTransforms, grid3D

    import numpy as np

    work = []
    for B in (137, 166):
        rng = np.random.default_rng(B)
        x = rng.standard_normal((2 * B,) * 3) + 1j * rng.standard_normal((2 * B,) * 3)
        grid, want = grid3D.wrap(x), DSOFTFourierCoefficients(B)
        FourierTransforms.DSOFT(grid, want)

        def loop(B=B, grid=grid, want=want):
            for _ in range(6):
                got = DSOFTFourierCoefficients(B)
                FourierTransforms.DSOFT(grid, got)
                assert np.array_equal(np.asarray(got.mem), np.asarray(want.mem))

        work.append(loop)
    _in_threads(work)
