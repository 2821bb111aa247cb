"""The split-precision kernel itself at every size, asked for with pfsoft_tune_split_bandwidth (a split plan takes
the FP64 kernels where those are faster): against the FP64 plan, the long-double oracle, several bandwidths in one
launch, and its bounded-wait exit above B = 16. That the kernel ran shows in the results, which are not the
FP64 kernels' bit for bit.

Tolerance: relative L2 error <= 1e-11 against FP64 results, the split path's stated bound."""
import contextlib
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SPLIT = 2
REL_TOL = 1e-11


def _rel(a, b):
    return (torch.linalg.vector_norm(a - b) / torch.linalg.vector_norm(b)).item()


@contextlib.contextmanager
def _split_everywhere(lib, bws):
    try:
        for B in set(bws):
            assert lib.pfsoft_tune_split_bandwidth(B, 1) == 0
        yield
    finally:
        lib.pfsoft_tune_split_bandwidth(0, 1)


def _ptrs(ts):
    return (ctypes.c_void_p * len(ts))(*[t.data_ptr() for t in ts])


def _run(lib, bws, coeffs, flags):
    s = torch.cuda.current_stream().cuda_stream
    grids = [torch.full((2 * B,) * 3, complex("nan"), dtype=torch.complex128, device="cuda") for B in bws]
    back = [torch.full_like(c, complex("nan")) for c in coeffs]
    plan = ctypes.c_void_p()
    assert lib.pfsoft_batch_create((ctypes.c_int * len(bws))(*bws), len(bws), 0, flags, ctypes.byref(plan)) == 0
    assert lib.pfsoft_batch_idsoft(plan, _ptrs(coeffs), _ptrs(grids), s) == 0
    assert lib.pfsoft_batch_dsoft(plan, _ptrs(grids), _ptrs(back), s) == 0
    torch.cuda.synchronize()
    assert lib.pfsoft_batch_status(plan) == 0
    lib.pfsoft_batch_destroy(plan)
    return grids, back


def _coeffs(lib, bws, seed0):
    out = []
    for i, B in enumerate(bws):
        c = torch.empty(B * (4 * B * B - 1) // 3, dtype=torch.complex128, device="cuda")
        assert lib.pfsoft_cuda_random_coeffs(c.data_ptr(), B, seed0 + i, 1, 1.0, torch.cuda.current_stream().cuda_stream) == 0
        out.append(c)
    return out


def _compare(lib, bws, seed0):
    cs = _coeffs(lib, bws, seed0)
    g64, c64 = _run(lib, bws, cs, 0)
    with _split_everywhere(lib, bws):
        gsp, csp = _run(lib, bws, cs, SPLIT)
    for t, B in enumerate(bws):
        assert _rel(gsp[t], g64[t]) <= REL_TOL and _rel(csp[t], c64[t]) <= REL_TOL, (t, B)
        assert _rel(csp[t], cs[t]) <= REL_TOL, (t, B)   # round trip
        assert not torch.equal(gsp[t], g64[t]), (t, B)


@pytest.mark.parametrize("B,T", [(3, 2), (17, 1), (32, 6), (37, 3), (64, 4), (100, 2), (128, 5), (192, 2), (256, 2)])
def test_split_kernel_matches_fp64(lib, B, T):
    _compare(lib, [B] * T, 1000 * B + T)


def test_several_bandwidths_in_one_launch(lib):
    _compare(lib, [16, 24, 32, 32, 40, 64, 64, 64, 64, 16, 97, 130, 130], 77)


def test_split_kernel_against_oracle(lib, oracle):
    from oracle import oracle as orc

    for B in (20, 33, 40):
        c = orc.coeffs_uniform(B, seed=B)
        dc = torch.from_numpy(c).to("cuda")
        with _split_everywhere(lib, [B]):
            grids, back = _run(lib, [B, B], [dc, dc], SPLIT)
        f_ref, g_ref = oracle.dsoft(grids[0].cpu().numpy()), oracle.idsoft(c, B)
        g64, _ = _run(lib, [B], [dc], 0)
        assert not torch.equal(g64[0], grids[0])
        for t in range(2):
            assert orc.rel_l2(grids[t].cpu().numpy(), g_ref) <= REL_TOL, B
        assert orc.rel_l2(back[0].cpu().numpy(), f_ref) <= REL_TOL, B


@pytest.mark.parametrize("B", [16, 64])
def test_bounded_wait_exit_of_the_forced_kernel(lib, B):
    bws = [B, B]
    cs = _coeffs(lib, bws, 5)
    grids = [torch.empty((2 * B,) * 3, dtype=torch.complex128, device="cuda") for _ in bws]
    plan = ctypes.c_void_p()
    with _split_everywhere(lib, bws):
        assert lib.pfsoft_batch_create((ctypes.c_int * 2)(*bws), 2, 0, SPLIT | 1, ctypes.byref(plan)) == 0
    try:
        assert lib.pfsoft_test_split_wait_ns(1_000_000) == 0      # 1 ms
        assert lib.pfsoft_batch_idsoft(plan, _ptrs(cs), _ptrs(grids), torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
    finally:
        lib.pfsoft_test_split_wait_ns(0)
    assert lib.pfsoft_batch_status(plan) == 3                       # PFSOFT_ETIMEOUT
    lib.pfsoft_batch_destroy(plan)
