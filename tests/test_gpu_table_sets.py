"""What the constant tables of a bandwidth hold on the device, call by call: weights, Wigner matrices, a slab's FFT
passes and a layer-wise DFT leave the small tables only, a split plan adds the split kernel's and not the
FP64 DWT's series (8/3 B^3 bytes), which the first FP64 transform then builds."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


# bandwidths of no other test: their tables are not there yet
@pytest.mark.parametrize("kind,B", [("weights", 233), ("wigner", 234), ("slab", 235), ("split", 236)])
def test_no_series_before_an_fp64_transform(lib, kind, B):
    from pfsoftlib_b200 import BatchPlan
    from pfsoftlib_b200.shard import ShardPlan

    N, series, s = 2 * B, 8 * B ** 3 // 3, torch.cuda.current_stream().cuda_stream
    grid = torch.zeros((N,) * 3, dtype=torch.complex128, device="cuda")
    coef = torch.empty(B * (4 * B * B - 1) // 3, dtype=torch.complex128, device="cuda")
    spectrum = torch.empty_like(grid)
    d = torch.empty((B, N), dtype=torch.float64, device="cuda")
    ws = torch.empty(lib.pfsoft_workspace_bytes(B) // 8, dtype=torch.float64, device="cuda")
    plan = ShardPlan(B, 1, 0)
    small = torch.zeros(2, dtype=torch.complex128, device="cuda")
    assert lib.pfsoft_cuda_layer_wise_dft2(2, 1, 1, small.data_ptr(), 1.0, s) == 0   # the device's first tables
    before = _free()
    if kind == "weights":
        assert lib.pfsoft_cuda_quadrature_weights(B, d.data_ptr(), s) == 0
    elif kind == "wigner":
        assert lib.pfsoft_cuda_wigner_d_matrix(B, 0, 0, 0, d.data_ptr(), s) == 0
    elif kind == "slab":
        plan.fft_forward(grid.view(-1), spectrum.view(-1))
    else:
        assert lib.pfsoft_tune_split_bandwidth(B, 1) == 0
        try:
            with BatchPlan([B], split=True) as p:
                p.idsoft([coef], [grid])
        finally:
            lib.pfsoft_tune_split_bandwidth(0, 1)
    kept = before - _free()
    split = 5 * B ** 3 if kind == "split" else 0   # its own tables: 24 bytes for each of B^3/6 steps, and a little
    assert kept < split + 0.5 * series, kept
    assert lib.pfsoft_cuda_dsoft(grid.data_ptr(), B, coef.data_ptr(), ws.data_ptr(), ws.numel() * 8, s) == 0
    added = before - kept - _free()
    assert 0.9 * series < added < 1.5 * series, added
