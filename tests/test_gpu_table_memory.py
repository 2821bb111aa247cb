"""The constant tables that a process keeps are those that its calls need: a split-mode server builds no
series tables of the FP64 DWT, which for the bandwidths of a serving mix add up to gigabytes, and each
DWT's tables are built once."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_split_server_builds_no_series_tables(lib):
    from pfsoftlib_b200 import DSOFTFourierCoefficients, FourierTransforms, grid3D
    from pfsoftlib_b200.serving import TransformServer

    B = 239   # no other test's bandwidth
    series = 8 * B ** 3 // 3
    grid, fc = grid3D(2 * B, device="cuda"), DSOFTFourierCoefficients(B, device="cuda")
    ws = torch.empty(lib.pfsoft_workspace_bytes(B) // 8, dtype=torch.float64, device="cuda")
    free = lambda: (torch.cuda.synchronize(), torch.cuda.mem_get_info()[0])[1]
    stream = torch.cuda.current_stream().cuda_stream
    dsoft = lambda: lib.pfsoft_cuda_dsoft(grid.mem.data_ptr(), B, fc.mem.data_ptr(), ws.data_ptr(), ws.numel() * 8, stream)
    before = free()
    with TransformServer(budget_bytes=8 << 30, max_batch=2, streams=1, split=True) as srv:
        srv.dsoft(grid.mem, fc.mem).wait(60)
    kept = before - free()
    assert kept < 3 * series, kept          # the split tables alone are 24 B^3 / 6 bytes and a little more
    assert dsoft() == 0
    added = before - kept - free()
    assert 0.9 * series < added < 1.5 * series, added
    assert dsoft() == 0
    assert before - kept - added - free() == 0
