"""A transform recorded into a CUDA graph after the bandwidth's first call of another kind (layer-wise DFT, weights,
Wigner matrix, a split plan): the tables it still needs are built beside the recording, which stays whole,
and the replay gives what a direct call gives, bit for bit."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _first_call(lib, kind, B, s):
    N = 2 * B
    if kind == "layers":
        a = torch.zeros(N * N, dtype=torch.complex128, device="cuda")
        return lib.pfsoft_cuda_layer_wise_dft2(N, N, 1, a.data_ptr(), 1.0, s)
    if kind == "weights":
        w = torch.empty(N, dtype=torch.float64, device="cuda")
        return lib.pfsoft_cuda_quadrature_weights(B, w.data_ptr(), s)
    if kind == "wigner":
        d = torch.empty((B, N), dtype=torch.float64, device="cuda")
        return lib.pfsoft_cuda_wigner_d_matrix(B, 0, 0, 0, d.data_ptr(), s)
    from pfsoftlib_b200 import BatchPlan

    assert lib.pfsoft_tune_split_bandwidth(B, 1) == 0
    try:
        BatchPlan([B], split=True).close()
    finally:
        lib.pfsoft_tune_split_bandwidth(0, 1)
    return 0


# bandwidths of no other test: their tables are not there yet
@pytest.mark.parametrize("kind,B", [("layers", 106), ("layers", 173), ("weights", 108), ("wigner", 179), ("split", 110), ("split", 181)])
@pytest.mark.parametrize("forward", [True, False])
def test_capture_after_another_first_call(lib, kind, B, forward):
    B = B if forward else B + 1
    n = B * (4 * B * B - 1) // 3
    g = torch.Generator(device="cuda")
    g.manual_seed(B)
    c = torch.randn(n, dtype=torch.complex128, device="cuda", generator=g)
    grid = torch.randn((2 * B,) * 3, dtype=torch.complex128, device="cuda", generator=g)
    ws = torch.empty(lib.pfsoft_workspace_bytes(B) // 8, dtype=torch.float64, device="cuda")
    out = torch.zeros_like(c if forward else grid)

    def call(s):
        if forward:
            return lib.pfsoft_cuda_dsoft(grid.data_ptr(), B, out.data_ptr(), ws.data_ptr(), ws.numel() * 8, s)
        return lib.pfsoft_cuda_idsoft(c.data_ptr(), B, out.data_ptr(), ws.data_ptr(), ws.numel() * 8, s)

    assert _first_call(lib, kind, B, torch.cuda.current_stream().cuda_stream) == 0, lib.pfsoft_last_error()
    torch.cuda.synchronize()
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        assert call(side.cuda_stream) == 0, lib.pfsoft_last_error()
    out.fill_(complex("nan"))
    graph.replay()
    torch.cuda.synchronize()
    got = out.clone()
    out.fill_(complex("nan"))
    assert call(torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert torch.equal(got, out)
