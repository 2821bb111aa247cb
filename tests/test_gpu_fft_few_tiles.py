"""Two-stage passes with few tiles (four vectors each from radix 17 on) against the same layers among many (eight
vectors), and the two sides of the line: bit for bit."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [136, 272, 320, 391, 448, 496, 512, 544, 640, 768, 900, 960, 1024])
def test_few_tiles_equal_many(lib, n):
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    s = torch.cuda.current_stream().cuda_stream
    for rows, cols in ((n, 21), (21, n)):
        x = torch.randn((170, cols, rows), dtype=torch.complex128, device="cuda", generator=g)
        for dft in (lib.pfsoft_cuda_layer_wise_dft2, lib.pfsoft_cuda_layer_wise_idft2):
            want = x.clone()
            assert dft(cols, rows, 170, want.data_ptr(), 0.5, s) == 0
            for first, lays in ((0, 1), (3, 9), (40, 49), (90, 57), (11, 65)):
                got = x[first:first + lays].clone()
                assert dft(cols, rows, lays, got.data_ptr(), 0.5, s) == 0
                assert torch.equal(got, want[first:first + lays]), (rows, cols, first, lays)
