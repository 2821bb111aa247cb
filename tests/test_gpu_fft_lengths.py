"""The layer-wise DFT at the lengths where its kernels change: the edges of every planned convolution
length of the chirp pass, even (split in two) and odd, with ragged vector counts, along the contiguous
and the strided direction; and every short length. Against torch.fft in FP64.

Tolerance: two transforms of length M = 2^10 at most and three products, 2 * 10 + 3 roundings of a few
2^-53 each on the relative L2 error, under 1e-14 in root mean square; 1e-13."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

REL_TOL = 1e-13
EVEN = [14, 22, 26, 34, 58, 62, 74, 94, 98, 118, 122, 126, 134, 158, 178, 182, 194, 254, 262, 302, 314, 326, 382, 386, 502, 514, 634,
        662, 1018, 1022]
ODD = [7, 13, 17, 31, 37, 47, 61, 67, 79, 97, 127, 131, 157, 191, 251, 257, 317, 331, 509]


def _check(rows, cols, lays, seed):
    from pfsoftlib_b200 import grid3D

    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = torch.randn((lays, cols, rows), dtype=torch.complex128, device="cuda", generator=g)
    for inverse in (False, True):
        y = grid3D.wrap(x.clone())
        (y.layer_wise_IDFT2 if inverse else y.layer_wise_DFT2)(0.5)
        f = torch.fft.ifft2(x, norm="forward") if inverse else torch.fft.fft2(x)
        err = (torch.linalg.vector_norm(y.mem - 0.5 * f) / torch.linalg.vector_norm(0.5 * f)).item()
        assert err <= REL_TOL, (rows, cols, lays, inverse, err)


@pytest.mark.parametrize("n", EVEN + ODD)
def test_chirp_lengths(lib, n):
    _check(n, 3, 5, n)     # contiguous elements, five vectors (layers) per column
    _check(3, n, 19, n)    # strided elements
    _check(19, n, 2, n)    # strided elements, ragged vectors


def test_every_short_length(lib):
    for n in range(1, 300):
        _check(n, 5, 3, n)
        _check(9, n, 2, n)


@pytest.mark.parametrize("n", [323, 361, 408, 456, 460, 496, 506, 529, 551, 713, 899, 961, 992])
def test_prime_radices_17_to_31(lib, n):
    _check(n, 3, 5, n)
    _check(3, n, 19, n)
    _check(19, n, 2, n)


@pytest.mark.parametrize("n", [38, 46, 86, 106, 111, 129, 185, 222, 259, 289, 333, 407, 444, 490, 505, 514, 578, 654, 1028])
def test_matrix_lengths(lib, n):
    """n = R p: the first and last p, every parity of the tiles of four and eight, R = 1 .. 12."""
    _check(n, 3, 5, n)
    _check(3, n, 19, n)
    _check(19, n, 2, n)
