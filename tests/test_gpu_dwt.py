"""The DWT stage alone (every order class's sums over beta and over the series in n), at the sizes
where its forms change: each compile-time DFT length, each MMA form's smallest and largest
bandwidth, partial tiles of 8, even and odd numbers of tiles. A few classes (the first, M' = 0,
M' = M, general ones, the last) against the long-double oracle, both directions.

Tolerance: a sum of up to N + B products of rounded factors is within (N + B + 8) 2^-53 of the exact
one relative to the 2-norms of its factors, 8.7e-14 at B = 256; 1e-13 on the relative L2 error."""
import numpy as np
import pytest

from oracle import oracle as orc

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

REL_TOL = 1e-13
SIZES = [1, 2, 7, 8, 9, 16, 17, 31, 32, 33, 40, 41, 63, 64, 65, 79, 80, 95, 96, 97, 100, 120, 127, 128, 129, 160, 192, 193,
         200, 256]


def _classes(B):
    def index(M, Mp):
        return M * (M + 1) // 2 + Mp

    pick = {(0, 0), (B - 1, 0), (B - 1, B - 1), (B // 2, 0), (B // 2, B // 2), (B // 2, B // 3), (B // 3, B // 4), (B - 1, B // 2)}
    return sorted({index(M, Mp) for M, Mp in pick})


@pytest.mark.parametrize("B", SIZES)
def test_dwt_matches_oracle_classes(lib, oracle, B):
    from pfsoftlib_b200.shard import ShardPlan

    N, cls = 2 * B, _classes(B)
    plan = ShardPlan(B, 1, 0)
    g = torch.Generator(device="cuda")
    g.manual_seed(900 + B)
    x = torch.randn(N ** 3, dtype=torch.complex128, device="cuda", generator=g)
    f = torch.full((orc.coef_count(B),), complex(np.nan, np.nan), dtype=torch.complex128, device="cuda")
    plan.dwt_forward(x, f)
    ref = oracle.dwt_forward(x.cpu().numpy(), B, cls, np.full(orc.coef_count(B), np.nan + 0j))
    at = ~np.isnan(ref)
    got = f.cpu().numpy()
    assert np.isfinite(got).all()
    assert orc.rel_l2(got[at], ref[at]) <= REL_TOL

    c = orc.coeffs_uniform(B, seed=B)
    x.fill_(complex(np.nan, np.nan))
    plan.dwt_inverse(torch.from_numpy(c).cuda(), x)
    ref = oracle.dwt_inverse(c, B, cls, np.full(N ** 3, np.nan + 0j))
    at = ~np.isnan(ref)
    assert orc.rel_l2(x.cpu().numpy()[at], ref[at]) <= REL_TOL


@pytest.mark.parametrize("B", [48, 49, 51, 57, 66, 75, 84, 104, 119, 121, 125, 130, 133, 143, 147, 169, 187, 196, 209, 225, 245, 255])
def test_dwt_dft_lengths(lib, oracle, B):
    """Compile-time DFT lengths of two and three radices, odd ones and the primes 7 .. 19 among them."""
    test_dwt_matches_oracle_classes(lib, oracle, B)
