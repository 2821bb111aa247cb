"""The DWT at bandwidths above 256 (beta sums by the matrix product, up to the last one, 512): every output
finite, and the coefficients and beta columns of a few orders, the extreme ones among them, against
sums in extended precision over the long-double oracle's Wigner rows.

Tolerance: a sum of up to N + B products of rounded factors is within (N + B + 8) 2^-53 of the exact one
relative to the product of its factors' 2-norms."""
import numpy as np
import pytest

from oracle import oracle as orc

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _orders(B):
    return [(0, 0), (B - 1, 0), (0, 1 - B), (1 - B, B - 1), (B - 1, B - 24), (B - 1, 23), (23, 1 - B), (B // 2, -(B // 3)),
            (-(B // 4), B // 2), (1, -2), (5, B // 2)]


def _rows(oracle, B, m1, m2):
    """The rows l = max(|m1|, |m2|) .. B - 1 that take the column of (m1, m2) to its coefficients, from those of the
    orders (M, M'), M >= M' >= 0: reversal in beta and signs as in class_case (common.cuh)."""
    M, Mp = max(abs(m1), abs(m2)), min(abs(m1), abs(m2))
    d = oracle.wigner_d(B, M, Mp).astype(np.longdouble)
    if (m1 < 0) != (m2 < 0):
        d = d[:, ::-1] * np.where((np.arange(M, B) - M) % 2, -1, 1)[:, None]
    x = m1 < 0 if abs(m1) == M else m2 > 0
    return d if x and (M - Mp) % 2 else -d


def _column(x, B, m1, m2):
    return x.view(2 * B, 2 * B, 2 * B)[m2 % (2 * B), m1 % (2 * B)]


@pytest.mark.parametrize("B", [257, 300, 511, 512])
def test_dwt_above_256(lib, oracle, B):
    from pfsoftlib_b200.shard import ShardPlan

    N, tol = 2 * B, (3 * B + 8) * 2.0 ** -53
    plan = ShardPlan(B, 1, 0)
    g = torch.Generator(device="cuda")
    g.manual_seed(B)
    x = torch.randn(N ** 3, dtype=torch.complex128, device="cuda", generator=g)
    f = torch.full((orc.coef_count(B),), complex(np.nan, np.nan), dtype=torch.complex128, device="cuda")
    plan.dwt_forward(x, f)
    assert torch.isfinite(torch.view_as_real(f)).all()
    w = oracle.weights(B).astype(np.longdouble)
    rows = {}
    for m1, m2 in _orders(B):
        d = rows[m1, m2] = _rows(oracle, B, m1, m2)
        l = np.arange(B - d.shape[0], B)
        got = f[torch.from_numpy(orc.coef_index(l, m1, m2)).cuda()].cpu().numpy()
        s = w * _column(x, B, m1, m2).cpu().numpy().astype(np.clongdouble)
        norm = np.pi / (2.0 * B * B)
        bound = tol * norm * np.sqrt((d * d).sum(1)) * np.sqrt((abs(s) ** 2).sum())
        assert (abs(got - norm * (d @ s)) <= bound).all(), (m1, m2)

    x.fill_(complex(np.nan, np.nan))
    f = torch.randn(orc.coef_count(B), dtype=torch.complex128, device="cuda", generator=g)
    plan.dwt_inverse(f, x)
    for m in range(N):   # every column but the Nyquist bins' (not written by this stage)
        row = torch.isfinite(torch.view_as_real(x.view(N, N, N)[m])).all(dim=2).all(dim=1)
        row[B] = True
        assert m == B or row.all(), m
    for m1, m2 in _orders(B):
        d = rows[m1, m2]
        l = np.arange(B - d.shape[0], B)
        c = f[torch.from_numpy(orc.coef_index(l, m1, m2)).cuda()].cpu().numpy().astype(np.clongdouble)
        norm = 2.0 * B * B / np.pi
        got = _column(x, B, m1, m2).cpu().numpy()
        err = np.sqrt((abs(got - norm * (d.T @ c)) ** 2).sum())
        assert err <= tol * norm * np.sqrt((d * d).sum() * (abs(c) ** 2).sum()), (m1, m2)
