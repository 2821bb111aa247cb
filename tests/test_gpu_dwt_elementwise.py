"""The error of single values of a beta column and of single coefficients. A Wigner row is a sum of l + 1 terms whose
sizes add up to at most sqrt((2l+1)/2), so a value of a row that is much smaller than that (a high order near a
pole) carries an absolute error, not a relative one:

  iDSOFT  |dS[k]| <= (N + B + 8) 2^-53 (2B^2/pi) sum_l sqrt((2l+1)/2) |f^l|
  DSOFT   |df^l|  <= (N + B + 8) 2^-53 (pi/(2B^2)) sqrt((2l+1)/2) sum_k w_k |S[k]|

Checked where it is sharpest: a single coefficient of the highest degree, and a single sample near a pole, whose
exact results pass through 100 and more orders of magnitude."""
import numpy as np
import pytest

from oracle import oracle as orc

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [9, 16, 40, 64, 100, 128, 137, 200, 251, 256])
def test_bound_at_single_values(lib, oracle, B):
    from pfsoftlib_b200.shard import ShardPlan

    N, u = 2 * B, (3 * B + 8) * 2.0 ** -53
    plan = ShardPlan(B, 1, 0)
    x = torch.zeros(N ** 3, dtype=torch.complex128, device="cuda")
    f = torch.zeros(orc.coef_count(B), dtype=torch.complex128, device="cuda")
    w, l = oracle.weights(B), B - 1
    scale = np.sqrt((2 * l + 1) / 2.0)
    # orders m1 >= |m2|, m2 >= 0: no reversal, sign -1 but for odd m1 - m2 (class_case, common.cuh)
    for m1, m2 in ((l, l), (l, 0), (l, B // 2), (l, l - 1), (B // 2, B // 3)):
        d = -oracle.wigner_d(B, m1, m2)[l - m1]
        column = x.view(N, N, N)[m2, m1]
        f.zero_()
        at = int(orc.coef_index(l, m1, m2))
        f[at] = 1.0 - 2.0j
        plan.dwt_inverse(f, x)
        norm = 2.0 * B * B / np.pi
        assert np.abs(column.cpu().numpy() - norm * d * (1 - 2j)).max() <= u * norm * scale * abs(1 - 2j), (m1, m2)
        for k in (0, B // 7, B, N - 1):
            x.zero_()
            column[k] = 1.0
            plan.dwt_forward(x, f)
            norm = np.pi / (2.0 * B * B)
            assert abs(f[at].item() - norm * w[k] * d[k]) <= u * norm * scale * w[k], (m1, m2, k)
