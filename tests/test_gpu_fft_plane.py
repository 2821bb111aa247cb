"""Both passes of a small transform in one launch: every N = 8 .. 52 around its range against the long-double
oracle, and bit for bit the same transform in a batch of one, two and three (two passes from N = 34 on).

Tolerance: the sums have at most N + B + 2 N products of rounded factors, so 1e-13 on the relative L2
error is above (3 N + B + 8) 2^-53 = 2.1e-14 at N = 52."""
import pytest

from oracle import oracle as orc

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

REL_TOL = 1e-13


@pytest.mark.parametrize("B", range(4, 27))
def test_small_transforms(lib, oracle, B):
    from pfsoftlib_b200 import BatchPlan, DSOFTFourierCoefficients, FourierTransforms, grid3D

    c = orc.coeffs_uniform(B, seed=40 + B)
    dc = torch.from_numpy(c).cuda()
    grid, back = grid3D(2 * B, device="cuda"), DSOFTFourierCoefficients(B, device="cuda")
    FourierTransforms.IDSOFT(DSOFTFourierCoefficients.wrap(dc, B), grid)
    FourierTransforms.DSOFT(grid, back)
    ref = oracle.idsoft(c, B)
    assert orc.rel_l2(grid.mem.cpu().numpy().reshape(ref.shape), ref) <= REL_TOL
    assert orc.rel_l2(back.mem.cpu().numpy(), oracle.dsoft(grid.mem.cpu().numpy())) <= REL_TOL
    for T in (1, 2, 3):
        grids = [torch.full_like(grid.mem, complex("nan")) for _ in range(T)]
        coefs = [torch.full_like(dc, complex("nan")) for _ in range(T)]
        with BatchPlan([B] * T) as plan:
            plan.idsoft([dc] * T, grids)
            plan.dsoft(grids, coefs)
        for t in range(T):
            assert torch.equal(grids[t], grid.mem) and torch.equal(coefs[t], back.mem)
