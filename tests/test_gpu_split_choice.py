"""pfsoft_tune_split_bandwidth for every bandwidth at once: 2 runs the split kernel in every group of a split plan, 0
the FP64 kernels in every group, 1 the default; a single bandwidth's choice goes before it."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

BANDS = [20, 33, 64, 64, 97, 128]


def _grids(lib, split):
    from pfsoftlib_b200 import BatchPlan

    out = [torch.full((2 * B,) * 3, complex("nan"), dtype=torch.complex128, device="cuda") for B in BANDS]
    coeffs = []
    for i, B in enumerate(BANDS):
        g = torch.Generator(device="cuda")
        g.manual_seed(i)
        coeffs.append(torch.randn(B * (4 * B * B - 1) // 3, dtype=torch.complex128, device="cuda", generator=g))
    with BatchPlan(BANDS, split=split) as plan:
        plan.idsoft(coeffs, out)
        torch.cuda.synchronize()
    return out


def test_choice_for_every_bandwidth(lib):
    fp64 = _grids(lib, False)

    def fp64_at():
        return [torch.equal(a, b) for a, b in zip(_grids(lib, True), fp64)]

    try:
        assert lib.pfsoft_tune_split_bandwidth(0, 2) == 0
        assert fp64_at() == [False] * len(BANDS)
        assert lib.pfsoft_tune_split_bandwidth(64, 0) == 0
        assert fp64_at() == [B == 64 for B in BANDS]
        assert lib.pfsoft_tune_split_bandwidth(0, 0) == 0
        assert fp64_at() == [True] * len(BANDS)
        assert lib.pfsoft_tune_split_bandwidth(33, 1) == 0
        assert fp64_at() == [B != 33 for B in BANDS]
        assert lib.pfsoft_tune_split_bandwidth(0, 1) == 0
        assert fp64_at() == [True] * len(BANDS)   # the faster form at these sizes
    finally:
        lib.pfsoft_tune_split_bandwidth(0, 1)
