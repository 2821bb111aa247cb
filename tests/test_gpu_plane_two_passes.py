"""Both passes of a small transform in one launch against the two passes of a one-rank slab on the same data, bit
for bit: the butterflies, twiddles and order are the same."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", range(4, 26))
def test_one_launch_equals_two_passes(lib, B):
    from pfsoftlib_b200 import DSOFTFourierCoefficients, FourierTransforms, grid3D
    from pfsoftlib_b200.shard import ShardPlan

    plan = ShardPlan(B, 1, 0)
    g = torch.Generator(device="cuda")
    g.manual_seed(B)
    x = torch.randn((2 * B,) * 3, dtype=torch.complex128, device="cuda", generator=g)
    fc = DSOFTFourierCoefficients(B, device="cuda")
    FourierTransforms.DSOFT(grid3D.wrap(x), fc)
    spectrum = torch.full((8 * B ** 3,), complex("nan"), dtype=torch.complex128, device="cuda")
    want = torch.full_like(fc.mem, complex("nan"))
    plan.fft_forward(x.reshape(-1), spectrum)
    plan.dwt_forward(spectrum, want)
    assert torch.equal(fc.mem, want)
    grid = grid3D(2 * B, device="cuda")
    FourierTransforms.IDSOFT(fc, grid)
    spectrum.fill_(complex("nan"))
    back = torch.full_like(x, complex("nan"))
    plan.dwt_inverse(want, spectrum)
    plan.fft_inverse(spectrum, back.view(-1))   # clears the Nyquist bins first
    assert torch.equal(grid.mem, back)
