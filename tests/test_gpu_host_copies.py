"""Transforms of pageable host arrays: copies of one chunk, of several, of more than the ring holds, with
ragged last chunks, against the same transform of device arrays, bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 8, 20, 21, 32, 41, 51, 64, 101, 128])
def test_host_transform_equals_device(lib, B):
    from pfsoftlib_b200 import DSOFTFourierCoefficients, FourierTransforms, grid3D

    rng = np.random.default_rng(B)
    n = B * (4 * B * B - 1) // 3
    c = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    hg, dg = grid3D(2 * B), grid3D(2 * B, device="cuda")
    FourierTransforms.IDSOFT(DSOFTFourierCoefficients.wrap(c, B), hg)
    FourierTransforms.IDSOFT(DSOFTFourierCoefficients.wrap(torch.from_numpy(c).cuda(), B), dg)
    assert np.array_equal(np.asarray(hg.mem), dg.mem.cpu().numpy())
    hc, dc = DSOFTFourierCoefficients(B), DSOFTFourierCoefficients(B, device="cuda")
    FourierTransforms.DSOFT(hg, hc)
    FourierTransforms.DSOFT(dg, dc)
    assert np.array_equal(np.asarray(hc.mem), dc.mem.cpu().numpy())
