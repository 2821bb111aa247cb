"""The '-split' workloads run the split-precision kernel: their round-trip error is that of the digit products, well
above the FP64 kernels' on the same inputs (about 1e-13 and more against 1e-16 and less)."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["batch-32x2", "batch-128x2"])
def test_split_workload_is_split(lib, name):
    from pfsoftlib_b200 import workloads

    fp64, split = workloads.run(name), workloads.run(name + "-split")
    assert fp64 < split < 1e-9
    assert workloads.run(name) == fp64   # and the default is back
