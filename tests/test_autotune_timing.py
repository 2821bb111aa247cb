"""The autotuner times only what the library lets it choose: transforms_per_cta has no effect in the present kernels, so
no plan is created for it (CPU, a fake library that refuses every call)."""
from pfsoftlib_b200 import autotune


def test_tune_batch_times_nothing():
    assert autotune.tune_batch(object(), [32, 64], [], [], [], use_cache=False) == (1, {})
