"""Launch-shape numbers that callers keep (mf_tune_get, mf_tune_set)."""
import pytest

from mid_fusion_b200 import build, capi


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def test_kept_integration_numbers_stand_for_a_fast_shape():
    """0..2 have always been shapes without the prefetch and 3..5 with it.
    Each is the kernel at four CTAs per SM, the residency at which no other is
    faster; 2 and 5 (1024 threads per SM) are what they were."""
    assert capi.tune_candidates(capi.TUNE_INTEGRATE) == 6
    for v in range(6):
        shape = capi.tune_describe(capi.TUNE_INTEGRATE, v)
        assert shape.startswith("integrate 4 x 256-thread CTAs per SM"), (v, shape)
        assert ("prefetched" in shape) == (v >= 3), (v, shape)
