"""Split-TF32x3 GEMMs of small groups have no work units: tuning such a plan keeps the
size in force (16) instead of caching whichever of four identical runs was quickest."""

import pytest

import skb_cuda

pytestmark = pytest.mark.gpu


def test_no_unit_size_is_chosen_where_there_are_no_units():
    skb_cuda.tune_cache_clear()
    for n, nz in ((64, 17), (64, 33), (64, 25), (128, 9)):
        flux = skb_cuda.Flux(n, nz, targets=3, members=1, mode=skb_cuda.FLUX_SPLIT_TF32X3)
        d_in = skb_cuda.DeviceArray(flux.input_elements * 8)
        d_out = skb_cuda.DeviceArray(flux.output_elements * 8)
        units = {k: v for k, v in flux.autotune(d_in.ptr, d_out.ptr).items() if "unit_tiles" in k}
        # The 3-target forward GEMM runs the small-group form at all of these sizes.
        (forward,) = [v for k, v in units.items() if " forward " in k]
        assert len(units) == 2 and forward[0] == 16 and forward[1] > 0
    skb_cuda.tune_cache_clear()
