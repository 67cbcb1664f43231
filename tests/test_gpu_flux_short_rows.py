"""The fused row kernel of 128- and 256-point rows (four or eight planes per
warp, TMA stages) with 8 and 16 planes per CTA: level counts around the chunk
width, both target counts, partial batches and the reported device status,
against the FP64 flux at the split path's 1e-6 relative L2."""

import numpy as np
import pytest

import skb_cuda
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("planes", [4, 8, 16])
@pytest.mark.parametrize("n,nz,targets,members", [(128, 4, 3, 1), (128, 16, 4, 2), (128, 33, 3, 3), (256, 7, 4, 1),
                                                  (256, 17, 3, 2), (256, 24, 4, 2)])
def test_short_rows_match_fp64(n, nz, targets, members, planes):
    skb_cuda.tune_cache_clear()
    options = dict(targets=targets, members=members, mode=skb_cuda.FLUX_SPLIT_TF32X3)
    flux = skb_cuda.Flux(n, nz, **options)
    rng = np.random.default_rng(n + nz)
    x = rng.uniform(-0.125, 0.125, flux.input_elements) + 1j * rng.uniform(-0.125, 0.125, flux.input_elements)
    x = x.astype(np.complex64)
    d_in = skb_cuda.DeviceArray.from_numpy(x)
    d_out = skb_cuda.DeviceArray(flux.output_elements * 8)
    key = [k for k in flux.autotune(d_in.ptr, d_out.ptr) if k.startswith("flux.rows.planes_per_cta")]
    assert len(key) == 1
    skb_cuda.tune_cache_store(key[0], planes, 0.0)  # 4 is an earlier tuner's choice: accepted
    flux = skb_cuda.Flux(n, nz, **options)
    expected = skb_cuda.Flux(n, nz, targets=targets, members=members).execute(x.astype(np.complex128))
    flux.execute_device(d_in.ptr, d_out.ptr)
    skb_cuda.synchronize()
    flux.check_device()
    assert orc.rel_l2_error(d_out.download(np.complex64, flux.output_elements), expected) <= 1e-6
    if members > 1:  # the first member only; the others' results stay
        d_out.upload(np.zeros(flux.output_elements, np.complex64))
        flux.execute_device(d_in.ptr, d_out.ptr, members=1)
        skb_cuda.synchronize()
        one = d_out.download(np.complex64, flux.output_elements)
        per = flux.output_elements // members
        assert orc.rel_l2_error(one[:per], expected[:per]) <= 1e-6
        assert not one[per:].any()
    skb_cuda.tune_cache_clear()


def test_register_band_columns_at_512():
    """The register-ended band columns as a 512-point tuner choice (form 9)."""
    skb_cuda.tune_cache_clear()
    n, nz, members = 512, 9, 1
    probe = skb_cuda.Flux(n, nz, members=members, mode=skb_cuda.FLUX_SPLIT_TF32X3)
    rng = np.random.default_rng(9)
    x = rng.uniform(-0.125, 0.125, probe.input_elements) + 1j * rng.uniform(-0.125, 0.125, probe.input_elements)
    x = x.astype(np.complex64)
    d_in = skb_cuda.DeviceArray.from_numpy(x)
    d_out = skb_cuda.DeviceArray(probe.output_elements * 8)
    band = [k for k in probe.autotune(d_in.ptr, d_out.ptr) if k.startswith("flux.columns_band.form")]
    for key in band:
        skb_cuda.tune_cache_store(key, 9, 0.0)
    flux = skb_cuda.Flux(n, nz, members=members, mode=skb_cuda.FLUX_SPLIT_TF32X3)
    expected = skb_cuda.Flux(n, nz, members=members).execute(x.astype(np.complex128))
    flux.execute_device(d_in.ptr, d_out.ptr)
    skb_cuda.synchronize()
    assert orc.rel_l2_error(d_out.download(np.complex64, flux.output_elements), expected) <= 1e-6
    skb_cuda.tune_cache_clear()
