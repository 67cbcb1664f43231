"""The staged flux's row product (derivative rows, pointwise product and target
rows in one kernel) at every row length, with plane counts around a CTA's
batch and members whose slots interleave, against the oracle.

Tolerances are the flux's own: 1e-12 relative L2 in FP64, 1e-5 in FP32."""

import numpy as np
import pytest

import skb_cuda
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nz,targets,members", [(2, 3, 3, 2), (4, 33, 4, 1), (8, 17, 3, 2), (16, 31, 4, 3), (32, 7, 3, 1),
                                                  (64, 9, 4, 2), (128, 8, 3, 1), (128, 5, 4, 3), (256, 6, 3, 2),
                                                  (512, 3, 4, 3), (512, 9, 3, 1), (1024, 3, 3, 1)])
@pytest.mark.parametrize("mode", ["fp64", "fp32"])
def test_every_row_length(n, nz, targets, members, mode):
    f64 = mode == "fp64"
    dtype = np.complex128 if f64 else np.complex64
    flux = skb_cuda.Flux(n, nz, targets=targets, members=members,
                         mode=skb_cuda.FLUX_FP64_PLAIN if f64 else skb_cuda.FLUX_FP32)
    rng = np.random.default_rng(n + nz)
    x = rng.uniform(-0.125, 0.125, flux.input_elements) + 1j * rng.uniform(-0.125, 0.125, flux.input_elements)
    d_in = skb_cuda.DeviceArray.from_numpy(x.astype(dtype))
    d_out = skb_cuda.DeviceArray.from_numpy(np.zeros(flux.output_elements, dtype))
    perIn, per = flux.input_elements // members, flux.output_elements // members
    for active in (members - 1, members):
        if active == 0:
            continue
        flux.execute_device(d_in.ptr, d_out.ptr, members=active)
        skb_cuda.synchronize()
        out = d_out.download(dtype, flux.output_elements)
        for m in range(members):
            if m < active:
                ref = orc.flux(n, nz, x[m * perIn:(m + 1) * perIn], targets=targets)
                assert orc.rel_l2_error(out[m * per:(m + 1) * per], ref) <= (1e-12 if f64 else 1e-5)
            else:
                assert not out[m * per:(m + 1) * per].any()
