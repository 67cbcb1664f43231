"""Plans of few planes: their bin arrays are blocks of 16 planes from 16 planes on and
hold just the plan's planes below.  Sizes of the scratch, and results on both sides of
that line (a flux's target array may lie below it and its scratch above).  A flux is
refused, before anything large is allocated, by the same sizes.

Tolerances as in test_gpu_horizontal.py and the flux tests: FP64 1e-12, FP32 1e-5."""

import numpy as np
import pytest

import skb_cuda
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _stored(planes):
    return planes if planes < 16 else (planes + 15) // 16 * 16


def _info(handle):
    info = handle.info() if callable(handle.info) else handle.info
    return info if isinstance(info, dict) else info.as_dict()


def _keep(n):
    return max(m.stored_kx for m in skb_cuda.retained_modes(skb_cuda.Workload(n, n, 2, 1))) + 1


@pytest.mark.parametrize("precision,size", [(skb_cuda.FP64, 8), (skb_cuda.FP32, 4)])
@pytest.mark.parametrize("nz,fields", [(1, 1), (3, 1), (5, 3), (16, 1), (17, 1)])
def test_scratch_of_few_planes(nz, fields, precision, size):
    w = skb_cuda.Workload(64, 32, nz, fields)
    assert _info(skb_cuda.FFTProvider(w, precision))["scratch_bytes"] == 32 * 33 * _stored(nz * fields) * 2 * size
    keep = max(m.stored_kx for m in skb_cuda.retained_modes(w)) + 1
    assert _info(skb_cuda.PrunedProvider(w, precision))["scratch_bytes"] == 32 * keep * _stored(nz * fields) * 2 * size


@pytest.mark.parametrize("precision,tol", [(skb_cuda.FP64, 1e-12), (skb_cuda.FP32, 1e-5)])
@pytest.mark.parametrize("nz,fields", [(1, 1), (1, 3), (3, 5), (4, 4), (7, 2)])
def test_pruned_results(nz, fields, precision, tol):
    w, o = skb_cuda.Workload(32, 64, nz, fields), orc.Workload(32, 64, nz, fields)
    modes = orc.retained_modes(32, 64)
    rng = np.random.default_rng(nz)
    retained = rng.standard_normal(len(modes) * nz * fields) + 1j * rng.standard_normal(len(modes) * nz * fields)
    pruned = skb_cuda.PrunedProvider(w, precision)
    want = orc.fft_c2r(o, orc.embed_retained(o, modes, retained))
    assert orc.rel_l2_error(pruned.inverse(retained), want) <= tol
    real = skb_cuda.make_fixture(w, "random", nz)
    assert orc.rel_l2_error(pruned.forward(real), orc.gather_retained(o, modes, orc.fft_r2c(o, real))) <= tol


def _staged_bytes(n, nz, targets, members):
    modes, keep = len(orc.retained_modes(n, n)), _keep(n)
    planes = 3 * members * nz
    return (16 * members * modes * nz * (3 + 4 * targets)  # physical values of every slot and target
            + 8 * n * n * planes  # U, V and W
            + 16 * n * keep * (_stored(planes) + _stored(members * nz)))


@pytest.mark.parametrize("n,nz,targets,members", [(8, 3, 3, 1), (16, 3, 4, 2), (32, 5, 3, 3), (16, 15, 3, 2)])
def test_staged_flux(n, nz, targets, members):
    flux = skb_cuda.Flux(n, nz, targets=targets, members=members)
    assert _info(flux)["scratch_bytes"] == _staged_bytes(n, nz, targets, members)
    rng = np.random.default_rng(n)
    x = rng.uniform(-0.125, 0.125, flux.input_elements) + 1j * rng.uniform(-0.125, 0.125, flux.input_elements)
    d_in = skb_cuda.DeviceArray.from_numpy(x)
    d_out = skb_cuda.DeviceArray(flux.output_elements * 16)
    per_in, per_out = flux.input_elements // members, flux.output_elements // members
    for active in range(1, members + 1):
        flux.execute_device(d_in.ptr, d_out.ptr, members=active)
        skb_cuda.synchronize()
        out = d_out.download(np.complex128, flux.output_elements)
        for m in range(active):
            ref = orc.flux(n, nz, x[m * per_in:(m + 1) * per_in], targets=targets)
            assert orc.rel_l2_error(out[m * per_out:(m + 1) * per_out], ref) <= 1e-12


@pytest.mark.parametrize("n,nz,targets", [(64, 3, 3), (128, 9, 4), (512, 5, 3)])
def test_fused_scratch(n, nz, targets):
    flux = skb_cuda.Flux(n, nz, targets=targets, members=2, mode=skb_cuda.FLUX_SPLIT_TF32X3)
    bins = 8 * n * _keep(n) * 2 * (3 + 4 * targets) * ((nz + 7) // 8 * 8)
    assert _info(flux)["scratch_bytes"] == bins + 8 * n * _keep(n)  # and the plan's one plane


def test_refusal_names_what_the_handle_would_hold():
    n, nz, targets, members = 1024, 48, 4, 42  # more than any device holds
    w = skb_cuda.Workload(n, n, nz, targets)
    matrices = 16 * len(skb_cuda.squared_wavenumber_groups(w)) * w.nj * nz
    with pytest.raises(MemoryError, match="flux workload needs %d device bytes" %
                       (_staged_bytes(n, nz, targets, members) + matrices)):
        skb_cuda.Flux(n, nz, targets=targets, members=members)
