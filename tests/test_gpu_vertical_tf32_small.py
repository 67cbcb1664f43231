"""The split-TF32x3 vertical GEMM of small groups (tiles of 32 columns) at the
edges of its tiles: rows of 16, inner chunks of 32 and steps of 8, columns of 4,
8 and 32, one common matrix, and cell-addressed operands with conjugates and
kx = 0 partners, against the oracle.

Tolerance 1e-6 relative L2, the split forms' own."""

import numpy as np
import pytest

import skb_cuda
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _values(rng, n):
    return rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n)


@pytest.mark.parametrize("nz,fields", [(3, 1), (5, 7), (9, 2), (16, 3), (17, 1), (25, 4), (32, 2), (33, 5), (48, 1),
                                       (49, 3), (64, 2), (65, 1), (80, 3), (96, 1), (97, 2), (113, 1), (128, 2),
                                       (129, 1)])
def test_tile_edges(nz, fields):
    w = skb_cuda.Workload(16, 16, nz, fields)
    o = orc.Workload(16, 16, nz, fields)
    fam = orc.k2_family(o)
    modes = len(orc.retained_modes(16, 16))
    gemm = skb_cuda.VerticalGemmProvider(w, skb_cuda.squared_wavenumber_groups(w), fam[0], fam[1],
                                         gemm_precision=skb_cuda.GEMM_TF32X3)
    rng = np.random.default_rng(nz)
    physical, modal = _values(rng, modes * fields * nz), _values(rng, modes * fields * w.nj)
    gemm.load_physical_input(physical)
    gemm.load_modal_input(modal)
    gemm.execute_forward()
    gemm.execute_inverse()
    assert orc.rel_l2_error(gemm.copy_forward_output(), orc.grouped_vertical(o, fam, "forward", physical)) <= 1e-6
    assert orc.rel_l2_error(gemm.copy_inverse_output(), orc.grouped_vertical(o, fam, "inverse", modal)) <= 1e-6


@pytest.mark.parametrize("nz,fields", [(7, 2), (33, 3), (66, 1)])
def test_wvm_cells(nz, fields):
    w = skb_cuda.Workload(16, 16, nz, fields)
    o = orc.Workload(16, 16, nz, fields)
    fam = orc.k2_family(o)
    direct = skb_cuda.WvmDirectVerticalProvider(w, skb_cuda.squared_wavenumber_groups(w), fam[0], fam[1],
                                                gemm_precision=skb_cuda.GEMM_TF32X3)
    rng = np.random.default_rng(nz)
    spectrum, modal = _values(rng, direct.spectrum_elements), _values(rng, direct.modal_elements)
    assert orc.rel_l2_error(direct.forward(spectrum), orc.wvm_direct_vertical(o, fam, "forward", spectrum)) <= 1e-6
    assert orc.rel_l2_error(direct.inverse(modal), orc.wvm_direct_vertical(o, fam, "inverse", modal)) <= 1e-6


def test_members_and_partial_batches():
    """A member's flux is bit-identical alone and in a batch of the same handle."""
    n, nz, members = 64, 17, 3
    flux = skb_cuda.Flux(n, nz, targets=3, members=members, mode=skb_cuda.FLUX_SPLIT_TF32X3)
    rng = np.random.default_rng(2)
    x = _values(rng, flux.input_elements).astype(np.complex64)
    d_in = skb_cuda.DeviceArray.from_numpy(x)
    d_out = skb_cuda.DeviceArray(flux.output_elements * 8)
    flux.execute_device(d_in.ptr, d_out.ptr)
    skb_cuda.synchronize()
    whole = d_out.download(np.complex64, flux.output_elements)
    expected = skb_cuda.Flux(n, nz, targets=3, members=members).execute(x.astype(np.complex128))
    assert orc.rel_l2_error(whole, expected) <= 1e-6
    for m in (1, 2):
        flux.execute_device(d_in.ptr, d_out.ptr, members=m)
        skb_cuda.synchronize()
        part = d_out.download(np.complex64, flux.output_elements)
        per = flux.output_elements // members
        assert np.array_equal(part[: m * per], whole[: m * per])
