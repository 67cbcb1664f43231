"""The tcgen05 pipeline of the tensor-core vertical GEMM, chosen or forced, at the
edges of its tiles (rows of 16, inner chunks of 32, columns of 64), and the failure
path of its device waits.

Small split-TF32x3 plans run a form without waits (vertical_tf32.cu), so the shapes
here assert the form that ran.  Tolerance 1e-6 relative L2, the split forms' own."""

import ctypes

import numpy as np
import pytest

import skb_cuda
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _provider(shape, precision=skb_cuda.GEMM_TF32X3):
    w = skb_cuda.Workload(*shape)
    fwd, inv, _ = skb_cuda.vertical_family(w)
    return skb_cuda.VerticalGemmProvider(w, skb_cuda.squared_wavenumber_groups(w), fwd, inv, gemm_precision=precision)


def _on_pipeline(gemm):
    forward, inverse = ctypes.c_int(-1), ctypes.c_int(-1)
    skb_cuda.check(skb_cuda.library().skb_vertical_uses_pipeline(gemm.h, ctypes.byref(forward), ctypes.byref(inverse)))
    return forward.value, inverse.value


def _force(gemm):
    skb_cuda.check(skb_cuda.library().skb_vertical_use_pipeline_for_test(gemm.h))


def _operands(shape):
    o = orc.Workload(*shape)
    fam = orc.k2_family(o)
    modes = len(orc.retained_modes(shape[0], shape[1]))
    rng = np.random.default_rng(shape[2])
    physical, modal = (rng.uniform(-1, 1, modes * shape[3] * n) + 1j * rng.uniform(-1, 1, modes * shape[3] * n)
                       for n in (shape[2], skb_cuda.Workload(*shape).nj))
    return o, fam, physical, modal


def _check_both(gemm, shape):
    o, fam, physical, modal = _operands(shape)
    gemm.load_physical_input(physical)
    gemm.load_modal_input(modal)
    gemm.execute_forward()
    gemm.execute_inverse()
    assert orc.rel_l2_error(gemm.copy_forward_output(), orc.grouped_vertical(o, fam, "forward", physical)) <= 1e-6
    assert orc.rel_l2_error(gemm.copy_inverse_output(), orc.grouped_vertical(o, fam, "inverse", modal)) <= 1e-6


@pytest.mark.parametrize("nz,fields", [(3, 1), (9, 2), (16, 3), (17, 1), (25, 4), (32, 2), (33, 5), (48, 1), (49, 17),
                                       (64, 2), (65, 16), (97, 2), (113, 1), (128, 2), (129, 1)])
def test_forced_pipeline_tile_edges(nz, fields):
    shape = (16, 16, nz, fields)
    gemm = _provider(shape)
    assert _on_pipeline(gemm) == (0, 0)
    _force(gemm)
    assert _on_pipeline(gemm) == (1, 1)
    _check_both(gemm, shape)


def test_forced_pipeline_with_one_common_matrix():
    w = skb_cuda.Workload(16, 16, 33, 3)
    fwd, inv, _ = skb_cuda.vertical_family(w, skb_cuda.FAMILY_COMMON_DCT2)
    modes = len(skb_cuda.retained_modes(w))
    groups = [skb_cuda.ModeGroup(0, 0, modes)]
    rng = np.random.default_rng(5)
    x = rng.uniform(-1, 1, modes * w.planes) + 1j * rng.uniform(-1, 1, modes * w.planes)
    want = (x.reshape(-1, w.nz) @ np.asarray(fwd).reshape(w.nj, w.nz).T).reshape(-1)
    gemm = skb_cuda.VerticalGemmProvider(w, groups, fwd, inv, gemm_precision=skb_cuda.GEMM_TF32X3)
    for forced in (False, True):
        if forced:
            _force(gemm)
        gemm.load_physical_input(x)
        gemm.execute_forward()
        assert orc.rel_l2_error(gemm.copy_forward_output(), want) <= 1e-6


@pytest.mark.parametrize("precision", [skb_cuda.GEMM_TF32X3, skb_cuda.GEMM_BF16X3], ids=["tf32x3", "bf16x3"])
def test_chosen_pipeline_matches_the_oracle(precision):
    shape = (64, 64, 17, 60)  # 264 columns a group
    gemm = _provider(shape, precision)
    assert _on_pipeline(gemm) == (1, 1)
    _check_both(gemm, shape)


@pytest.mark.parametrize("shape,precision", [((64, 64, 17, 2), skb_cuda.GEMM_BF16X3), ((64, 64, 17, 60), skb_cuda.GEMM_TF32X3),
                                             ((64, 64, 17, 2), skb_cuda.GEMM_TF32X3)])
def test_expired_wait_of_the_pipeline(shape, precision):
    gemm = _provider(shape, precision)
    skb_cuda.check(skb_cuda.library().skb_vertical_expire_wait_for_test(gemm.h, ctypes.c_int(1)))
    assert _on_pipeline(gemm) == (1, 1)
    o, fam, physical, _ = _operands(shape)
    gemm.load_physical_input(physical)
    with pytest.raises(RuntimeError, match="bounded device wait expired"):
        gemm.execute_forward()
    gemm.close()
    fresh = _provider(shape, precision)
    fresh.load_physical_input(physical)
    fresh.execute_forward()
    assert orc.rel_l2_error(fresh.copy_forward_output(), orc.grouped_vertical(o, fam, "forward", physical)) <= 1e-6


def test_switches_are_refused_where_no_pipeline_serves():
    gemm = _provider((16, 16, 9, 2), skb_cuda.GEMM_FP64)
    assert _on_pipeline(gemm) == (0, 0)
    with pytest.raises(ValueError):
        _force(gemm)
