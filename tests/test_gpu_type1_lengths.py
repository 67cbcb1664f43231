"""Register-ended type-I transforms at every length they serve (2(nz-1) = 8 to
512, and 1024 of the kernel that stays), with row counts around the columns of a
CTA and mixed kinds in one arena, against the oracle.

Tolerances as in test_gpu_type1.py: FP64 1e-12, FP32 1e-5 (relative L2)."""

import numpy as np
import pytest

import skb_cuda
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [(skb_cuda.FP64, 1e-12), (skb_cuda.FP32, 1e-5)])
@pytest.mark.parametrize("rows", [1, 5, 43])
@pytest.mark.parametrize("nz", [5, 9, 17, 33, 65, 129, 257, 513])
def test_lengths(nz, rows, precision, tol):
    rng = np.random.default_rng(nz + rows)
    x = rng.standard_normal((rows, 3, nz)) + 1j * rng.standard_normal((rows, 3, nz))
    plans = skb_cuda.ConstantStratificationVertical(rows, nz, precision)
    for kind, name in ((skb_cuda.TYPE1_DCT, "dct"), (skb_cuda.TYPE1_DST, "dst")):
        for normalize in (False, True):
            y = plans.transform(x, kind, 3, 1, 2, normalize)
            expected = orc.type1_transform(x, name, 3, 1, 2, normalize)
            assert orc.rel_l2_error(y.reshape(-1), np.asarray(expected).reshape(-1)) <= tol, (name, normalize)
    a1 = rng.standard_normal((rows, 1, nz)) + 1j * rng.standard_normal((rows, 1, nz))
    got = plans.schedule(x, a1)
    for y, expected in zip(got, orc.type1_schedule(x, a1)):
        assert orc.rel_l2_error(y.reshape(-1), np.asarray(expected).reshape(-1)) <= tol
