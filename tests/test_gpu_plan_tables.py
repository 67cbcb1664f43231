"""Plans hold the tables that their path reads and no others: creating a plan costs an
allocation and a copy for each, in calls whose own time is tens of microseconds."""

import pytest

import skb_cuda

pytestmark = pytest.mark.gpu


def _persistent(handle):
    info = handle.info() if callable(handle.info) else handle.info
    return (info if isinstance(info, dict) else info.as_dict())["persistent_bytes"]


@pytest.mark.parametrize("precision,size", [(skb_cuda.FP64, 8), (skb_cuda.FP32, 4)])
def test_horizontal_plans(precision, size):
    w = skb_cuda.Workload(64, 32, 5, 2)
    modes = skb_cuda.retained_modes(w)
    # Rows of 64: the 64-point table and two orders of the 32-point one (its first
    # radix, 8 forward and 4 inverse, takes no twiddles); columns of 32: radix 8 first.
    twiddles = 64 + (32 - 8) + (32 - 4) + (32 - 8)
    for plan, columns in ((skb_cuda.FFTProvider(w, precision), 33),
                          (skb_cuda.PrunedProvider(w, precision), max(m.stored_kx for m in modes) + 1)):
        maps = 4 * (2 * columns * 32 + columns + 1 + 2 * len(modes)) + 9 * len(modes)
        assert _persistent(plan) == maps + 2 * size * twiddles


@pytest.mark.parametrize("nz,entries", [(129, 256 - 16), (33, 64 - 8), (513, 1024), (50, 98)])
def test_type1_plans(nz, entries):
    assert _persistent(skb_cuda.ConstantStratificationVertical(10, nz)) == 16 * entries
    assert _persistent(skb_cuda.ConstantStratificationVertical(10, nz, skb_cuda.FP32)) == 8 * entries
