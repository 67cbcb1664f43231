"""Every row and column length of the register-ended transforms against the
oracle, at plane counts around the kernels' plane batches (8 to 32 planes per
CTA; 16-plane scratch blocks) and with chunks that run across field views.

Tolerances as in test_gpu_horizontal.py: FP64 1e-12 (max-relative and
relative-L2), FP32 1e-5 relative-L2.
"""

import numpy as np
import pytest

import skb_cuda
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
LENGTHS = [2, 4, 8, 16, 32, 64, 128, 256, 512, 1024]


def close(actual, expected, precision):
    if precision == skb_cuda.FP64:
        return max(orc.rel_l2_error(actual, expected), orc.max_rel_error(actual, expected)) <= 1e-12
    return orc.rel_l2_error(actual, expected) <= 1e-5


@pytest.mark.parametrize("precision", [skb_cuda.FP64, skb_cuda.FP32])
@pytest.mark.parametrize("planes", [(1, 1), (17, 1), (3, 11)])
@pytest.mark.parametrize("n", LENGTHS)
def test_fft_lengths(n, planes, precision):
    for nx, ny in ((n, 4), (4, n)):
        w = skb_cuda.Workload(nx, ny, *planes)
        o = orc.Workload(nx, ny, *planes)
        real = skb_cuda.make_fixture(w, "random", 3 * n + planes[0])
        fft = skb_cuda.FFTProvider(w, precision)
        spec = fft.forward(real)
        expected = orc.fft_r2c(o, real)
        assert close(spec, expected, precision), (nx, ny)
        # An arbitrary spectrum: bins that no real field has are read as FFTW reads them.
        rng = np.random.default_rng(n)
        any_spec = rng.standard_normal(expected.size) + 1j * rng.standard_normal(expected.size)
        assert close(fft.inverse(any_spec), orc.fft_c2r(o, any_spec), precision), (nx, ny)


@pytest.mark.parametrize("precision", [skb_cuda.FP64, skb_cuda.FP32])
@pytest.mark.parametrize("nx,ny", [(n, 16) for n in LENGTHS[3:]] + [(32, n) for n in LENGTHS[3:]])
def test_pruned_lengths(nx, ny, precision):
    w = skb_cuda.Workload(nx, ny, 5, 7)  # 35 planes: chunks cross the views
    o = orc.Workload(nx, ny, 5, 7)
    modes = orc.retained_modes(nx, ny)
    rng = np.random.default_rng(nx + ny)
    retained = rng.standard_normal(len(modes) * 35) + 1j * rng.standard_normal(len(modes) * 35)
    pruned = skb_cuda.PrunedProvider(w, precision)
    real = pruned.inverse(retained)
    assert close(real, orc.fft_c2r(o, orc.embed_retained(o, modes, retained)), precision)
    real = skb_cuda.make_fixture(w, "random", nx)
    assert close(pruned.forward(real), orc.gather_retained(o, modes, orc.fft_r2c(o, real)), precision)
