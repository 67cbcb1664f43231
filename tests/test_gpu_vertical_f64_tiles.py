"""The FP64 matrix-instruction form of the grouped vertical GEMM at the edges of
its tiles (8 rows, 4 and 32 complex columns, chunks of 28 inner steps and their
rows of 4), in both layouts, against the oracle.

Tolerance 1e-12 (max-relative and relative-L2), as for every FP64 path.
"""

import numpy as np
import pytest

import skb_cuda
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
TOL = 1e-12


# Nz from 3 (one output level) to the largest with up to 288 output rows; Nj = floor(2 (Nz-1) / 3)
# gives both directions other remainders.
@pytest.mark.parametrize("layout", [skb_cuda.INTERLEAVED, skb_cuda.SPLIT])
@pytest.mark.parametrize("nz,fields", [(3, 4), (5, 5), (8, 1), (12, 2), (16, 3), (28, 1), (29, 2), (33, 1),
                                       (41, 3), (56, 2), (57, 1), (64, 5), (73, 1), (90, 2), (112, 1), (129, 6),
                                       (145, 1), (208, 2), (288, 1)])
def test_f64_tile_edges(nz, fields, layout):
    w = skb_cuda.Workload(16, 16, nz, fields)
    o = orc.Workload(16, 16, nz, fields)
    fam = orc.k2_family(o)
    modes = len(orc.retained_modes(16, 16))
    groups = skb_cuda.squared_wavenumber_groups(w)
    gemm = skb_cuda.VerticalGemmProvider(w, groups, fam[0], fam[1], layout)
    rng = np.random.default_rng(nz)

    def values(n):
        return rng.standard_normal(modes * fields * n) + 1j * rng.standard_normal(modes * fields * n)

    physical, modal = values(nz), values(w.nj)
    if layout == skb_cuda.SPLIT:
        gemm.load_physical_input_split(physical.real.copy(), physical.imag.copy())
        gemm.load_modal_input_split(modal.real.copy(), modal.imag.copy())
        gemm.execute_forward()
        gemm.execute_inverse()
        f = gemm.copy_forward_output_split()
        i = gemm.copy_inverse_output_split()
        forward, inverse = f[0] + 1j * f[1], i[0] + 1j * i[1]
    else:
        gemm.load_physical_input(physical)
        gemm.load_modal_input(modal)
        gemm.execute_forward()
        gemm.execute_inverse()
        forward, inverse = gemm.copy_forward_output(), gemm.copy_inverse_output()
    for actual, direction, data in ((forward, "forward", physical), (inverse, "inverse", modal)):
        expected = orc.grouped_vertical(o, fam, direction, data)
        assert orc.rel_l2_error(actual, expected) <= TOL
        assert orc.max_rel_error(actual, expected) <= TOL
