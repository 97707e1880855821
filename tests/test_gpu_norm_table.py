"""Norm of a gridding call where the rows that the table of tap sums is built
from fit into shared memory all together, in part, and one at a time (the
largest support and oversampling accepted).  The sums are the reference's, in its order,
so the norm of one point is the oracle's to the bit."""
import numpy as np
import pytest

import fpga_gridding_b200 as fg
from fpga_gridding_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("single", [True, False])
@pytest.mark.parametrize("support,oversample", [
    (1, 1), (4, 4), (36, 4), (40, 31), (99, 32), (127, 32)])
def test_norm_of_one_point(oracle, support, oversample, single):
    rng = np.random.default_rng(support)
    sup = np.array([support], np.int32)
    csh = W.min_conv_size_half(sup, oversample) + 1
    real = np.float32 if single else np.float64
    g = 2 * support + 40
    for off in (0.0, 0.49, -0.27):
        w = dict(num_w_planes=1, support=sup, oversample=oversample,
                 conv_size_half=csh,
                 conv_func=rng.standard_normal(2 * csh * csh, dtype=real),
                 uu=np.array([off / g], real), vv=np.array([-off / g], real),
                 ww=np.zeros(1, real), vis=np.ones(2, real),
                 weight=np.ones(1, real), cell_size_rad=1.0, w_scale=1.0,
                 grid_size=g)
        run = oracle.grid_f if single else oracle.grid_d
        s1, n1, _ = run(w)
        s2, n2, _ = fg.grid_workload(w, single=single)
        assert s1 == s2 == 0
        assert n1 == n2
