"""Columns of 4096 complex points, two to a block (with scalar sums in single): one,
two and more blocks, both ways, in place, and under the real DFT's odd row pitch."""
import numpy as np
import pytest

import minfft_b200
from conftest import rel_l2, tolerance
from test_gpu_parity import expected, gpu_apply, make_input

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("single", [False, True], ids=["f64", "f32"])
@pytest.mark.parametrize("op,dims", [("dft", (4096, 2)), ("dft", (4096, 8)), ("invdft", (4096, 4)), ("dft", (2, 4096, 4)),
                                     ("realdft", (4096, 8)), ("invrealdft", (4096, 8)), ("realdft", (16384, 32))])
def test_columns(op, dims, single):
    _, rep, _ = minfft_b200.engine(single).plan_selfcheck(op, dims)
    assert "L=4096,col" in rep, rep
    x = make_input(op, dims, np.random.default_rng(4), single)
    ref = expected(op, x, dims)
    for inplace in (False, True):
        assert rel_l2(gpu_apply(op, x, dims, single, inplace=inplace), ref) <= tolerance(single, dims), inplace
