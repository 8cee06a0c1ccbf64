"""Single lines and small batches at the lengths where the planner changes radix (512
and 1024 complex points) and at the longest that fit a block: every real kind against
the oracle."""
import numpy as np
import pytest

from conftest import rel_l2, tolerance
from minfft_b200 import OPS
from test_gpu_parity import expected, gpu_apply, make_input

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("single", [False, True], ids=["f64", "f32"])
@pytest.mark.parametrize("dims", [(1024,), (2048,), (8192,), (16384,), (2, 2048), (1024, 4), (2048, 4)],
                         ids=lambda d: "x".join(map(str, d)))
def test_matches_oracle(dims, single):
    rng = np.random.default_rng(sum(dims))
    for op in OPS:
        if op in ("dft", "invdft"):
            continue
        x = make_input(op, dims, rng, single)
        ref = expected(op, x, dims)
        for inplace in (False, True):
            assert rel_l2(gpu_apply(op, x, dims, single, inplace=inplace), ref) <= tolerance(single, dims), (op, inplace)
