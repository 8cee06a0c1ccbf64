"""Which complex arrays beyond the L2 run their inner axes slab by slab: with three
steps inside a slab always, with two below 384 MiB, unless one of them is a pass over
512-point columns that streams as one launch; in a tensor-core mode with two below 256
MiB, and not where there are no other axes."""
import pytest

import minfft_b200


@pytest.mark.parametrize("single,dims,howmany,precision,slabs", [
    (True, (256, 256), 300, "fp32", True), (True, (256, 256), 300, "tc_f16", False), (True, (256, 256), 300, "tc_bf16", False),
    (True, (256, 256), 255, "fp32", False), (True, (256, 256), 256, "fp32", True), (True, (256, 256), 767, "fp32", True),
    (True, (256, 256), 768, "fp32", False), (False, (64, 64, 64), 300, "fp32", True), (False, (512, 512), 64, "fp32", False),
    (True, (512, 512), 64, "fp32", True), (True, (512, 512), 128, "fp32", False), (True, (512, 512, 512), 1, "fp32", False),
    (True, (16, 512, 512), 8, "fp32", True), (True, (256, 256, 256), 1, "fp32", True), (True, (256, 256, 256), 1, "tc_f16", True),
    (True, (256, 256, 256), 2, "fp32", True), (True, (256, 256, 256), 2, "tc_bf16", False), (True, (256, 256, 256), 3, "tc_f16", False)])
def test_slabs(single, dims, howmany, precision, slabs):
    for op in ("dft", "invdft"):
        bad, rep, n = minfft_b200.engine(single).plan_selfcheck(op, dims, howmany, precision=precision)
        assert bad == 0, rep
        assert (n > len(dims)) == slabs, rep
