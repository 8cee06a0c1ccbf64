"""The streamed column pass where the planner takes it by itself: 512-point
columns of arrays of 128 MiB (256 MiB in single) and more, the smallest such
batch and one that leaves the last round of tiles ragged, and 256-point columns
of rows 2 MiB apart; one line fewer, or rows half as long, keep the one-tile
pass.  Outputs against torch's double-precision FFT with the repository's bars."""
import numpy as np
import pytest

import minfft_b200
from conftest import tolerance

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("single,dims,howmany,length,streamed", [
    (False, (1 << 18,), 31, 512, False), (False, (1 << 18,), 32, 512, True), (False, (1 << 18,), 37, 512, True),
    (True, (1 << 18,), 127, 512, False), (True, (1 << 18,), 131, 512, True),
    (False, (256, 1 << 16), 1, 256, False), (False, (256, 1 << 17), 1, 256, True), (True, (256, 1 << 18), 1, 256, True)])
def test_planned_streamed_columns(single, dims, howmany, length, streamed):
    eng = minfft_b200.engine(single)
    _, rep, _ = eng.plan_selfcheck("dft", dims, howmany)
    assert ("stream_pass<cplx,L=%d,col" % length in rep) == streamed, rep
    g = torch.Generator(device="cuda").manual_seed(9)
    x = torch.randn((howmany,) + dims, dtype=torch.complex64 if single else torch.complex128, device="cuda", generator=g)
    y, z = torch.full_like(x, float("nan")), torch.full_like(x, float("nan"))
    plan = eng.plan("dft", dims)
    plan.batch("dft", x.data_ptr(), y.data_ptr(), howmany)
    plan.batch("invdft", y.data_ptr(), z.data_ptr(), howmany)
    torch.cuda.synchronize()
    plan.free()
    for i in sorted({0, howmany // 2, howmany - 1}):
        ref = torch.fft.fftn(x[i].to(torch.complex128))
        err = torch.linalg.vector_norm(y[i] - ref) / torch.linalg.vector_norm(ref)
        assert err.item() <= tolerance(single, dims), i
    back = torch.linalg.vector_norm(z / float(np.prod(dims)) - x) / torch.linalg.vector_norm(x)
    assert back.item() <= 2 * tolerance(single, dims)
