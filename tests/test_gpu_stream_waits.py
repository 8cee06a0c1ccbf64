"""The waits between the groups of a streamed column pass: a group that waits for
another group's refill outlasts a long one, and where its limit does run out the
launch ends, says so, and leaves the plan usable.  64 lines of 2^18 points: their
first pass keeps three tiles in flight for two groups, so each refill serves the
other group."""
import pytest

import minfft_b200
from conftest import tolerance

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
LINE, LINES = 1 << 18, 64


@pytest.fixture
def lines():
    eng = minfft_b200.engine(False)
    assert "stream_pass<cplx,L=512,col" in eng.plan_selfcheck("dft", (LINE,), LINES)[1]
    x = torch.randn((LINES, LINE), dtype=torch.complex128, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    plan = eng.plan("dft", (LINE,))
    y = torch.full_like(x, float("nan"))
    yield eng, plan, x, y
    assert eng.lib.minfft_b200_test_stream_stall(0, 0) == 0
    torch.cuda.synchronize()
    plan.free()


def right(x, y):
    ref = torch.fft.fft(x)
    return (torch.linalg.vector_norm(y - ref) / torch.linalg.vector_norm(ref)).item() <= tolerance(False, (LINE,))


def test_waits_outlast_a_slow_refill(lines):
    eng, plan, x, y = lines
    assert eng.lib.minfft_b200_test_stream_stall(1000000, 0) == 0  # about a second
    plan.batch("dft", x.data_ptr(), y.data_ptr(), LINES)
    eng.device_status(plan.aux)
    assert right(x, y)


def test_a_wait_that_runs_out_is_reported_and_the_plan_recovers(lines):
    eng, plan, x, y = lines
    assert eng.lib.minfft_b200_test_stream_stall(100000, 1000) == 0
    plan.batch("dft", x.data_ptr(), y.data_ptr(), LINES)
    assert eng.lib.minfft_b200_device_status(plan.aux) == 5  # MINFFT_B200_ETIMEOUT
    eng.last_error()
    assert eng.lib.minfft_b200_test_stream_stall(0, 0) == 0
    plan.batch("dft", x.data_ptr(), y.data_ptr(), LINES)
    eng.device_status(plan.aux)
    assert right(x, y)
