"""A streamed tensor-core launch that gives up while the next tile's copy is in flight
waits for that copy and no other: with matrix operations withheld it ends in
milliseconds.  (A wait for a copy already used lasts the whole poll limit, 2^22 polls
of 4 us.)  3200 tiles, more than can be resident, so that every thread block has
refilled its stage; one stage and two."""
import os
import subprocess
import sys

import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

PROGRAM = """
import time, torch, minfft_b200
eng = minfft_b200.engine(True)
x = torch.randn(100, 256, 256, dtype=torch.complex64, device="cuda")
y = torch.empty_like(x)
plan = eng.plan("dft", (256, 256))
eng.set_precision(plan.aux, "tc_f16")
plan.batch("dft", x.data_ptr(), y.data_ptr(), 100)
eng.device_status(plan.aux)
assert eng.lib.minfft_b200_test_tc_withhold(256) == 0
t = time.perf_counter()
plan.batch("dft", x.data_ptr(), y.data_ptr(), 100)
assert eng.lib.minfft_b200_device_status(plan.aux) == 5  # MINFFT_B200_ETIMEOUT
t = time.perf_counter() - t
eng.last_error()
assert eng.lib.minfft_b200_test_tc_withhold(0) == 0
plan.batch("dft", x.data_ptr(), y.data_ptr(), 100)
eng.device_status(plan.aux)
ref = torch.fft.fft2(x.to(torch.complex128))
assert (torch.linalg.vector_norm(y - ref) / torch.linalg.vector_norm(ref)).item() <= 1e-6
assert t < 2.0, t
"""


@pytest.mark.parametrize("stages", [1, 2])
def test_give_up_with_a_refill_in_flight(stages):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", PROGRAM], env=dict(os.environ, MINFFT_B200_TC_STAGES=str(stages)), cwd=root,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
