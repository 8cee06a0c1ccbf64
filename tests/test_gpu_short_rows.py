"""Batches of the shortest rows, which share a block by the hundred: counts around the
128 and 256 rows of a block, and around the 24 MiB from which rows of 128 bytes take
256.  Forward results against torch's double-precision FFT, then back."""
import pytest

import minfft_b200
from conftest import tolerance

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
MANY = (24 << 20) // 128


@pytest.mark.parametrize("single", [False, True], ids=["f64", "f32"])
@pytest.mark.parametrize("family,lengths", [("dft", (2, 4, 8)), ("realdft", (2, 4, 8)), ("t2t3", (2, 4, 8)), ("t4", (2, 4, 8))])
def test_counts_around_a_block(family, lengths, single):
    for n in lengths:
        for howmany in (1, 63, 64, 65, 127, 128, 129, 255, 256, 257, 1001):
            check(family, n, howmany, single)


@pytest.mark.parametrize("family", ["realdft", "t2t3"])
@pytest.mark.parametrize("howmany", [MANY - 1, MANY, MANY + 257])
@pytest.mark.parametrize("single,n", [(False, 16), (True, 32)], ids=["f64", "f32"])
def test_rows_of_128_bytes(family, howmany, single, n):
    check(family, n, howmany, single)


def check(family, n, howmany, single):
    eng = minfft_b200.engine(single)
    rdt, cdt = (torch.float32, torch.complex64) if single else (torch.float64, torch.complex128)
    fwd, inv = {"dft": ("dft", "invdft"), "realdft": ("realdft", "invrealdft"), "t2t3": ("dst2", "dst3"),
                "t4": ("dct4", "dct4")}[family]
    x = torch.randn((howmany, n), dtype=cdt if family == "dft" else rdt, device="cuda",
                    generator=torch.Generator("cuda").manual_seed(n))
    y = torch.full((howmany, n // 2 + 1 if family == "realdft" else n), float("nan"), dtype=rdt if family[0] == "t" else cdt,
                   device="cuda")
    z = torch.full_like(x, float("nan"))
    plan = eng.plan(family, (n,))
    plan.batch(fwd, x.data_ptr(), y.data_ptr(), howmany)
    plan.batch(inv, y.data_ptr(), z.data_ptr(), howmany)
    torch.cuda.synchronize()
    plan.free()
    scale = n * (2.0 if family[0] == "t" else 1.0)
    back = torch.linalg.vector_norm(z / scale - x) / torch.linalg.vector_norm(x)
    assert back.item() <= 2 * tolerance(single, (n,)), (family, n, howmany)
    if family[0] != "t":
        ref = torch.fft.fft(x.to(torch.complex128)) if family == "dft" else torch.fft.rfft(x.double())
        err = torch.linalg.vector_norm(y - ref) / torch.linalg.vector_norm(ref)
        assert err.item() <= tolerance(single, (n,)), (family, n, howmany)
