"""Slabs under the real DFT: the complex steps of batched 3-D arrays whose spectra are
beyond the L2, both ways, out of place and in place, the last slab shorter; spectra of
an odd number of columns.  Against torch's double-precision FFT."""
import numpy as np
import pytest

import minfft_b200
from conftest import tolerance

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("single,dims,howmany", [(False, (64, 64, 64), 70), (True, (32, 128, 128), 77)], ids=["f64", "f32"])
def test_real_dft_of_batched_arrays(single, dims, howmany):
    eng = minfft_b200.engine(single)
    for op in ("realdft", "invrealdft"):
        bad, rep, n = eng.plan_selfcheck(op, dims, howmany)
        assert bad == 0 and n > 4, rep
    rdt, cdt = (torch.float32, torch.complex64) if single else (torch.float64, torch.complex128)
    spec = dims[:-1] + (dims[-1] // 2 + 1,)
    x = torch.randn((howmany,) + dims, dtype=rdt, device="cuda", generator=torch.Generator("cuda").manual_seed(6))
    y = torch.full((howmany,) + spec, float("nan"), dtype=cdt, device="cuda")
    z = torch.full_like(x, float("nan"))
    plan = eng.plan("realdft", dims)
    plan.batch("realdft", x.data_ptr(), y.data_ptr(), howmany)
    w = y.clone()  # the inverse reads its input only
    plan.batch("invrealdft", y.data_ptr(), z.data_ptr(), howmany)
    torch.cuda.synchronize()
    assert torch.equal(w, y)
    for i in (0, howmany // 2, howmany - 1):
        ref = torch.fft.rfftn(x[i].double())
        assert (torch.linalg.vector_norm(y[i] - ref) / torch.linalg.vector_norm(ref)).item() <= tolerance(single, dims), i
    scale = float(np.prod(dims))
    back = torch.linalg.vector_norm(z / scale - x) / torch.linalg.vector_norm(x)
    assert back.item() <= 2 * tolerance(single, dims)
    # in place: one array of spectra that starts as the reals
    buf = torch.zeros_like(y)
    reals = torch.view_as_real(buf).flatten()[:x.numel()]
    reals.copy_(x.flatten())
    plan.batch("realdft", buf.data_ptr(), buf.data_ptr(), howmany)
    torch.cuda.synchronize()
    assert torch.equal(buf, y)
    plan.batch("invrealdft", buf.data_ptr(), buf.data_ptr(), howmany)
    torch.cuda.synchronize()
    plan.free()
    assert torch.equal(reals.view_as(z), z)
