"""Rounding of the short radix-8 kernels and of the steps fused into long lines and the
long jobs of mixed batches: round trips on normal data, four seeds, relative error
against the input.  The bars are what the kernels they replaced (radix 16,
element-wise steps) measured on the same data, and 3% for the spread."""
import numpy as np
import pytest

import minfft_b200

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

PAIRS = {"t2t3": ("dct2", "dct3"), "t4": ("dct4", "dct4"), "realdft": ("realdft", "invrealdft")}


def round_trip(family, single, dims, howmany):
    eng = minfft_b200.engine(single)
    fwd, inv = PAIRS[family]
    rdt, cdt = (torch.float32, torch.complex64) if single else (torch.float64, torch.complex128)
    plan = eng.plan(family, dims)
    mid = dims[:-1] + ((dims[-1] // 2 + 1,) if family == "realdft" else dims[-1:])
    y = torch.empty((howmany,) + mid, dtype=cdt if family == "realdft" else rdt, device="cuda")
    scale = float(np.prod(dims)) * (1 if family == "realdft" else 2.0 ** len(dims))
    errors = []
    for seed in range(1, 5):
        x = torch.randn((howmany,) + dims, dtype=rdt, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))
        z = torch.empty_like(x)
        plan.batch(fwd, x.data_ptr(), y.data_ptr(), howmany)
        plan.batch(inv, y.data_ptr(), z.data_ptr(), howmany)
        torch.cuda.synchronize()
        errors.append((torch.linalg.vector_norm(z.double() / scale - x) / torch.linalg.vector_norm(x.double())).item())
    plan.free()
    return sum(errors) / len(errors)


@pytest.mark.parametrize("family,single,dims,howmany,bar", [
    ("t4", True, (64,), 1500, 1.65e-7), ("t4", True, (64, 64), 30, 2.63e-7), ("t4", True, (256, 256), 2, 3.19e-7),
    ("t2t3", True, (64, 64), 30, 2.76e-7), ("t2t3", True, (256, 256), 2, 3.18e-7),
    ("t4", False, (64, 32, 64), 1, 4.37e-16), ("t4", False, (16, 64), 100, 3.34e-16)])
def test_short_lines(family, single, dims, howmany, bar):
    assert round_trip(family, single, dims, howmany) <= 1.03 * bar


@pytest.mark.parametrize("family,single,dims,howmany,bar", [
    ("t2t3", True, (1 << 16,), 4, 3.21e-7), ("t2t3", True, (1 << 18,), 1, 3.5e-7), ("realdft", True, (1 << 15,), 8, 2.95e-7),
    ("realdft", True, (1 << 18,), 1, 3.4e-7), ("t2t3", False, (1 << 15,), 8, 5.28e-16)])
def test_long_lines(family, single, dims, howmany, bar):
    assert round_trip(family, single, dims, howmany) <= 1.03 * bar


def mixed_round_trip(single, n, count):
    eng = minfft_b200.engine(single)
    rdt = torch.float32 if single else torch.float64
    errors = []
    for seed in range(1, 5):
        x = torch.randn(count, n, dtype=rdt, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))
        y, z = torch.empty_like(x), torch.empty_like(x)
        for src, dst, ops in ((x, y, ("dct4", "dct2")), (y, z, ("dct4", "dct3"))):
            h = eng.mixed_plan([(ops[i % 2], n, src[i].data_ptr(), dst[i].data_ptr()) for i in range(count)])
            eng.mixed_execute(h)
            torch.cuda.synchronize()
            eng.mixed_free(h)
        errors.append((torch.linalg.vector_norm(z.double() / (2.0 * n) - x) / torch.linalg.vector_norm(x.double())).item())
    return sum(errors) / len(errors)


@pytest.mark.parametrize("single,n,bar", [(True, 1 << 15, 2.98e-7), (True, 1 << 16, 3.12e-7), (False, 1 << 16, 5.11e-16)])
def test_long_jobs_of_mixed_batches(single, n, bar):
    assert mixed_round_trip(single, n, 16) <= 1.03 * bar
