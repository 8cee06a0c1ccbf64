"""The long transforms of a mixed batch: the wait for their tiles where it runs out,
the wait for a scratch slot (more transforms of one length than slots), and real rows
that are not aligned for pairs."""
import numpy as np
import pytest

import minfft_b200
from conftest import tolerance
from minfft_b200 import MinfftError
from test_gpu_mixed import check_batch, make_batch

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
precisions = pytest.mark.parametrize("single", [False, True], ids=["f64", "f32"])


@precisions
def test_a_wait_that_runs_out_is_reported(single):
    eng = minfft_b200.engine(single)
    pool, jobs, host = make_batch(single, [("dft", 1 << 15)] * 4 + [("dct2", 256)] * 20, np.random.default_rng(4))
    assert eng.lib.minfft_b200_test_mixed_withhold(1000) == 0
    try:
        h = eng.mixed_plan(jobs)
    finally:
        assert eng.lib.minfft_b200_test_mixed_withhold(0) == 0
    try:
        eng.mixed_execute(h)
        torch.cuda.synchronize()
        with pytest.raises(MinfftError) as e:
            eng.mixed_execute(h)
        assert e.value.code == 5  # MINFFT_B200_ETIMEOUT
        torch.cuda.synchronize()
    finally:
        eng.mixed_free(h)
    h = eng.mixed_plan(jobs)
    try:
        eng.mixed_execute(h)
        torch.cuda.synchronize()
        check_batch(single, pool, host)
        eng.mixed_execute(h)  # nothing is left of the report
        torch.cuda.synchronize()
    finally:
        eng.mixed_free(h)


@precisions
@pytest.mark.parametrize("n", [1 << 14, 1 << 16])
def test_more_transforms_than_scratch_slots(single, n):
    """Slots of one length take 32 MiB: each is used two to three times here."""
    eng = minfft_b200.engine(single)
    cdt = torch.complex64 if single else torch.complex128
    slots = (32 << 20) // (n * (8 if single else 16))
    count = 2 * slots + slots // 2 + 1
    x = torch.randn((count, n), dtype=cdt, device="cuda", generator=torch.Generator("cuda").manual_seed(n))
    y = torch.full_like(x, float("nan"))
    h = eng.mixed_plan([("dft", n, x[i].data_ptr(), y[i].data_ptr()) for i in range(count)])
    try:
        eng.mixed_execute(h)
        eng.mixed_execute(h)
        torch.cuda.synchronize()
    finally:
        eng.mixed_free(h)
    ref = torch.fft.fft(x.to(torch.complex128))
    err = torch.linalg.vector_norm(y - ref, dim=1) / torch.linalg.vector_norm(ref, dim=1)
    assert err.max().item() <= tolerance(single, (n,))


@precisions
@pytest.mark.parametrize("n", [1 << 13, 1 << 14])
def test_real_rows_not_aligned_for_pairs(single, n):
    """2^14 reals are the longest rows that may start at any real: one past an
    aligned address here, both ways."""
    eng = minfft_b200.engine(single)
    rdt, cdt = (torch.float32, torch.complex64) if single else (torch.float64, torch.complex128)
    g = torch.Generator("cuda").manual_seed(n)
    x = torch.randn(3, n + 1, dtype=rdt, device="cuda", generator=g)[:, 1:]
    y = torch.empty(3, n // 2 + 1, dtype=cdt, device="cuda")
    z = torch.empty(3, n + 1, dtype=rdt, device="cuda")[:, 1:]
    rows = range(0, 3, 2)  # (the odd row length aligns every other row)
    for op, src, dst in (("realdft", x, y), ("invrealdft", y, z)):
        h = eng.mixed_plan([(op, n, src[i].data_ptr(), dst[i].data_ptr()) for i in rows])
        try:
            eng.mixed_execute(h)
            torch.cuda.synchronize()
        finally:
            eng.mixed_free(h)
    for i in rows:
        ref = torch.fft.rfft(x[i].double())
        assert (torch.linalg.vector_norm(y[i] - ref) / torch.linalg.vector_norm(ref)).item() <= tolerance(single, (n,))
        back = torch.linalg.vector_norm(z[i] / n - x[i]) / torch.linalg.vector_norm(x[i])
        assert back.item() <= 2 * tolerance(single, (n,))


@precisions
def test_transforms_of_8192_points_take_one_block_each(single):
    """One item a transform, between shorter and longer jobs and alone; every kind."""
    eng = minfft_b200.engine(single)
    rng = np.random.default_rng(8)
    wide = [(op, 1 << (13 if op in ("dft", "invdft") else 14)) for op in minfft_b200.OPS] * 3
    for specs, items in ((wide, len(wide)), (wide + [("dct2", 64)] * 8 + [("dft", 1 << 15)], None)):
        pool, jobs, host = make_batch(single, specs, rng)
        h = eng.mixed_plan(jobs)
        try:
            assert items is None or eng.mixed_items(h) == items
            eng.mixed_execute(h)
            eng.mixed_execute(h)
            torch.cuda.synchronize()
            check_batch(single, pool, host)
        finally:
            eng.mixed_free(h)


@precisions
def test_item_counts_around_one_and_two_grids(single):
    """Without long transforms a block's first two items are dealt by index and the
    rest come from the counter: one job an item, counts around the grid's size."""
    eng = minfft_b200.engine(single)
    cdt = torch.complex64 if single else torch.complex128
    n, grid = 4096, torch.cuda.get_device_properties(0).multi_processor_count * (4 if single else 2)
    x = torch.randn(2 * grid + 3, n, dtype=cdt, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    ref = torch.fft.fft(x.to(torch.complex128))
    for count in (1, grid - 1, grid, grid + 1, 2 * grid, 2 * grid + 1, 2 * grid + 3):
        y = torch.full_like(x[:count], float("nan"))
        h = eng.mixed_plan([("dft", n, x[i].data_ptr(), y[i].data_ptr()) for i in range(count)])
        try:
            assert eng.mixed_items(h) == count
            eng.mixed_execute(h)
            torch.cuda.synchronize()
        finally:
            eng.mixed_free(h)
        err = torch.linalg.vector_norm(y - ref[:count], dim=1) / torch.linalg.vector_norm(ref[:count], dim=1)
        assert err.max().item() <= tolerance(single, (n,)), count
