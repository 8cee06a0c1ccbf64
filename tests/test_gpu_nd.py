"""Small multi-dimensional arrays run all their axes in one launch (nd_pass.cu):
every transform against the oracle with the repository's bars, at the edges of
that route -- axes of 2 points, the longest axes, the largest arrays, spectra of
one column more than a round, three and four axes, the longest batch and one more,
in-place calls and real arrays that are not aligned for pairs -- and the shapes
just outside it, which keep one launch per axis."""
import numpy as np
import pytest

import minfft_b200
from conftest import rel_l2, tolerance
from minfft_b200 import OP_FAMILY, OPS, shapes
from test_gpu_parity import expected, gpu_apply, make_input

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SHAPES = [(2, 2), (2, 128), (128, 2), (4, 256), (64, 64), (64, 128), (128, 128), (128, 32), (2, 4, 8), (16, 16, 16),
          (32, 16, 32), (8, 2, 4, 16)]


@pytest.mark.parametrize("single", [False, True], ids=["f64", "f32"])
@pytest.mark.parametrize("dims", SHAPES, ids=lambda d: "x".join(map(str, d)))
def test_one_launch_matches_oracle(dims, single):
    eng = minfft_b200.engine(single)
    rng = np.random.default_rng(sum(dims))
    for op in OPS:
        x = make_input(op, dims, rng, single)
        ref = expected(op, x, dims)
        for inplace in (False, True):
            err = rel_l2(gpu_apply(op, x, dims, single, inplace=inplace), ref)
            assert err <= tolerance(single, dims), (op, dims, inplace, err)


@pytest.mark.parametrize("single", [False, True], ids=["f64", "f32"])
@pytest.mark.parametrize("howmany", [3, 18, 19])
def test_batches_and_offsets(howmany, single):
    eng = minfft_b200.engine(single)
    rng = np.random.default_rng(howmany)
    dims = (8, 16)
    rdt, cdt = (torch.float32, torch.complex64) if single else (torch.float64, torch.complex128)
    for op in ("invdft", "realdft", "invrealdft", "dst2", "dct3", "dct4"):
        _, in_c, out_shape, out_c = shapes(op, dims)
        x = np.stack([make_input(op, dims, rng, single) for _ in range(howmany)])
        ref = np.stack([expected(op, v, dims) for v in x])
        skip = 0 if in_c or out_c and op != "realdft" else 1  # real input one element past an aligned address
        src = torch.zeros(x.size + 1, dtype=cdt if in_c else rdt, device="cuda")
        src[skip:skip + x.size] = torch.from_numpy(x.ravel()).cuda()
        y = torch.full((howmany,) + tuple(out_shape), float("nan"), dtype=cdt if out_c else rdt, device="cuda")
        plan = eng.plan(OP_FAMILY[op], dims)
        plan.batch(op, src.data_ptr() + skip * src.element_size(), y.data_ptr(), howmany)
        torch.cuda.synchronize()
        plan.free()
        assert rel_l2(y.cpu().numpy(), ref) <= tolerance(single, dims), (op, howmany)


@pytest.mark.parametrize("op,dims,single,one", [
    ("dft", (64, 128), True, True), ("dft", (128, 128), True, False), ("dft", (64, 64), False, True),
    ("dft", (64, 128), False, False), ("realdft", (128, 128), True, True), ("dct2", (64, 64), False, True),
    ("dct3", (32, 64), True, False), ("dst2", (16, 32), False, True), ("dct4", (32, 64), False, True),
    ("dft", (256, 16), True, False), ("dft", (32, 32, 32), True, False), ("dft", (1, 64), True, False)])
def test_which_shapes_take_one_launch(op, dims, single, one):
    _, rep, n = minfft_b200.engine(single).plan_selfcheck(op, dims)
    assert ("nd_pass" in rep and n == 1) == one, rep


@pytest.mark.parametrize("single,dims,howmany", [(True, (64, 64, 64), 67), (False, (256, 8, 4096), 1)],
                         ids=["f32-batch", "f64-3d"])
def test_slabs_of_arrays_beyond_the_l2(single, dims, howmany):
    """Complex arrays above 128 MiB run their inner axes slab by slab (the last
    slab of the batch shorter than the others); the first, a middle and the
    last array or plane against the oracle, in place too."""
    eng = minfft_b200.engine(single)
    _, _, n = eng.plan_selfcheck("dft", dims, howmany)
    assert n > len(dims)
    cdt = torch.complex64 if single else torch.complex128
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn((howmany,) + dims, dtype=cdt, device="cuda", generator=g)
    y = torch.full_like(x, float("nan"))
    plan = eng.plan("dft", dims)
    plan.batch("dft", x.data_ptr(), y.data_ptr(), howmany)
    torch.cuda.synchronize()
    pick = (0, howmany // 2, howmany - 1) if howmany > 1 else (0,)
    for i in pick:
        ref = expected("dft", x[i].cpu().numpy(), dims)
        assert rel_l2(y[i].cpu().numpy(), ref) <= tolerance(single, dims), i
    plan.batch("invdft", y.data_ptr(), y.data_ptr(), howmany)
    torch.cuda.synchronize()
    plan.free()
    scale = float(np.prod(dims))
    err = (torch.linalg.vector_norm(y / scale - x) / torch.linalg.vector_norm(x)).item()
    assert err <= 2 * tolerance(single, dims)
