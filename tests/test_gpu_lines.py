"""Long 1-D real lines whose pre- and post-processing runs inside the first
and last pass of their half-length chain (the *Line load and store stages of
axis_pass.cuh), against the oracle with the repository's bars: chains of two
and three passes of 128 to 1024 points (the shortest chain, uneven pass
lengths, the first three-pass one), several lines of a 2-D array, arrays that
start one real past a 16-byte boundary, in-place calls, and the tensor-core
chains that fuse one end or both."""
import numpy as np
import pytest

import minfft_b200
from conftest import rel_l2, tolerance
from minfft_b200 import OP_FAMILY
from test_gpu_parity import expected, gpu_apply, make_input

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

FUSED = {"realdft": ("r2cunpack",), "invrealdft": ("c2rpack",), "dct2": ("dct2pre", "dct2post"),
         "dst2": ("dct2pre", "dct2post"), "dct3": ("dct3pre", "dct3post"), "dst3": ("dct3pre", "dct3post")}


@pytest.mark.parametrize("single", [False, True], ids=["f64", "f32"])
@pytest.mark.parametrize("dims", [(1 << 15,), (1 << 18,), (1 << 21,), (1 << 22,), (3, 1 << 15)],
                         ids=lambda d: "x".join(map(str, d)))
def test_fused_lines_match_oracle(dims, single):
    eng = minfft_b200.engine(single)
    rng = np.random.default_rng(len(dims) + dims[-1])
    for op, steps in FUSED.items():
        if len(dims) > 1 and dims[0] == 3:
            x = np.stack([make_input(op, dims[1:], rng, single) for _ in range(3)])
            fam = OP_FAMILY[op]
            plan = eng.plan(fam, dims[1:])
            xt = torch.from_numpy(x).cuda()
            refs = np.stack([expected(op, v, dims[1:]) for v in x])
            y = torch.full(refs.shape, float("nan"), device="cuda",
                           dtype={"f": torch.float32, "d": torch.float64, "F": torch.complex64,
                                  "D": torch.complex128}[np.dtype(
                                      (np.complex64 if single else np.complex128) if np.iscomplexobj(refs)
                                      else (np.float32 if single else np.float64)).char])
            plan.batch(op, xt.data_ptr(), y.data_ptr(), 3)
            torch.cuda.synchronize()
            plan.free()
            got, ref = y.cpu().numpy(), refs
        else:
            _, rep, _ = eng.plan_selfcheck(op, dims)
            assert all(s in rep for s in steps) and "line<" not in rep, rep
            x = make_input(op, dims, rng, single)
            got, ref = gpu_apply(op, x, dims, single), expected(op, x, dims)
        err = rel_l2(got, ref)
        assert err <= tolerance(single, dims[-1:]), (op, dims, err)


@pytest.mark.parametrize("single", [False, True], ids=["f64", "f32"])
def test_fused_lines_offset_and_in_place(single):
    eng = minfft_b200.engine(single)
    rng = np.random.default_rng(8)
    n = 1 << 16
    tdt = torch.float32 if single else torch.float64
    for op in ("dct2", "dst2", "dct3", "dst3"):
        x = make_input(op, (n,), rng, single)
        ref = expected(op, x, (n,))
        src = torch.zeros(n + 1, dtype=tdt, device="cuda")
        src[1:] = torch.from_numpy(x).cuda()
        dst = torch.full((n + 1,), float("nan"), dtype=tdt, device="cuda")
        plan = eng.plan("t2t3", (n,))
        plan(op, src.data_ptr() + src.element_size(), dst.data_ptr() + dst.element_size())
        torch.cuda.synchronize()
        plan.free()
        assert rel_l2(dst[1:].cpu().numpy(), ref) <= tolerance(single, (n,)), op
    for op in FUSED:
        x = make_input(op, (n,), rng, single)
        err = rel_l2(gpu_apply(op, x, (n,), single, inplace=True), expected(op, x, (n,)))
        assert err <= tolerance(single, (n,)), (op, err)


@pytest.mark.parametrize("precision", ["tc_f16", "tc_bf16"])
@pytest.mark.parametrize("bits", [15, 17, 20, 21])
def test_fused_lines_tensor_core_chains(bits, precision):
    """Chains of 2^14 (256 x 64), 2^16 (16 x 256 x 16), 2^19 (64 x 256 x 32) and 2^20 (64 x 256 x 64) points; 1e-6 as the
    tensor-core modes' bar."""
    eng = minfft_b200.engine(True)
    rng = np.random.default_rng(bits)
    dims = (1 << bits,)
    for op in FUSED:
        x = make_input(op, dims, rng, True)
        xt = torch.from_numpy(x).cuda()
        ref = expected(op, x, dims)
        y = torch.full(ref.shape, float("nan"), dtype=torch.complex64 if np.iscomplexobj(ref) else torch.float32,
                       device="cuda")
        plan = eng.plan(OP_FAMILY[op], dims)
        eng.set_precision(plan.aux, precision)
        plan(op, xt.data_ptr(), y.data_ptr())
        torch.cuda.synchronize()
        eng.tc_status(plan.aux)
        plan.free()
        assert rel_l2(y.cpu().numpy(), ref) <= 1e-6, (op, bits)
