"""The work that a user of this engine has it do, as cases that can be timed and compared.

A case is one pass of a user's program: a forward transform of the arrays at hand and the inverse transform of the
result (spectral solvers, convolutions and codecs always run both), on device-resident torch tensors through the plan
API, or one mixed batch.  Plans, mixed batches, inputs and output buffers are made by ``prepare``, as such a program
makes them once and keeps them.  ``exact`` gives the same outputs from torch's double-precision FFT.

Lengths are powers of two (all that minfft's plans take); batch counts, job counts and aspect ratios are not.
"""
import numpy as np
import torch

from minfft_b200 import OP_CODES, engine, shapes

#: family -> (forward, inverse), and the sine variants of the real symmetric families
PAIRS = {
    ("dft", False): ("dft", "invdft"),
    ("realdft", False): ("realdft", "invrealdft"),
    ("t2t3", False): ("dct2", "dct3"),
    ("t2t3", True): ("dst2", "dst3"),
    ("t4", False): ("dct4", "dct4"),
    ("t4", True): ("dst4", "dst4"),
}
MIXED_OPS = ("dft", "realdft", "dct2", "dst2", "dct3", "dst3", "dct4", "dst4")


def _case(family, precision, dims, howmany=1, sine=False, arith="fp32", name=None):
    c = {"family": family, "precision": precision, "dims": "x".join(str(n) for n in dims), "howmany": int(howmany),
         "sine": bool(sine), "arith": arith}
    return c if name is None else dict(c, name=name)


def _mixed(precision, jobs, lo, hi, name=None):
    c = {"family": "mixed", "precision": precision, "jobs": int(jobs), "lo": int(lo), "hi": int(hi)}
    return c if name is None else dict(c, name=name)


def listed():
    return [
        # one short signal at a time, in the library's default precision: latency and launches
        _case("realdft", "f64", (1024,), name="realdft_1k_f64"),
        # one small image or block of a field: two axes of short lines, latency again
        _case("t2t3", "f32", (64, 64), name="dct23_64x64_f32"),
        # frames of audio or subbands, an odd number of them, sine variant
        _case("t4", "f32", (512,), howmany=1001, sine=True, name="dst4_512_x1001_f32"),
        # 1024 independent 4096-point complex DFTs in double: channelisers, ensembles
        _case("dft", "f64", (4096,), howmany=1024, name="dft_4k_x1024_f64"),
        # a 2-D real field in double: spectral solvers
        _case("realdft", "f64", (2048, 2048), name="realdft_2048x2048_f64"),
        # a 2-D field with even boundaries in single (Poisson solvers, image transforms)
        _case("t2t3", "f32", (2048, 2048), name="dct23_2048x2048_f32"),
        # a 3-D complex field in single: molecular dynamics, cosmology
        _case("dft", "f32", (256, 256, 256), name="dft_256x256x256_f32"),
        # the same in the split-precision tensor-core mode
        _case("dft", "f32", (256, 256, 256), arith="tc_f16", name="dft_256x256x256_tc_f16"),
        # thousands of independent transforms of uneven lengths and kinds in one launch
        _mixed("f32", 20000, 4, 16, name="mixed_20000_f32"),
        # one huge complex signal in double: the largest call, several passes over memory
        _case("dft", "f64", (1 << 26,), name="dft_64m_f64"),
        # one long line with mixed boundaries in single
        _case("t4", "f32", (1 << 24,), name="dct4_16m_f32"),
        # one long line with even boundaries in double
        _case("t2t3", "f64", (1 << 22,), name="dct23_4m_f64"),
    ]


def draw(rng):
    """One more case of the same ranges: 2^8 .. 2^25 points in one to three dimensions, single or batched."""
    family = rng.choice(("dft", "dft", "realdft", "realdft", "t2t3", "t2t3", "t4", "mixed"))
    precision = rng.choice(("f32", "f64"))
    if family == "mixed":
        return _mixed(precision, 2 ** rng.uniform(8, 14), 4, rng.randint(10, 16))
    nd = rng.choice((1, 1, 2, 2, 3))
    bits = rng.randint(8, 25)
    if nd == 1:
        n = rng.randint(4, bits)  # a batch of shorter lines, or one line of them all
        dims = (1 << n,)
        left = bits - n
        howmany = 1 if left == 0 else max(1, int(2 ** left * rng.uniform(0.5, 1.0)))
    else:
        cuts = [bits // nd + (1 if i < bits % nd else 0) for i in range(nd)]
        a, b = rng.sample(range(nd), 2)
        shift = rng.randint(0, min(3, cuts[a] - 1))  # uneven aspect ratios
        cuts[a] -= shift
        cuts[b] += shift
        dims = tuple(1 << c for c in cuts)
        howmany = rng.choice((1, 1, 1, 3)) if bits <= 23 else 1
    sine = family in ("t2t3", "t4") and rng.random() < 0.4
    arith = "fp32"
    if family == "dft" and precision == "f32" and rng.random() < 0.4:
        arith = rng.choice(("tc_f16", "tc_bf16"))
    return _case(family, precision, dims, howmany, sine, arith)


def _dims(case):
    return tuple(int(n) for n in case["dims"].split("x"))


def _job_list(case):
    """The jobs of a mixed batch: (op, n, offset of the input, offset of the output) in reals."""
    r = np.random.RandomState(case["jobs"])
    ops = r.randint(0, len(MIXED_OPS), case["jobs"])
    lens = 1 << r.randint(case["lo"], case["hi"] + 1, case["jobs"])
    jobs, i, o = [], 0, 0
    for k, n in zip(ops.tolist(), lens.tolist()):
        op = MIXED_OPS[k]
        jobs.append((op, n, i, o))
        i += 2 * n if op == "dft" else n
        o += 2 * n if op == "dft" else n + 2 if op == "realdft" else n
    return jobs, i, o


def _input(case, seed):
    """Seeded values as the paths meet them: uniform in [-1, 1) for complex signals, normal for real ones."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    real = torch.float32 if case["precision"] == "f32" else torch.float64
    if case["family"] == "mixed":
        return torch.randn(_job_list(case)[1], dtype=real, device="cuda", generator=g)
    shape = (case["howmany"],) + _dims(case)
    if case["family"] == "dft":
        return torch.view_as_complex(torch.rand(shape + (2,), dtype=real, device="cuda", generator=g) * 2 - 1)
    return torch.randn(shape, dtype=real, device="cuda", generator=g)


class _Mixed:
    """A mixed batch that is given back with the state that holds it."""

    def __init__(self, eng, jobs):
        self.eng, self.handle = eng, eng.mixed_plan(jobs)

    def __del__(self):
        self.eng.mixed_free(self.handle)


def prepare(case, seed):
    eng = engine(case["precision"] == "f32")
    x = _input(case, seed)
    if case["family"] == "mixed":
        jobs, _, n_out = _job_list(case)
        y = torch.zeros(n_out, dtype=x.dtype, device="cuda")
        size = x.element_size()
        batch = _Mixed(eng, [(OP_CODES[op], n, x.data_ptr() + i * size, y.data_ptr() + o * size) for op, n, i, o in jobs])
        return {"mixed": batch, "eng": eng, "x": x, "y": y}
    dims, howmany = _dims(case), case["howmany"]
    fwd, inv = PAIRS[case["family"], case["sine"]]
    plan = eng.plan(case["family"], dims)
    if case["arith"] != "fp32":
        eng.set_precision(plan.aux, case["arith"])
    cplx = torch.complex64 if case["precision"] == "f32" else torch.complex128
    real = torch.float32 if case["precision"] == "f32" else torch.float64
    _, _, shape, is_c = shapes(fwd, dims)
    y = torch.empty((howmany,) + tuple(shape), dtype=cplx if is_c else real, device="cuda")
    return {"plan": plan, "fwd": fwd, "inv": inv, "howmany": howmany, "x": x, "y": y, "z": torch.empty_like(x)}


def run(state):
    if "mixed" in state:
        state["eng"].mixed_execute(state["mixed"].handle)
        return [state["y"]]
    plan, x, y, z = state["plan"], state["x"], state["y"], state["z"]
    if state["howmany"] == 1:
        plan(state["fwd"], x.data_ptr(), y.data_ptr())
        plan(state["inv"], y.data_ptr(), z.data_ptr())
    else:
        plan.batch(state["fwd"], x.data_ptr(), y.data_ptr(), state["howmany"])
        plan.batch(state["inv"], y.data_ptr(), z.data_ptr(), state["howmany"])
    return [y, z]


def _one_way(op, n_real, n_cplx, points, length_bits):
    """(values moved, flops) of one transform: 5 N log2 N for complex data, half of that for real data."""
    if op == "dft":
        return 4 * n_cplx, float(5 * points * length_bits)
    if op == "realdft":
        return n_real + 2 * n_cplx, float(2.5 * points * length_bits)
    return 2 * n_real, float(2.5 * points * length_bits)


def work(case):
    size = 4 if case["precision"] == "f32" else 8
    if case["family"] == "mixed":
        moved, flops = 0, 0.0
        for op, n, _, _ in _job_list(case)[0]:
            m, f = _one_way(op, n, n if op == "dft" else n // 2 + 1, n, np.log2(n))
            moved, flops = moved + m, flops + f
        return {"bytes": float(moved * size), "flops": float(flops)}
    dims, howmany = _dims(case), case["howmany"]
    points = int(np.prod(dims))
    n_cplx = points if case["family"] == "dft" else points // dims[-1] * (dims[-1] // 2 + 1)
    moved, flops = _one_way(case["family"], points, n_cplx, points, np.log2(points))
    return {"bytes": 2.0 * howmany * moved * size, "flops": 2.0 * howmany * flops}


# ------------------------------------------------------------------ double-precision values
def _roots(num, den, n, device):
    """exp(-i pi num(k) / den) for k < n."""
    k = torch.arange(n, dtype=torch.float64, device=device)
    a = num(k) * (np.pi / den)
    return torch.complex(torch.cos(a), -torch.sin(a))


def _alternate(n, device):
    return 1.0 - 2.0 * (torch.arange(n, device=device) % 2).to(torch.float64)


def _last_axis(op, x):
    """Transform `op` of a real symmetric family along the last axis, unnormalised (FFTW's definitions)."""
    n, dev = x.shape[-1], x.device
    if op == "dst2":
        return _last_axis("dct2", x * _alternate(n, dev)).flip(-1)
    if op == "dst3":
        return _last_axis("dct3", x.flip(-1)) * _alternate(n, dev)
    if op == "dst4":
        return _last_axis("dct4", x.flip(-1)) * _alternate(n, dev)
    if op == "dct2":
        v = torch.cat((x[..., 0::2], x[..., 1::2].flip(-1)), -1)
        return 2 * (torch.fft.fft(v) * _roots(lambda k: k, 2 * n, n, dev)).real
    if op == "dct3":
        rest = torch.cat((torch.zeros_like(x[..., :1]), x[..., 1:].flip(-1)), -1)
        v = n * torch.fft.ifft(torch.complex(x, -rest) * _roots(lambda k: k, 2 * n, n, dev).conj()).real
        y = torch.empty_like(x)
        y[..., 0::2] = v[..., : n // 2]
        y[..., 1::2] = v[..., n // 2:].flip(-1)
        return y
    t = torch.complex(x[..., 0::2], x[..., 1::2].flip(-1)) * _roots(lambda k: 4 * k + 1, 4 * n, n // 2, dev)
    t = torch.fft.fft(t) * _roots(lambda k: k, n, n // 2, dev)
    y = torch.empty_like(x)
    y[..., 0::2] = 2 * t.real
    y[..., 1::2] = -2 * t.imag.flip(-1)
    return y


def _transform(op, x, axes):
    """Transform `op` of double-precision data along the last `axes` axes."""
    dims = tuple(range(-axes, 0))
    if op == "dft":
        return torch.fft.fftn(x, dim=dims)
    if op == "realdft":
        return torch.fft.rfftn(x, dim=dims)
    for d in dims:
        x = _last_axis(op, x.movedim(d, -1)).movedim(-1, d)
    return x.contiguous()


def exact(case, seed):
    x = _input(case, seed)
    x = x.to(torch.complex128 if x.is_complex() else torch.float64)
    if case["family"] == "mixed":
        jobs, _, n_out = _job_list(case)
        y = torch.zeros(n_out, dtype=torch.float64, device=x.device)
        groups = {}
        for op, n, i, o in jobs:
            groups.setdefault((op, n), []).append((i, o))
        for (op, n), at in groups.items():
            i, o = (torch.tensor(v, device=x.device)[:, None] for v in zip(*at))
            v = x[i + torch.arange(2 * n if op == "dft" else n, device=x.device)]
            if op == "dft":
                v = torch.view_as_complex(v.reshape(len(at), n, 2))
            v = _transform(op, v, 1)
            if v.is_complex():
                v = torch.view_as_real(v).reshape(len(at), -1)
            y[o + torch.arange(v.shape[1], device=x.device)] = v
        return [y]
    dims = _dims(case)
    fwd, _ = PAIRS[case["family"], case["sine"]]
    points = float(np.prod(dims))
    # the unnormalised inverse of the exact result: N x for the DFTs, (2N per axis) x for the symmetric families
    back = points if case["family"] in ("dft", "realdft") else points * 2.0 ** len(dims)
    return [_transform(fwd, x, len(dims)), x * back]
