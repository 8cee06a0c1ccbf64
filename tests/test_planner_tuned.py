"""Saved tuning entries of single axis launches still count where the planner by itself
runs those axes in one launch (small arrays) or slab by slab (large ones)."""
import os

import pytest

import minfft_b200


# entry: combo, length, columns, 0, 0, batch, inner, inner, inner, then form, transforms per block, radix
@pytest.mark.parametrize("single,op,dims,entry,launches,by_itself", [
    (True, "dft", (64, 64), "0 64 0 0 0 64 1 1 1 0 4 16", 2, 1), (False, "dct2", (32, 32), "3 16 1 0 0 32 32 32 32 0 4 8", 2, 1),
    (True, "realdft", (32, 64), "1 32 0 0 0 32 1 1 1 0 2 16", 2, 1),
    (True, "dft", (256, 256, 256), "0 256 0 0 0 65536 1 1 1 0 4 16", 3, 5),
    (False, "invdft", (256, 256, 256), "0 256 1 0 0 65536 256 256 256 1 8 16", 3, 9)])
def test_entries_keep_their_launches(single, op, dims, entry, launches, by_itself):
    eng = minfft_b200.engine(single)
    d = os.path.join(os.path.dirname(os.path.abspath(__file__)), "_build", "tune")  # git-ignored
    os.makedirs(d, exist_ok=True)
    path = os.path.join(d, "axes.txt")
    assert eng.plan_selfcheck(op, dims)[2] == by_itself
    with open(path, "w") as f:
        f.write(entry + "\n")
    try:
        eng.tune_clear()
        eng.tune_load(path)
        bad, rep, n = eng.plan_selfcheck(op, dims)
        assert bad == 0 and n == launches, rep
        if entry.split()[9] == "1":
            assert "axis_pipe<cplx,L=256,col>" in rep, rep
    finally:
        eng.tune_clear()
    assert eng.plan_selfcheck(op, dims)[2] == by_itself
