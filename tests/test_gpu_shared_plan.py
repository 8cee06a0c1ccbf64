"""A plan shared by threads: each finds the launch list of its own call."""
import os
import shutil
import subprocess

import pytest

from test_c_api_program import OUT, ROOT, engine_lib

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(shutil.which("gcc") is None, reason="gcc not found")]


@pytest.mark.parametrize("single", [False, True], ids=["f64", "f32"])
def test_threads_find_their_own_launch_lists(single):
    lib = engine_lib(single)
    exe = os.path.join(OUT, f"shared_plan_{int(single)}")
    os.makedirs(OUT, exist_ok=True)
    d, name = os.path.split(lib)
    subprocess.run(["gcc", "-O2", "-std=c99", "-Wall", "-Wextra", "-Werror", "-pthread", f"-DMINFFT_SINGLE={int(single)}",
                    os.path.join(ROOT, "tests", "c_api", "shared_plan.c"), "-I", os.path.join(ROOT, "include"), "-L", d,
                    f"-l:{name}", f"-Wl,-rpath,{d}", "-lm", "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
