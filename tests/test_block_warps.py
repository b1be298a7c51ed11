"""Builds with other blocks than four warps (the tuning macro GLP_GEN_WARPS): teams of
warps are offered only where a block holds them whole, and the kernels of teams that
it does not hold do not compile."""
import subprocess

import pytest

from glphase_gb300 import build as B

WIDEST = {1: 32, 2: 64, 3: 32, 4: 128}


def compile_with(tmp_path, warps, src):
    f = tmp_path / "w.cu"
    f.write_text('#include "glp_launch.h"\n' + src)
    return subprocess.run([B.nvcc(), B.ARCH, *B.FLAGS, "-DGLP_GEN_WARPS=%d" % warps, "-I", B.CSRC,
                           "-c", str(f), "-o", str(tmp_path / "w.o")], capture_output=True, text=True)


@pytest.mark.parametrize("warps", [1, 2, 3, 4])
def test_widest(tmp_path, warps):
    r = compile_with(tmp_path, warps, "static_assert(glp::kWidest == %d, \"\");\n" % WIDEST[warps])
    assert r.returncode == 0, r.stderr


def test_teams_that_do_not_fit(tmp_path):
    r = compile_with(tmp_path, 2, """
namespace glp {
SingleFn f() { return generation_kernel<128, EmitF32, 1>; }
}
""")
    assert r.returncode != 0 and "whole teams" in r.stderr
