"""Device functions of the library compiled with a test's own launcher: the
kernels' headers are included as they are, with the library's compiler flags."""
import ctypes as C
import subprocess

from glphase_gb300 import build as B


def compile_launcher(directory, src):
    """src: CUDA C++ with extern "C" launchers; returns the loaded library."""
    cu, so = directory / "launcher.cu", directory / "liblauncher.so"
    cu.write_text(src)
    subprocess.run([B.nvcc(), B.ARCH, *B.FLAGS, "-shared", "-I", B.CSRC, str(cu), "-o", str(so)],
                   check=True)
    return C.CDLL(str(so))
