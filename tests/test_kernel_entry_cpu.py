"""Entry points of the kernel library with arguments that leave nothing to do: host code, checked without a GPU (the launch
itself may answer with an error here; the process must not end)."""
import subprocess
import sys

import pytest

from tinyinfinitrain_b200._build import CSRC, CUDA_HOME, CXX, KERNEL_LIB


def _run(call):
    code = f"""
import ctypes
lib = ctypes.CDLL({str(KERNEL_LIB)!r})
null, f = None, ctypes.c_float
print("rc", {call})
"""
    return subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120)


@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("B,T,H,hd", [(2, 3, 0, 64), (2, 3, 4, 0), (0, 3, 4, 64), (2, 0, 4, 64)])
def test_rope_of_nothing(B, T, H, hd, dtype):
    r = _run(f"lib.titb_rope_strided(null, null, {B}, {T}, {H}, {hd}, ctypes.c_longlong(64), 0, f(1e4), 0, {dtype}, null)")
    assert r.returncode == 0 and "rc 0" in r.stdout, (r.returncode, r.stdout, r.stderr[-500:])


def test_split_planner_keeps_its_signature(tmp_path):
    """Callers outside the library size their workspace with it."""
    src = tmp_path / "caller.cc"
    src.write_text('#include <type_traits>\n#include "api.h"\n'
                   "static_assert(std::is_same<decltype(&titb_gemm_pick_splits), int (*)(int, int, int)>::value, \"\");\n")
    r = subprocess.run([CXX, "-std=c++17", "-fsyntax-only", f"-I{CSRC / 'kernels'}", f"-I{CUDA_HOME / 'include'}", str(src)],
                       capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
    # a weight gradient of few tiles and a long reduction is split, in the output and through a workspace
    for name in ("titb_gemm_pick_splits", "titb_gemm_pick_splits_workspace"):
        r = _run(f"lib.{name}(768, 768, 8192)")
        assert int(r.stdout.split()[1]) > 1
