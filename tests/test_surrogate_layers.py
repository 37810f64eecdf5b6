"""The calls that launch a network pass's kernels, on the host: what they hand
to the layers' own entry points (a shim in their place records it)."""
import ctypes
import shutil
import subprocess
import sys
import textwrap

import pytest

from eemd4cuda_b200 import _sg

SHIM = """
#include <stdint.h>
int64_t rec[64];
int n = 0;
int32_t eemd_sg_wgrad(const void* dy, const void* x, float* dw, float* db, int32_t B, int32_t T, int32_t n_rows,
                      int32_t c, int32_t nv, int32_t cv, int32_t dil, int32_t tensor_cores, int32_t* err,
                      int64_t spin, void* stream) {
    rec[n++] = 1; rec[n++] = (int64_t)(intptr_t)dy; rec[n++] = (int64_t)(intptr_t)err; return 0;
}
int32_t eemd_sg_conv(const void* x, const void* w, const float* bias, void* y, int32_t B, int32_t T, int32_t cin,
                     int32_t cout, int32_t dil, int32_t dir, int32_t relu, const void* mask, int32_t tensor_cores,
                     int32_t* err, int64_t spin, void* stream) {
    rec[n++] = 2; rec[n++] = (int64_t)(intptr_t)x; rec[n++] = (int64_t)(intptr_t)err; return 0;
}
"""

CALL = """
import ctypes, sys
shim = ctypes.CDLL(sys.argv[1], mode=ctypes.RTLD_GLOBAL)
lib = ctypes.CDLL(sys.argv[2])
fn = getattr(lib, sys.argv[3])
rows = [int(v) for v in sys.argv[4].split(",")]
n_layers = int(sys.argv[5])
rc = fn((ctypes.c_int64 * len(rows))(*rows), ctypes.c_int32(n_layers), ctypes.c_int32(1), ctypes.c_int32(128),
        ctypes.c_int32(4), ctypes.c_void_p(0x7770), ctypes.c_void_p(0))
n = ctypes.c_int.in_dll(shim, "n").value
print(rc, *(ctypes.c_int64 * 64).in_dll(shim, "rec")[:n])
"""


@pytest.mark.skipif(shutil.which("gcc") is None, reason="builds a shim with gcc")
@pytest.mark.parametrize("fn,rows,kinds", [
    ("eemd_sg_forward_layers", [[16, 32, 48, 64, 0, 16, 64, 1, 1, 1], [64, 32, 48, 80, 0, 64, 16, 2, 1, 0]], [2, 2]),
    ("eemd_sg_backward_layers", [[16, 32, 48, 64, 80, 96, 16, 64, 11, 64, 1], [96, 32, 48, 64, 80, 0, 64, 16, 64, 11, 1]],
     [1, 2, 1])])
def test_every_kernel_of_a_pass_gets_the_error_word(tmp_path, fn, rows, kinds):
    src, so = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(textwrap.dedent(SHIM))
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(so), str(src)], check=True)
    out = subprocess.run([sys.executable, "-c", CALL, str(so), str(_sg.lib_path()), fn,
                          ",".join(str(v) for r in rows for v in r), str(len(rows))],
                         capture_output=True, text=True, check=True).stdout.split()
    got = [int(v) for v in out]
    assert got[0] == 0
    assert got[1::3] == kinds
    assert got[3::3] == [0x7770] * len(kinds)
