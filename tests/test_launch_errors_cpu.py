"""A launch that the runtime refuses is reported by the launcher (no device: the
object is linked against a runtime whose launches fail)."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fzgpumodules_b200", "csrc")

RUNTIME = """
static int last, refuse = %d;
int cudaGetLastError(void) { int e = last; last = 0; return e; }
int cudaLaunchKernel(void) { return last = refuse; }
int cudaLaunchKernelExC(void) { return last = refuse; }
int __cudaPushCallConfiguration(void) { return 0; }
int __cudaPopCallConfiguration(void) { return 0; }
void **__cudaRegisterFatBinary(void *p) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **h) {}
void __cudaUnregisterFatBinary(void **h) {}
void __cudaRegisterFunction(void) {}
void __cudaRegisterVar(void) {}
"""


@pytest.mark.parametrize("code", [0, 1, 700])
def test_tile_launch_reports_what_the_runtime_said(tmp_path, code):
    obj = "_build/fzb_tiles.o"
    subprocess.run(["make", "-C", CSRC, obj], check=True, capture_output=True)
    (tmp_path / "runtime.c").write_text(RUNTIME % code)
    so = str(tmp_path / f"tiles{code}.so")
    subprocess.run(["gcc", "-w", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-o", so, str(tmp_path / "runtime.c"),
                    os.path.join(CSRC, obj), "-lstdc++"], check=True)  # its own runtime, whatever else is loaded
    launch = C.CDLL(so)["_ZN3fzb15launch_lq_tilesERKNS_7FwdArgsEP11CUstream_st"]
    launch.restype = C.c_int
    assert launch(C.create_string_buffer(4096), None) == code  # a field of no extents
