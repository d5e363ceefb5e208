"""A launch that the CUDA runtime refuses: the call returns the error and leaves none behind.  The library is loaded
on a fake runtime (a stub of every entry point it imports) whose launch fails, in a process of its own."""
import re
import subprocess
import sys

from sageattention_rdna3_b200 import _native

_CHILD = """
import ctypes, sys
fake = ctypes.CDLL(sys.argv[1], mode=ctypes.RTLD_GLOBAL)
lib = ctypes.CDLL(sys.argv[2])
lib.sage_last_error.restype = ctypes.c_char_p
class Strided(ctypes.Structure):
    _fields_ = [("ptr", ctypes.c_void_p), ("b", ctypes.c_int64), ("h", ctypes.c_int64), ("s", ctypes.c_int64)]
k = Strided(0x1000, 2048, 1024, 64)
lib.sage_mean_seq.argtypes = [ctypes.POINTER(Strided)] + [ctypes.c_int] * 5 + [ctypes.c_void_p] * 2
lib.sage_v_to_f16.argtypes = lib.sage_mean_seq.argtypes
for fn in (lib.sage_mean_seq, lib.sage_v_to_f16):
    rc = fn(ctypes.byref(k), 0, 1, 2, 16, 64, 0x2000, None)
    print(rc, fake.launches(), fake.cudaPeekAtLastError(), lib.sage_last_error().decode())
"""


def test_the_error_of_a_refused_launch_is_returned_once(tmp_path):
    listed = subprocess.run(["nm", "-D", "-u", str(_native.ABI_PATH)], check=True, capture_output=True, text=True).stdout
    names = sorted(set(re.findall(r"\b((?:__)?cuda\w+)", listed)))
    assert "cudaLaunchKernelExC" in names
    own = {"cudaLaunchKernelExC": "{ ++n; return last = 9; }",           # cudaErrorInvalidConfiguration
           "cudaGetLastError": "{ int e = last; last = 0; return e; }", "cudaPeekAtLastError": "{ return last; }"}
    lines = ["static int last = 0, n = 0;", 'extern "C" {', "int launches() { return n; }",
             'const char* cudaGetErrorString(int) { return "refused"; }', "void* __cudaRegisterFatBinary(void*) { static void* h; return &h; }"]
    for name in sorted((set(names) | set(own)) - {"cudaGetErrorString", "__cudaRegisterFatBinary"}):
        lines.append(f"int {name}() {own.get(name, '{ return 0; }')}")
    (tmp_path / "fake.cpp").write_text("\n".join(lines + ["}"]))
    fake = tmp_path / "libcudart.so.12"
    (tmp_path / "versions").write_text("libcudart.so.12 { global: *; };")
    subprocess.run(["g++", "-shared", "-fPIC", "-Wl,-soname,libcudart.so.12", f"-Wl,--version-script={tmp_path}/versions",
                    "-o", str(fake), str(tmp_path / "fake.cpp")], check=True)
    out = subprocess.run([sys.executable, "-c", _CHILD, str(fake), str(_native.ABI_PATH)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stderr
    lines = out.stdout.splitlines()
    assert len(lines) == 2
    for i, line in enumerate(lines, 1):
        rc, launches, left, message = line.split(" ", 3)
        assert (int(rc), int(launches)) == (2, i) and "refused" in message
        assert int(left) == 0, "the error is still pending"
