"""libdiffsoup_b200.so on the recording CUDA runtime of fake_cudart.cpp, for tests of what the host code asks of the
runtime.  Imported in a process of its own (`run`), which never loads the real runtime."""

import ctypes as C
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
LIB = os.path.join(os.path.dirname(HERE), "diffsoup_b200", "libdiffsoup_b200.so")
STREAM = 0x77


def build(directory) -> str:
    """Compiles the runtime into `directory`; returns its path."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    out, script = os.path.join(directory, "libcudart.so.12"), os.path.join(directory, "versions")
    with open(script, "w") as f:
        f.write("libcudart.so.12 { global: *; };\n")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", include, "-o", out,
                           os.path.join(HERE, "fake_cudart.cpp"), "-Wl,-soname,libcudart.so.12",
                           f"-Wl,--version-script={script}"])
    return out


def run(directory, body: str) -> str:
    """The output of `body` in a new process, with this module's names in it."""
    code = f"import sys; sys.path.insert(0, {HERE!r})\nfrom fake_runtime import *\nload({build(directory)!r})\n{body}"
    p = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0, p.stdout + p.stderr
    return p.stdout


fake = lib = None


def load(path: str) -> None:
    global fake, lib
    fake = C.CDLL(path, mode=C.RTLD_GLOBAL)
    lib = C.CDLL(LIB)
    fake.fake_take.restype = C.c_char_p
    lib.ds_last_error.restype = C.c_char_p
    for name in ("ds_tiles_workspace_size", "ds_train_step_workspace_size", "ds_render_workspace_size",
                 "ds_split_soup_workspace_size"):
        getattr(lib, name).restype = C.c_size_t
    import __main__
    __main__.fake, __main__.lib = fake, lib


def call(name: str, *args) -> list:
    """A library call with integers as ints, floats as floats and "p" as a device pointer; the recorded calls."""
    fake.fake_take()
    got = getattr(lib, name)(*[C.c_void_p(0x40000000 + 0x1000000 * i) if a == "p" else
                               C.c_float(a) if isinstance(a, float) else a for i, a in enumerate(args)])
    assert got == 0, lib.ds_last_error()
    return [line.split() for line in fake.fake_take().decode().splitlines()]


def i64(v: int):
    return C.c_int64(v)


def stream():
    return C.c_void_p(STREAM)


def feats(lo: int, hi: int) -> int:
    return sum(3 if k == 0 else ((1 << k - 1) + 1) * ((1 << k) + 1) for k in range(lo, hi + 1))


class StepConfig(C.Structure):
    """ds_step_config of include/diffsoup_b200.h."""
    _fields_ = [(n, C.c_float if n in ("thr_const", "frag_records") else C.c_int32) for n in
                ("B", "T", "V", "C", "min_level", "max_level", "hidden", "n_layers", "stochastic", "thr_const",
                 "frag_records", "precision", "block_shape", "view_enc", "target_u8", "shade_mode")]


def train_step(B=2, T=3000, H=96, W=128, C_=8, hi=2, hidden=16, layers=1, frag_records=2.0, precision=1) -> list:
    """The calls of one ds_train_step."""
    c = StepConfig(B, T, 3 * T, C_, 0, hi, hidden, layers, 1, 0.5, frag_records, precision, 0, 0, 0, 0)
    nt, cap = B * ((W + 15) // 16) * ((H + 15) // 16), i64(8 * B * T)
    need = lib.ds_train_step_workspace_size(C.byref(c), nt, i64(B * H * W), cap)
    return call("ds_train_step", C.byref(c), "p", nt, i64(B * H * W), *["p"] * 17, C.c_size_t(need), cap, "p", stream())
