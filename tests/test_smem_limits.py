"""The dynamic shared memory limit that a kernel's launches need is not lowered by a call of another size in between,
as another thread may make one."""

import pytest

from fake_runtime import run

LEVELS = """
def forward(T, hi, C, b=0x40000000):
    S = sum(3 if l == 0 else ((1 << l - 1) + 1) * ((1 << l) + 1) for l in range(hi + 1))
    ST = 3 if hi == 0 else ((1 << hi - 1) + 1) * ((1 << hi) + 1)
    return lib.ds_accumulate_to_level_forward(T, 0, hi, hi, S, ST, C, p(b), p(2 * b), stream())
def p(v): import ctypes; return ctypes.c_void_p(v)
"""


def test_level_operators(tmp_path):
    out = run(tmp_path, LEVELS + """
assert forward(20000, 3, 7) == 0
fake.fake_take()
inner = C.CFUNCTYPE(None)(lambda: print("inner", forward(50000, 2, 1)))
fake.fake_before_launch(inner)
print("outer", forward(20000, 3, 7), lib.ds_last_error().decode())
smem = [int(l.split()[3]) for l in fake.fake_take().decode().splitlines() if l.startswith("launch")]
print("sizes", *smem)
""")
    lines = dict(line.split(" ", 1) for line in out.splitlines())
    assert lines["inner"] == "0" and lines["outer"].split()[0] == "0", out
    small, large = map(int, lines["sizes"].split())
    assert small < large and large > 48 * 1024  # the two calls share a kernel and differ in size


def test_training_step(tmp_path):
    """Two steps of one model with other levels: a step's forward and adjoint kernels launch with their own sizes."""
    out = run(tmp_path, """
wide = dict(C_=16, hidden=64, layers=2, precision=0)
train_step(hi=3, **wide)
sizes = lambda log: sorted({int(x[3]) for x in log if x[0] == "launch" and "accum_tab" in x[4]})
inner = C.CFUNCTYPE(None)(lambda: print("inner", *sizes(train_step(hi=2, **wide))))
fake.fake_before_launch(inner)  # before the level accumulation, the step's first launch
print("outer", *sizes(train_step(hi=3, **wide)))
""")
    lines = dict(line.split(" ", 1) for line in out.splitlines())
    inner, outer = ([int(v) for v in lines[k].split()] for k in ("inner", "outer"))
    assert inner and outer and inner[0] < outer[0] and inner[-1] < outer[-1]
