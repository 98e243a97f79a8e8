"""The bounds within which a product is handed to the kernels that read its operands themselves, against the index arithmetic of those kernels.  No
GPU is needed: the rules are functions of the sizes and strides alone."""
import ctypes as C
import os
import re

import pytest

from vkml_b200 import _abi

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vkml_b200", "csrc")
FITS = "_ZN4b20016gemm_inline_fitsERKNS_11GemmProblemEb"  # b200::gemm_inline_fits(const GemmProblem&, bool tf32)


def read(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


class Problem(C.Structure):
    _fields_ = [("a", C.c_void_p), ("b", C.c_void_p), ("out", C.c_void_p), ("b0", C.c_int64), ("b1", C.c_int64), ("m", C.c_int64),
                ("n", C.c_int64), ("k", C.c_int64), ("a_s", C.c_int64 * 4), ("b_s", C.c_int64 * 4)]


def fits(a_s, b_s, tf32, m=320, n=512, k=1024):
    rule = getattr(_abi.load(), FITS)
    rule.restype, rule.argtypes = C.c_bool, [C.c_void_p, C.c_bool]
    p = Problem(None, None, None, 1, 1, m, n, k, (C.c_int64 * 4)(0, 0, *a_s), (C.c_int64 * 4)(0, 0, *b_s))
    return bool(rule(C.byref(p), tf32))


def row_steps(tf32):
    """How many rows a converter's loads lie apart, by form: quads along K, quads along the other axis, single floats."""
    block = 32 if tf32 else 64
    steps = [2 * rows // (block // 4) for rows in (64, 128)] + [2 * rows // (rows // 4) for rows in (64, 128)]
    return steps + ([2] + [rows // 16 for rows in (64, 128)] if tf32 else [])


@pytest.mark.parametrize("tf32", [False, True])
@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("side", ["a", "b"])
def test_rows_of_a_thread_are_within_32_bits(tf32, sign, side):
    served = []
    for pitch in [1024, 1 << 20] + [(1 << e) + d for e in (23, 24, 25, 26) for d in (-4, -1, 0, 1, 4)] + [20_000_000, 1 << 31]:
        ok = fits((sign * pitch, 1), (512, 1), tf32) if side == "a" else fits((1024, 1), (1, sign * pitch), tf32)
        if ok:
            served.append(pitch)
            assert max(row_steps(tf32)) * pitch * 4 < 1 << 31, pitch
    assert max(served) == (1 << (24 if tf32 else 25)) - 1  # and nothing below is given up


@pytest.mark.parametrize("name", [f for f in sorted(os.listdir(CSRC)) if f.endswith(".cu") and "= unit_plan(" in read(f)])
def test_unit_walkers_leave_room_for_a_pending_all_reduce(name):
    """A kernel whose CTAs stay on their SMs takes none of those that a gradient span's all-reduce has set aside."""
    launchers = [f for f in re.split(r"\n}\n", read(name)) if "= unit_plan(" in f]
    assert launchers
    for f in launchers:
        assert "in_grad_sync_span && ctx->comm_pending" in f and "comm_sms" in f, f[-300:]
