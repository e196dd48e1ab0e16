"""Which host memory a copy kernel may be given (host logic, no GPU): whole ranges of the library's own page-locked allocations only.  A buffer that begins in
page-locked memory and ends outside it would be an access out of range on the GPU."""
import ctypes as C
import re
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def r(tmp_path_factory):
    out = tmp_path_factory.mktemp("hr") / "libhost_ranges.so"
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-o", str(out), str(ROOT / "tests" / "cpp" / "host_ranges.cpp")], check=True)
    lib = C.CDLL(str(out))
    for f in (lib.hr_add, lib.hr_drop, lib.hr_inside):
        f.argtypes = [C.c_uint64] * (1 if f is lib.hr_drop else 2)
    return lib


def test_ranges(r):
    r.hr_add(0x10000, 4096)
    r.hr_add(0x11000, 64)                       # adjoins the first: still another allocation
    r.hr_add(0x20000, 256)
    assert r.hr_inside(0x10000, 4096) and r.hr_inside(0x10000, 1) and r.hr_inside(0x10ff0, 16) and r.hr_inside(0x20010, 240)
    assert not r.hr_inside(0x10000, 4097)       # ends outside
    assert not r.hr_inside(0x10ff8, 16)         # ends in the next allocation
    assert not r.hr_inside(0xfff0, 32)          # begins outside
    assert not r.hr_inside(0x20000, 257) and not r.hr_inside(0x20101, 1) and not r.hr_inside(0x30000, 16) and not r.hr_inside(0, 16)
    assert not r.hr_inside(0x20010, 2 ** 64 - 1)
    r.hr_drop(0x10000)
    assert not r.hr_inside(0x10000, 16) and r.hr_inside(0x11000, 64)
    r.hr_drop(0x10000)                          # twice, or memory of somebody else: no effect
    r.hr_drop(0x20010)
    assert r.hr_inside(0x20000, 256)


def test_kernels_are_given_no_other_host_memory():
    """By reading: the copy kernel's host address is the staging buffer's or one that was looked up with its whole length."""
    code = re.sub(r"//[^\n]*", "", (ROOT / "pyre_b200" / "csrc" / "pb_api.cu").read_text())
    assert "devicePointer" not in code
    assert re.findall(r"\bdev = ([^;]*);", code) == [
        "stage ? ctx->pin + off : (bytes <= PB_COPY_IN && g_host.inside(src, bytes) ? src : nullptr)",
        "g_host.inside(dst, bytes) ? dst : nullptr",
        "ctx->pin + off",
    ]
