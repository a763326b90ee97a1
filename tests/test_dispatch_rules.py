"""The rules by which calls are sent to kernels (csrc/rules.h), compiled for the
host and checked at their limits.  CPU only."""
import ctypes
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "trove_gb300" / "csrc"

SHIM = """
#include "rules.h"
extern "C" {
int slab() { return trv::kSlab; }
unsigned most_pass_words() { return trv::kMostPassWords; }
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-shared", "-fPIC", f"-I{CSRC}", str(d / "shim.cpp"), "-o",
                    str(d / "rules.so")], check=True)
    lib = ctypes.CDLL(str(d / "rules.so"))
    lib.most_pass_words.restype = ctypes.c_uint32
    return lib


def test_rows_in_parts_keep_32_bit_offsets(rules):
    """A slab of the widest rows that go in parts: the words of the whole slab and
    a round past them, which the kernel counts in 32 bits with a sign."""
    most = rules.most_pass_words()
    in_flight = 32 * 8  # words that a round of a warp covers
    assert rules.slab() * most + 2 * in_flight <= 2**31 - 1
    assert most * 16 >= 200  # every width that goes in parts by default, in words of any size
