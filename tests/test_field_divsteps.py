"""The divsteps inversion, built for the CPU from the kernels' own header and
checked against Python integers mod p = 2^255 - 19, and the start points'
table against its generator (no GPU needed)."""
import ctypes
import os
import random
import subprocess
import sys

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "lxmf-vanity_b200", "csrc")
P = 2**255 - 19


@pytest.fixture(scope="module")
def invert(tmp_path_factory):
    d = tmp_path_factory.mktemp("divsteps")
    src = d / "inv.cpp"
    src.write_text('#include "fe_divsteps.h"\nextern "C" void inv(const uint32_t* z, uint32_t* o) { fed_invert(z, o); }\n')
    so = d / "inv.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", str(so), str(src)], check=True)
    lib = ctypes.CDLL(str(so))

    def call(z):
        a = (ctypes.c_uint32 * 8)(*[(z >> (32 * i)) & 0xFFFFFFFF for i in range(8)])
        o = (ctypes.c_uint32 * 8)()
        lib.inv(a, o)
        return sum(o[i] << (32 * i) for i in range(8))

    return call


@pytest.mark.parametrize("name", ["edges", "powers of two", "near p", "random"])
def test_divsteps_inverse(invert, name):
    rng = random.Random(17)
    values = {"edges": [0, 1, 2, 18, 19, 20, P - 2, P - 1, (P - 1) // 2, (P + 1) // 2, 2**255 - 20],
              "powers of two": [2**i for i in range(255)],
              "near p": [P - 2**i for i in range(255)] + [2**255 - 2**i for i in range(5, 255)],
              "random": [rng.randrange(P) for _ in range(5000)]}[name]
    for z in values:
        assert invert(z) == pow(z, P - 2, P), hex(z)  # canonical, and 0 for 0


def test_fold_of_a_difference(tmp_path):
    """fe_sub_canon's common case: whenever it accepts, the value is a - b mod
    p, canonical; it refuses only near the ends of limb 0 or of the top limb."""
    src = tmp_path / "fold.cpp"
    src.write_text('#include "fe_fold.h"\nextern "C" int fold(uint32_t* d, uint32_t b) { return fef_fold(d, b); }\n')
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", str(tmp_path / "f.so"), str(src)], check=True)
    lib = ctypes.CDLL(str(tmp_path / "f.so"))
    rng = random.Random(23)
    ends = [0, 1, 18, 19, 37, 38, 63, 64, 65, 127, 2**32 - 66, 2**32 - 65, 2**32 - 64, 2**32 - 20, 2**32 - 1, P - 1, P, P + 1,
            2**255 - 1, 2**255, 2**255 + 64, 2**256 - 65, 2**256 - 1] + [rng.getrandbits(256) for _ in range(40)]
    values = ends + [(x + rng.getrandbits(256)) % 2**256 for x in ends] + [(x << 224) % 2**256 for x in ends]
    accepted = 0
    for a in values:
        for b in values:
            diff = (a - b) % 2**256
            d = (ctypes.c_uint32 * 8)(*[(diff >> (32 * i)) & 0xFFFFFFFF for i in range(8)])
            if lib.fold(d, 0xFFFFFFFF if a < b else 0):
                accepted += 1
                assert sum(d[i] << (32 * i) for i in range(8)) == (a - b) % P, (hex(a), hex(b))
            else:
                assert (diff + 64) % 2**32 < 128 or (diff >> 224) % 2**31 == 2**31 - 1
    assert accepted > len(values) ** 2 // 2


def test_comb_table_is_current():
    out = subprocess.run([sys.executable, os.path.join(CSRC, "gen_comb_table.py")], capture_output=True, text=True, check=True)
    assert out.stdout == open(os.path.join(CSRC, "comb_table.cuh")).read()
