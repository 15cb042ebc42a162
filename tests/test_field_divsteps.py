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


@pytest.fixture(scope="module")
def rows(tmp_path_factory):
    d = tmp_path_factory.mktemp("rows")
    src = d / "rows.cpp"
    src.write_text("""#include "fe_divsteps.h"
extern "C" {
void fg(const int32_t* m, uint32_t* f, uint32_t* g) { fed_apply_fg(f, g, fed_row(m[0], m[1]), fed_row(m[2], m[3])); }
void de(const int32_t* m, FedResidue* d, FedResidue* e) { fed_apply_de(*d, *e, fed_row(m[0], m[1]), fed_row(m[2], m[3]), m); }
}
""")
    so = d / "rows.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", str(so), str(src)], check=True)
    return ctypes.CDLL(str(so))


ROWS = [(1 << 30, 0), (0, -(1 << 30)), (-(1 << 30), 0), (1 << 29, -(1 << 29)), (-(1 << 29), -(1 << 29)), (0, 0), (1, 0),
        (0, -1), (-1, 1), ((1 << 30) - 1, 1), (-1, (1 << 30) - 1), (1, 1 - (1 << 30)), (123456789, -987654)]


class Residue(ctypes.Structure):
    _fields_ = [("w", ctypes.c_uint32 * 8), ("c", ctypes.c_int32)]


def _words(x):
    return (ctypes.c_uint32 * 8)(*[(x >> (32 * i)) & 0xFFFFFFFF for i in range(8)])


def _value(w):
    return sum(w[i] << (32 * i) for i in range(8))


@pytest.mark.parametrize("i", range(len(ROWS)))
def test_updates_of_a_batch(rows, i):
    """A batch's two updates at the ends of their ranges, against integers: the
    rows over 2^30, rounded down (exact where the rows are divsteps'), of
    256-bit signed f and g; and any 256 bits with any pending carry as
    residues."""
    rng = random.Random(i)
    m = ROWS[i] + ROWS[(i + 5) % len(ROWS)]
    cm = (ctypes.c_int32 * 4)(*m)
    ends = [0, 1, -1, 2, P, -P, 2**255 - 1, 1 - 2**255, 2**224, -(2**224), 2**32 - 1] + \
           [rng.randrange(-(2**255) + 1, 2**255) for _ in range(8)]
    for f in ends:
        for g in ends:
            a, b = _words(f), _words(g)
            rows.fg(cm, a, b)
            assert _value(a) == (m[0] * f + m[1] * g >> 30) % 2**256, (f, g)
            assert _value(b) == (m[2] * f + m[3] * g >> 30) % 2**256, (f, g)
    ends = [0, 1, 18, 19, 37, 38, P, 2 * P, 2**255, 2**256 - 1, 2**256 - 38, 2**64 - 1, 2**256 - 2**64] + \
           [rng.getrandbits(256) for _ in range(8)]
    for x in ends:
        for y in ends:
            for xc, yc in ((0, 0), (1, -1), (-1, 1), (-1, -1), (1, 1)):
                d, e = Residue(_words(x), xc), Residue(_words(y), yc)
                rows.de(cm, ctypes.byref(d), ctypes.byref(e))
                dv, ev = x + (xc << 64), y + (yc << 64)
                for got, want in ((d, m[0] * dv + m[1] * ev), (e, m[2] * dv + m[3] * ev)):
                    assert got.c in (-1, 0, 1) and (_value(got.w) + (got.c << 64) - want) % P == 0, (x, y, xc, yc)
