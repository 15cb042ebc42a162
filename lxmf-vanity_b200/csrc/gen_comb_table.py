#!/usr/bin/env python3
"""Generates comb_table.cuh: the multiples of Q = 8B that fixed-base scalar
multiplication adds up, on the twisted Edwards form of Curve25519
(-x^2 + y^2 = 1 + d x^2 y^2; u = (1 + y) / (1 - y), v = c u / x with
c^2 = -486664, the birational map of RFC 7748, section 4.1).

Entry (i, j), i < 32, 1 <= j <= 8, is the point j 256^i Q as the three field
elements that a mixed addition takes: y + x, y - x and 2 d x y.

Run from this directory: python gen_comb_table.py > comb_table.cuh
"""
P = 2**255 - 19
D = -121665 * pow(121666, P - 2, P) % P
# u(8B), and v(8B) as the even square root of u^3 + 486662 u^2 + u.
QU = int.from_bytes(bytes.fromhex("6899c948ed6f71f11ea974adcaed787aa15cb6c84d883bd82d5cd6aad7a65f27"), "little")


def inv(x: int) -> int:
    return pow(x, P - 2, P)


def sqrt_even(a: int) -> int:
    """The even square root mod p (p = 5 mod 8)."""
    r = pow(a, (P + 3) // 8, P)
    if r * r % P != a % P:
        r = r * pow(2, (P - 1) // 4, P) % P
    assert r * r % P == a % P
    return r if r % 2 == 0 else P - r


C = sqrt_even(-486664)
QV = sqrt_even(QU**3 + 486662 * QU**2 + QU)


def add(p, q):
    x1, y1 = p
    x2, y2 = q
    t = D * x1 * x2 * y1 * y2 % P
    return (x1 * y2 + x2 * y1) * inv(1 + t) % P, (y1 * y2 + x1 * x2) * inv(1 - t) % P


def words(x: int) -> str:
    return ", ".join(f"0x{x >> 32 * i & 0xffffffff:08x}" for i in range(8))


def main() -> None:
    base = (C * QU * inv(QV) % P, (QU - 1) * inv(QU + 1) % P)
    x, y = base
    assert (-x * x + y * y - 1 - D * x * x * y * y) % P == 0
    print("// Generated by gen_comb_table.py: do not edit by hand.")
    print("// [32][8][3][8]: j 256^i Q (j = 1..8) as y + x, y - x, 2 d x y.")
    print("#pragma once")
    print("#include <cstdint>")
    print()
    print(f"#define LXK_COMB_C {{{words(C)}}}")
    print(f"#define LXK_COMB_2D {{{words(2 * D % P)}}}")
    print()
    print("static __device__ const uint32_t kCombTable[32 * 8 * 24] __attribute__((aligned(16))) = {")
    for _ in range(32):
        p = base
        for _ in range(8):
            x, y = p
            for e in ((y + x) % P, (y - x) % P, 2 * D * x * y % P):
                print(f"    {words(e)},")
            p = add(p, base)
        for _ in range(8):
            base = add(base, base)
    print("};")


if __name__ == "__main__":
    main()
