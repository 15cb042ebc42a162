#!/usr/bin/env python3
"""Generates fe25519_ptx.cuh: GF(2^255-19) multiply and square on 8 x 32-bit
limbs as single inline-PTX blocks, so that each carry chain stays inside one
asm statement (the carry flag is not preserved between asm statements).

Representation: a field element is any 256-bit value x (8 little-endian
32-bit words) standing for x mod p, p = 2^255 - 19.  Products are reduced
with 2^256 = 38 (mod p) to another 256-bit value; only fe_canon (in
fe25519.cuh) maps to [0, p).

Run from this directory: python gen_fe_ptx.py > fe25519_ptx.cuh
"""


def _product(A: list[str], B: list[str], square: bool) -> list[str]:
    """The columns of a * b (or, square, of the cross products a_i a_j with
    i < j) into two accumulators: e<k> holds words of weight k, o<k> words of
    weight k + 1.  A product a_i b_j with i + j even adds to the aligned pair
    (e[i+j], e[i+j+1]), one with i + j odd to (o[i+j-1], o[i+j]), so a row is
    two chains of mad.lo.cc / madc.hi.cc over the same operands and an aligned
    register pair: one 32 x 32 + 64 multiply-add with carry each, where a row
    of low halves and a row of high halves take two and a carry add."""
    L = []
    defined = set()

    def chain(acc, items):
        regs = [(f"{acc}{k}", f"{acc}{k + 1}", x, y) for k, x, y in items]
        if not any(lo in defined for lo, _, _, _ in regs):
            for lo, hi, x, y in regs:
                L.append(f"mul.lo.u32 {lo}, {x}, {y};")
                L.append(f"mul.hi.u32 {hi}, {x}, {y};")
                defined.update((lo, hi))
            return
        for n, (lo, hi, x, y) in enumerate(regs):
            last = n == len(regs) - 1
            # The last pair of a row that reaches a new word cannot carry out
            # of it: the partial sum is below 2^(32 (k+2)) of its weight.
            grows = hi not in defined
            assert last or not grows
            L.append(f"{'madc' if n else 'mad'}.lo.cc.u32 {lo}, {x}, {y}, {lo if lo in defined else 0};")
            L.append(f"madc.hi{'' if grows else '.cc'}.u32 {hi}, {x}, {y}, {0 if grows else hi};")
            defined.update((lo, hi))
            if last and not grows:
                L.append(f"addc.u32 {acc}{items[-1][0] + 2}, 0, 0;")
                defined.add(f"{acc}{items[-1][0] + 2}")

    for i in range(8):
        js = range(i + 1 if square else 0, 8)
        for acc, odd in (("e", 0), ("o", 1)):
            items = [(i + j - odd, A[i], B[j]) for j in js if (i + j) % 2 == odd]
            if items:
                chain(acc, items)
    return L


def mul_body(square: bool) -> list[str]:
    """PTX lines computing a * b (or a * a) into %0..%7.  Inputs are %8..%15
    (a) and %16..%23 (b)."""
    A = [f"%{8 + i}" for i in range(8)]
    B = A if square else [f"%{16 + i}" for i in range(8)]
    L = [".reg .u32 e<16>;", ".reg .u32 o<16>;", ".reg .u32 c, t;", ".reg .pred p;"]
    L.extend(_product(A, B, square))
    if not square:
        # High half: e8..e15 += o7..o14.  The low halves stay apart until the
        # fold has added to both.
        L.append("add.cc.u32 e8, e8, o7;")
        for k in range(9, 15):
            L.append(f"addc.cc.u32 e{k}, e{k}, o{k - 1};")
        L.append("addc.u32 e15, e15, o14;")
    else:
        # The cross sum (words 1..14, below 2^480) doubled into e1..e15, then
        # the squares a_i^2 at words 2i, 2i + 1: aligned pairs again.
        L.append("add.cc.u32 e2, e2, o1;")
        for k in range(3, 14):
            L.append(f"addc.cc.u32 e{k}, e{k}, o{k - 1};")
        L.append("addc.u32 e14, 0, o13;")
        L.append("shf.l.wrap.b32 e15, e14, 0, 1;")
        for k in range(14, 2, -1):
            L.append(f"shf.l.wrap.b32 e{k}, e{k - 1}, e{k}, 1;")
        L.append("shf.l.wrap.b32 e2, o0, e2, 1;")
        L.append("shl.b32 e1, o0, 1;")
        L.append(f"mul.lo.u32 e0, {A[0]}, {A[0]};")
        L.append(f"mad.hi.cc.u32 e1, {A[0]}, {A[0]}, e1;")
        for i in range(1, 8):
            L.append(f"madc.lo.cc.u32 e{2 * i}, {A[i]}, {A[i]}, e{2 * i};")
            L.append(f"madc.hi{'.cc' if i < 7 else ''}.u32 e{2 * i + 1}, {A[i]}, {A[i]}, e{2 * i + 1};")
    L.extend(reduce_lines(square))
    return L


def reduce_lines(square: bool) -> list[str]:
    """e0..e15 plus (a product only) o0..o6 at weights 1..7 -> %0..%7 with
    2^256 = 38; result < 2^256."""
    L = []
    # 38 e8, 38 e10, ... on the pairs of e0..e7; their carry into c.
    for k in range(0, 8, 2):
        L.append(f"{'madc' if k else 'mad'}.lo.cc.u32 e{k}, e{k + 8}, 38, e{k};")
        L.append(f"madc.hi.cc.u32 e{k + 1}, e{k + 8}, 38, e{k + 1};")
    L.append("addc.u32 c, 0, 0;")
    # 38 e9, 38 e11, ... on the pairs of o0..o7 (o7, of weight 8, is new).
    for k in range(0, 8, 2):
        if square:
            L.append(f"mul.lo.u32 o{k}, e{k + 9}, 38;")
            L.append(f"mul.hi.u32 o{k + 1}, e{k + 9}, 38;")
        else:
            L.append(f"{'madc' if k else 'mad'}.lo.cc.u32 o{k}, e{k + 9}, 38, o{k};")
            L.append(f"madc.hi{'.cc' if k < 6 else ''}.u32 o{k + 1}, e{k + 9}, 38, {f'o{k + 1}' if k < 6 else 0};")
    L.append("add.cc.u32 e1, e1, o0;")
    for k in range(2, 8):
        L.append(f"addc.cc.u32 e{k}, e{k}, o{k - 1};")
    L.append("addc.u32 c, c, o7;")
    # value = e0..e7 + c 2^256 with c <= 40: fold c once more.  The add into
    # e0 carries into e1 with probability below 2^-21, so that chain is a
    # branch the common case skips.
    L.append("mul.lo.u32 t, c, 38;")
    L.append("add.cc.u32 e0, e0, t;")
    L.append("addc.u32 c, 0, 0;")
    L.append("setp.eq.u32 p, c, 0;")
    L.append("@p bra FOLDED;")
    L.append("add.cc.u32 e1, e1, 1;")
    for k in range(2, 8):
        L.append(f"addc.cc.u32 e{k}, e{k}, 0;")
    L.append("addc.u32 c, 0, 0;")
    # A carry here leaves e0..e7 < 38 * 40: adding 38 cannot carry.
    L.append("mad.lo.u32 e0, c, 38, e0;")
    L.append("FOLDED:")
    for k in range(8):
        L.append(f"mov.u32 %{k}, e{k};")
    return L


def emit_asm(name: str, lines: list[str], square: bool) -> str:
    out = []
    params = "fe& o, const fe& a" if square else "fe& o, const fe& a, const fe& b"
    out.append(f"__device__ __forceinline__ void {name}({params}) {{")
    out.append("    asm(\"{\\n\\t\"")
    for ln in lines:
        out.append(f"        \"{ln}\\n\\t\"")
    out.append("        \"}\"")
    outs = ", ".join(f'"=r"(o.v[{i}])' for i in range(8))
    ins_a = ", ".join(f'"r"(a.v[{i}])' for i in range(8))
    if square:
        out.append(f"        : {outs}")
        out.append(f"        : {ins_a});")
    else:
        ins_b = ", ".join(f'"r"(b.v[{i}])' for i in range(8))
        out.append(f"        : {outs}")
        out.append(f"        : {ins_a},")
        out.append(f"          {ins_b});")
    out.append("}")
    return "\n".join(out)


def main() -> None:
    print("// Generated by gen_fe_ptx.py: do not edit by hand.")
    print("// 8 x 32-bit limb multiply and square mod 2^255-19 (2^256 = 38), one")
    print("// inline-PTX block each so every carry chain stays in one asm statement.")
    print("#pragma once")
    print()
    print(emit_asm("fe_mul_ptx", mul_body(False), False))
    print()
    print(emit_asm("fe_sqr_ptx", mul_body(True), True))


if __name__ == "__main__":
    main()
