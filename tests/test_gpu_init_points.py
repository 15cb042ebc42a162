"""Grouped walk from public keys near the point at infinity (Backend.init
takes any): a centre that is a table point up to sign has a denominator of
zero, and the batch inversion then makes every inverse of its group zero, in
however many parts the group is walked."""
import numpy as np
import pytest

P = 2**255 - 19
A = 486662
U = int.from_bytes(np.array([0x48C99968, 0xF1716FED, 0xAD74A91E, 0x7A78EDCA, 0xC8B65CA1, 0xD83B884D, 0xAAD65C2D, 0x275FA6D7],
                            "<u4").tobytes(), "little")  # u(8B)


def _sqrt(a):
    r = pow(a, (P + 3) // 8, P)
    if r * r % P != a:
        r = r * pow(2, (P - 1) // 4, P) % P
    assert r * r % P == a
    return r if r % 2 == 0 else P - r


Q = (U, _sqrt((U**3 + A * U * U + U) % P))


def _add(p, q):
    if p == q:
        l = (3 * p[0] * p[0] + 2 * A * p[0] + 1) * pow(2 * p[1], -1, P) % P
    else:
        l = (q[1] - p[1]) * pow(q[0] - p[0], -1, P) % P
    u = (l * l - A - p[0] - q[0]) % P
    return u, (l * (p[0] - u) - p[1]) % P


def _multiples(n):
    t = [None, Q]
    while len(t) <= n:
        t.append(_add(t[-1], Q))
    return t


def _walk(start, m, groups, table):
    """The keys of `groups` groups from P = start Q, as the walk computes
    them: with a zero among a group's denominators, every inverse is zero."""
    centre = table[abs(start + m)]
    if start + m < 0:
        centre = (centre[0], P - centre[1])
    keys = []
    for _ in range(groups):
        uc, vc = centre
        points = [table[2 * m]] + table[1:m + 1]
        dens = [(u - uc) % P for u, _ in points]
        inv = [0 if 0 in dens else pow(d, -1, P) for d in dens]
        up = [((v - vc) * i * (v - vc) * i - A - uc - u) % P for (u, v), i in zip(points, inv)]
        um = [((v + vc) * i * (v + vc) * i - A - uc - u) % P for (u, v), i in zip(points, inv)]
        keys += um[:0:-1] + [uc] + up[1:m]
        l = (points[0][1] - vc) * inv[0] % P
        centre = (up[0], (l * (uc - up[0]) - vc) % P)
    return keys


@pytest.mark.gpu
@pytest.mark.parametrize("lanes,batch", [(32, 64), (33, 1024), (1000, 256), (148 * 512, 64)])
def test_walks_through_infinity_by_parts(lx, lanes, batch):
    m = batch // 2
    table = _multiples(2 * m + 8)
    starts = [-5, 7, 1 - m, -1]  # zero denominators at i = m - 5, none, at i = 1, at i = m - 1
    words = np.zeros((lanes, 16), np.uint32)
    for t in range(lanes):
        s = starts[t % 4]
        for half, n in ((0, s - 1), (8, s)):
            words[t, half:half + 8] = np.frombuffer(table[abs(n)][0].to_bytes(32, "little"), "<u4")
    want = [_walk(s, m, 2, table) for s in starts]
    with lx.Backend(device=0, lanes=lanes, batch=batch) as b:
        b.init(words)
        got = []
        for _ in range(2):  # one group per launch, so that the stored state is seen too
            args = lx.make_launch_args(1, bytes(32), lx.prefix_parse("ffffffff"), dump_threads=32, dump_keys=batch)
            _, dump, _, _ = b.launch(args, want_dump=True)
            got.append(dump.reshape(32, batch, 8).view(np.uint8).reshape(32, batch, 32))
    for t in range(32):
        keys = [int.from_bytes(k.tobytes(), "little") for g in got for k in g[t]]
        assert keys == want[t % 4], (t, [i for i in range(2 * batch) if keys[i] != want[t % 4][i]][:5])
