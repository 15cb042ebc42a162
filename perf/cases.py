"""The work that a user of this library has it do, as measurable cases.

The library walks X25519 keys k, k+8, k+16, ... on many lanes, hashes every
key to its LXMF destination hash and reports those that start with a prefix.
Programs reach it through the ctypes bindings over the C ABI: `Backend` (one
search), `Pool` (many searches at once) and a few array entry points.

A case is a dict of plain values; `kind` says which entry points it calls:

  search  Backend.launch on an open, initialised handle: one launch of the walk
          and its hits, as the command line's search loop runs it;
  check   the same with a dump of the first lanes' keys and hashes (the self-test);
  start   Backend.init_from_scalars, then the first launch: a new search on an
          open handle;
  keys    Backend.first_public_keys: start points in the layout Backend.init takes;
  batch   Pool.step and Pool.poll on a resident mix of searches;
  serve   one turn of a serving loop: admit what arrived, step, poll, retire;
  hash    Backend.address_chain on public keys in host memory;
  invert  fe_batch_invert_static on device buffers.

Hits come from an atomic queue in no fixed order, so they are returned sorted,
in an array of a fixed number of rows (the unused ones are -1).
"""
import hashlib
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "lxmf-vanity_b200"))

import lxmfv as lx  # noqa: E402
import lxmfv_serve as serving  # noqa: E402

HEX = "0123456789abcdef"
P = 2**255 - 19

# One wave of the default launch shape (512 threads on each of 148 SMs), and the
# two waves that the benchmark walks.
ONE_WAVE = 75776
TWO_WAVES = 151552


def listed():
    return [
        # The self-test: 256 lanes x one batch of 512, every key and hash dumped
        # and a 2-digit prefix; the smallest launch a program makes.
        {"name": "self_test", "kind": "check", "walk": 0, "lanes": 256, "batch": 512, "block": 0, "flags": 0,
         "iters": 1, "nibbles": 2, "dump": 256},
        # A search on few walkers, the size of the smoke run (--lanes 2048).
        {"name": "few_lanes", "kind": "search", "walk": 0, "lanes": 2048, "batch": 1024, "block": 0, "flags": 0,
         "iters": 1, "nibbles": 5},
        # The command line's search: one wave of the default shape, launches of about a tenth of a second.
        {"name": "default", "kind": "search", "walk": 0, "lanes": ONE_WAVE, "batch": 1024, "block": 0, "flags": 0,
         "iters": 4, "nibbles": 5},
        # A walker count that is no multiple of a wave, a block or a warp (--lanes 100003).
        {"name": "ragged_lanes", "kind": "search", "walk": 0, "lanes": 100003, "batch": 1024, "block": 0, "flags": 0,
         "iters": 2, "nibbles": 5},
        # The benchmark's lanes, at the 64 keys per inversion of the reference kernel.
        {"name": "two_waves_g64", "kind": "search", "walk": 0, "lanes": TWO_WAVES, "batch": 64, "block": 0, "flags": 0,
         "iters": 64, "nibbles": 5},
        # The x-only walk (the reference's algorithm) at 64 keys per inversion, in the benchmark's shape.
        {"name": "xonly_b64", "kind": "search", "walk": 1, "lanes": TWO_WAVES, "batch": 64, "block": 512, "flags": 0,
         "iters": 16, "nibbles": 5},
        # A new search on an open handle: start points for one wave, then the first launch.
        {"name": "start", "kind": "start", "walk": 0, "lanes": ONE_WAVE, "batch": 1024, "block": 0, "flags": 0,
         "iters": 1, "nibbles": 5},
        # Start points for one wave as arrays, for programs that keep their own (the reference's interface).
        {"name": "first_keys", "kind": "keys", "count": ONE_WAVE},
        # The batched workload: 256 mixed searches of 1,184 lanes in one pool.
        {"name": "pool_256", "kind": "batch", "searches": 256, "lanes": 1184, "batch": 1024, "groups": 1,
         "min_nibbles": 4, "max_nibbles": 10},
        # The serving loop in its usual state: a dozen small searches and a larger one resident, two arriving.
        {"name": "serve_turn", "kind": "serve", "small": 12, "medium": 2, "large": 1, "arrive": 2, "batch": 1024},
        # Destination hashes of public keys that a program already has.
        {"name": "hash_keys", "kind": "hash", "count": 1 << 20},
        # Batch inversion on a host runtime's own device buffers, at the most a call takes.
        {"name": "invert", "kind": "invert", "count": 131072, "group": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _nibbles(keys):
    """A prefix length that some dozens to hundreds of the keys of a pass match."""
    n = 1
    while keys / 16.0**n > 600 and n < 9:
        n += 1
    return n


def draw(rng):
    kind = rng.choice(["search", "search", "search", "check", "start", "keys", "batch", "serve", "hash", "invert"])
    if kind in ("search", "check", "start"):
        walk = 1 if rng.random() < 0.25 else 0
        batch = rng.choice([16, 32, 64, 128] if walk else [32, 64, 128, 256, 512, 1024, 1024, 1024])
        lanes = _log_int(rng, 33, 4096 if kind == "check" else TWO_WAVES)
        block, flags = rng.choice([(0, 0), (0, 0), (128, 0), (256, 0), (256, 1), (512, 0), (512, 1)])
        # 2^17 .. 2^27 keys, and no lane longer than four batches of 1024.
        per_lane = min(4096, max(1, _log_int(rng, 1 << 17, 1 << 27) // lanes))
        iters = 1 if kind == "check" else max(1, per_lane // batch)
        case = {"kind": kind, "walk": walk, "lanes": lanes, "batch": batch, "block": block, "flags": flags,
                "iters": iters, "nibbles": _nibbles(lanes * batch * iters)}
        if kind == "check":
            case["dump"] = max(1, lanes // rng.choice([1, 3, 16]))
        return case
    if kind == "keys":
        return {"kind": "keys", "count": _log_int(rng, 1, TWO_WAVES)}
    if kind == "batch":
        searches = _log_int(rng, 1, 256)
        lanes = 32 * _log_int(rng, 1, min(512, 9472 // searches))
        batch = rng.choice([64, 128, 256, 512, 1024, 1024])
        return {"kind": "batch", "searches": searches, "lanes": lanes, "batch": batch, "groups": rng.choice([1, 2, 4])
                if searches * lanes < TWO_WAVES // 2 else 1, "min_nibbles": 4, "max_nibbles": 8}
    if kind == "serve":
        return {"kind": "serve", "small": _log_int(rng, 1, 64), "medium": rng.randrange(0, 6),
                "large": rng.randrange(0, 3), "arrive": rng.randrange(1, 7), "batch": rng.choice([256, 512, 1024, 1024])}
    if kind == "hash":
        return {"kind": "hash", "count": _log_int(rng, 1, 1 << 20)}
    return {"kind": "invert", "count": _log_int(rng, 1, 131072), "group": _log_int(rng, 1, 256)}


def _prefix(rng, nibbles):
    return "".join(rng.choice(HEX) for _ in range(nibbles))


def _spec(rng, nibbles, lanes):
    return serving.SearchSpec.seeded(rng.getrandbits(40), _prefix(rng, nibbles), rng.choice(serving.ASPECTS), lanes)


def prepare(case, seed):
    rng = random.Random("%s %d" % (sorted((k, v) for k, v in case.items() if k != "name"), seed))
    kind = case["kind"]
    if kind in ("search", "check", "start"):
        b = lx.Backend(device=0, lanes=case["lanes"], batch=case["batch"], block=case["block"], walk=case["walk"],
                       flags=case["flags"])
        setup = lx.seeded_setup(rng.getrandbits(40), case["lanes"])
        if kind != "start":
            b.init_from_scalars(setup.scalars)
        dump = case.get("dump", 0)
        args = lx.make_launch_args(case["iters"], setup.ed_pub, lx.prefix_parse(_prefix(rng, case["nibbles"])),
                                   dump_threads=dump)
        return {"kind": kind, "backend": b, "scalars": setup.scalars, "args": args}
    if kind == "keys":
        scalars, _ = lx.seeded_scalars(rng.getrandbits(40), 0, case["count"])
        return {"kind": kind, "backend": lx.Backend(device=0, lanes=256), "scalars": scalars}
    if kind == "batch":
        pool = serving.Pool(device=0, capacity_lanes=case["searches"] * case["lanes"], batch=case["batch"])
        pool.submit_many([_spec(rng, rng.randint(case["min_nibbles"], case["max_nibbles"]), case["lanes"])
                          for _ in range(case["searches"])])
        return {"kind": kind, "pool": pool, "groups": case["groups"]}
    if kind == "serve":
        # Lanes by difficulty (64 for 5 digits and fewer, 1,024 for 6, 16,384 for 7), as the serving loop gives them.
        pool = serving.Pool(device=0, capacity_lanes=262144, batch=case["batch"])
        lengths = [rng.choice((4, 5)) for _ in range(case["small"])] + [6] * case["medium"] + [7] * case["large"]
        pool.submit_many([_spec(rng, n, serving.lanes_by_difficulty(n)) for n in lengths])
        arrive = [_spec(rng, n, serving.lanes_by_difficulty(n)) for n in (rng.choice((3, 4, 5))
                                                                          for _ in range(case["arrive"]))]
        return {"kind": kind, "pool": pool, "arrive": arrive}
    if kind == "hash":
        keys = np.random.default_rng(rng.getrandbits(60)).integers(0, 256, (case["count"], 64), np.uint8)
        return {"kind": kind, "backend": lx.Backend(device=0, lanes=256), "keys": keys, "name_hash": lx.name_hash()}
    a = torch.from_numpy(_elements(case, rng).view(np.int32)).cuda()
    return {"kind": kind, "a": a, "out": torch.empty_like(a), "group": case["group"]}


def _elements(case, rng):
    """Nonzero field elements as 8 little-endian words."""
    a = np.random.default_rng(rng.getrandbits(60)).integers(0, 2**32, (case["count"], 8), np.uint32)
    a[:, 0] |= 1
    a[:, 7] >>= 2
    return a


def _rows(hits, width):
    rows = np.full((lx.MAX_HITS, width), -1, np.int64)
    if hits:
        rows[:len(hits)] = sorted(hits)
    return rows


def run(state):
    kind = state["kind"]
    if kind == "search":
        hits, _, _, n = state["backend"].launch(state["args"])
        return {"hits": _rows(hits, 2), "count": n}
    if kind == "check":
        hits, keys, hashes, n = state["backend"].launch(state["args"], want_dump=True, want_dump_addr=True)
        return {"hits": _rows(hits, 2), "count": n, "keys": keys, "hashes": hashes}
    if kind == "start":
        state["backend"].init_from_scalars(state["scalars"])
        hits, _, _, n = state["backend"].launch(state["args"])
        return {"hits": _rows(hits, 2), "count": n}
    if kind == "keys":
        return state["backend"].first_public_keys(state["scalars"])
    if kind == "batch":
        state["pool"].step(state["groups"])
        hits, n = state["pool"].poll()
        return {"hits": _rows(hits, 3), "count": n}
    if kind == "serve":
        pool = state["pool"]
        ids = pool.submit_many(state["arrive"])
        pool.step(1)
        hits, n = pool.poll()
        for i in ids:
            pool.retire(i)
        return {"ids": ids, "hits": _rows(hits, 3), "count": n}
    if kind == "hash":
        return state["backend"].address_chain(state["keys"], state["name_hash"])
    # In order with the caller's other work on its current stream.
    lx.fe_batch_invert_static(state["a"].data_ptr(), state["out"].data_ptr(), state["a"].shape[0], state["group"],
                              torch.cuda.current_stream().cuda_stream)
    return state["out"]


# 32-bit integer operations that the path cannot do without.  A hash: three
# compressions of 64 rounds (6 rotates, 4 logic functions, 7 sums), two message
# schedules of 48 words (4 rotates, 2 shifts, 2 logic functions, 3 sums).  A
# field multiply: 64 products, 8 for the reduction, a multiply and an add each.
HASH_OPS = 3 * 64 * 17 + 2 * 48 * 11
MUL_OPS = 2 * 72
SQR_OPS = 2 * 44
# An inversion by Fermat's chain, and a start point by a ladder of 253 steps.
INV_OPS = 254 * SQR_OPS + 11 * MUL_OPS
START_OPS = 253 * (5 * MUL_OPS + 4 * SQR_OPS) + INV_OPS


def work(case):
    kind = case["kind"]
    if kind in ("search", "check", "start"):
        lanes, batch = case["lanes"], case["batch"]
        keys = lanes * batch * case["iters"]
        if case["walk"]:
            per_key, state = 8 * MUL_OPS + 2 * SQR_OPS, 2 * 136
        else:
            per_key, state = 2.5 * MUL_OPS + SQR_OPS, 2 * 72
        ops = keys * (HASH_OPS + per_key) + lanes * case["iters"] * INV_OPS
        moved = lanes * state + 48 * case.get("dump", 0) * batch
        if kind == "start":
            ops += lanes * START_OPS
            moved += 32 * lanes
        return {"bytes": moved, "flops": ops}
    if kind == "keys":
        return {"bytes": 96 * case["count"], "flops": case["count"] * START_OPS}
    if kind in ("batch", "serve"):
        if kind == "batch":
            lanes, new, groups = case["searches"] * case["lanes"], 0, case["groups"]
        else:
            new, groups = 64 * case["arrive"], 1
            lanes = 64 * case["small"] + 1024 * case["medium"] + 16384 * case["large"] + new
        keys = lanes * case["batch"] * groups
        return {"bytes": 144 * lanes + 32 * new, "flops": keys * (HASH_OPS + 2.5 * MUL_OPS + SQR_OPS)
                + lanes * groups * INV_OPS + new * START_OPS}
    if kind == "hash":
        return {"bytes": 80 * case["count"], "flops": case["count"] * HASH_OPS}
    groups = -(-case["count"] // case["group"])
    return {"bytes": 64 * case["count"], "flops": case["count"] * 3 * MUL_OPS + groups * INV_OPS}


def exact(case, seed):
    """The hashes by hashlib and the inverses by Python integers; the walks'
    outputs are whole numbers that a reference of this kind takes minutes for."""
    kind = case["kind"]
    if kind not in ("hash", "invert"):
        return None
    rng = random.Random("%s %d" % (sorted((k, v) for k, v in case.items() if k != "name"), seed))
    if kind == "hash":
        keys = np.random.default_rng(rng.getrandbits(60)).integers(0, 256, (case["count"], 64), np.uint8).tobytes()
        name = hashlib.sha256(b"lxmf.delivery").digest()[:10]
        sha = hashlib.sha256
        got = b"".join(sha(name + sha(keys[i:i + 64]).digest()[:16]).digest()[:16] for i in range(0, len(keys), 64))
        return np.frombuffer(got, np.uint8).reshape(-1, 16)
    a = [int.from_bytes(row.tobytes(), "little") for row in _elements(case, rng)]
    prefix, acc = [], 1
    for x in a:
        prefix.append(acc)
        acc = acc * x % P
    inv, out = pow(acc, P - 2, P), [b""] * len(a)
    for i in range(len(a) - 1, -1, -1):
        out[i] = (inv * prefix[i] % P).to_bytes(32, "little")
        inv = inv * a[i] % P
    return np.frombuffer(b"".join(out), np.int32).reshape(-1, 8)
