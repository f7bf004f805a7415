"""Performance cases of the engine, each through an entry point that a
program calls: the api.h drop-in, the one-shot and the reusable batches of
include/cuspx.h, and several parameter sets in one graph launch.

Sizes follow bench.py (4096 x 64-B messages under one key, 1024 signatures of
256 B per set, 16 .. 1024-B served messages with 10% corrupted signatures,
log-uniform 1 B .. 64 KiB requests over two sets and many keys, messages of a
megabyte) and the widths in between.  Every output is bytes, verdicts or
statuses; there are no floating-point results.
"""
import ctypes
import math

import numpy as np
import torch

import cuspx_gb300 as c

# (n, h, d, a, k) of the parameter sets, by size
SIZES = {"128s": (16, 63, 7, 12, 14), "128f": (16, 66, 22, 6, 33), "192s": (24, 63, 7, 14, 17),
         "192f": (24, 66, 22, 8, 33), "256s": (32, 64, 8, 14, 22), "256f": (32, 68, 17, 9, 35)}
SET_NAMES = ["%s-%s-%s" % (h, s, m) for h in ("sha256", "shake256") for s in SIZES for m in ("simple", "robust")]
# 32-bit integer operations of one hash unit, as bench.py counts them: a
# SHA-256 compression or a Keccak-f[1600] permutation
OPS = {"sha256": 1384, "shake256": 4560}


def listed():
    return [
        # one call at a time through the NIST api.h drop-in: a program that
        # was linked against the reference and now links this library
        {"name": "api sign 1", "kind": "api_sign", "set": "sha256-128f-simple", "count": 1, "keys": 1,
         "min_len": 33, "max_len": 33},
        {"name": "api open 1", "kind": "api_open", "set": "sha256-128f-simple", "count": 1, "keys": 1,
         "min_len": 1024, "max_len": 1024},
        # the headline batch: one signing service, one key, 4096 short messages
        {"name": "sign 4096", "kind": "sign", "set": "sha256-128f-simple", "count": 4096, "keys": 1,
         "min_len": 64, "max_len": 64},
        # ... and the verification of such a batch
        {"name": "verify 4096", "kind": "verify", "set": "sha256-128f-simple", "count": 4096, "keys": 1,
         "min_len": 64, "max_len": 64},
        # provisioning: a key pair for each of 4096 seeds
        {"name": "keygen 4096", "kind": "keygen", "set": "sha256-128f-simple", "count": 4096, "keys": 4096,
         "min_len": 0, "max_len": 0},
        # a small burst of requests under keys of their own, ragged lengths, one-shot call
        {"name": "oneshot sign 37", "kind": "oneshot_sign", "set": "sha256-192f-simple", "count": 37, "keys": 37,
         "min_len": 1, "max_len": 1024},
        # verification traffic of a few hundred requests over some keys, 10% of them forged
        {"name": "verify 301", "kind": "verify", "set": "sha256-128f-simple", "count": 301, "keys": 17,
         "min_len": 16, "max_len": 1024},
        # SHAKE-256 at the widest set, one key
        {"name": "sign shake 1024", "kind": "sign", "set": "shake256-256f-simple", "count": 1024, "keys": 1,
         "min_len": 256, "max_len": 256},
        # verify-heavy traffic of the robust SHAKE-256 set, a key per request
        {"name": "verify shake robust 2048", "kind": "verify", "set": "shake256-256f-robust", "count": 2048,
         "keys": 2048, "min_len": 16, "max_len": 1024},
        # small signatures (s set, tall subtrees), robust, every request under its own key
        {"name": "sign 256s robust 100", "kind": "sign", "set": "sha256-256s-robust", "count": 100, "keys": 100,
         "min_len": 16, "max_len": 1024},
        # documents of about a megabyte, where hashing the message is the work
        {"name": "oneshot sign long 3", "kind": "oneshot_sign", "set": "sha256-128f-simple", "count": 3, "keys": 3,
         "min_len": 900001, "max_len": 1048577},
        # uneven requests of two parameter sets over 16 keys each, in one graph launch
        {"name": "mixed 256", "kind": "mixed", "set": "sha256-128s-simple", "set2": "sha256-192f-robust",
         "count": 256, "keys": 16, "min_len": 1, "max_len": 65536},
    ]


# ---------------------------------------------------------------------------
# work of one pass
# ---------------------------------------------------------------------------
def _shape(name):
    h, size, mode = name.split("-")
    n, hh, d, a, k = SIZES[size]
    return h, n, hh, d, a, k, hh // d, 2 * n + 3, mode == "robust"


def _sig_bytes(name):
    _, n, hh, d, a, k, hp, ln, _ = _shape(name)
    return n * (1 + k * (a + 1) + d * ln + hh)


def _msg_units(name, sign, mlen):
    h, n, hh, d, a, k, hp, ln, _ = _shape(name)
    dgst = (k * a + 7) // 8 + (hh - hp + 7) // 8 + (hp + 7) // 8
    if h == "shake256":
        return (3 * n + mlen) // 136 + 1 + ((2 * n + mlen) // 136 + 1 if sign else 0)
    return (3 * n + mlen + 72) // 64 + (dgst + 31) // 32 + (3 + (n + mlen + 72) // 64 if sign else 0)


def _units(name, kind, count, keys, mlen):
    """Hash units of `count` requests over `keys` keys.  Requests of one key
    share subtrees towards the top of the hypertree, where a subtree that
    several of them need counts once (its expected number of distinct ones)."""
    h, n, hh, d, a, k, hp, ln, robust = _shape(name)

    def th(m):  # T_m of m n-byte values
        if h == "shake256":
            return (n + 32 + m * n) // 136 + 1 + (-(-m * n // 136) if robust else 0)
        return (22 + m * n + 72) // 64 + (-(-m * n // 32) * ((n + 26 + 72) // 64) if robust else 0)

    leaf = ln * (1 + 15 * th(1)) + th(ln)
    tree = (leaf << hp) + ((1 << hp) - 1) * th(2)
    if kind == "keygen":
        return count * tree
    if kind in ("verify", "api_open"):
        steps = 7.5 * (2 * n) + 3 * 7.5
        return count * (_msg_units(name, False, mlen) + k * (th(1) + a * th(2)) + th(k) +
                        d * (steps * th(1) + th(ln) + hp * th(2)))
    per = count / keys
    trees = 0.0
    for layer in range(d):
        there = 2.0 ** (hp * (d - 1 - layer))
        trees += keys * (there * -math.expm1(per * math.log1p(-1.0 / there)) if there > 1 else 1.0)
    fors = k * ((1 + th(1) << a) + ((1 << a) - 1) * th(2)) + th(k)
    return count * (_msg_units(name, True, mlen) + fors) + trees * tree


def _mean_len(case):
    lo, hi = case["min_len"], case["max_len"]
    return hi if lo == hi else int((hi - lo) / math.log(hi / max(lo, 1)))


def _parts(case):
    """(set, count, keys) of each parameter set in the case"""
    if case["kind"] == "mixed":
        half = case["count"] // 2
        return [(case["set"], case["count"] - half, case["keys"]), (case["set2"], half, case["keys"])]
    return [(case["set"], case["count"], case["keys"])]


def work(case):
    """bytes: inputs and outputs; flops: 32-bit integer operations of the hash units"""
    kind, mlen = case["kind"], _mean_len(case)
    nbytes = ops = 0.0
    for name, count, keys in _parts(case):
        n = _shape(name)[1]
        ops += _units(name, kind, count, min(keys, count), mlen) * OPS[name.split("-")[0]]
        nbytes += count * 9 * n if kind == "keygen" else count * (mlen + _sig_bytes(name)) + min(keys, count) * 4 * n
    return {"bytes": nbytes, "flops": ops}


# ---------------------------------------------------------------------------
# drawn cases
# ---------------------------------------------------------------------------
def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    limit = max(work(x)["flops"] for x in listed())
    kind = rng.choice(["api_sign", "api_open", "sign", "sign", "verify", "verify", "keygen", "oneshot_sign", "long",
                       "mixed"])
    name = rng.choice(SET_NAMES)
    lo = rng.randint(1, 64)
    case = {"kind": kind, "set": name, "count": 1, "keys": 1, "min_len": lo, "max_len": lo + rng.randint(0, 1000)}
    if kind == "long":
        size = _log_int(rng, 2048, 1 << 20)
        case.update(kind="oneshot_sign", count=rng.randint(1, 8), min_len=size - rng.randint(0, 999), max_len=size)
    elif kind == "oneshot_sign":
        case["count"] = _log_int(rng, 2, 256)
    elif kind == "mixed":
        case.update(set2=rng.choice([x for x in SET_NAMES if x != name]), count=_log_int(rng, 4, 512), max_len=65536)
    elif kind in ("sign", "verify", "keygen"):
        case["count"] = _log_int(rng, 6 if kind == "verify" else 2, 4096)

    def cost(x):  # verify inputs are signed first
        return work(dict(x, kind="sign"))["flops"] if x["kind"] == "verify" else work(x)["flops"]

    case["keys"] = case["count"]
    while case["count"] > 1 and cost(case) > limit:
        case["count"] = case["keys"] = case["count"] * 3 // 4
    if kind == "keygen":
        case["min_len"] = case["max_len"] = 0
    else:
        case["keys"] = rng.choice([1, _log_int(rng, 1, case["count"]), case["count"]])
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
_engine = None
_dropins = {}


def _eng():
    global _engine
    if _engine is None:
        _engine = c.Engine(0)
    return _engine


def _dropin(name):
    if name not in _dropins:
        L = ctypes.CDLL(c.dropin_path(name))
        p, z = ctypes.c_void_p, ctypes.c_size_t
        L.crypto_sign_signature.argtypes = [p, ctypes.POINTER(z), p, z, p]
        L.crypto_sign_open.argtypes = [p, ctypes.POINTER(ctypes.c_ulonglong), p, ctypes.c_ulonglong, p]
        _dropins[name] = L
    return _dropins[name]


def _pinned(nbytes):
    return torch.empty(max(1, nbytes), dtype=torch.uint8, pin_memory=True).numpy()


def _at(a):
    return ctypes.c_void_p(a.ctypes.data)


class _Requests:
    """Seeded keys and messages of `count` requests of one set, in pinned host
    buffers: key rows and the row of each request, and a message slab with
    16-byte aligned offsets."""

    def __init__(self, rng, name, count, keys, lo, hi):
        eng = _eng()
        self.name, self.sid, self.count, self.nkeys = name, c.set_id(name), count, min(keys, count)
        self.z = z = c.set_sizes(self.sid)
        seeds = [rng.bytes(z["seed"]) for _ in range(self.nkeys)]
        pks, sks = eng.keypair_batch(self.sid, seeds)
        self.pks = _pinned(self.nkeys * z["pk"])
        self.sks = _pinned(self.nkeys * z["sk"])
        self.pks[:] = np.frombuffer(b"".join(pks), np.uint8)
        self.sks[:] = np.frombuffer(b"".join(sks), np.uint8)
        self.row = np.arange(count, dtype=np.uint32) if self.nkeys == count else \
            rng.integers(0, self.nkeys, count, dtype=np.uint32)
        if lo == hi:
            self.lens = np.full(count, lo, np.uint64)
        else:
            self.lens = np.floor(np.exp(rng.uniform(math.log(max(lo, 1)), math.log(hi + 1), count))).astype(np.uint64)
        step = (self.lens + np.uint64(15)) & ~np.uint64(15)
        self.offs = np.zeros(count, np.uint64)
        self.offs[1:] = np.cumsum(step)[:-1]
        self.slab = _pinned(int(step.sum()) + 16)
        self.slab[:] = np.frombuffer(rng.bytes(self.slab.size), np.uint8)
        self.sigs = _pinned(count * z["sig"])
        self.status = torch.zeros(count, dtype=torch.int32, pin_memory=True).numpy()

    def batch(self, op):
        return _eng().batch(op, self.sid, self.count, self.slab.size, self.nkeys)

    def sign_into(self, b):
        b.upload(self.count, self.sks, self.nkeys, self.row, self.slab, self.slab.size, self.offs, self.lens)
        b.run()
        b.download(self.sigs, None, self.status)

    def corrupt(self, rng):
        """one byte of each tenth signature (of every second one in a small batch)"""
        bad = np.nonzero(rng.random(self.count) < (0.1 if self.count >= 32 else 0.5))[0]
        at = bad * self.z["sig"] + rng.integers(0, self.z["sig"], bad.size)
        self.sigs[at] ^= 1


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind, lo, hi = case["kind"], case["min_len"], case["max_len"]
    if kind == "mixed":
        parts = [_Requests(rng, name, count, keys, lo, hi) for name, count, keys in _parts(case)]
        ids, sks, msgs = [], [], []
        for r in parts:
            for i in range(r.count):
                o, k = int(r.offs[i]), int(r.row[i]) * r.z["sk"]
                ids.append(r.sid)
                sks.append(r.sks[k:k + r.z["sk"]].tobytes())
                msgs.append(r.slab[o:o + int(r.lens[i])].tobytes())
        order = rng.permutation(len(ids))
        return {"kind": kind, "signer": c.MixedSigner(_eng()), "ids": [ids[i] for i in order],
                "sks": [sks[i] for i in order], "msgs": [msgs[i] for i in order]}
    if kind == "keygen":
        sid = c.set_id(case["set"])
        z = c.set_sizes(sid)
        rows = _pinned(case["count"] * z["sk"])   # a key row carries the seed in its first 3n bytes
        rows[:] = np.frombuffer(rng.bytes(rows.size), np.uint8)
        return {"kind": kind, "batch": _eng().batch(c.OP_KEYGEN, sid, case["count"], 0, case["count"]), "rows": rows,
                "count": case["count"], "sk": _pinned(case["count"] * z["sk"]), "pk": _pinned(case["count"] * z["pk"])}
    r = _Requests(rng, case["set"], case["count"], case["keys"], lo, hi)
    s = {"kind": kind, "r": r}
    if kind in ("verify", "api_open"):
        b = r.batch(c.OP_SIGN)
        r.sign_into(b)
        b.close()
        if kind == "verify":
            r.corrupt(rng)
            s["batch"] = r.batch(c.OP_VERIFY)
        else:
            s["sm"] = np.concatenate([r.sigs, r.slab[:int(r.lens[0])]])
            s["m"] = np.zeros_like(s["sm"])
    elif kind == "sign":
        s["batch"] = r.batch(c.OP_SIGN)
    else:
        s["rows"] = np.ascontiguousarray(r.sks.reshape(-1, r.z["sk"])[r.row])   # a row per request
    if kind.startswith("api"):
        s["lib"] = _dropin(case["set"])
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "mixed":
        sigs, status, _ = state["signer"].sign(state["ids"], state["sks"], state["msgs"])
        return [np.frombuffer(b"".join(sigs), np.uint8), status]
    if kind == "keygen":
        b = state["batch"]
        b.upload(state["count"], state["rows"], state["count"])
        b.run()
        b.download(state["sk"], state["pk"])
        return [state["sk"], state["pk"]]
    r = state["r"]
    if kind == "sign":
        r.sign_into(state["batch"])
        return [r.sigs, r.status]
    if kind == "verify":
        b = state["batch"]
        b.upload(r.count, r.pks, r.nkeys, r.row, r.slab, r.slab.size, r.offs, r.lens, r.sigs)
        b.run()
        b.download(None, None, r.status)
        return [r.status]
    if kind == "oneshot_sign":
        eng = _eng()
        rc = eng.L.cuspx_sign_batch(eng.h, r.sid, r.count, _at(state["rows"]), _at(r.slab), _at(r.offs), _at(r.lens),
                                    None, _at(r.sigs), _at(r.status))
        return [rc, r.sigs, r.status]
    if kind == "api_sign":
        n = ctypes.c_size_t()
        rc = state["lib"].crypto_sign_signature(_at(r.sigs), ctypes.byref(n), _at(r.slab), int(r.lens[0]),
                                                _at(state["rows"]))
        return [rc, n.value, r.sigs]
    n, m, sm = ctypes.c_ulonglong(), state["m"], state["sm"]
    rc = state["lib"].crypto_sign_open(_at(m), ctypes.byref(n), _at(sm), sm.size, _at(r.pks))
    return [rc, n.value, m[:n.value]]


def exact(case, seed):
    """Outputs are bytes and verdicts: none has a value in 64-bit floating point."""
    return None
