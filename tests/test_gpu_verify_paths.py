"""Verify batches through the sorted layers, the fused blocks and the speculative
walk, by groups of lanes, a warp and a thread per item, at the sizes where a block, a warp or
an item group is part full: good signatures pass, a signature with one byte
changed anywhere is rejected, and its neighbours are not disturbed.
"""
import random

import pytest

pytestmark = pytest.mark.gpu

SETS = ["%s-%s-%s" % (h, s, m) for h in ("sha256", "shake256") for s in ("128s", "128f", "192s", "192f", "256s", "256f")
        for m in ("simple", "robust")]


@pytest.fixture(scope="module")
def engine():
    import cuspx_gb300
    eng = cuspx_gb300.Engine(0)
    yield eng
    eng.close()


@pytest.fixture(scope="module")
def pool(engine):
    """64 signed messages of a set, two of them checked against the oracle (f sets; the s
    sets' signatures are in test_gpu_sign_paths.py)"""
    import spx_oracle
    made = {}

    def get(setname):
        if setname not in made:
            sid = engine.set_id(setname)
            rng = random.Random(3)
            o = spx_oracle.Oracle(setname)
            pks, sks = engine.keypair_batch(sid, [rng.randbytes(o.p.seed_bytes) for _ in range(3)])
            msgs = [rng.randbytes(rng.randrange(0, 300)) for _ in range(64)]
            sigs, st = engine.sign_batch(sid, [sks[i % 3] for i in range(64)], msgs)
            assert not any(st)
            for i in (0, 63) if setname.split("-")[1].endswith("f") else ():
                assert sigs[i] == o.sign(msgs[i], sks[i % 3])
            made[setname] = [(pks[i % 3], msgs[i], sigs[i]) for i in range(64)]
        return made[setname]

    return get


def _check(engine, sid, items, count, seed):
    rng = random.Random(seed)
    pk, msg, sig, want = [], [], [], []
    for i in range(count):
        p, m, s = items[i % len(items)]
        bad = rng.random() < 0.4
        if bad:
            s = bytearray(s)
            s[rng.randrange(len(s))] ^= 1 << rng.randrange(8)
        pk.append(p)
        msg.append(m)
        sig.append(bytes(s))
        want.append(-1 if bad else 0)
    assert list(engine.verify_batch(sid, pk, msg, sig)) == want


@pytest.mark.parametrize("setname", SETS)
def test_sorted_layers(engine, pool, setname):
    sid = engine.set_id(setname)
    saved = engine.get_tuning(sid)
    try:
        for count, groups in ((1, 1), (7, 1), (9, 2), (65, 4), (301, 1), (1300, 2)):
            engine.set_tuning(sid, verify_spec_max=0, verify_item_max=0, verify_mode=3, verify_groups=groups)
            _check(engine, sid, pool(setname), count, count)
    finally:
        engine.set_tuning(sid, **saved)


@pytest.mark.parametrize("setname,count", [("sha256-128f-simple", 2049), ("sha256-192f-simple", 2500),
                                           ("sha256-256s-simple", 2049), ("sha256-128s-robust", 4097),
                                           ("sha256-192s-robust", 4100), ("sha256-256s-robust", 4097)])
def test_sorted_layers_thread_per_item(engine, pool, setname, count):
    """the first sizes past the lanes-per-item layer kernel"""
    _check(engine, engine.set_id(setname), pool(setname), count, count)


@pytest.mark.parametrize("setname", SETS)
def test_default_mapping_edges(engine, pool, setname):
    """the sizes at which the default mapping changes (of 152 SMs)"""
    for count in (32, 33, 64, 65, 129, 305, 609, 1023):
        _check(engine, engine.set_id(setname), pool(setname), count, count)


@pytest.mark.parametrize("setname", SETS)
def test_speculative_walk(engine, pool, setname):
    sid = engine.set_id(setname)
    saved = engine.get_tuning(sid)
    try:
        engine.set_tuning(sid, verify_spec_max=64)
        for count in (1, 2, 33, 64):
            _check(engine, sid, pool(setname), count, count)
    finally:
        engine.set_tuning(sid, **saved)


@pytest.mark.parametrize("setname,counts", [("sha256-128f-simple", (1499, 1500, 8192, 8193)),
                                            ("sha256-192f-simple", (1500, 3001)),
                                            ("sha256-256f-simple", (3072, 3073)),
                                            ("sha256-128f-robust", (4097,)), ("sha256-192s-robust", (4097,)),
                                            ("sha256-256s-robust", (2999, 3000)), ("sha256-256f-robust", (3001,))])
def test_lanes_in_item_groups(engine, pool, setname, counts):
    """the sizes between which several item groups run with lanes in the layer kernel"""
    for count in counts:
        _check(engine, engine.set_id(setname), pool(setname), count, count)


@pytest.mark.parametrize("setname,count", [("sha256-128f-simple", 2049), ("sha256-192s-simple", 2049),
                                           ("sha256-256f-simple", 2049), ("sha256-128s-robust", 4097),
                                           ("sha256-192s-robust", 4097), ("sha256-256f-robust", 4097),
                                           ("shake256-128f-simple", 2049), ("shake256-192s-simple", 2049),
                                           ("shake256-256s-simple", 2049), ("shake256-128s-robust", 8193),
                                           ("shake256-192s-robust", 8193), ("shake256-256s-robust", 8193)])
def test_layer_thread_per_item(engine, pool, setname, count):
    """one item group past the sizes of the lanes and warps per item: a thread
    per item in the layer kernel, its last block part full"""
    sid = engine.set_id(setname)
    saved = engine.get_tuning(sid)
    try:
        engine.set_tuning(sid, verify_groups=1)
        _check(engine, sid, pool(setname), count, count)
    finally:
        engine.set_tuning(sid, **saved)


@pytest.mark.parametrize("setname", ["sha256-128f-simple", "sha256-256s-robust", "shake256-192f-robust"])
def test_sorted_min_below_spec_max(engine, pool, setname):
    """verify_sorted_min decides whatever verify_mode says, also for batches that
    the speculative chains would take, and only from its size on"""
    import numpy as np
    import cuspx_gb300 as c
    sid = engine.set_id(setname)
    z = c.set_sizes(sid)
    saved = engine.get_tuning(sid)
    ran = {}
    try:
        engine.set_tuning(sid, verify_sorted_min=8, verify_spec_max=16, verify_item_max=0)
        for count in (7, 8, 16):
            items = pool(setname)[:count]
            slab, offs, lens = c.pack_messages([m for _, m, _ in items])
            sigs = np.frombuffer(b"".join(s for _, _, s in items), np.uint8).reshape(count, z["sig"]).copy()
            sigs[1, 3] ^= 1
            b = engine.batch(c.OP_VERIFY, sid, count, len(slab), count)
            got = np.zeros(count, np.int32)
            try:
                b.profile()
                b.upload(count, b"".join(p for p, _, _ in items), count, None, slab, len(slab), offs, lens,
                         sigs.reshape(-1))
                b.run()
                ran[count] = {k for k, _, _ in b.kernel_ms()}
                b.download(None, None, got)
            finally:
                b.close()
            assert [int(x) for x in got] == [-1 if i == 1 else 0 for i in range(count)]
    finally:
        engine.set_tuning(sid, **saved)
    assert "k_vspec_walk" in ran[7]
    assert all("k_vsort_layer" in ran[n] and "k_vspec_walk" not in ran[n] for n in (8, 16))


@pytest.mark.parametrize("setname", ["shake256-128f-simple", "shake256-192f-robust", "shake256-256s-simple"])
@pytest.mark.parametrize("slots,block", [(1, 32), (2, 128)])
def test_persistent_kernel_refills_slots(engine, pool, setname, slots, block):
    """more items than all resident warps hold at once (152 SMs x 32 blocks of
    a warp, or x 16 warps of two items), a wrong-length signature in five: warps
    take new items as theirs finish"""
    import numpy as np
    import cuspx_gb300 as c
    count, items = 6000, pool(setname)
    sid = engine.set_id(setname)
    z = c.set_sizes(sid)
    slab, offs, lens = c.pack_messages([items[i % 64][1] for i in range(count)])
    sigs = np.frombuffer(b"".join(s for _, _, s in items), np.uint8).reshape(64, -1)[np.arange(count) % 64].copy()
    rng = np.random.default_rng(count + slots)
    bad = rng.random(count) < 0.4
    sigs[bad, rng.integers(0, z["sig"], count)[bad]] ^= 1
    short = rng.random(count) < 0.2
    siglen = np.where(short, z["sig"] - 1, z["sig"]).astype(np.uint64)
    saved = engine.get_tuning(sid)
    b = engine.batch(c.OP_VERIFY, sid, count, len(slab), count)
    got = np.zeros(count, np.int32)
    try:
        engine.set_tuning(sid, verify_mode=2, verify_sorted_min=0, verify_spec_max=0, verify_item_max=0,
                          verify_slots=slots, verify_block=block)
        b.profile()
        b.upload(count, b"".join(items[i % 64][0] for i in range(count)), count, None, slab, len(slab), offs, lens,
                 sigs.reshape(-1), siglen)
        b.run()
        names = [k for k, _, _ in b.kernel_ms()]
        b.download(None, None, got)
    finally:
        b.close()
        engine.set_tuning(sid, **saved)
    assert "k_verify_hyper" in names
    assert np.array_equal(got, np.where(bad | short, -1, 0))
