"""Sign batches through each way their work is laid out: chain lanes with the
streaming T_len (batches above chain_mode_max) in one or more chunks of trees,
trees that items share computed once, and FORS trees spread over more lanes
than a warp.  All of them are byte-identical to the small-batch path, which
test_gpu_parity.py pins to the oracle, and to the oracle itself.
"""
import random

import pytest

pytestmark = pytest.mark.gpu

HASHES = ("sha256", "shake256")
SETS = ["%s-%s-%s" % (h, s, m) for h in HASHES for s in ("128s", "128f", "192s", "192f", "256s", "256f")
        for m in ("simple", "robust")]


@pytest.fixture(scope="module")
def engine():
    import cuspx_gb300
    eng = cuspx_gb300.Engine(0)
    yield eng
    eng.close()


def _oracle(name):
    import spx_oracle
    return spx_oracle.Oracle(name)


def _requests(engine, sid, count, keys, seed):
    import cuspx_gb300 as c
    rng = random.Random(seed)
    n = c.set_sizes(sid)["seed"]
    pks, sks = engine.keypair_batch(sid, [rng.randbytes(n) for _ in range(keys)])
    row = [i % keys if keys == count else rng.randrange(keys) for i in range(count)]
    msgs = [rng.randbytes(rng.randrange(0, 150)) for _ in range(count)]
    return [pks[r] for r in row], [sks[r] for r in row], msgs


def _in_pieces(engine, sid, sks, msgs, piece=60):
    """signatures through batches small enough for the latency mapping"""
    out = []
    for i in range(0, len(msgs), piece):
        sigs, st = engine.sign_batch(sid, sks[i:i + piece], msgs[i:i + piece])
        assert not any(st)
        out += sigs
    return out


@pytest.mark.parametrize("setname", SETS)
def test_streaming_leaves_match_latency_path(engine, setname):
    sid = engine.set_id(setname)
    pks, sks, msgs = _requests(engine, sid, 65, 65, 5)
    sigs, st = engine.sign_batch(sid, sks, msgs)
    assert not any(st)
    assert sigs == _in_pieces(engine, sid, sks, msgs)
    assert sigs[64] == _oracle(setname).sign(msgs[64], sks[64])


@pytest.mark.parametrize("setname,count", [("sha256-128s-simple", 140), ("shake256-192s-simple", 70)])
def test_leaf_chunks(engine, setname, count):
    """more trees than the chain-end scratch holds (256 MiB: 935 trees of
    128s, 428 of 192s), the last chunk part full"""
    sid = engine.set_id(setname)
    pks, sks, msgs = _requests(engine, sid, count, count, 6)
    sigs, st = engine.sign_batch(sid, sks, msgs)
    assert not any(st)
    assert sigs == _in_pieces(engine, sid, sks, msgs, 30)


@pytest.mark.parametrize("setname,count", [("sha256-128f-simple", 65), ("sha256-128f-simple", 1000),
                                           ("sha256-192f-robust", 130), ("shake256-256f-simple", 130),
                                           ("sha256-128s-simple", 100)])
@pytest.mark.parametrize("keys", [1, 3, 0])
def test_shared_trees(engine, setname, count, keys):
    """one key, a few, and a key per item; some messages twice, so that items
    share even their lowest leaf"""
    sid = engine.set_id(setname)
    pks, sks, msgs = _requests(engine, sid, count, keys or count, 7)
    for i in range(5):
        sks[count - 1 - i], pks[count - 1 - i], msgs[count - 1 - i] = sks[i], pks[i], msgs[i]
    sigs, st = engine.sign_batch(sid, sks, msgs)
    assert not any(st)
    assert sigs == _in_pieces(engine, sid, sks, msgs)
    assert sigs[count // 2] == _oracle(setname).sign(msgs[count // 2], sks[count // 2])
    assert not any(engine.verify_batch(sid, pks, msgs, sigs))


def test_shared_trees_by_key_index_and_wrong_root(engine):
    """rows of a key table picked by index; a row whose ROOT is not its own is
    reported for its items alone, whose seeds they share with a good row"""
    import numpy as np
    import cuspx_gb300 as c
    sid = engine.set_id("sha256-128f-simple")
    z = c.set_sizes(sid)
    pks, sks, msgs = _requests(engine, sid, 200, 1, 8)
    bad = bytearray(sks[0])
    bad[-1] ^= 1
    table = np.frombuffer(sks[0] + bytes(bad), np.uint8)
    idx = np.array([i % 7 == 3 for i in range(200)], np.uint32)
    slab, offs, lens = c.pack_messages(msgs)
    b = engine.batch(c.OP_SIGN, sid, 200, len(slab), 2)
    out, st = np.zeros(200 * z["sig"], np.uint8), np.zeros(200, np.int32)
    for _ in range(3):   # direct launch, capture, replay
        b.upload(200, table, 2, idx, slab, len(slab), offs, lens)
        b.run()
        b.download(out, None, st)
        assert list(st) == [-2 if x else 0 for x in idx]
        want = _in_pieces(engine, sid, [sks[0]] * 60, msgs[:60])
        for i in range(60):
            if not idx[i]:
                assert out[i * z["sig"]:(i + 1) * z["sig"]].tobytes() == want[i]
    b.close()


@pytest.mark.parametrize("setname,count", [("sha256-192f-simple", 1), ("sha256-192f-robust", 20),
                                           ("shake256-256f-simple", 1), ("sha256-128s-robust", 1),
                                           ("shake256-128s-simple", 2), ("sha256-256s-simple", 30),
                                           ("sha256-192s-simple", 150), ("sha256-192s-simple", 300)])
def test_fors_lane_spread(engine, setname, count):
    """2^8 (a whole tree of 192f), 2^9, 2^10 and down to 2^6 lanes per tree"""
    sid = engine.set_id(setname)
    pks, sks, msgs = _requests(engine, sid, count, count, 9)
    sigs, st = engine.sign_batch(sid, sks, msgs)
    assert not any(st)
    assert sigs[count - 1] == _oracle(setname).sign(msgs[count - 1], sks[count - 1])
    assert not any(engine.verify_batch(sid, pks, msgs, sigs))


@pytest.mark.parametrize("count", [17, 18, 40])
def test_chain_block_cap(engine, count):
    """256f-robust below, at and above 16 chain blocks an SM (152 of them),
    where the chain blocks' number per SM is capped"""
    sid = engine.set_id("sha256-256f-robust")
    pks, sks, msgs = _requests(engine, sid, count, count, 10)
    sigs, st = engine.sign_batch(sid, sks, msgs)
    assert not any(st)
    assert sigs == _in_pieces(engine, sid, sks, msgs, 9)
    assert sigs[count - 1] == _oracle("sha256-256f-robust").sign(msgs[count - 1], sks[count - 1])


@pytest.mark.parametrize("setname,count", [("sha256-128f-simple", 1), ("sha256-192f-robust", 127),
                                           ("sha256-256f-simple", 129), ("shake256-128f-simple", 129)])
def test_keygen_midstates(engine, setname, count):
    """a key, the last of a block of keys and the first of the next: as the
    oracle's, and as each key by itself"""
    import cuspx_gb300 as c
    rng = random.Random(11)
    sid = engine.set_id(setname)
    seeds = [rng.randbytes(c.set_sizes(sid)["seed"]) for _ in range(count)]
    pks, sks = engine.keypair_batch(sid, seeds)
    for i in sorted({0, count // 2, count - 1}):
        assert (pks[i], sks[i]) == _oracle(setname).seed_keypair(seeds[i])
        assert ([pks[i]], [sks[i]]) == engine.keypair_batch(sid, [seeds[i]])


@pytest.mark.parametrize("setname", ["sha256-128f-simple", "sha256-192f-robust", "sha256-256f-simple",
                                     "shake256-128f-simple", "shake256-192f-simple", "shake256-256f-robust"])
@pytest.mark.parametrize("edge", [256, 1024, 1536])
def test_message_kernels_around_threshold(engine, setname, edge):
    """messages about the lengths from which the long-message kernels take
    them, alone in a batch and beside short and longer ones"""
    rng = random.Random(edge)
    sid, o = engine.set_id(setname), _oracle(setname)
    pk, sk = o.seed_keypair(rng.randbytes(3 * o.p.n))
    msgs = [rng.randbytes(x) for x in (edge - 1, edge, edge + 1, 0, 3 * edge, 77)]
    for some in ([msgs[0]], [msgs[1]], msgs):
        sigs, st = engine.sign_batch(sid, [sk] * len(some), some)
        assert not any(st)
        assert sigs == [o.sign(m, sk) for m in some]
        wrong = [m[:-1] + bytes([m[-1] ^ 1]) for m in some if m]
        keep = [s for m, s in zip(some, sigs) if m]
        got = engine.verify_batch(sid, [pk] * (len(some) + len(wrong)), some + wrong, sigs + keep)
        assert list(got) == [0] * len(some) + [-1] * len(wrong)


@pytest.mark.parametrize("setname", ["sha256-128f-simple", "sha256-192f-robust", "sha256-256f-simple"])
def test_message_warps(engine, setname):
    """a warp per message: the padding about a block's end, one and two rounds
    of 32 blocks, and lengths about that from which the batch's long messages
    are hashed apart, alone and with a wrong-length signature beside them"""
    rng = random.Random(12)
    sid, o = engine.set_id(setname), _oracle(setname)
    n = o.p.n
    pk, sk = o.seed_keypair(rng.randbytes(3 * n))
    lens = [0, 1, 3, 4]
    for pre in (n, 3 * n):
        for blocks in (2, 32, 33):
            lens += [64 * blocks - 9 - pre + x for x in (-1, 0, 1)]
    for some in (lens + [4095], lens + [1023, 1024, 4095, 4096, 4097, 9000], [4096]):
        msgs = [rng.randbytes(x) for x in some]
        sigs, st = engine.sign_batch(sid, [sk] * len(msgs), msgs)
        assert not any(st)
        assert sigs == [o.sign(m, sk) for m in msgs]
        vm, vs = msgs + msgs[-1:] * 2, sigs + [sigs[-1], bytes([sigs[-1][0] ^ 1]) + sigs[-1][1:]]
        got = engine.verify_batch(sid, [pk] * len(vm), vm, vs,
                                  siglens=[len(x) for x in sigs] + [len(sigs[0]) - 1, len(sigs[0])])
        assert list(got) == [0] * len(msgs) + [-1, -1]


@pytest.mark.parametrize("count", [608, 609])
def test_message_warps_batch_limit(engine, count):
    """the last batch with a warp a message and the first with a thread each"""
    sid = engine.set_id("sha256-128f-simple")
    pks, sks, msgs = _requests(engine, sid, count, 5, 13)
    sigs, st = engine.sign_batch(sid, sks, msgs)
    assert not any(st)
    assert sigs == _in_pieces(engine, sid, sks, msgs)
    assert sigs[-1] == _oracle("sha256-128f-simple").sign(msgs[-1], sks[-1])
    assert not any(engine.verify_batch(sid, pks, msgs, sigs))


@pytest.mark.parametrize("setname,count", [("sha256-128f-simple", 4096), ("shake256-192f-robust", 300)])
@pytest.mark.parametrize("part", [0, 2])
def test_shared_trees_of_keys_with_alike_seeds(engine, setname, count, part):
    """a key per item whose seeds differ in the last two bytes of SK_SEED or of
    PUB_SEED alone: the search for trees that items share takes no longer than
    with random seeds (five times as long at most, where a walk over all the
    batch's keys takes ten to a hundred times) and the signatures are the keys' own"""
    import numpy as np
    import cuspx_gb300 as c
    rng = random.Random(14)
    sid = engine.set_id(setname)
    z = c.set_sizes(sid)
    n = z["n"]
    base = rng.randbytes(3 * n)
    alike = [base[:(part + 1) * n - 2] + i.to_bytes(2, "big") + base[(part + 1) * n:] for i in range(count)]
    apart = [rng.randbytes(3 * n) for _ in range(count)]
    msgs = [rng.randbytes(20) for _ in range(count)]
    slab, offs, lens = c.pack_messages(msgs)
    b = engine.batch(c.OP_SIGN, sid, count, len(slab), count)
    b.profile()
    took = []
    for seeds in (apart, alike):
        pks, sks = engine.keypair_batch(sid, seeds)
        best = None
        for _ in range(4):
            b.upload(count, b"".join(sks), count, None, slab, len(slab), offs, lens)
            b.profile()
            b.run()
            ms = dict((k, t) for k, t, _ in b.kernel_ms())["k_share"]
            best = ms if best is None else min(best, ms)
        took.append(best)
    out, st = np.zeros(count * z["sig"], np.uint8), np.zeros(count, np.int32)
    b.download(out, None, st)
    b.close()
    assert not st.any()
    sigs = [out[i * z["sig"]:(i + 1) * z["sig"]].tobytes() for i in range(count)]
    assert sigs[:60] == _in_pieces(engine, sid, sks[:60], msgs[:60])
    assert sigs[-1] == _oracle(setname).sign(msgs[-1], sks[-1])
    assert took[1] < 5 * took[0], took


@pytest.mark.parametrize("count,kernel", [(256, "k_leaves"), (257, "k_leaf_chains")])
def test_chain_mode_max_decides_up_to_256_items(engine, count, kernel):
    """chain_mode_max 0, as tuning files may hold it for any batch size: a lane
    per leaf where the knob decides, chain lanes and shared trees above"""
    import numpy as np
    import cuspx_gb300 as c
    sid = engine.set_id("sha256-128f-simple")
    z = c.set_sizes(sid)
    pks, sks, msgs = _requests(engine, sid, count, 1, 15)
    slab, offs, lens = c.pack_messages(msgs)
    saved = engine.get_tuning(sid)
    b = engine.batch(c.OP_SIGN, sid, count, len(slab), 1)
    try:
        engine.set_tuning(sid, chain_mode_max=0)
        b.profile()
        b.upload(count, sks[0], 1, np.zeros(count, np.uint32), slab, len(slab), offs, lens)
        b.run()
        names = [k for k, _, _ in b.kernel_ms()]
        out = np.zeros(count * z["sig"], np.uint8)
        b.download(out)
    finally:
        b.close()
        engine.set_tuning(sid, **saved)
    assert kernel in names and ("k_share" in names) == (count > 256)
    assert [out[i * z["sig"]:(i + 1) * z["sig"]].tobytes() for i in range(count)] == _in_pieces(engine, sid, sks, msgs)


@pytest.mark.parametrize("setname", ["sha256-128f-simple", "shake256-192f-robust"])
def test_oneshot_inputs_packed_and_apart(setname):
    """one engine's calls whose inputs go up in one copy, in a growing one and
    buffer by buffer (above 1 MiB), there and back, with and without
    randomisers; each shape three times (launched, captured, replayed), a key
    row with a wrong root and a signature of a wrong length among them"""
    import cuspx_gb300
    rng = random.Random(16)
    o = _oracle(setname)
    eng = cuspx_gb300.Engine(0)
    try:
        sid = eng.set_id(setname)
        pk, sk = o.seed_keypair(rng.randbytes(o.p.seed_bytes))
        bad = sk[:-1] + bytes([sk[-1] ^ 1])
        for count, size, opt in ((3, 40, False), (3, 900, True), (2, 40, True), (3, 400_000, True), (3, 40, True),
                                 (3, 40, False), (3, 400_000, False), (2, 900, False)):
            msgs = [rng.randbytes(size + i) for i in range(count)]
            rand = [rng.randbytes(o.p.n) for _ in range(count)] if opt else None
            want = [o.sign(m, sk, rand[i] if opt else None) for i, m in enumerate(msgs[:-1])]
            for _ in range(3):
                sigs, st = eng.sign_batch(sid, [sk] * (count - 1) + [bad], msgs, rand)
                assert list(st) == [0] * (count - 1) + [-2] and sigs[:-1] == want
                got = eng.verify_batch(sid, [pk] * (2 * count - 2), msgs[:-1] * 2, want * 2,
                                       siglens=[len(x) for x in want] + [len(x) - 1 for x in want])
                assert list(got) == [0] * (count - 1) + [-1] * (count - 1)
    finally:
        eng.close()


@pytest.mark.parametrize("count", [256, 257])
def test_chain_mode_max_above_256_items(engine, count):
    """a chain_mode_max above the sizes that it decides about: larger batches
    still share trees"""
    import numpy as np
    import cuspx_gb300 as c
    sid = engine.set_id("sha256-128f-simple")
    z = c.set_sizes(sid)
    pks, sks, msgs = _requests(engine, sid, count, 1, 16)
    slab, offs, lens = c.pack_messages(msgs)
    saved = engine.get_tuning(sid)
    b = engine.batch(c.OP_SIGN, sid, count, len(slab), 1)
    try:
        engine.set_tuning(sid, chain_mode_max=4096)
        b.profile()
        b.upload(count, sks[0], 1, np.zeros(count, np.uint32), slab, len(slab), offs, lens)
        b.run()
        names = [k for k, _, _ in b.kernel_ms()]
        out = np.zeros(count * z["sig"], np.uint8)
        b.download(out)
    finally:
        b.close()
        engine.set_tuning(sid, **saved)
    assert ("k_share" in names) == (count > 256)
    assert [out[i * z["sig"]:(i + 1) * z["sig"]].tobytes() for i in range(count)] == _in_pieces(engine, sid, sks, msgs)
