"""The engine's host code (batches, graphs, one-shot calls) over a CUDA runtime
in host memory (fake_cuda/): which inputs a launch reads, and whether they are
live memory of its device.  Needs nvcc, no GPU.
"""
import ctypes
import os
import shutil
import subprocess
import threading

import numpy as np
import pytest

from conftest import ROOT

FAKE = os.path.join(ROOT, "tests", "fake_cuda")


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    """cuspx_gb300 over the built engine objects, the fake runtime and fake
    hash families in place of the CUDA ones"""
    import cuspx_gb300 as c
    from cuspx_gb300 import build
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("needs nvcc")
    build.build()
    out = str(tmp_path_factory.mktemp("fake"))
    inc = "-I" + os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    fam, rt, so = (os.path.join(out, x) for x in ("family.o", "cudart.o", "libfake.so"))
    subprocess.run([nvcc] + build.NVCC_FLAGS + ["-c", os.path.join(FAKE, "family.cu"), "-o", fam], check=True)
    subprocess.run(["g++"] + build.CXX_FLAGS + [inc, "-c", os.path.join(FAKE, "cudart.cpp"), "-o", rt], check=True)
    objs = [os.path.join(build.BUILD, x + ".o") for x in ("engine", "serve", "noalloc", "calib", "drbg")]
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-Wl,-z,defs", "-o", so, fam, rt] + objs + ["-lpthread"],
                   check=True)
    saved = c._lib, c.LIB_PATH
    c._lib, c.LIB_PATH = None, so
    c.lib()
    yield c
    c._lib, c.LIB_PATH = saved


@pytest.fixture
def engine(fake, monkeypatch, tmp_path):
    monkeypatch.setenv("CUSPX_TUNE_CACHE", str(tmp_path / "none.tsv"))
    fake.lib().cudaSetDevice(0)
    eng = fake.Engine(0)
    yield eng
    eng.close()
    assert fake.lib().fake_faults() == 0


SETS = ("sha256-128f-simple", "shake256-128s-robust")


def _rows(z, count, seed):
    return np.random.default_rng(seed).integers(0, 256, (count, z), dtype=np.uint8)


def _upload(c, b, count, sks, nkeys=None, idx=None, opt=None):
    slab, offs, lens = c.pack_messages([b"m%d" % i for i in range(count)])
    b.upload(count, sks, nkeys or count, idx, slab, len(slab), offs, lens, opt)


def _signed(c, b, count):
    z = c.set_sizes(b.sid)
    out = np.zeros(count * z["sig"], np.uint8)
    b.download(out)
    rows = out.reshape(count, z["sig"])
    return rows[:, :z["n"]], rows[:, z["n"]:2 * z["n"]]


def test_group_run_reads_this_uploads_inputs(engine, fake):
    """sign batches of the same sizes with and without randomisers and key
    indices, in every order and each twice: the present upload's are used"""
    c, count = fake, 5
    sid = [engine.set_id(s) for s in SETS]
    z = [c.set_sizes(s) for s in sid]
    bs = [engine.batch(c.OP_SIGN, s, 8, 4096, 8) for s in sid]
    sks = [_rows(z[k]["sk"], count, k) for k in range(2)]
    idx = np.array([4, 0, 3, 3, 1], np.uint32)
    steps = [(None, None), (7, None), (None, None), (8, None), (8, idx), (None, idx), (None, None), (9, idx)]
    for seed, ix in [s for s in steps for _ in range(2)]:
        opt = [None if seed is None else _rows(z[k]["n"], count, seed + k) for k in range(2)]
        for k in range(2):
            _upload(c, bs[k], count, sks[k], count, ix, opt[k])
        c.group_run(engine, bs)
        for k in range(2):
            n = z[k]["n"]
            r, prf = _signed(c, bs[k], count)
            assert np.array_equal(r, opt[k] if seed else np.full((count, n), 0xad, np.uint8))
            assert np.array_equal(prf, (sks[k] if ix is None else sks[k][ix])[:, n:2 * n])
    for b in bs:
        b.close()


def test_group_run_reads_bound_keys_and_lengths(engine, fake):
    """verify batches with and without signature lengths, and a key table
    bound, changed and unbound between runs of the same sizes"""
    c, count = fake, 3
    L = c.lib()
    sid = engine.set_id(SETS[0])
    z = c.set_sizes(sid)
    b = engine.batch(c.OP_VERIFY, sid, 4, 4096, 4)
    pks = _rows(z["pk"], count, 1)
    sigs = _rows(z["sig"], count, 2)
    sigs[:, z["n"]:2 * z["n"]] = pks[:, :z["n"]]
    slab, offs, lens = c.pack_messages([b"x"] * count)
    tables = []
    for t in (pks, _rows(z["pk"], count, 3)):
        p = ctypes.c_void_p()
        assert L.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(t.size)) == 0
        assert L.cudaMemcpy(p, t.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(t.size), 1) == 0
        tables.append(p)
    good, short = np.full(count, z["sig"], np.uint64), np.array([z["sig"], z["sig"] - 1, z["sig"]], np.uint64)
    for table, siglens, want in [(None, None, [0, 0, 0]), (None, short, [0, -1, 0]), (None, good, [0, 0, 0]),
                                 (0, good, [0, 0, 0]), (1, good, [-1, -1, -1]), (0, short, [0, -1, 0]),
                                 (None, good, [0, 0, 0])]:
        L.cuspx_batch_bind_keys(ctypes.c_void_p(b.h.value), tables[table] if table is not None else None,
                                ctypes.c_size_t(count))
        keys = pks if table is None else None
        b.upload(count, keys, count if table is None else 0, None, slab, len(slab), offs, lens, sigs, siglens)
        c.group_run(engine, [b])
        st = np.zeros(count, np.int32)
        b.download(None, None, st)
        assert list(st) == want
    b.close()


def test_group_graphs_go_with_their_batches(engine, fake):
    """a graph launches into its batches' memory: none may be left, and none
    found for a new batch at the old one's address, once a batch is gone"""
    c, live = fake, fake.lib().fake_live_execs
    sid = [engine.set_id(s) for s in SETS]
    bs = [engine.batch(c.OP_SIGN, s, 4, 4096, 4) for s in sid]
    for count in (2, 3, 4):
        for k in range(2):
            _upload(c, bs[k], count, _rows(c.set_sizes(sid[k])["sk"], count, k))
        c.group_run(engine, bs)
        c.group_run(engine, bs[1:])
    assert live() == 6
    bs[0].close()
    assert live() == 3
    c.group_run(engine, bs[1:])
    assert live() == 3
    bs[1].close()
    assert live() == 0


def test_mixed_signer_grows_and_shrinks(engine, fake):
    """batches that are replaced by larger ones, then used at the old sizes"""
    c = fake
    ms = c.MixedSigner(engine)
    sid = [engine.set_id(s) for s in SETS]
    for step, count in enumerate((10, 20, 10, 10, 20, 33, 10, 20)):
        sks, msgs = [], []
        for k in range(2):
            sks += [r.tobytes() for r in _rows(c.set_sizes(sid[k])["sk"], count, 10 * step + k)]
            msgs += [b"%d" % i for i in range(count)]
        ids = [sid[0]] * count + [sid[1]] * count
        sigs, status, _ = ms.sign(ids, sks, msgs)
        for s, sk, sig, st in zip(ids, sks, sigs, status):
            n = c.set_sizes(s)["n"]
            assert st == 0 and sig[:n] == b"\xad" * n and sig[n:2 * n] == sk[n:2 * n]
    ms.close()
    assert c.lib().fake_live_execs() == 0


def test_batches_outlive_their_engine(fake):
    c = fake
    eng = c.Engine(0)
    b = eng.batch(c.OP_SIGN, eng.set_id(SETS[0]), 4, 4096, 4)
    _upload(c, b, 2, _rows(c.set_sizes(b.sid)["sk"], 2, 1))
    c.group_run(eng, [b])
    eng.close()
    b.close()
    assert c.lib().fake_live_execs() == 0 and c.lib().fake_faults() == 0


def test_oneshot_memory_is_on_the_engines_device(fake):
    """calls from threads whose current device is another one (each new
    thread's is device 0), whose packed input grows with and without a new batch"""
    c = fake
    c.lib().cudaSetDevice(0)
    eng = c.Engine(1)
    sid = eng.set_id(SETS[0])
    z = c.set_sizes(sid)
    res = []

    def call(count, size):
        msgs = [b"m" * size] * count
        c.lib().cudaSetDevice(0)
        sks = [r.tobytes() for r in _rows(z["sk"], count, count)]
        opt = [r.tobytes() for r in _rows(z["n"], count, 99)]
        sigs, st = eng.sign_batch(sid, sks, msgs, opt)
        ok = list(st) == [0] * count and [s[:z["n"]] for s in sigs] == opt
        got = eng.verify_batch(sid, [s[z["n"]:2 * z["n"]] + bytes(z["n"]) for s in sigs], msgs, sigs)
        res.append(ok and list(got) == [0] * count)

    try:
        for count, size in ((5, 40), (3, 0), (5, 800), (9, 40), (70, 100), (2, 3000), (70, 112)):
            t = threading.Thread(target=call, args=(count, size))
            t.start()
            t.join()
        assert res == [True] * 7 and c.lib().fake_faults() == 0
    finally:
        eng.close()
        c.lib().cudaSetDevice(0)


@pytest.mark.parametrize("setname", ["sha256-128f-simple", "sha256-256s-robust", "shake256-128f-simple",
                                     "shake256-256f-robust"])
def test_served_verify_request_counts_its_device_bytes(engine, fake, setname):
    """what a verify request is admitted with is what an item more takes in a
    batch, within the 64 bytes set aside for its offsets, indices and status"""
    c = fake
    live = c.lib().fake_live_bytes
    live.restype = ctypes.c_size_t
    sid = engine.set_id(setname)
    z = c.set_sizes(sid)

    def batch_bytes(items):
        before = live()
        b = engine.batch(c.OP_VERIFY, sid, items, 4096, 1)
        got = live() - before
        b.close()
        return got

    item = batch_bytes(101) - batch_bytes(100)
    srv = c.Server(engine, max_batch=16, max_inflight=1)
    try:
        kid = srv.add_pubkeys(sid, [bytes(z["pk"])])[0]
        assert srv.wait(srv.submit(c.OP_VERIFY, sid, kid, b"x" * 16, bytes(z["sig"])), 10_000_000)[1] == 0
        counted = srv.stats()["bytes_peak"] - 16
    finally:
        srv.close()
    assert item <= counted <= item + 64
