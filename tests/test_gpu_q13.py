"""Q13 (customer distribution) on the GPU against the CPU oracle, bit-exact: SF-1 sizes,
other word pairs, hand-written comments at the pattern's edge cases (adjacent words, words
in the wrong order, a word cut by the 80-byte slot end, one-letter words, empty comments),
customers without orders, orders of unknown customers, and the count and word limits."""
import ctypes as C

import numpy as np
import pytest

from gpudbmetalbenchmark_b200 import capi

pytestmark = pytest.mark.gpu


def run(engine, cu, od, *words, cu_key_max=None):
    tc = engine.upload("customer", cu, key_max=None if cu_key_max is None else {"key": cu_key_max})
    to = engine.upload("orders", od)
    try:
        return engine.q13(tc, to, *words)
    finally:
        engine.free(tc)
        engine.free(to)


@pytest.mark.parametrize("n_cu,n_or,seed", [(150_000, 1_500_000, 42), (20_000, 90_000, 3), (1, 1, 5), (7, 0, 6)])
def test_q13_matches_oracle(engine, orc, n_cu, n_or, seed):
    cu, od = orc.q13_tables(n_cu, max(n_or, 1), seed)
    if n_or == 0:
        od = {k: v[:0] for k, v in od.items()}
    assert run(engine, cu, od) == orc.q13(cu, od)


@pytest.mark.parametrize("w1,w2", [(b"pinto", b"beans"), (b"s", b"s"), (b"even", b"bold"), (b"y", b"e"),
                                   (b"instructions", b"instructions")])
def test_q13_other_words(engine, orc, w1, w2):
    cu, od = orc.q13_tables(3000, 40_000, 11)
    assert run(engine, cu, od, w1, w2) == orc.q13(cu, od, w1, w2)


def test_q13_hand_written_comments(engine, orc):
    texts = [b"special requests", b"requests special", b"specialrequests", b"xspecialx yrequestsy",
             b"special", b"requests", b"", b"spe cial requests", b"special reque sts",
             b"a" * 72 + b"special",                      # word 1 ends at the slot's last text byte
             b"special " + b"b" * 63 + b"requests",        # 79 characters, word 2 at the very end
             b"special " + b"b" * 64 + b"request",         # word 2 cut off
             b"sspecial rrequests", b"special special requests requests"]
    n = len(texts)
    od = dict(cust_key=np.arange(n, dtype=np.int32) % 4, comment=np.array(texts, dtype="S80"))
    cu = dict(cust_key=np.arange(6, dtype=np.int32))   # customers 4 and 5 have no orders
    got = run(engine, cu, od)
    assert got == orc.q13(cu, od)
    # direct count: the comments that are NOT LIKE '%special%requests%'
    keep = [t for t in texts if not (b"special" in t and b"requests" in t.split(b"special", 1)[1])]
    assert sum(c * d for c, d in got) == len(keep)


def test_q13_orders_of_unknown_customers(engine, orc):
    cu, od = orc.q13_tables(500, 20_000, 13)
    od = dict(od)
    ck = od["cust_key"].copy()
    ck[::5] = 900      # beyond the customers' key range: counted for nobody
    ck[1::9] = -3
    od["cust_key"] = ck
    assert run(engine, cu, od) == orc.q13(cu, od)
    # sparse customer keys: only the listed customers are in the distribution
    cu2 = dict(cust_key=np.arange(0, 500, 3, dtype=np.int32))
    assert run(engine, cu2, od) == orc.q13(cu2, od, cu_key_max=499)


def test_q13_limits(engine, orc):
    od = dict(cust_key=np.zeros(1024, np.int32), comment=np.array([b"x"] * 1024, dtype="S80"))
    cu = dict(cust_key=np.arange(3, dtype=np.int32))
    with pytest.raises(capi.GpudbError) as e:      # one customer with 1024 > GPUDB_Q13_MAX_COUNT orders
        run(engine, cu, od)
    assert e.value.code == capi.E_CAPACITY
    od1 = dict(cust_key=od["cust_key"][:1023], comment=od["comment"][:1023])
    assert run(engine, cu, od1) == [(0, 2), (1023, 1)]
    with pytest.raises(capi.GpudbError) as e:
        run(engine, cu, od1, b"", b"requests")
    assert e.value.code == capi.E_INVALID


@pytest.mark.parametrize("n_or", [1, 31, 32, 33, 257, 8 * 32 * 4 * 148 + 5])
@pytest.mark.parametrize("w1,w2", [(b"special", b"requests"), (b"spe", b"requests"), (b"aaaaaaa", b"aaaaaaaaaaaaaaa")])
def test_q13_tiles_and_candidates(engine, orc, n_or, w1, w2):
    """Orders that fill no warp tile evenly, and comments whose candidates do not verify: word
    prefixes before and after the words, at every alignment, and periodic words."""
    rng = np.random.default_rng(n_or)
    w1s, w2s = w1.decode(), w2.decode()
    bits = [w1s, w2s, w1s[:-1], w1s[1:], w2s[:5], w2s[1:], "a", "aaaa", " ", "xy"]
    pool = []
    for _ in range(600):
        s = "".join(bits[i] for i in rng.integers(0, len(bits), rng.integers(0, 12)))
        pool.append(s[:79].encode())
    for pad in range(80 - len(w1s + w2s)):
        pool.append(b"q" * pad + w1 + w2)
        pool.append(w1 + b"q" * pad + w2)
    pool = np.array(pool, dtype="S80")
    od = dict(cust_key=rng.integers(-1, 1001, n_or).astype(np.int32), comment=pool[rng.integers(0, len(pool), n_or)])
    cu = dict(cust_key=np.arange(1000, dtype=np.int32))
    assert run(engine, cu, od, w1, w2) == orc.q13(cu, od, w1, w2)


class _Repeated:
    """An address range of `size` bytes over `chunk` bytes of memory mapped again and again, its last
    `tail` bytes over memory of their own."""

    class _Prop(C.Structure):
        _fields_ = [("type", C.c_int), ("handle", C.c_int), ("loc", C.c_int * 2), ("win32", C.c_void_p),
                    ("flags", C.c_uint8 * 8)]

    class _Access(C.Structure):
        _fields_ = [("loc", C.c_int * 2), ("flags", C.c_int)]

    def __init__(self, size, chunk, tail):
        self.cu = C.CDLL("libcuda.so.1")
        self.size, self.maps, self.handles, self.va = size, [], [], C.c_uint64(0)
        assert (size - tail) % chunk == 0
        self.check("cuMemAddressReserve", C.byref(self.va), C.c_size_t(size), C.c_size_t(0), C.c_uint64(0), C.c_ulonglong(0))
        body, end = self.alloc(chunk), self.alloc(tail)
        for at in range(0, size - tail, chunk):
            self.map(at, chunk, body)
        self.map(size - tail, tail, end)
        acc = self._Access((C.c_int * 2)(1, 0), 3)   # device 0, read and write
        self.check("cuMemSetAccess", self.va, C.c_size_t(size), C.byref(acc), C.c_size_t(1))

    def check(self, name, *args):
        rc = getattr(self.cu, name)(*args)
        assert rc == 0, (name, rc)

    def alloc(self, size):
        prop = self._Prop(type=1, loc=(C.c_int * 2)(1, 0))   # pinned, device 0
        h = C.c_uint64(0)
        self.check("cuMemCreate", C.byref(h), C.c_size_t(size), C.byref(prop), C.c_ulonglong(0))
        self.handles.append(h)
        return h

    def map(self, at, size, handle):
        self.check("cuMemMap", C.c_uint64(self.va.value + at), C.c_size_t(size), C.c_size_t(0), handle, C.c_ulonglong(0))
        self.maps.append((at, size))

    def close(self):
        for at, size in self.maps:
            self.check("cuMemUnmap", C.c_uint64(self.va.value + at), C.c_size_t(size))
        for h in self.handles:
            self.check("cuMemRelease", h)
        self.check("cuMemAddressFree", self.va, C.c_size_t(self.size))


def test_q13_more_than_2_to_the_32_orders(engine, orc):
    """Orders from row 2^32 on are matched with their own comments (344 GB of comments, the first 2^32
    of them one block of memory mapped 512 times: no comment, no known customer)."""
    head, tail, period = 1 << 32, 1 << 19, 1 << 23
    text = _Repeated((head + tail) * 80, period * 80, tail * 80)
    cust = _Repeated((head + tail) * 4, period * 4, tail * 4)
    try:
        zeros, none = np.zeros(period * 80, np.uint8), np.full(period, -1, np.int32)
        comments = np.where(np.arange(tail) % 3 == 0, np.array(b"special requests", "S80"),
                            np.array(b"special packages", "S80")).astype("S80")
        ck = (np.arange(tail) % 1000).astype(np.int32)
        for dst, src in ((text.va.value, zeros), (text.va.value + head * 80, comments),
                         (cust.va.value, none), (cust.va.value + head * 4, ck)):
            engine._check(engine.lib.gpudb_copy(engine.ctx, dst, src.ctypes.data, src.nbytes))
        cu = dict(cust_key=np.arange(1000, dtype=np.int32))
        tc = engine.upload("customer", cu)
        got = engine.q13(tc, _View(capi.Orders(n_rows=head + tail, cust_key=cust.va.value, comment=text.va.value,
                                               key_max=-1, cust_key_max=999)))
        engine.free(tc)
        assert got == orc.q13(cu, dict(cust_key=ck, comment=comments))
    finally:
        engine.sync()
        text.close()
        cust.close()


class _View:
    """A table given as its C struct."""

    def __init__(self, s):
        self.s = s

    def struct(self):
        return self.s


@pytest.mark.parametrize("w1,w2", [(b"a", b"a"), (b"q", b"zz"), (b"ab", b"ba"), (b"aa", b"a"), (b"zz", b"special"),
                                   (b"a", b"aaaaaaaaaaaaaaa")])
def test_q13_first_word_of_one_or_two_letters(engine, orc, w1, w2):
    """Such orders are matched without a queue: the words at every pair of places, next to each
    other and overlapping, at the ends of the slot, and comments without the first word."""
    rng = np.random.default_rng(len(w1) * 16 + len(w2))
    texts = [b"", b"b" * 79, w1, w2, w2 + w1, w1 + w2, w1[:1] * 79, w2[:1] * 80]
    for at in range(80 - len(w1) + 1):
        for gap in (0, 1, 2, 3, 7, 40):
            t = b"-" * at + w1 + b"-" * gap + w2
            texts += [t[:80], t[:79], (b"-" * at + w1)[:80]]
        texts.append((w2 + b"-" * at + w1)[:80])
    alphabet = np.frombuffer(w1 + w2 + b"- ", np.uint8)
    texts += [bytes(rng.choice(alphabet, int(rng.integers(0, 81)))) for _ in range(3000)]
    n = len(texts)
    od = dict(cust_key=rng.integers(-1, 301, n).astype(np.int32), comment=np.array(texts, dtype="S80"))
    cu = dict(cust_key=np.arange(300, dtype=np.int32))
    assert run(engine, cu, od, w1, w2) == orc.q13(cu, od, w1, w2)


@pytest.mark.parametrize("w1,w2", [(b"special", b"requests"), (b"pinto", b"beans"), (b"s", b"t")])
@pytest.mark.parametrize("shift,key_shift", [(0, 1), (1, 0), (4, 0), (8, 3), (2, 2)])
def test_q13_columns_off_16_bytes(engine, orc, w1, w2, shift, key_shift):
    """Comments that start `shift` bytes (customer keys: rows) off a 16-byte boundary: no bulk
    copies, and comments read byte by byte."""
    cu, od = orc.q13_tables(300, 20_011, 17)
    tc = engine.upload("customer", cu)
    text = np.concatenate([np.zeros(shift, np.uint8), np.ascontiguousarray(od["comment"], "S80").view(np.uint8)])
    keys = np.concatenate([np.full(key_shift, 7, np.int32), od["cust_key"]])
    dt, dk = engine.to_device(text), engine.to_device(keys)
    view = _View(capi.Orders(n_rows=len(od["cust_key"]), cust_key=dk + 4 * key_shift, comment=dt + shift, key_max=-1,
                             cust_key_max=299))
    try:
        assert engine.q13(tc, view, w1, w2) == orc.q13(cu, od, w1, w2)
    finally:
        engine.free(tc)
        engine.device_free(dt)
        engine.device_free(dk)
