"""The work a user of this library has it do, as measurable cases.

Every case is one pass through a public entry point of the C ABI
(include/mpzmm_b200.h, by way of rforest_b200.api and rforest_b200._lib):

  one      one product, host arrays in, host arrays out (mpzmm_matmul_batch
           with one product: what mpz_rmatrix_mult_fft runs)
  noalloc  one product on device buffers (mpzmm_matmul_noalloc)
  batch    many products of uneven shapes in one call, host to host
  plan     a batch kept on the device: execute and read the results back
  fixed_b  a plan that keeps B's transforms: new A, execute, results
  chain    X_0 X_1 ... left to right, the running product on the device
  mod      x mod d for many x and one d

Sizes are the repository's own configurations (rforest_b200/workloads.py,
bench.py, the tests) or lie in the ranges those name: 2 to 64 rows, 2^8 to
2^20-bit entries, single operands of 10^7 bits.  Entry values are uniform
with random signs; "ragged" operands mix lengths and hold zeros.
"""
import ctypes as C
import math
import random

import numpy as np
import torch

from rforest_b200 import _lib, api

# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------


def listed():
    return [
        # the smallest call: a few launches over a few kilobytes, device buffers
        dict(name="noalloc_2x2x2_1kb", kind="noalloc", m=2, k=2, n=2, bits=1024, ragged=False),
        # the first configuration: 4 x 4 of signed 4096-bit integers, one call
        dict(name="one_4x4x4_4kb", kind="one", m=4, k=4, n=4, bits=4096, ragged=False,
             pinned=False),
        # odd dimensions, odd bit length, zeros and short entries, device buffers
        dict(name="noalloc_5x7x3_20011b", kind="noalloc", m=5, k=7, n=3, bits=20011, ragged=True),
        # the second configuration's product on device buffers
        dict(name="noalloc_8x8x8_64kb", kind="noalloc", m=8, k=8, n=8, bits=65536, ragged=False),
        # and as an ordinary call from ordinary (pageable) host memory
        dict(name="one_8x8x8_64kb", kind="one", m=8, k=8, n=8, bits=65536, ragged=False,
             pinned=False),
        # a remainder-tree level: 16 matrices multiplied on the device
        dict(name="chain_16_8x8_64kb", kind="chain", count=16, dim=8, bits=65536),
        # the batched configuration (2..16 rows, 2^10..2^18 bits), its first
        # eighth end to end from pinned host memory
        dict(name="batch_512_mixed", kind="batch", count=512, dim_lo=2, dim_hi=16, lg_lo=10,
             lg_hi=18, pinned=True, shapes=1),
        # the same mix resident on the device, replayed as a CUDA graph
        dict(name="plan_256_mixed_graph", kind="plan", count=256, dim_lo=2, dim_hi=16, lg_lo=10,
             lg_hi=18, graph=True, tc=False, shapes=2),
        # one B against many A
        dict(name="fixed_b_64_4x16x16_32kb", kind="fixed_b", count=64, m=4, k=16, n=16,
             bits=32768),
        # many residues of one modulus
        dict(name="mod_2000_20kb_by_10kb", kind="mod", count=2000, x_bits=20000, d_bits=10007),
        # long operands: the reference's benchmark size
        dict(name="one_2x2x2_10mb", kind="one", m=2, k=2, n=2, bits=10_000_000, ragged=False,
             pinned=True),
        # the large dense configuration on the tensor cores
        dict(name="plan_64x64x64_1mb_tc", kind="plan", count=1, dim_lo=64, dim_hi=64, lg_lo=20,
             lg_hi=20, graph=False, tc=True, shapes=3),
    ]


def _log_int(rng, lo, hi):
    """An integer in [lo, hi], uniform in its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["one", "one", "noalloc", "noalloc", "batch", "plan", "fixed_b", "chain",
                       "mod"])
    if kind == "one":
        if rng.random() < 0.25:  # few long operands
            return dict(kind="one", m=rng.randint(1, 2), k=rng.randint(1, 3), n=rng.randint(1, 2),
                        bits=_log_int(rng, 1 << 20, 10_000_000), ragged=False, pinned=True)
        return dict(kind="one", m=rng.randint(1, 32), k=rng.randint(1, 32), n=rng.randint(1, 32),
                    bits=_log_int(rng, 256, 1 << 17), ragged=rng.random() < 0.3,
                    pinned=rng.random() < 0.5)
    if kind == "noalloc":
        # at most 300 entries of 2^15 bits, or fewer longer ones: the entry
        # point's scratch holds them
        m, k, n = (rng.randint(1, 10) for _ in range(3))
        entries = m * k + k * n + m * n
        top = min(1 << 17, (1 << 15) * 300 // max(entries, 75))
        return dict(kind="noalloc", m=m, k=k, n=n, bits=_log_int(rng, 256, top),
                    ragged=rng.random() < 0.3)
    if kind == "batch":
        return dict(kind="batch", count=_log_int(rng, 8, 400), dim_lo=2, dim_hi=16, lg_lo=8,
                    lg_hi=18, pinned=rng.random() < 0.7, shapes=rng.randrange(1 << 20))
    if kind == "plan":
        tc = rng.random() < 0.4
        hi = rng.choice([8, 16, 32])
        return dict(kind="plan", count=_log_int(rng, 1, 64), dim_lo=2, dim_hi=hi, lg_lo=8,
                    lg_hi=17, graph=rng.random() < 0.5, tc=tc, shapes=rng.randrange(1 << 20))
    if kind == "fixed_b":
        return dict(kind="fixed_b", count=_log_int(rng, 1, 64), m=rng.randint(1, 16),
                    k=rng.randint(2, 16), n=rng.randint(2, 16), bits=_log_int(rng, 1024, 1 << 16))
    if kind == "chain":
        return dict(kind="chain", count=rng.randint(3, 16), dim=rng.randint(2, 8),
                    bits=_log_int(rng, 1024, 1 << 16))
    d = _log_int(rng, 1024, 1 << 17)
    return dict(kind="mod", count=_log_int(rng, 16, 1000), x_bits=2 * d - rng.randint(0, 64),
                d_bits=d)


def _shapes(case):
    """(m, k, n, bits) of every product of a batch or plan case."""
    if case["kind"] == "fixed_b":
        return [(case["m"], case["k"], case["n"], case["bits"])] * case["count"]
    if case["kind"] in ("one", "noalloc"):
        return [(case["m"], case["k"], case["n"], case["bits"])]
    r = random.Random(case["shapes"])
    out = []
    for _ in range(case["count"]):
        m, k, n = (r.randint(case["dim_lo"], case["dim_hi"]) for _ in range(3))
        if case["lg_hi"] > case["lg_lo"]:
            bits = int(2.0 ** r.uniform(case["lg_lo"], case["lg_hi"]))
        else:
            bits = 1 << case["lg_lo"]
        out.append((m, k, n, bits))
    return out


# ---------------------------------------------------------------------------
# host memory and entries
# ---------------------------------------------------------------------------


class _Pinned:
    """A block from mpzmm_host_alloc that lives as long as an array on it."""

    def __init__(self, words):
        p = C.c_void_p()
        _lib.check(_lib.lib().mpzmm_host_alloc(8 * words, C.byref(p)))
        self.ptr = p.value
        self.__array_interface__ = dict(shape=(words,), typestr="<u8", data=(self.ptr, False),
                                        version=3)

    def __del__(self):
        _lib.lib().mpzmm_host_free(C.c_void_p(self.ptr))


def _words(count, pinned):
    count = max(int(count), 1)
    a = np.asarray(_Pinned(count)) if pinned else np.empty(count, np.uint64)
    return a


def _fill(rng, dst, entries, bits, ragged, positive=False):
    """Writes `entries` random integers of exactly `bits` bits (ragged: some
    shorter, some zero) into dst, evenly spaced; returns their signed sizes."""
    nl = (bits + 63) // 64
    top = bits - 64 * (nl - 1)
    v = dst[:entries * nl].reshape(entries, nl)
    step = max(1, (1 << 22) // nl)
    for e in range(0, entries, step):
        rows = v[e:e + step]
        rows[...] = rng.integers(0, 1 << 64, size=rows.shape, dtype=np.uint64)
    if top < 64:
        v[:, nl - 1] &= np.uint64((1 << top) - 1)
    v[:, nl - 1] |= np.uint64(1 << (top - 1))
    sizes = np.full(entries, nl, np.int32)
    if ragged and entries > 1:
        sizes[1:] = rng.integers((nl + 1) // 2, nl + 1, size=entries - 1)
        sizes[1:][rng.random(entries - 1) < 0.1] = 0
        for e in range(1, entries):
            if sizes[e]:
                v[e, sizes[e] - 1] |= np.uint64(1 << 40)
    if not positive:
        sizes = np.where(rng.random(entries) < 0.5, -sizes, sizes).astype(np.int32)
    return sizes


def _p(a, t):
    return a.ctypes.data_as(t)


class _Products:
    """Host arrays of a list of products, laid out once: one block of operand
    limbs, one of result limbs, one of result sizes."""

    def __init__(self, shapes, seed, ragged, pinned):
        rng = np.random.default_rng(seed)
        self.shapes = shapes
        limbs = [((b + 63) // 64) for (_, _, _, b) in shapes]
        caps = [api.output_limbs(k, b, b) for (_, k, _, b) in shapes]
        self.ins = _words(sum((m * k + k * n) * w for (m, k, n, _), w in zip(shapes, limbs)),
                          pinned)
        self.outs = _words(sum(m * n * c for (m, _, n, _), c in zip(shapes, caps)), pinned)
        self.outs[...] = 0
        self.sizes = np.zeros(sum(m * n for (m, _, n, _) in shapes), np.int32)
        self.keep = []
        self.arr = (_lib.Product * len(shapes))()
        pos = cpos = spos = 0
        for t, ((m, k, n, b), w, cap) in enumerate(zip(shapes, limbs, caps)):
            a = self.ins[pos:pos + m * k * w]
            pos += m * k * w
            bb = self.ins[pos:pos + k * n * w]
            pos += k * n * w
            asz = _fill(rng, a, m * k, b, ragged)
            bsz = _fill(rng, bb, k * n, b, ragged)
            ao = np.arange(m * k, dtype=np.int64) * w
            bo = np.arange(k * n, dtype=np.int64) * w
            co = np.arange(m * n, dtype=np.int64) * cap
            cc = np.full(m * n, cap, np.int64)
            cl = self.outs[cpos:cpos + m * n * cap]
            cs = self.sizes[spos:spos + m * n]
            cpos += m * n * cap
            spos += m * n
            self.keep.append((a, ao, asz, bb, bo, bsz, cl, co, cc, cs, cap))
            self.arr[t] = _lib.Product(m, k, n, _p(a, _lib.u64p), _p(ao, _lib.i64p),
                                       _p(asz, _lib.i32p), _p(bb, _lib.u64p), _p(bo, _lib.i64p),
                                       _p(bsz, _lib.i32p), _p(cl, _lib.u64p), _p(co, _lib.i64p),
                                       _p(cc, _lib.i64p), _p(cs, _lib.i32p))

    def results(self):
        return [self.outs.view(np.int64), self.sizes]


class _Plan:
    """A plan handle over _Products."""

    def __init__(self, products, fixed_b=False, graph=False, tc=False):
        self.products = products
        self.handle = C.c_void_p()
        L = _lib.lib()
        # a plan keeps the contraction engine it was built with
        before = api.contract_mode()
        api.set_contract_mode(2 if tc else before)
        try:
            create = L.mpzmm_plan_create_fixed_b if fixed_b else L.mpzmm_plan_create
            _lib.check(create(C.byref(self.handle), len(products.shapes), products.arr, None))
        finally:
            api.set_contract_mode(before)
        if graph:
            _lib.check(L.mpzmm_plan_set_graph(self.handle, 1))

    def __del__(self):
        if self.handle:
            _lib.lib().mpzmm_plan_destroy(self.handle)


class _NoAlloc:
    """One product on device buffers, and the host arrays that describe it."""

    def __init__(self, shape, seed, ragged):
        m, k, n, b = shape
        rng = np.random.default_rng(seed)
        w = (b + 63) // 64
        a, bb = _words(m * k * w, False), _words(k * n * w, False)
        self.dims = (m, k, n)
        self.asz = _fill(rng, a, m * k, b, ragged)
        self.bsz = _fill(rng, bb, k * n, b, ragged)
        self.ao = np.arange(m * k, dtype=np.int64) * w
        self.bo = np.arange(k * n, dtype=np.int64) * w
        cap = api.output_limbs(k, 64 * w, 64 * w)
        self.co = np.arange(m * n, dtype=np.int64) * cap
        self.cc = np.full(m * n, cap, np.int64)
        self.da = torch.from_numpy(a.view(np.int64)).cuda()
        self.db = torch.from_numpy(bb.view(np.int64)).cuda()
        self.dc = torch.zeros(m * n * cap, dtype=torch.int64, device="cuda")
        self.dsz = torch.zeros(m * n, dtype=torch.int32, device="cuda")

    def run(self):
        m, k, n = self.dims
        _lib.check(_lib.lib().mpzmm_matmul_noalloc(
            m, k, n, self.da.data_ptr(), _p(self.ao, _lib.i64p), _p(self.asz, _lib.i32p),
            self.db.data_ptr(), _p(self.bo, _lib.i64p), _p(self.bsz, _lib.i32p),
            self.dc.data_ptr(), _p(self.co, _lib.i64p), _p(self.cc, _lib.i64p),
            self.dsz.data_ptr(), torch.cuda.current_stream().cuda_stream))
        return [self.dc, self.dsz]


class _Chain:
    """Host arrays of a chain of square matrices and its result."""

    def __init__(self, count, dim, bits, seed):
        rng = np.random.default_rng(seed)
        w = (bits + 63) // 64
        self.keep = []
        self.arr = (_lib.Matrix * count)()
        for i in range(count):
            x = _words(dim * dim * w, False)
            sz = _fill(rng, x, dim * dim, bits, False)
            off = np.arange(dim * dim, dtype=np.int64) * w
            self.keep.append((x, off, sz))
            self.arr[i] = _lib.Matrix(dim, dim, _p(x, _lib.u64p), _p(off, _lib.i64p),
                                      _p(sz, _lib.i32p))
        self.count = count
        cap = int(_lib.lib().mpzmm_chain_output_limbs(count, self.arr))
        self.out = np.zeros(dim * dim * cap, np.uint64)
        self.co = np.arange(dim * dim, dtype=np.int64) * cap
        self.cc = np.full(dim * dim, cap, np.int64)
        self.sizes = np.zeros(dim * dim, np.int32)

    def run(self):
        _lib.check(_lib.lib().mpzmm_chain(self.count, self.arr, _p(self.out, _lib.u64p),
                                          _p(self.co, _lib.i64p), _p(self.cc, _lib.i64p),
                                          _p(self.sizes, _lib.i32p), None))
        return [self.out.view(np.int64), self.sizes]


class _Mod:
    """A modulus handle, the numbers to reduce and their remainders."""

    def __init__(self, count, x_bits, d_bits, seed):
        rng = np.random.default_rng(seed)
        L = _lib.lib()
        d = _words((d_bits + 63) // 64, False)
        dsz = _fill(rng, d, 1, d_bits, False, positive=True)
        w = (x_bits + 63) // 64
        self.x = _words(count * w, False)
        self.xs = _fill(rng, self.x, count, x_bits, False)
        self.xo = np.arange(count, dtype=np.int64) * w
        self.handle = C.c_void_p()
        _lib.check(L.mpzmm_mod_create(C.byref(self.handle), _p(d, _lib.u64p), int(dsz[0]), w))
        nd = int(L.mpzmm_mod_limbs(self.handle))
        self.d = d
        self.r = np.zeros(count * nd, np.uint64)
        self.ro = np.arange(count, dtype=np.int64) * nd
        self.rc = np.full(count, nd, np.int64)
        self.rs = np.zeros(count, np.int32)
        self.count = count

    def run(self):
        _lib.check(_lib.lib().mpzmm_mod_batch(self.handle, self.count, _p(self.x, _lib.u64p),
                                              _p(self.xo, _lib.i64p), _p(self.xs, _lib.i32p),
                                              _p(self.r, _lib.u64p), _p(self.ro, _lib.i64p),
                                              _p(self.rc, _lib.i64p), _p(self.rs, _lib.i32p),
                                              None))
        return [self.r.view(np.int64), self.rs]

    def __del__(self):
        if self.handle:
            _lib.lib().mpzmm_mod_destroy(self.handle)


# ---------------------------------------------------------------------------
# prepare, run, work, exact
# ---------------------------------------------------------------------------


def prepare(case, seed):
    api.setup(0)
    kind = case["kind"]
    if kind == "noalloc":
        return kind, _NoAlloc(_shapes(case)[0], seed, case["ragged"])
    if kind == "chain":
        return kind, _Chain(case["count"], case["dim"], case["bits"], seed)
    if kind == "mod":
        return kind, _Mod(case["count"], case["x_bits"], case["d_bits"], seed)
    products = _Products(_shapes(case), seed, case.get("ragged", False), case.get("pinned", True))
    if kind in ("one", "batch"):
        return kind, products
    return kind, _Plan(products, fixed_b=kind == "fixed_b", graph=case.get("graph", False),
                       tc=case.get("tc", False))


def run(state):
    kind, s = state
    L = _lib.lib()
    if kind in ("noalloc", "chain", "mod"):
        return s.run()
    if kind in ("one", "batch"):
        _lib.check(L.mpzmm_matmul_batch(len(s.shapes), s.arr, None))
        return s.results()
    if kind == "fixed_b":
        _lib.check(L.mpzmm_plan_upload_a(s.handle, None))
    _lib.check(L.mpzmm_plan_execute(s.handle, None))
    _lib.check(L.mpzmm_plan_download(s.handle, None))
    return s.products.results()


def work(case):
    """Operand limbs read once, result limbs written once (the arithmetic is
    integer work without a fixed operation count)."""
    kind = case["kind"]
    if kind == "mod":
        words = case["count"] * ((case["x_bits"] + 63) // 64 + (case["d_bits"] + 63) // 64)
    elif kind == "chain":
        words = case["count"] * case["dim"] ** 2 * ((case["bits"] + 63) // 64) * 2
    else:
        words = 0
        for m, k, n, b in _shapes(case):
            w = (b + 63) // 64
            a_words = 0 if kind == "plan" else m * k * w
            b_words = 0 if kind in ("plan", "fixed_b") else k * n * w
            if kind == "plan":  # operands resident on the device, still read
                a_words, b_words = m * k * w, k * n * w
            words += a_words + b_words + m * n * api.output_limbs(k, b, b)
    return {"bytes": 8 * words, "flops": 0}


def _ints(limbs, offs, sizes):
    out = []
    for o, s in zip(offs, sizes):
        v = int.from_bytes(limbs[o:o + abs(int(s))].astype("<u8").tobytes(), "little")
        out.append(-v if s < 0 else v)
    return out


def _pack(values, cap):
    limbs = np.zeros(len(values) * cap, np.uint64)
    sizes = np.zeros(len(values), np.int32)
    for e, v in enumerate(values):
        mag = abs(v)
        nl = (mag.bit_length() + 63) // 64
        limbs[e * cap:e * cap + nl] = np.frombuffer(mag.to_bytes(8 * nl, "little"), "<u8")
        sizes[e] = -nl if v < 0 else nl
    return [limbs.view(np.int64), sizes]


def exact(case, seed):
    """The results by Python integers, for the cases that are quick that way."""
    kind = case["kind"]
    if kind == "mod":
        if case["count"] * case["x_bits"] * case["d_bits"] > 1 << 40:
            return None
        s = _Mod(case["count"], case["x_bits"], case["d_bits"], seed)
        d = int.from_bytes(s.d.astype("<u8").tobytes(), "little")
        return _pack([x % d for x in _ints(s.x, s.xo, s.xs)], s.d.size)
    if kind not in ("one", "noalloc"):
        return None
    m, k, n, b = _shapes(case)[0]
    if m * k * n * float(b) ** 1.6 > 4e11:
        return None
    if kind == "noalloc":
        s = _NoAlloc((m, k, n, b), seed, case["ragged"])
        A = _ints(s.da.cpu().numpy().view(np.uint64), s.ao, s.asz)
        B = _ints(s.db.cpu().numpy().view(np.uint64), s.bo, s.bsz)
        cap = int(s.cc[0])
    else:
        s = _Products([(m, k, n, b)], seed, case["ragged"], False)
        a, ao, asz, bb, bo, bsz, _, _, _, _, cap = s.keep[0]
        A, B = _ints(a, ao, asz), _ints(bb, bo, bsz)
    vals = [sum(A[i * k + q] * B[q * n + j] for q in range(k)) for i in range(m)
            for j in range(n)]
    return _pack(vals, cap)
