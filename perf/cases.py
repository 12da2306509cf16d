"""Workloads of the off-target search, through the C ABI of libcof.so.

Each case is one call (or one stream of results) that a user of the library
makes on a genome that is already resident on the GPU: small and large
genomes, one guide and a whole guide library, 3' and 5' PAMs, one request and
a batch of them, rows, raw matches, bulges, and the allocation-free entry
point.  Genomes are seeded: i.i.d. bases at 41 % GC, runs of N, and planted
near-target sites of every guide (substitutions, and inserted or deleted bases
where the request allows bulges).  They reach the library as .2bit files, the
form in which genomes are shipped.
"""
import ctypes
import math
import os
import struct
import sys
import tempfile
import weakref

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "cas-offinder-rust-old_b200"))
import cof  # noqa: E402

# PAM by name: (cells, whether it precedes the guide)
PAMS = {"NRG": ("NRG", False), "NNGRRT": ("NNGRRT", False), "NNNRRT": ("NNNRRT", False),
        "TTTN": ("TTTN", True)}
IUPAC = {"A": "A", "C": "C", "G": "G", "T": "T", "N": "ACGT", "R": "AG", "Y": "CT"}
BASES = "ACGT"  # codes 0..3 here; a base and its complement add up to 3


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def _case(name, call, nt, records, guides, mm, pam="NRG", guide_len=20, requests=1, db=0, rb=0):
    """call: search (rows as text), stream (rows collected by the sink of a
    streamed search), sites (the match records of a streamed search), count (a
    streamed search whose sink counts), raw (search()'s Match lines) or
    noalloc (cof_search_seq_noalloc).  guides: per request."""
    c = dict(call=call, nt=nt, records=records, guides=guides, mm=mm, pam=pam,
             guide_len=guide_len, requests=requests, db=db, rb=rb)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one guide against a plasmid or an amplicon: launches and host waits
        _case("plasmid_20k_1guide", "search", 20011, 1, 1, 3),
        # the plain small benchmark: one guide, a small genome of four records
        _case("small_10m_1guide", "search", 10_000_000, 4, 1, 3),
        # one guide against a whole human-size genome
        _case("genome_3100m_1guide", "search", 3_100_000_000, 24, 1, 3),
        # the headline benchmark: 100 guides against a human-size genome, its
        # 124 MB of rows collected while the search goes on
        _case("genome_3100m_100guides", "stream", 3_100_000_000, 24, 100, 6),
        # two guide sets with different PAMs (3' and 5') in one batched pass
        _case("mixed_pam_310m_2x50guides", "search", 310_000_007, 24, 50, 6, pam="3'+5'",
              guide_len=25, requests=2),
        # a guide library against one chromosome
        _case("library_100m_1200guides", "search", 100_000_019, 1, 1200, 4),
        # a server's pass: many small requests of mixed lengths, PAMs and limits
        _case("serving_310m_64requests", "search", 310_000_007, 24, 0, 4, pam="mixed",
              guide_len=0, requests=64),
        # search()'s own output, before the writer: every window, no PAM filter
        _case("raw_10m_4guides", "raw", 10_000_019, 4, 4, 4),
        # one guide with a DNA and an RNA bulge against a viral genome
        _case("bulge_50k_1guide", "search", 50_021, 1, 1, 3, db=1, rb=1),
        # a guide panel with bulges against a targeted region
        _case("bulge_150k_20guides", "sites", 150_013, 2, 20, 4, db=2, rb=2),
        # the bulge benchmark's guides and limits on a larger genome, streamed:
        # more rows than one device row buffer holds
        _case("bulge_25m_20guides", "count", 25_000_013, 5, 20, 4, db=2, rb=2),
        # a sequence that the caller holds on the device, no allocation allowed
        _case("noalloc_50m_8guides", "noalloc", 50_000_017, 1, 8, 4),
    ]


def draw(rng):
    def log_int(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    kind = rng.choice(["one", "one", "set", "set", "set", "batch", "bulge", "bulge", "raw",
                       "noalloc"])
    if kind == "one":  # a few guides, any genome
        return _case(None, "search", log_int(5_000, 1_500_000_000), rng.randint(1, 24),
                     rng.randint(1, 4), rng.randint(2, 4), pam=rng.choice(sorted(PAMS)),
                     guide_len=rng.randint(18, 25))
    if kind == "set":  # a guide set; genome x guides at most the listed ones'
        guides = log_int(4, 1200)
        nt = log_int(200_000, int(min(1_000_000_000, 2.0e11 / guides)))
        glen = rng.randint(18, 25)
        return _case(None, rng.choice(["search", "stream"]), nt, rng.randint(1, 24), guides,
                     rng.randint(3, 6 if glen >= 20 else 4), pam=rng.choice(sorted(PAMS)),
                     guide_len=glen)
    if kind == "batch":
        return _case(None, "search", log_int(1_000_000, 310_000_000), rng.randint(1, 24), 0,
                     rng.randint(2, 4), pam="mixed", guide_len=0, requests=log_int(4, 128))
    if kind == "bulge":
        db, rb = rng.choice([(1, 0), (0, 1), (1, 1), (2, 1), (1, 2), (2, 2)])
        guides = rng.randint(1, 20)
        nt = log_int(20_000, int(4.0e8 / guides / (1 if db + rb > 2 else 0.5)))
        call = "search" if nt * guides < 60_000 else "sites" if nt * guides < 6_000_000 else "count"
        return _case(None, call, nt, rng.randint(1, 5), guides, rng.randint(1, 4),
                     pam=rng.choice(sorted(PAMS)), guide_len=rng.randint(19, 24), db=db, rb=rb)
    if kind == "raw":
        return _case(None, "raw", log_int(50_000, 30_000_000), rng.randint(1, 6),
                     rng.randint(1, 8), rng.randint(2, 4), pam=rng.choice(sorted(PAMS)),
                     guide_len=rng.randint(20, 24))
    return _case(None, "noalloc", log_int(100_000, 200_000_000), 1, rng.randint(1, 64),
                 rng.randint(2, 4), pam=rng.choice(sorted(PAMS)), guide_len=rng.randint(18, 25))


# ---------------------------------------------------------------------------
# the library's C structures (include/cof.h)
# ---------------------------------------------------------------------------

class _Request(ctypes.Structure):
    _fields_ = [("search_filter", ctypes.c_char_p), ("pattern_len", ctypes.c_size_t),
                ("patterns", ctypes.POINTER(ctypes.c_char_p)), ("n_patterns", ctypes.c_size_t),
                ("max_mismatches", ctypes.c_uint32), ("max_dna_bulges", ctypes.c_uint32),
                ("max_rna_bulges", ctypes.c_uint32), ("flags", ctypes.c_uint32),
                ("chunks_per_search", ctypes.c_uint32)]


class _Result(ctypes.Structure):
    _fields_ = [("text", ctypes.c_void_p), ("text_len", ctypes.c_size_t),
                ("n_rows", ctypes.c_uint64), ("device_ms", ctypes.c_double)]


class _Piece(ctypes.Structure):
    _fields_ = [("request", ctypes.c_size_t), ("text", ctypes.c_void_p),
                ("text_len", ctypes.c_size_t), ("n_rows", ctypes.c_uint64),
                ("matches", ctypes.c_void_p)]


_MATCH = np.dtype([("chrom_idx", "i8"), ("text_offset", "i8"), ("record", "i4"),
                   ("pattern_idx", "i4"), ("mismatches", "u1"), ("dna", "u1"), ("rna", "u1"),
                   ("is_forward", "u1"), ("pad", "i4")])
_SINK = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p, ctypes.POINTER(_Piece))
_lib = None


def _abi():
    """A handle of libcof.so of this file's own (its argument types are not
    the binding's)."""
    global _lib
    if _lib is None:
        _lib = ctypes.CDLL(cof.LIB_PATH)
        _lib.cof_last_error.restype = ctypes.c_char_p
        _lib.cof_genome_free.restype = None
        _lib.cof_result_free.restype = None
    return _lib


def _ok(rc):
    if rc:
        raise RuntimeError("cof error %d: %s" % (rc, _abi().cof_last_error().decode()))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _codes(s):
    return np.array([BASES.index(c) for c in s], dtype=np.uint8)


def _requests(case, rng):
    """(filter, patterns, mm, db, rb) of every request; guides are random."""
    out = []
    for i in range(case["requests"]):
        name, glen, n, mm = case["pam"], case["guide_len"], case["guides"], case["mm"]
        if name == "3'+5'":
            name = ("NNGRRT", "TTTN")[i % 2]
        elif name == "mixed":
            name = sorted(PAMS)[int(rng.integers(0, 4))]
        glen = glen or int(rng.integers(17, 26))
        if not n:
            n = int(rng.integers(1, 5))
            mm = int(rng.integers(0, mm + 1))
        pam, lead = PAMS[name]
        rest = "N" * len(pam)
        g = ["".join(BASES[b] for b in x) for x in rng.integers(0, 4, size=(n, glen))]
        out.append((pam + "N" * glen if lead else "N" * glen + pam,
                    [rest + x if lead else x + rest for x in g], mm, case["db"], case["rb"]))
    return out


def _sites(rng, filt, patterns, per, mm, db, rb):
    """`per` near-target sites of every pattern, as base codes: 0..mm
    substitutions, a PAM of the filter's set, and in two thirds of the sites
    of a bulge request an inserted or a deleted cell; half of them reverse
    complemented."""
    L = len(filt)
    base = np.repeat(np.array([[BASES.find(c) & 0xFF for c in p] for p in patterns], dtype=np.int64),
                     per, axis=0)
    n = len(base)
    site = base.copy()
    for c in range(L):
        if patterns[0][c] == "N":
            opts = _codes(IUPAC[filt[c]])
            site[:, c] = opts[rng.integers(0, len(opts), n)]
    cells = np.array([c for c in range(L) if patterns[0][c] != "N"])
    k = rng.integers(0, mm + 1, n)
    order = np.argsort(rng.random((n, len(cells))), axis=1)
    sub = order < k[:, None]
    site[:, cells] = np.where(sub, (site[:, cells] + rng.integers(1, 4, sub.shape)) % 4,
                              site[:, cells])
    if db or rb:
        # the cell next to the PAM stays where it is, the far end gives or
        # takes a base; written for a PAM that ends the pattern
        lead = patterns[0][0] == "N"
        x = site[:, ::-1] if lead else site
        j = rng.integers(2, len(cells) - 2, n)[:, None]
        at = np.arange(L)[None, :]
        extra = rng.integers(0, 4, (n, 1))
        gone = np.where(at > j, x, np.where(at == 0, extra,
                                            np.take_along_axis(x, np.maximum(at - 1, 0), 1)))
        more = np.where(at > j, x, np.where(at == j, extra, np.take_along_axis(
            x, np.minimum(at + 1, L - 1), 1)))
        kind = rng.integers(0, 3, n)[:, None]
        x = np.where((kind == 1) & (rb > 0), gone, np.where((kind == 2) & (db > 0), more, x))
        site = x[:, ::-1] if lead else x
    rc = rng.integers(0, 2, n).astype(bool)
    site[rc] = 3 - site[rc][:, ::-1]
    return site.astype(np.uint8)


def _planted(nt, guides):
    """Near-target sites per guide."""
    return max(1, min(50, nt // 4000 // guides))


def _genome(case, seed, reqs):
    """Record lengths, base codes on the GPU (one uint8 per nucleotide), and
    runs of N as (record, start, length)."""
    rng = np.random.default_rng([seed, 7])
    nt, nrec = case["nt"], case["records"]
    w = rng.uniform(50, 250, nrec)
    lens = np.maximum(64, (w / w.sum() * nt).astype(np.int64))
    lens[-1] = max(64, nt - int(lens[:-1].sum()))
    nt = int(lens.sum())
    g = torch.Generator(device="cuda").manual_seed(seed)
    codes = torch.empty(nt, dtype=torch.uint8, device="cuda")
    step = 1 << 28
    for a in range(0, nt, step):
        r = torch.randint(0, 256, (min(step, nt - a),), dtype=torch.uint8, device="cuda", generator=g)
        c = codes[a:a + step]
        torch.ge(r, 76, out=c.view(torch.bool))
        c += r >= 128
        c += r >= 180
        del r
    first = np.concatenate([[0], np.cumsum(lens)[:-1]])
    per = _planted(nt, sum(len(r[1]) for r in reqs))
    taken = np.zeros(0, np.int64)  # sites lie in 64-nt cells of their own
    for filt, pats, mm, db, rb in reqs:
        s = _sites(rng, filt, pats, per, mm, db, rb)
        cell = np.setdiff1d(rng.integers(0, nt // 64, len(s)), taken)
        taken = np.concatenate([taken, cell])
        s = s[rng.permutation(len(s))[:len(cell)]]
        at = torch.from_numpy(64 * cell[:, None] + np.arange(s.shape[1])[None, :]).cuda().reshape(-1)
        codes[at] = torch.from_numpy(s).cuda().reshape(-1)
    runs = []
    left = int(0.05 * nt) if nt >= 1_000_000 else 0
    while left > 0 and len(runs) < 400:
        rec = int(rng.integers(0, nrec))
        ln = int(min(np.exp(rng.uniform(np.log(500), np.log(3_000_000))), lens[rec] // 4, left))
        if ln < 1:
            break
        runs.append((rec, int(rng.integers(0, lens[rec] - ln)), ln))
        left -= ln
    return lens, first, codes, runs


def _merged(runs, rec):
    """The record's N runs as sorted, disjoint (start, length) arrays."""
    out = []
    for a, n in sorted((a, n) for r, a, n in runs if r == rec):
        if out and a <= out[-1][0] + out[-1][1]:
            out[-1][1] = max(out[-1][1], a + n - out[-1][0])
        else:
            out.append([a, n])
    return np.array([x[0] for x in out], "<u4"), np.array([x[1] for x in out], "<u4")


def _scratch_dir(need):
    for d in ("/dev/shm", tempfile.gettempdir()):
        try:
            v = os.statvfs(d)
            if os.access(d, os.W_OK) and v.f_bavail * v.f_frsize > 2 * need:
                return d
        except OSError:
            pass
    return tempfile.gettempdir()


def _write_2bit(path, lens, first, codes, runs):
    """UCSC .2bit, version 0: T=0 C=1 A=2 G=3, first base in the high bits."""
    names = [b"chr%d" % (i + 1) for i in range(len(lens))]
    blocks = [_merged(runs, i) for i in range(len(lens))]
    off = 16 + sum(1 + len(n) + 4 for n in names)
    with open(path, "wb") as f:
        f.write(struct.pack("<IIII", 0x1A412743, 0, len(names), 0))
        for n, ln, (st, sz) in zip(names, lens, blocks):
            f.write(bytes([len(n)]) + n + struct.pack("<I", off))
            off += 16 + 8 * len(st) + (int(ln) + 3) // 4
        for ln, a, (st, sz) in zip(lens, first, blocks):
            ln, a = int(ln), int(a)
            f.write(struct.pack("<II", ln, len(st)) + st.tobytes() + sz.tobytes() +
                    struct.pack("<II", 0, 0))
            c = codes[a:a + ln]
            if ln % 4:
                c = torch.cat([c, c.new_full((4 - ln % 4,), 3)])
            c = c.view(-1, 4)
            packed = torch.zeros(len(c), dtype=torch.uint8, device="cuda")
            for k in range(4):  # A C G T = 0 1 2 3 here, 2 1 3 0 in the file
                b = c[:, k]
                packed |= (((b & 1) ^ 1) << 1 | ((b ^ (b >> 1)) & 1)) << (6 - 2 * k)
            f.write(memoryview(packed.cpu().numpy()))


class _State:
    pass


def prepare(case, seed):
    lib = _abi()
    rng = np.random.default_rng([seed, 11])
    reqs = _requests(case, rng)
    lens, first, codes, runs = _genome(case, seed, reqs)
    s = _State()
    s.call = case["call"]
    if s.call == "noalloc":
        return _prepare_noalloc(s, case, first, codes, runs, reqs[0])
    fd, path = tempfile.mkstemp(suffix=".2bit", dir=_scratch_dir(int(lens.sum()) // 4))
    os.close(fd)
    h = ctypes.c_void_p()
    _ok(lib.cof_genome_create(0, ctypes.byref(h)))
    s.genome = h
    weakref.finalize(s, lib.cof_genome_free, h)
    try:
        _write_2bit(path, lens, first, codes, runs)
        del codes
        _ok(lib.cof_genome_load(h, path.encode()))
        _ok(lib.cof_genome_upload(h))
    finally:
        os.unlink(path)
    s.keep = []
    s.n = len(reqs)
    s.reqs = (_Request * len(reqs))()
    for r, (filt, pats, mm, db, rb) in zip(s.reqs, reqs):
        arr = (ctypes.c_char_p * len(pats))(*[p.encode() for p in pats])
        s.keep.append(arr)
        r.search_filter, r.pattern_len = filt.encode(), len(filt)
        r.patterns, r.n_patterns = arr, len(pats)
        r.max_mismatches, r.max_dna_bulges, r.max_rna_bulges = mm, db, rb
        r.flags = cof.COF_F_ADD_REVCOMP | (cof.COF_F_RAW_MATCHES if s.call == "raw" else 0)
    s.by_line = bool(case["db"] or case["rb"])
    rows = _row_room(case)
    if s.call == "sites":
        s.sites = np.zeros(rows, _MATCH)
    elif s.call != "count":
        s.text = torch.zeros(rows * (2 * (case["guide_len"] or 25) + 62), dtype=torch.uint8)
    return s


def _prepare_noalloc(s, case, first, codes, runs, req):
    """The sequence as bit4 nibbles in a tensor of the caller's."""
    filt, pats, mm, _, _ = req
    n = len(codes)
    nib = torch.tensor([4, 2, 8, 1], dtype=torch.uint8, device="cuda")[codes.to(torch.int32)]
    for rec, a, ln in runs:
        nib[first[rec] + a:first[rec] + a + ln] = 15
    if n % 2:
        nib = torch.cat([nib, nib.new_zeros(1)])
    s.bit4 = nib[0::2] | (nib[1::2] << 4)
    s.nt = n
    comp = str.maketrans("ACGTN", "TGCAN")
    full = pats + [p.translate(comp)[::-1] for p in pats]
    s.patterns = (ctypes.c_char_p * len(full))(*[p.encode() for p in full])
    s.filter, s.mm = filt.encode(), mm
    s.rows = torch.zeros((_row_room(case), 3), dtype=torch.int32, device="cuda")
    s.out = torch.zeros_like(s.rows)
    return s


def _row_room(case):
    """Rows the caller keeps room for: several times what i.i.d. bases give,
    and what the planted sites add."""
    guides = sum(g for _, _, g, _ in _requests_shape(case))
    if case["db"] or case["rb"]:
        return int(0.3 * case["nt"] * guides + 25000 * guides * _planted(case["nt"], int(guides)) + 1000)
    per = 50 if case["guides"] else 250
    return int((1.2 + 4 / math.sqrt(guides)) * _expected_rows(case) + per * guides + 1000)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _collect(s, at, p, n):
    """Copies n bytes of row text at address p into the caller's buffer."""
    if at + n > len(s.text):
        raise RuntimeError("%d bytes of rows, room for %d" % (at + n, len(s.text)))
    if n >= 1 << 20:  # a copy on several threads
        s.text[at:at + n].copy_(torch.frombuffer((ctypes.c_uint8 * n).from_address(p), dtype=torch.uint8))
    elif n:
        ctypes.memmove(s.text.data_ptr() + at, p, n)


def _run_search(s):
    lib = _abi()
    outs = (_Result * s.n)()
    _ok(lib.cof_search_batch(s.genome, s.reqs, ctypes.c_size_t(s.n), outs))
    rows, size, at = np.empty(s.n, np.int64), np.empty(s.n, np.int64), 0
    for i, o in enumerate(outs):
        rows[i], size[i] = o.n_rows, o.text_len
        if s.by_line and o.text_len:  # the alignments of one site come in any order
            text = b"".join(sorted(ctypes.string_at(o.text, o.text_len).splitlines(True)))
            ctypes.memmove(o.text, text, len(text))
        _collect(s, at, o.text, o.text_len)
        at += o.text_len
        lib.cof_result_free(ctypes.byref(o))
    return rows, size, s.text


def _run_stream(s):
    lib = _abi()
    rows, size, err = np.zeros(s.n, np.int64), np.zeros(s.n, np.int64), []

    def piece(_user, p):
        p = p.contents
        try:
            if s.call == "stream":  # one request: its pieces come in order
                _collect(s, int(size[0]), p.text, p.text_len)
            elif s.call == "sites" and p.n_rows:
                at = int(rows.sum())
                if at + p.n_rows > len(s.sites):
                    raise RuntimeError("room for %d sites only" % len(s.sites))
                ctypes.memmove(s.sites[at:].ctypes.data, p.matches, p.n_rows * _MATCH.itemsize)
            rows[p.request] += p.n_rows
            size[p.request] += p.text_len
            return 0
        except Exception as e:
            err.append(e)
            return 1

    fn = _SINK(piece)
    n = (ctypes.c_uint64 * s.n)()
    rc = lib.cof_search_stream(s.genome, s.reqs, ctypes.c_size_t(s.n),
                               cof.COF_STREAM_MATCHES if s.call == "sites" else 0, fn, None, n)
    if err:
        raise err[0]
    _ok(rc)
    if s.call == "count":
        return rows, size, np.array(n, dtype=np.uint64).astype(np.int64)
    if s.call == "stream":
        return rows, size, s.text
    m = s.sites
    return rows, size, m["chrom_idx"], m["record"], m["pattern_idx"], m["is_forward"]


def _run_noalloc(s):
    n = ctypes.c_uint32()
    _ok(_abi().cof_search_seq_noalloc(
        ctypes.c_void_p(s.bit4.data_ptr()), ctypes.c_uint64(s.nt), s.filter, s.patterns,
        ctypes.c_size_t(len(s.patterns)), ctypes.c_uint32(s.mm), ctypes.c_void_p(s.rows.data_ptr()),
        ctypes.c_uint32(len(s.rows)), ctypes.byref(n),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    r = s.rows[:n.value]  # in no particular order: sorted by start, then pattern
    torch.index_select(r, 0, torch.argsort(r[:, 0].long() * 1024 + r[:, 1]), out=s.out[:n.value])
    return n.value, s.out


def run(state):
    if state.call == "noalloc":
        return _run_noalloc(state)
    if state.call in ("stream", "sites", "count"):
        return _run_stream(state)
    return _run_search(state)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _requests_shape(case):
    """(PAM pass rate, guide length, guides, mm) of every request, or of a
    typical one where they are drawn from the seed."""
    def rate(pam):
        return math.prod(len(IUPAC[c]) / 4 for c in PAMS[pam][0])
    names = {"3'+5'": ["NNGRRT", "TTTN"], "mixed": sorted(PAMS)}.get(case["pam"], [case["pam"]])
    return [(rate(names[i % len(names)]), case["guide_len"] or 21, case["guides"] or 2.5,
             case["mm"] if case["guides"] else case["mm"] / 2) for i in range(case["requests"])]


def _expected_rows(case):
    """Rows of random bases at equal frequencies."""
    rows = 0.0
    for rate, glen, guides, mm in _requests_shape(case):
        hit = sum(math.comb(glen, k) * 0.75 ** k * 0.25 ** (glen - k) for k in range(int(mm) + 1))
        rows += 2.0 * case["nt"] * guides * (1 if case["call"] == "raw" else rate) * hit
        if case["db"] or case["rb"]:  # an alignment's gaps go to many places
            rows *= 30 ** (case["db"] + case["rb"]) / 2
    return rows


def work(case):
    nt, ops = case["nt"], 0.0
    for rate, _, guides, _ in _requests_shape(case):
        if case["db"] or case["rb"]:
            ops += 2.0 * nt * guides * 12  # a bit-parallel edit distance column per position
        else:  # two differences, a count and a comparison per window
            ops += 4 * 2.0 * nt * guides * (1 if case["call"] == "raw" else rate)
    # bases at 2 bits and a mask bit (4 bits in the caller's own buffer)
    read = nt * (0.5 if case["call"] == "noalloc" else 0.375)
    return {"bytes": read + _expected_rows(case) * (12 if case["call"] == "noalloc" else 75),
            "flops": ops}
