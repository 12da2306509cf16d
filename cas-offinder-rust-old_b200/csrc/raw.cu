// raw.cu -- search()'s raw Match stream for the popcount path
// (COF_F_RAW_MATCHES): every window whose masked popcount count passes the
// threshold, as search_chunk_cpu emits it (search.rs:378-463), kept by
// convert_matches (search.rs:1428-1488), before the CLI writer's PAM filter
// and mismatch recount.  There is no PAM prefilter on this stream, so every
// window start is compared with every pattern.
//
//   raw_screen_kernel few mismatches: a bit-parallel bound from the planes, one
//                     lane per 32 starts, and the exact count of the few starts
//                     within it
//   raw_scan_kernel   otherwise; one thread per (32 window starts, pattern): the bit4
//                     window words (N masked to 0, zero past the batch end)
//                     funnel-shifted to each start, popcount against the
//                     pattern's bit4 words; emits starts with count <= max_mm
//   raw_verify_kernel convert_matches' ownership and record-end rules
//   raw_len/raw_write Match lines: name, chrom_idx, pattern index, strand,
//                     max(count, 0), 0, 0, rna_seq, dna_seq (NUL bytes kept)
#include <cub/cub.cuh>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "cof_engine.h"
#include "engine_dev.cuh"
#include "shares.h"

namespace cof {

namespace {

struct RawSeg {
    uint64_t lo, hi;       // global window starts [lo, hi)
    uint64_t base, clip;   // batch base and end
    uint64_t blk_begin;    // prefix of 32-start blocks
    uint32_t batch, pad;
};

struct RawPattern {
    uint32_t w[8];         // bit4 cells, 8 per word, zero past L (L <= 64)
    uint32_t strand, pad[3];
};

// 32-bit word of masked, clipped bit4 nibbles of nucleotides [8j, 8j + 8).
__device__ __forceinline__ uint32_t masked_word(const uint8_t *bit4, uint64_t j, uint64_t clip) {
    const uint64_t n0 = 8 * j;
    if (n0 >= clip) return 0;
    uint32_t x = __ldg(reinterpret_cast<const uint32_t *>(bit4) + j);
    if (n0 + 8 > clip) x &= (1u << (4 * (clip - n0))) - 1u;
    // genome N (0xF) -> 0 (mask_genome_n_to_zero_inplace, search.rs:512-531)
    const uint32_t t = x & (x >> 1) & (x >> 2) & (x >> 3) & 0x11111111u;
    return x & ~(t * 0xFu);
}

// NWD: pattern words compared (4: patterns of <= 32 cells, 8: <= 64)
template <int NWD>
__global__ void raw_scan_kernel(const uint8_t *__restrict__ bit4, const RawSeg *__restrict__ segs,
                                uint32_t nseg, uint64_t n_blocks, const RawPattern *__restrict__ pats,
                                uint32_t npat, uint32_t L, int max_mm, Hit *hits, uint32_t cap,
                                Counters *ctr) {
    const uint32_t nw = (L + 7) / 8;
    const uint64_t items = n_blocks * npat;
    for (uint64_t it = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; it < items;
         it += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t blk = it / npat;
        const uint32_t p = (uint32_t)(it % npat);
        uint32_t si = 0;
        while (si + 1 < nseg && blk >= segs[si + 1].blk_begin) ++si;
        const RawSeg S = segs[si];
        const uint64_t p0 = (S.lo & ~31ull) + 32 * (blk - S.blk_begin);  // 32-aligned
        uint32_t W[NWD + 5];
#pragma unroll
        for (int k = 0; k < NWD + 5; ++k) W[k] = masked_word(bit4, p0 / 8 + k, S.clip);
        const RawPattern P = pats[p];
#pragma unroll
        for (int o = 0; o < 32; ++o) {
            const uint64_t st = p0 + o;
            const int sh = 4 * (o & 7);
            int matches = 0;
#pragma unroll
            for (int j = 0; j < NWD; ++j) {
                if (j < (int)nw) {
                    const uint32_t w = __funnelshift_r(W[(o >> 3) + j], W[(o >> 3) + j + 1], sh);
                    matches += __popc(w & P.w[j]);
                }
            }
            if ((int)L - matches <= max_mm && st >= S.lo && st < S.hi) {
                const uint32_t i = atomicAdd(&ctr->hits, 1u);
                if (i < cap) hits[i] = Hit{(uint32_t)(st - S.base), p, S.batch, (uint32_t)((int)L - matches)};
                else ctr->overflow = 1;
            }
        }
    }
}

// Patterns of at most 32 cells that share kRawCells single-base cells, and few
// mismatches: one lane per 32 starts counts a pattern's differing cells among
// those for all of them at once, one bit per start (bit planes summed by full
// adders), and compares the starts left in full.  The differing single-base
// cells bound a start's mismatches from below while every cell of its window is
// a base of the batch (S clear, before the batch's end); windows with other
// cells, and the starts within the limit, are counted on the bit4 words, as
// raw_scan_kernel does for every start and pattern with four POPCs each.
// 10 Mbp x 4 guides: scan 0.049 ms, 0.103 with raw_scan_kernel; one POPC per
// start and pattern in a loop per lane took 0.143.
constexpr int kRawCells = 12;
constexpr uint32_t kRawMaxK = 4;
struct RawScreen {
    uint32_t ph[kRawCells], pl[kRawCells];  // code bits of the screened cells, as masks
    uint32_t h, l, care, pad;               // scan form: code bits, single-base cells
};
struct RawScreenParams {
    const uint8_t *bit4;
    const uint32_t *H, *L, *S;
    const RawSeg *segs;
    const RawPattern *pats;
    const RawScreen *screen;
    Hit *hits;
    Counters *ctr;
    uint64_t n_blocks;
    uint32_t nseg, npat, len, cap;
    int max_mm;
    uint32_t shift[kRawCells], kb[4];
};

__device__ __forceinline__ void raw_add(uint32_t a, uint32_t b, uint32_t c, uint32_t &s, uint32_t &y) {
    s = a ^ b ^ c;
    y = (a & b) | (c & (a | b));
}

__global__ void __launch_bounds__(256) raw_screen_kernel(const __grid_constant__ RawScreenParams P) {
    const uint32_t L = P.len, nw = (L + 7) / 8;
    // the block's share of the patterns
    const uint32_t p_lo = share_begin(P.npat, blockIdx.y, gridDim.y),
                   p_hi = share_begin(P.npat, blockIdx.y + 1, gridDim.y);
    for (uint64_t blk = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; blk < P.n_blocks;
         blk += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t si = 0;
        while (si + 1 < P.nseg && blk >= P.segs[si + 1].blk_begin) ++si;
        const RawSeg G = P.segs[si];
        const uint64_t p0 = (G.lo & ~31ull) + 32 * (blk - G.blk_begin);  // 32-aligned
        const uint64_t w = p0 / 32 + 1;  // (the planes begin with one padding word)
        const uint32_t h0 = __ldg(P.H + w), h1 = __ldg(P.H + w + 1), l0 = __ldg(P.L + w),
                       l1 = __ldg(P.L + w + 1), s0 = __ldg(P.S + w), s1 = __ldg(P.S + w + 1);
        // the starts of the range, and those whose window has a cell that is
        // no base: bit o of the OR of S over cells o .. o + L - 1
        uint32_t in = ~0u;
        if (p0 < G.lo) in &= ~0u << (uint32_t)(G.lo - p0);
        if (p0 + 32 > G.hi) in &= G.hi > p0 ? ~0u >> (uint32_t)(32 - (G.hi - p0)) : 0u;
        uint64_t z = ((uint64_t)s1 << 32) | s0;
        for (uint32_t have = 1; have < L;) {
            const uint32_t step = min(have, L - have);
            z |= z >> step;
            have += step;
        }
        uint32_t odd = (uint32_t)z;
        if (p0 + 31 + L > G.clip)  // windows past the batch's end
            odd |= G.clip >= p0 + L ? ~1u << (uint32_t)(G.clip - p0 - L) : ~0u;
        odd &= in;
        // a start's window words on the bit4 stream, N and what lies past the
        // batch zero
        uint32_t x[4];
        auto words = [&](uint64_t st) {
            uint32_t a = masked_word(P.bit4, st / 8, G.clip);
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                x[j] = 0;
                if (j >= nw) continue;
                const uint32_t b = masked_word(P.bit4, st / 8 + j + 1, G.clip);
                x[j] = __funnelshift_r(a, b, 4 * (uint32_t)(st & 7));
                a = b;
            }
        };
        auto exact = [&](uint64_t st, uint32_t p) {
            int matches = 0;
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j)
                if (j < nw) matches += __popc(x[j] & P.pats[p].w[j]);
            if ((int)L - matches > P.max_mm) return;
            const uint32_t i = atomicAdd(&P.ctr->hits, 1u);
            if (i < P.cap)
                P.hits[i] = Hit{(uint32_t)(st - G.base), p, G.batch, (uint32_t)((int)L - matches)};
            else
                P.ctr->overflow = 1;
        };
        // (a window of N only is zero and matches nothing; the next word's N
        // are not looked at again for it)
        for (uint32_t m = odd; m; m &= m - 1) {
            const uint64_t st = p0 + __ffs(m) - 1;
            words(st);
            if (!(x[0] | x[1] | x[2] | x[3])) continue;
            for (uint32_t p = p_lo; p < p_hi; ++p) exact(st, p);
        }
        const uint32_t in_bases = in & ~odd;
        uint32_t hs[kRawCells], ls[kRawCells];
#pragma unroll
        for (int i = 0; i < kRawCells; ++i) {
            hs[i] = __funnelshift_r(h0, h1, P.shift[i]);
            ls[i] = __funnelshift_r(l0, l1, P.shift[i]);
        }
        for (uint32_t p = p_lo; p < p_hi; ++p) {
            const uint4 *q = reinterpret_cast<const uint4 *>(P.screen + p);
            uint32_t y[kRawCells];
#pragma unroll
            for (int i = 0; i < kRawCells / 4; ++i) {
                const uint4 a = __ldg(q + i), b = __ldg(q + kRawCells / 4 + i);
                y[4 * i] = (hs[4 * i] ^ a.x) | (ls[4 * i] ^ b.x);
                y[4 * i + 1] = (hs[4 * i + 1] ^ a.y) | (ls[4 * i + 1] ^ b.y);
                y[4 * i + 2] = (hs[4 * i + 2] ^ a.z) | (ls[4 * i + 2] ^ b.z);
                y[4 * i + 3] = (hs[4 * i + 3] ^ a.w) | (ls[4 * i + 3] ^ b.w);
            }
            uint32_t s1_, s2, s3, s4, s5, c1, c2, c3, c4, c5, t1, t2, d1, d2, b2, b3;
            raw_add(y[0], y[1], y[2], s1_, c1);
            raw_add(y[3], y[4], y[5], s2, c2);
            raw_add(y[6], y[7], y[8], s3, c3);
            raw_add(y[9], y[10], y[11], s4, c4);
            raw_add(s1_, s2, s3, s5, c5);
            const uint32_t b0 = s5 ^ s4, c6 = s5 & s4;
            raw_add(c1, c2, c3, t1, d1);
            raw_add(c4, c5, c6, t2, d2);
            const uint32_t b1 = t1 ^ t2, d3 = t1 & t2;
            raw_add(d1, d2, d3, b2, b3);
            uint32_t gt = b0 & ~P.kb[0];  // count > max_mm, from the low bit up
            gt = (b1 & ~P.kb[1]) | (~(b1 ^ P.kb[1]) & gt);
            gt = (b2 & ~P.kb[2]) | (~(b2 ^ P.kb[2]) & gt);
            gt = (b3 & ~P.kb[3]) | (~(b3 ^ P.kb[3]) & gt);
            uint32_t m = in_bases & ~gt;
            if (!m) continue;
            const uint4 f = __ldg(q + 2 * (kRawCells / 4));  // h, l, care
            for (; m; m &= m - 1) {
                const uint32_t o = __ffs(m) - 1;
                const uint32_t wh = __funnelshift_r(h0, h1, o), wl = __funnelshift_r(l0, l1, o);
                if ((int)__popc(((wh ^ f.x) | (wl ^ f.y)) & f.z) > P.max_mm) continue;
                words(p0 + o);
                exact(p0 + o, p);
            }
        }
    }
}

// (the scan's hit count is read here, so that the host waits once for both)
__global__ void raw_verify_kernel(GenomeDev G, const BatchDev *__restrict__ batches,
                                  const Hit *__restrict__ hits, uint32_t hit_cap, uint32_t L,
                                  Row *rows, uint64_t *keys, uint32_t *vals, uint32_t row_cap,
                                  Counters *ctr) {
    const uint32_t n_hits = min(*(volatile const uint32_t *)&ctr->hits, hit_cap);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_hits; i += gridDim.x * blockDim.x) {
        const Hit h = hits[i];
        const BatchDev B = batches[h.batch];
        const uint64_t sg = B.base + h.s_local;
        const uint64_t gbyte = sg >> 1;
        uint32_t lo = B.first, hi = B.first + B.nch;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (G.boff[mid] <= gbyte) lo = mid; else hi = mid;
        }
        const uint32_t k = lo;
        const uint64_t pos = G.start[k] + (sg - 2 * G.boff[k]);
        const bool end_chrom = (k == B.first + B.nch - 1) || G.start[k + 1] == 0;
        if (end_chrom && pos + L > G.end[k]) continue;
        const int kmm = (int)h.pad;
        const uint32_t r = atomicAdd(&ctr->rows, 1u);
        if (r >= row_cap) continue;  // counted: the host makes room and asks again
        rows[r] = Row{sg, B.base + B.valid, pos, k, h.pattern, (uint32_t)(kmm > 0 ? kmm : 0), 0};
        keys[r] = ((uint64_t)h.pattern << 34) | sg;
        vals[r] = r;
    }
}

__global__ void raw_len_kernel(GenomeDev G, const Row *__restrict__ rows, const uint32_t *order,
                               uint32_t n, uint32_t L, uint32_t *len) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const Row w = rows[order[i]];
        const uint32_t ni = G.name_idx[w.chunk];
        len[i] = (G.name_off[ni + 1] - G.name_off[ni]) + 1 + ndigits(w.pos) + 1 +
                 ndigits(w.pattern) + 3 + ndigits(w.mm) + 5 + L + 1 + L + 1;
    }
}

__global__ void raw_write_kernel(GenomeDev G, const Row *__restrict__ rows, const uint32_t *order,
                                 uint32_t n, uint32_t L, const RawPattern *__restrict__ pats,
                                 const uint64_t *off, char *text) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const Row w = rows[order[i]];
        const RawPattern &P = pats[w.pattern];
        const bool fwd = P.strand == 0;
        char *o = text + off[i];
        const uint32_t ni = G.name_idx[w.chunk];
        for (uint32_t c = G.name_off[ni]; c < G.name_off[ni + 1]; ++c) *o++ = G.names[c];
        *o++ = '\t';
        o = put_u64(o, w.pos);
        *o++ = '\t';
        o = put_u64(o, w.pattern);
        *o++ = '\t';
        *o++ = fwd ? '+' : '-';
        *o++ = '\t';
        o = put_u64(o, w.mm);
        *o++ = '\t';
        *o++ = '0';
        *o++ = '\t';
        *o++ = '0';
        *o++ = '\t';
        char *rna = o, *dna = o + L + 1;
        for (uint32_t c = 0; c < L; ++c) {
            const uint32_t sc = fwd ? c : L - 1 - c;
            const uint64_t gi = w.s_global + sc;
            uint8_t g = gi < w.clip ? nib(G.bit4, gi) : 0;
            if (g == 0xF) g = 0;
            uint8_t p = (uint8_t)((P.w[sc >> 3] >> (4 * (sc & 7))) & 0xF);
            if (!fwd) {
                g = dcomp4(g);
                p = dcomp4(p);
            }
            rna[c] = b4char(p);
            dna[c] = b4char(g);  // NUL for N and padding, as in the reference
        }
        o += L;
        *o++ = '\t';
        o += L;
        *o++ = '\n';
    }
}

}  // namespace

int Engine::run_raw(const Request &r, Result &out, Error &err, const SearchRange &range) {
    DeviceGenome &d = *dev_;
    const HostGenome &h = host_;
    const Bit4Tables &t = bit4();
    cudaStream_t s = d.stream;
    const uint32_t L = (uint32_t)r.filter.size();
    const auto hb = make_batches(h.n_chunks(), r.cps);
    std::vector<BatchDev> batches;
    std::vector<RawSeg> segs;
    uint64_t blocks = 0;
    for (size_t bi = 0; bi < hb.size(); ++bi) {
        const HostBatch &b = hb[bi];
        BatchDev x{};
        x.base = 2 * h.boff[b.first];
        x.valid = (uint32_t)(2 * (h.boff[b.last + 1] - h.boff[b.first]));
        x.first = (uint32_t)b.first;
        x.nch = (uint32_t)(b.last - b.first + 1);
        batches.push_back(x);
        const uint64_t c1 = b.has_head ? 2 * (h.boff[b.first + 1] - h.boff[b.first]) : 0;
        const uint64_t msmin = c1 > L - 1 ? c1 - (L - 1) : 0;  // search.rs:540-546
        RawSeg sg{};
        sg.lo = std::max(x.base + msmin, range.lo);
        sg.hi = std::min<uint64_t>(x.base + x.valid, range.hi);
        if (sg.hi <= sg.lo) continue;
        sg.base = x.base;
        sg.clip = x.base + x.valid;
        sg.blk_begin = blocks;
        sg.batch = (uint32_t)bi;
        blocks += (sg.hi - (sg.lo & ~31ull) + 31) / 32;
        segs.push_back(sg);
    }
    std::vector<RawPattern> pats;
    std::vector<RawScreen> screen;
    const size_t np = r.patterns.size(), nfwd = np / 2;
    for (size_t p = 0; p < np; ++p) {
        RawPattern rp{};
        rp.strand = p >= nfwd;
        RawScreen rf{};
        for (uint32_t c = 0; c < L; ++c) {
            const uint8_t v = t.str2b4[1][(uint8_t)r.patterns[p][c]];
            rp.w[c / 8] |= (uint32_t)v << (4 * (c % 8));
            if (c < 32 && v && !(v & (v - 1))) {
                const uint32_t cd = code2(v);
                rf.care |= 1u << c;
                rf.h |= ((cd >> 1) & 1u) << c;
                rf.l |= (cd & 1u) << c;
            }
        }
        pats.push_back(rp);
        screen.push_back(rf);
    }
    out = Result();
    if (segs.empty()) return kOk;
    // the screened cells, where all patterns share enough of them
    RawScreenParams sq{};
    uint32_t common = L <= 32 && r.max_mm <= kRawMaxK ? ~0u : 0u;
    for (const RawScreen &x : screen) common &= x.care;
    const bool screened = __builtin_popcount(common) >= kRawCells;
    if (screened) {
        for (int i = 0; i < kRawCells; ++i, common &= common - 1) {
            const uint32_t c = (uint32_t)__builtin_ctz(common);
            sq.shift[i] = c;
            for (RawScreen &x : screen) {
                x.ph[i] = (x.h >> c) & 1 ? ~0u : 0u;
                x.pl[i] = (x.l >> c) & 1 ? ~0u : 0u;
            }
        }
        for (int b = 0; b < 4; ++b) sq.kb[b] = (r.max_mm >> b) & 1 ? ~0u : 0u;
    }
    TablePack tp;
    const size_t o_b = tp.add(batches), o_s = tp.add(segs), o_p = tp.add(pats), o_f = tp.add(screen);
    if (d.tables.ensure(tp.buf.size(), err)) return err.code;
    CU(cudaMemcpyAsync(d.tables.p, tp.buf.data(), tp.buf.size(), cudaMemcpyHostToDevice, s));
    auto tab = [&](size_t o) { return (const void *)(d.tables.p + o); };
    if (d.ctr.ensure(1, err)) return err.code;
    if (d.hits.cap == 0 && d.hits.ensure(1u << 22, err)) return err.code;
    Counters hc{};
    for (int attempt = 0; attempt < 2; ++attempt) {
        CU(cudaMemsetAsync(d.ctr.p, 0, sizeof(Counters), s));
        CU(cudaEventRecord(d.ev[1], s));
        const uint32_t hit_cap = (uint32_t)std::min<size_t>(d.hits.cap, 0xFFFFFFF0u);
        if (screened) {
            const uint64_t pw = d.n_words + 1;
            sq.bit4 = d.bit4.p;
            sq.H = d.planes.p;
            sq.L = d.planes.p + pw;
            sq.S = d.planes.p + 2 * pw;
            sq.segs = (const RawSeg *)tab(o_s);
            sq.pats = (const RawPattern *)tab(o_p);
            sq.screen = (const RawScreen *)tab(o_f);
            sq.hits = d.hits.p;
            sq.ctr = d.ctr.p;
            sq.n_blocks = blocks;
            sq.nseg = (uint32_t)segs.size();
            sq.npat = (uint32_t)np;
            sq.len = L;
            sq.cap = hit_cap;
            sq.max_mm = (int)r.max_mm;
            const unsigned gb = (unsigned)std::max<uint64_t>(
                1, std::min<uint64_t>((blocks + 255) / 256, (uint64_t)d.n_sm * 32));
            // small genomes: the patterns split over blocks, to fill the GPU (whole
            // call of 50 kb x 12 patterns: 0.118 ms, 0.139 without, 0.127 with
            // raw_scan_kernel)
            const unsigned gy = (unsigned)std::max<size_t>(
                1, std::min<size_t>(np, (size_t)d.n_sm * 8 / gb));
            raw_screen_kernel<<<dim3(gb, gy), 256, 0, s>>>(sq);
        } else {
            const uint64_t items = blocks * np;
            const unsigned gb = (unsigned)std::max<uint64_t>(
                1, std::min<uint64_t>((items + 255) / 256, (uint64_t)d.n_sm * 16));
            auto scan_fn = L > 32 ? raw_scan_kernel<8> : raw_scan_kernel<4>;
            scan_fn<<<gb, 256, 0, s>>>(d.bit4.p, (const RawSeg *)tab(o_s), (uint32_t)segs.size(), blocks,
                                       (const RawPattern *)tab(o_p), (uint32_t)np, L, (int)r.max_mm,
                                       d.hits.p, hit_cap, d.ctr.p);
        }
        CU(cudaGetLastError());
        CU(cudaEventRecord(d.ev[2], s));
        // room for the rows of most calls; a call with more is verified again
        for (size_t room = size_t(1) << 12;; room = (size_t)hc.rows + 1) {
            if (d.rows.ensure(room, err) || d.keys.ensure(room, err) || d.keys2.ensure(room, err) ||
                d.vals.ensure(room, err) || d.vals2.ensure(room, err))
                return err.code;
            const uint32_t row_cap = (uint32_t)std::min<size_t>(
                std::min({d.rows.cap, d.keys.cap, d.keys2.cap, d.vals.cap, d.vals2.cap}), 0xFFFFFFF0u);
            raw_verify_kernel<<<d.n_sm * 8, 256, 0, s>>>(d.view(), (const BatchDev *)tab(o_b), d.hits.p,
                                                         hit_cap, L, d.rows.p, d.keys.p, d.vals.p,
                                                         row_cap, d.ctr.p);
            CU(cudaGetLastError());
            ++times_.kernel_launches;
            CU(cudaMemcpyAsync(&hc, d.ctr.p, sizeof(Counters), cudaMemcpyDeviceToHost, s));
            CU(cudaStreamSynchronize(s));
            if (hc.rows <= row_cap) break;
            CU(cudaMemsetAsync(&d.ctr.p->rows, 0, sizeof(uint32_t), s));
        }
        ++times_.kernel_launches;
        if (!hc.overflow && hc.hits <= d.hits.cap) break;
        if (attempt == 1) {
            err = {kOom, "raw match buffer overflow after resize"};
            return err.code;
        }
        if (d.hits.ensure((size_t)hc.hits + hc.hits / 4 + 1024, err)) return err.code;
    }
    float ms = 0;
    cudaEventElapsedTime(&ms, d.ev[1], d.ev[2]);
    times_.scan_ms += ms;
    times_.raw_hits += hc.hits;
    const uint32_t nr = hc.rows;
    times_.rows += nr;
    if (!nr) return kOk;
    if (d.lens.ensure(nr + 1, err) || d.offs.ensure(nr + 1, err)) return err.code;
    // pattern << 34 | start: the bits in use
    int key_bits = 34;
    while (key_bits < 64 && (np >> (key_bits - 34))) ++key_bits;
    size_t tmp = 0, tmp2 = 0;
    CU(cub::DeviceRadixSort::SortPairs(nullptr, tmp, d.keys.p, d.keys2.p, d.vals.p, d.vals2.p,
                                       (int)nr, 0, key_bits, s));
    CU(cub::DeviceScan::ExclusiveSum(nullptr, tmp2, d.lens.p, d.offs.p, (int)nr + 1, s));
    if (d.cub_tmp.ensure(std::max(tmp, tmp2), err)) return err.code;
    tmp = d.cub_tmp.cap;
    CU(cub::DeviceRadixSort::SortPairs(d.cub_tmp.p, tmp, d.keys.p, d.keys2.p, d.vals.p, d.vals2.p,
                                       (int)nr, 0, key_bits, s));
    const unsigned fb = (unsigned)std::min<uint64_t>((nr + 255) / 256, (uint64_t)d.n_sm * 8);
    raw_len_kernel<<<fb, 256, 0, s>>>(d.view(), d.rows.p, d.vals2.p, nr, L, d.lens.p);
    CU(cudaGetLastError());
    CU(cudaMemsetAsync(d.lens.p + nr, 0, 4, s));
    tmp2 = d.cub_tmp.cap;
    CU(cub::DeviceScan::ExclusiveSum(d.cub_tmp.p, tmp2, d.lens.p, d.offs.p, (int)nr + 1, s));
    uint64_t bytes = 0;
    CU(cudaMemcpyAsync(&bytes, d.offs.p + nr, 8, cudaMemcpyDeviceToHost, s));
    CU(cudaStreamSynchronize(s));
    if (d.text.ensure(bytes + 1, err)) return err.code;
    raw_write_kernel<<<fb, 256, 0, s>>>(d.view(), d.rows.p, d.vals2.p, nr, L,
                                        (const RawPattern *)tab(o_p), d.offs.p, d.text.p);
    CU(cudaGetLastError());
    times_.kernel_launches += 4;
    out.owned.resize(bytes);
    CU(cudaMemcpyAsync(&out.owned[0], d.text.p, bytes, cudaMemcpyDeviceToHost, s));
    CU(cudaStreamSynchronize(s));
    out.text = out.owned.data();
    out.text_len = bytes;
    out.n_rows = nr;
    return kOk;
}

}  // namespace cof
