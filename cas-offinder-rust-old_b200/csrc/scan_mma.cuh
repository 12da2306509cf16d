// scan_mma.cuh -- the popcount scan's window x pattern comparison as a matrix
// product on the tensor cores (tcgen05, sm_100a).  Included by engine.cu after
// the scan's device structures.
//
// A base's 2-bit code (H, L) is written as the three signs (-1)^H, (-1)^L and
// (-1)^(H^L).  The product of two bases' sign triples is 3 when they are equal
// and -1 when they differ, so over the c cells that a pattern compares, m of
// them equal, the dot product is 4m - c.  A pattern row carries a bias of
// -(3c - 4k - 2) beside its signs: the sum is at least 2 exactly when at most
// k cells differ, and at most -2 otherwise.  A hit is an accumulator whose
// sign bit is clear.  Signs are the e4m3 bytes 0x38 and 0xB8, cells that a
// pattern does not compare are 0, the bias sits in spare columns as one
// multiple of 16 and one whole number up to 15 (both exact in e4m3), and
// every partial sum of 96 such products is a whole number below 2048, exact in
// the 16-bit accumulators that halve the registers to read.
//
// Cells that are no single base (S plane) are tested in the PAM only; in a
// guide they count by whatever code their union of bits gives, never less
// equal than the writer's recount takes them.  So the hits are a superset of
// the rows, as those of the other scan kernels, and verify_kernel decides.  Windows
// without a base, which a guide of one base repeated would meet by the code of N,
// are left out where no PAM cell does it (100 Mbp with 5 Mbp of N, 100 guides of an
// all-N filter, one with 15 Ts: 72 k hits instead of 5.1 M).
//
// Why: a POPC compares one window with one pattern and the XU pipe does 16 per
// SM and clock; products of 128 windows, 64 patterns and K = 64 take 106 clocks each
// back to back (intpeak.cu), 77 comparisons per clock.  Scan of 100 Mbp, NRG, against
// the POPC scan: 64 guides 0.328 ms (0.456), 100 0.441 (0.656), 200 0.665 (1.182), 400
// 1.037 (2.215), 1200 2.043 (7.334; 41 comparisons per SM and clock).  What bounds it:
// with hundreds of patterns the products and the wait for each; at 100 the issue of
// what a row block costs before any comparison (of 436 warp instructions per 32
// windows, about 160 to find and list them, 70 to write them as rows, 110 to read
// the accumulators; 66 % of the issue slots, the tensor pipe busy 17 % of the time).
// A team finds its windows together: when each of its warps walked tiles of its
// own, one of the four nearly always had a new tile to test while the others
// waited for its rows (40 % of all warp time; 0.494 and 2.34 ms at 100 and 1200
// guides, 0.424 and 2.00 together).
// Tried and slower than those: one CTA of four warps per 128 accumulator columns
// (0.62 ms at 100 guides), producer, issuer and reader warps apart with a ring of row
// tiles (0.72: an instruction of one warp takes about 13 clocks, so the few
// issuers and readers set the pace), 128 columns shared by two teams (0.52, and
// 3.1 ms at 1200 guides), a ring of windows drained by ballots instead of the
// list of starts (0.535 and 2.57, with tiles per warp), and taking the next
// block's windows while a product runs (0.447 and 2.18: the registers it holds
// spill, and the next columns' product starts later).
#pragma once

#include <cstdint>

#include "mma_f8.cuh"

namespace cof {

// One CTA per SM of eight teams of four warps.  A team's warps drain PAM-passing
// starts into a row block of 32 windows each; the four blocks are the 128 rows
// of a product, and each warp reads the accumulators of its own rows.  The
// teams share the group's pattern rows.
constexpr uint32_t kMmaTeams = 8;
constexpr uint32_t kMmaWarps = 4 * kMmaTeams;
constexpr int kMmaThreads = 32 * kMmaWarps;
constexpr uint32_t kMmaCols = 64;     // columns of a team's accumulator
constexpr uint32_t kMmaWaitLimit = 1u << 22;  // polls of a barrier before giving up

// A set of patterns: one strand of every request whose filter has the same non-N
// cells at the same place, over all batches (a ScanGroup without its split into
// care classes and runs of segments), or a part of a large one.
struct MmaGroup {
    uint32_t n_pam, pat_begin, pat_end, seg_begin, seg_end;
    uint32_t cell0;  // window cell of the first compared cell
    uint32_t b_off;  // byte offset of the group's pattern rows in MmaParams::bmat
    uint32_t n_pad;  // pattern rows, a multiple of 16
    PamCell pam[kMaxPamCells];
};

struct MmaParams {
    const uint32_t *H, *L, *S;
    const MmaGroup *groups;
    const ScanSeg *segs;         // of the groups, tiles counted from each one's first
    const uint64_t *item_begin;  // per group: first work item; [n_groups] = total
    uint32_t n_groups;
    uint32_t span_tiles;         // 1024-start tiles per work item
    const unsigned char *bmat;   // the groups' pattern rows
    uint32_t rows;               // most pattern rows of a group
    uint32_t hit_cap;
    const uint32_t *pat_off;     // window offset of each pattern's first cell
    Hit *hits;
    Counters *ctr;
};

// K = 32 columns per instruction: two steps hold 20 cells (60 signs and four
// spare columns), three hold 31 (93 and three)
__host__ __device__ constexpr uint32_t mma_cells(int steps) { return steps == 2 ? 20u : 31u; }
// most pattern rows of a group: what shared memory holds beside the windows
constexpr uint32_t mma_pats(int steps) { return steps == 2 ? 1216u : 608u; }
// byte offsets in shared memory with `rows` pattern rows: the teams' window
// rows, the patterns, and per team the step's words (H, L pairs) and the places
// of its PAM-passing starts
struct MmaLayout {
    uint32_t a, b, words, ent, total;
};
__host__ __device__ inline MmaLayout mma_layout(int steps, uint32_t rows) {
    MmaLayout o{};
    o.a = 0;
    o.b = o.a + kMmaTeams * 128 * 32 * steps;
    o.words = o.b + rows * 32 * steps;
    o.ent = o.words + kMmaTeams * 130 * 8;
    o.total = o.ent + kMmaTeams * 4096 * 2;
    return o;
}

// Column (K index) of sign bit p: a window's sign bits are spread over its
// row by word i = (v << i) & 0x80808080, so bit 8 b + 7 - i of a 32-bit
// group is byte b of word i.
constexpr uint32_t mma_column(uint32_t p) {
    return 32 * (p / 32) + 4 * (7 - p % 8) + (p % 32) / 8;
}
// sign bit of plane d (H, L, H ^ L) of compared cell c, and spare bit j
constexpr uint32_t mma_bit(int steps, uint32_t d, uint32_t c) {
    return steps == 2 ? 20 * d + c : 32 * d + c;
}
constexpr uint32_t mma_spare(int steps, uint32_t j) { return steps == 2 ? 60 + j : 31 + 32 * j; }

// e4m3 of a whole number of at most 15, or of a multiple of 16 up to 240
inline uint8_t e4m3(int v) {
    const uint8_t sign = v < 0 ? 0x80 : 0;
    uint32_t a = (uint32_t)(v < 0 ? -v : v);
    if (!a) return sign;
    uint32_t e = 0;
    while ((a >> e) > 1) ++e;
    const uint32_t frac = e >= 3 ? (a >> (e - 3)) & 7 : (a << (3 - e)) & 7;
    return (uint8_t)(sign | ((e + 7) << 3) | frac);
}

// Writes the row of pattern `row` into a group's B operand of n_pad rows:
// 16-byte pieces, each piece's rows one after the other (the K-major layout
// without swizzle whose 8 x 16-byte core matrices are contiguous).  h, l:
// 2-bit code bits; care: compared cells; both shifted so that cell 0 is bit 0.
inline void mma_pattern_row(uint8_t *b, uint32_t n_pad, uint32_t row, int steps, uint32_t h,
                            uint32_t l, uint32_t care, int k) {
    auto put = [&](uint32_t p, uint8_t v) {
        const uint32_t col = mma_column(p);
        b[(size_t)(col / 16) * n_pad * 16 + row * 16 + col % 16] = v;
    };
    int c = 0;
    for (uint32_t i = 0; i < mma_cells(steps); ++i) {
        if (!((care >> i) & 1)) continue;
        ++c;
        const uint32_t hb = (h >> i) & 1, lb = (l >> i) & 1;
        put(mma_bit(steps, 0, i), hb ? 0xB8 : 0x38);
        put(mma_bit(steps, 1, i), lb ? 0xB8 : 0x38);
        put(mma_bit(steps, 2, i), hb ^ lb ? 0xB8 : 0x38);
    }
    const int bias = -(3 * c - 4 * k - 2);
    const int whole = bias / 16 * 16;  // toward zero: the rest is below 16
    put(mma_spare(steps, 0), e4m3(whole));
    put(mma_spare(steps, 1), e4m3(bias - whole));
}
// a padding row: no cell, a negative bias
inline void mma_padding_row(uint8_t *b, uint32_t n_pad, uint32_t row, int steps) {
    const uint32_t col = mma_column(mma_spare(steps, 0));
    b[(size_t)(col / 16) * n_pad * 16 + row * 16 + col % 16] = e4m3(-16);
}

// the votes of a team's 128 threads at their barrier.  (The aligned forms want a
// warp's lanes together; what comes before may have parted them.)
__device__ __forceinline__ uint32_t team_count(uint32_t team, bool vote) {
    uint32_t n;
    __syncwarp();
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t"
        "barrier.cta.red.popc.aligned.u32 %0, %1, 128, p;\n\t}"
        : "=r"(n)
        : "r"(team + 1), "r"((uint32_t)vote)
        : "memory");
    return n;
}

__device__ __forceinline__ void team_sync(uint32_t team) {
    __syncwarp();
    asm volatile("barrier.cta.sync.aligned %0, 128;" ::"r"(team + 1) : "memory");
}

// The warp's 32 lanes of 16, 32 or 64 accumulator columns, two columns (f16) per
// register.  Load and wait are one statement, so that no use of the registers
// can move between them.
__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t *r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.pack::16b.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7])
        : "r"(addr));
}
__device__ __forceinline__ void tmem_ld32(uint32_t addr, uint32_t *r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.pack::16b.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
        "[%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr));
}
__device__ __forceinline__ void tmem_ld64(uint32_t addr, uint32_t *r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.pack::16b.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, "
        "%18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, "
        "[%32];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
          "=r"(r[31])
        : "r"(addr));
}
// the AND of n registers, as four chains
template <int n>
__device__ __forceinline__ uint32_t and_all(const uint32_t *r) {
    uint32_t v[4] = {r[0] & r[1], r[2] & r[3], r[4] & r[5], r[6] & r[7]};
#pragma unroll
    for (int j = 8; j < n; j += 8)
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = v[k] & r[j + 2 * k] & r[j + 2 * k + 1];
    return v[0] & v[1] & v[2] & v[3];
}

// Bit b: none of the cells b .. b + 31 of two S words is a base.
__device__ __forceinline__ uint32_t mma_no_base(uint32_t s0, uint32_t s1) {
    uint64_t z = ((uint64_t)s1 << 32) | s0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) z &= z >> o;
    return (uint32_t)z;
}

// Appends the hits of a warp's 32 rows in n (a multiple of 16, at most 64)
// accumulator columns of patterns pat .. pat + n.  Reads the columns again: few
// row blocks have a hit, and the others need not keep their registers.
__device__ __forceinline__ void mma_hits(const MmaParams &P, uint32_t tmem, uint32_t n, bool dead,
                                      uint32_t pat, uint32_t row_off, uint32_t batch) {
#pragma unroll 1
    for (uint32_t c = 0; c < n; c += 16) {
        uint32_t r[8];
        tmem_ld16(tmem + c, r);
        uint32_t mk = 0;  // bit 2 j + 16 k: half k of register j, column 2 j + k
        if (!dead && (~and_all<8>(r) & 0x80008000u)) {
#pragma unroll
            for (int j = 0; j < 8; ++j) mk |= (~r[j] & 0x80008000u) >> (15 - 2 * j);
        }
        for (; mk; mk &= mk - 1) {
            const uint32_t b = __ffs(mk) - 1;
            const uint32_t p = pat + c + (b & 15) + (b >> 4);
            const uint32_t i = atomicAdd(&P.ctr->hits, 1u);
            if (i < P.hit_cap) P.hits[i] = Hit{row_off + __ldg(P.pat_off + p), p, batch, 0};
            else P.ctr->overflow = 1;
        }
        __syncwarp();  // every lane, hit or not, before the next aligned load
    }
}

// the row words of 32 sign bits: bytes +1 or -1
__device__ __forceinline__ void mma_spread(uint32_t v, uint4 &a, uint4 &b) {
    auto word = [v](int i) { return ((v << i) & 0x80808080u) | 0x38383838u; };
    a = make_uint4(word(0), word(1), word(2), word(3));
    b = make_uint4(word(4), word(5), word(6), word(7));
}

// Persistent scan over strand groups, group by group (a CTA takes the first
// group that any of its teams holds a work item of).
//
// Each team takes work items (spans of tiles), four 1024-start tiles a step, one
// per warp: the lanes test their 32 starts' PAM cells and list the passing
// starts at places from a prefix sum over the team.  The listed windows are
// taken 128 at a time, one per thread (windows left over wait in the threads'
// registers for the next step's), and written as the rows of the team's operand.
// One thread multiplies them with the group's pattern rows, kMmaCols at a time,
// and the warps combine the sign bits of their rows' accumulators; only a block
// with a hit looks at single columns.  While a team waits for its product, the
// others work.  A warp that does not see its product in kWaitLimit polls waits,
// reads and multiplies no more; the team leaves at the vote before its next row
// block, the CTA at the group's end.  (A vote at every product cost 4 % of the scan
// with 1,200 patterns, a limit from the parameters 2 %.)
template <int kSteps, uint32_t kWaitLimit>
__global__ void __launch_bounds__(kMmaThreads, 1)
scan_mma_kernel(const __grid_constant__ MmaParams P) {
    constexpr uint32_t kPieces = 2 * kSteps;
    extern __shared__ __align__(128) unsigned char mma_smem_raw[];
    const MmaLayout lay = mma_layout(kSteps, P.rows);
    __shared__ uint4 s_cm[kMaxPamCells];
    __shared__ uint32_t s_ci[kMaxPamCells];
    __shared__ __align__(8) uint64_t s_done[kMmaTeams];  // a team's product is there
    __shared__ uint4 s_count[kMmaTeams];     // passing starts of the step's four tiles
    __shared__ unsigned long long s_item[kMmaTeams];
    __shared__ uint32_t s_tmem, s_next[kMmaTeams];
    __shared__ int s_bad;

    const uint32_t full = 0xFFFFFFFFu;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, team = warp >> 2,
                   q = warp & 3, row = tid & 127;
    unsigned char *sA = mma_smem_raw + lay.a + team * (kPieces * 128 * 16),
                  *sB = mma_smem_raw + lay.b;
    uint2 *words = reinterpret_cast<uint2 *>(mma_smem_raw + lay.words) + team * 130;
    uint16_t *ent = reinterpret_cast<uint16_t *>(mma_smem_raw + lay.ent) + team * 4096;
    const uint32_t done = (uint32_t)__cvta_generic_to_shared(&s_done[team]);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(&s_tmem)),
                     "r"(kMmaCols * kMmaTeams)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) s_bad = 0;
    if (tid < kMmaTeams) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(&s_done[tid]))
                     : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem + team * kMmaCols, tmem_row = tmem + ((q * 32) << 16);

    // the team's work item: tiles [t, t_end) of group ig
    const uint64_t total_items = P.item_begin[P.n_groups];
    uint64_t t = 0, t_end = 0;
    unsigned long long ahead = 0;  // row 0: the item after it, asked for early
    if (row == 0) ahead = atomicAdd(&P.ctr->mma_next, 1ull);
    uint32_t ig = P.n_groups, sidx = 0, phase = 0;
    bool bad = false;  // the warp gave up a wait
    // (between two calls the team meets at a step's barriers)
    auto fetch = [&]() {
        if (row == 0) {
            s_item[team] = ahead;
            ahead = atomicAdd(&P.ctr->mma_next, 1ull);
        }
        team_sync(team);
        const uint64_t it = s_item[team];
        ig = P.n_groups;
        if (it >= total_items) return;
        uint32_t lo = 0, hi = P.n_groups;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (__ldg(P.item_begin + mid) <= it) lo = mid; else hi = mid;
        }
        ig = lo;
        const ScanSeg &last = P.segs[P.groups[ig].seg_end - 1];
        const uint64_t tiles = last.tile_begin + ((last.hi - last.w0 * 32 + 1023) >> 10);
        t = (it - __ldg(P.item_begin + lo)) * P.span_tiles;
        t_end = min(t + P.span_tiles, tiles);
        const ScanSeg *segs = P.segs + P.groups[ig].seg_begin;
        sidx = 0;  // the segment of tile t
        for (uint32_t end = P.groups[ig].seg_end - P.groups[ig].seg_begin; end - sidx > 1;) {
            const uint32_t mid = (sidx + end) >> 1;
            if (segs[mid].tile_begin <= t) sidx = mid; else end = mid;
        }
    };
    fetch();

    for (;;) {
        if (row == 0) s_next[team] = ig;
        __syncthreads();
        const uint32_t cur = __reduce_min_sync(full, s_next[lane % kMmaTeams]);
        if (cur >= P.n_groups || *(volatile int *)&s_bad) break;
        const MmaGroup &G = P.groups[cur];
        const uint32_t n_pam = G.n_pam, n_pad = G.n_pad, cell0 = G.cell0;
        {
            const uint4 *src = reinterpret_cast<const uint4 *>(P.bmat + G.b_off);
            uint4 *dst = reinterpret_cast<uint4 *>(sB);
            for (uint32_t i = tid; i < n_pad * kPieces; i += kMmaThreads) dst[i] = __ldg(src + i);
            if (tid < n_pam) {
                const PamCell c = G.pam[tid];
                s_cm[tid] = make_uint4(c.fa, c.fc, c.fg, c.ft);
                s_ci[tid] = c.cell;
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();

        const uint32_t desc_a = mma_desc((uint32_t)__cvta_generic_to_shared(sA), 2048),
                       desc_b = mma_desc((uint32_t)__cvta_generic_to_shared(sB), n_pad * 16);
        // the current run of tiles (of one segment) and the lane's place in it
        uint32_t run = 0, pos = 0, seg_lo = 0, seg_hi = 0, offb = 0, sbatch = 0;
        uint64_t w = 0;
        auto next_run = [&]() -> bool {
            if (ig != cur) return false;
            if (t >= t_end) {
                fetch();
                if (ig != cur) return false;
            }
            const ScanSeg *segs = P.segs + G.seg_begin;
            const uint32_t nseg = G.seg_end - G.seg_begin;
            while (sidx + 1 < nseg && t >= segs[sidx + 1].tile_begin) ++sidx;
            const ScanSeg &sg = segs[sidx];
            uint64_t e = t_end;
            if (sidx + 1 < nseg) e = min(e, segs[sidx + 1].tile_begin);
            run = (uint32_t)(e - t);
            const uint64_t p0s = sg.w0 * 32;
            pos = (uint32_t)(t - sg.tile_begin) * 1024u;
            seg_lo = (uint32_t)(sg.lo - p0s);
            seg_hi = (uint32_t)(sg.hi - p0s);
            offb = (uint32_t)(p0s - sg.base);
            sbatch = sg.batch;
            w = sg.w0 + (t - sg.tile_begin) * 32 + row;
            t = e;
            return true;
        };

        uint32_t left = 0, at = 0, off0 = 0;  // the step's list: entries left, the next one
        uint32_t qbatch = 0xFFFFFFFFu, ncand = 0;
        for (;;) {
            // -- the next row block: 128 windows, one per thread (n, left and the
            // run are the same in all of the team's threads)
            uint32_t n = 0, row_off = 0, h = 0, l = 0;
            while (n < 128) {
                if (!left) {
                    if (run == 0 && !next_run()) break;
                    if (sbatch != qbatch) {  // a row block is of one batch
                        if (n) break;
                        qbatch = sbatch;
                    }
                    const bool on = q < run;  // the warp has a tile
                    uint32_t m = 0, h0 = 0, h1 = 0, l0 = 0, l1 = 0;
                    if (on) {
                        h0 = __ldg(P.H + w), h1 = __ldg(P.H + w + 1);
                        l0 = __ldg(P.L + w), l1 = __ldg(P.L + w + 1);
                        const uint32_t s0 = __ldg(P.S + w), s1 = __ldg(P.S + w + 1);
                        m = pos >= seg_lo && pos + 4096u <= seg_hi
                                ? full
                                : range_mask32(pos + row * 32u, seg_lo, seg_hi);
                        m = pam_mask_staged(s_cm, s_ci, n_pam, m, h0, h1, l0, l1, s0, s1);
                        // (no PAM to turn down a run of N: windows of nothing else)
                        if (!n_pam) m &= ~mma_no_base(s0, s1);
                        if (q + 4 < run) {  // the next step's words
                            asm volatile("prefetch.global.L1 [%0];" ::"l"(P.H + w + 128));
                            asm volatile("prefetch.global.L1 [%0];" ::"l"(P.L + w + 128));
                            asm volatile("prefetch.global.L1 [%0];" ::"l"(P.S + w + 128));
                        }
                    }
                    const uint32_t k = __popc(m);
                    uint32_t incl = k;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const uint32_t y = __shfl_up_sync(full, incl, o);
                        if ((int)lane >= o) incl += y;
                    }
                    if (lane == 31) reinterpret_cast<uint32_t *>(&s_count[team])[q] = incl;
                    team_sync(team);  // the counts are there, the list before is used up
                    const uint4 c4 = s_count[team];
                    const uint32_t c01 = c4.x + c4.y, c012 = c01 + c4.z;
                    uint16_t *e = ent + (incl - k) + (q == 0 ? 0u : q == 1 ? c4.x : q == 2 ? c01 : c012);
                    if (on) {
                        words[row] = make_uint2(h0, l0);
                        if (lane == 31 && (q == 3 || q + 1 == run)) words[row + 1] = make_uint2(h1, l1);
                    }
                    for (; m; ++e) {
                        const uint32_t b = 31 - __clz(m);
                        m ^= 1u << b;
                        *e = (uint16_t)(row * 32 + b);
                    }
                    left = c012 + c4.w;
                    at = 0;
                    ncand += left;
                    off0 = offb + pos;
                    pos += 4096u;
                    w += 128;
                    run -= min(run, 4u);
                    team_sync(team);  // the list is there
                    continue;
                }
                const uint32_t take = min(128u - n, left);
                if (row - n < take) {
                    const uint32_t p = ent[at + row - n];
                    const uint2 x = words[p >> 5], y = words[(p >> 5) + 1];
                    row_off = off0 + p;
                    h = __funnelshift_r(x.x, y.x, p);
                    l = __funnelshift_r(x.y, y.y, p);
                }
                n += take;
                at += take;
                left -= take;
            }
            if (!n) break;
            // -- its rows: sign bits spread to e4m3 bytes
            {
                h >>= cell0;
                l >>= cell0;
                uint32_t v[3];
                if (kSteps == 2) {
                    v[0] = (h & 0xFFFFFu) | (l << 20);
                    v[1] = ((l >> 12) & 0xFFu) | (((h ^ l) << 8) & 0x0FFFFF00u);
                } else {
                    v[0] = h & 0x7FFFFFFFu;
                    v[1] = l & 0x7FFFFFFFu;
                    v[2] = (h ^ l) & 0x7FFFFFFFu;
                }
                uint4 *dst = reinterpret_cast<uint4 *>(sA) + row;
#pragma unroll
                for (int s = 0; s < kSteps; ++s)
                    mma_spread(v[s], dst[2 * s * 128], dst[(2 * s + 1) * 128]);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
            if (team_count(team, bad)) {
                s_bad = 1;
                break;
            }
            const bool dead = row >= n;
            for (uint32_t c = 0; c < n_pad; c += kMmaCols) {
                const uint32_t cols = min(kMmaCols, n_pad - c);
                // (warps of one q share a scheduler: the teams' issuers differ in it)
                if (q == (team & 3)) {
                    if (lane == 0) {
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const uint32_t idesc = mma_f8_desc(cols);
                        const uint32_t db = desc_b + c;
                        mma_f8<false>(tmem, desc_a, db, idesc);
#pragma unroll
                        for (int s = 1; s < kSteps; ++s)
                            mma_f8<true>(tmem, desc_a + s * 256, db + s * 2 * n_pad, idesc);
                        mma_commit(done);
                    }
                    __syncwarp();
                }
                if (!mma_wait(done, phase, kWaitLimit)) {
                    // given up: the warp only keeps the team's barriers, and issues
                    // no product into an accumulator that this one may still write
                    bad = true;
                    for (; c + kMmaCols < n_pad; c += kMmaCols) team_count(team, false);
                    break;
                }
                phase ^= 1;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (q * 32 < n) {
                    uint32_t v = ~0u;
                    if (cols == 64) {
                        uint32_t r[32];
                        tmem_ld64(tmem_row, r);
                        v = and_all<32>(r);
                    } else {
                        if (cols & 32) {
                            uint32_t r[16];
                            tmem_ld32(tmem_row, r);
                            v = and_all<16>(r);
                        }
                        if (cols & 16) {
                            uint32_t r[8];
                            tmem_ld16(tmem_row + (cols & 32), r);
                            v &= and_all<8>(r);
                        }
                    }
                    if (__any_sync(full, (~v & 0x80008000u) && !dead))
                        mma_hits(P, tmem_row, cols, dead, G.pat_begin + c, row_off, qbatch);
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                // the next columns' product overwrites the accumulator
                if (c + kMmaCols < n_pad) team_count(team, false);
            }
        }
        if (row == 0 && ncand) {
            atomicAdd(&P.ctr->candidates, (unsigned long long)ncand);
            atomicAdd(&P.ctr->pairs, (unsigned long long)ncand * (G.pat_end - G.pat_begin));
        }
        if (bad) s_bad = 1;
        __syncthreads();  // every team is done with the group
    }
    if (tid == 0 && s_bad) P.ctr->fault = 1;
    // the product that the issuing warp gave up on may still write the team's
    // accumulator: it is waited for once more before the TMEM goes back
    if (bad && q == (team & 3)) mma_wait(done, phase, kMmaWaitLimit);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(s_tmem),
                     "r"(kMmaCols * kMmaTeams));
    }
}

}  // namespace cof
