// noalloc.cu -- popcount search over one caller-resident sequence that
// allocates no memory (cof_search_seq_noalloc, declared in include/cof.h).
//
// Some callers cannot call cudaMalloc: a host application that owns the whole
// device memory through its own pool allocator and only hands out pointers
// into it (an allocation from this library would bypass its accounting or
// fail once the pool holds the memory), or a serving process that must not
// allocate on its request path because an allocation can synchronise the
// device and stall unrelated work.  This entry point takes the caller's device
// buffers for its input (the bit4 sequence) and its output (the rows), and keeps
// everything else -- counters, pattern tables, the candidate list -- in one
// fixed file-scope device array, `g_noalloc_scratch`, that exists on every GPU
// that loads libcof.so until the process exits.
//
// It is a variant of the genome scan of engine.cu (same PAM prefilter and
// popcount lower bound, same exact decision of the reference writer,
// search.rs:378-463 + main.rs:159-222) restricted to a single record: every
// window start s with s + L <= n_nucl, the record-end drop of
// convert_matches (search.rs:1449-1454).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstring>
#include <mutex>
#include <string>

#include "../../include/cof.h"
#include "cof_engine.h"

namespace {

constexpr uint32_t kNaMaxPatterns = 512;                 // fwd + reverse patterns
constexpr size_t kNaScratchBytes = 8u << 20;              // 8 MiB per GPU
constexpr size_t kNaCounterBytes = 256;
constexpr size_t kNaTableBytes = 32u << 10;
constexpr size_t kNaCandOffset = kNaCounterBytes + kNaTableBytes;
constexpr uint32_t kNaMaxCandidates =
    (uint32_t)((kNaScratchBytes - kNaCandOffset) / sizeof(uint2));  // 1,044,448
// rows a call may count before its 32-bit row counter could wrap
constexpr uint32_t kNaRowCountLimit = 0xFFFFFFF0u;

struct NaPam {
    uint32_t cell, fa, fc, fg, ft;
};
struct NaFast {
    uint32_t h, l, care;
    int32_t k;
};
struct NaTables {
    uint32_t L, n_fwd, n_pat, max_mm;
    uint32_t n_pam[2];
    uint32_t pad[2];
    NaPam pam[2][32];
    uint8_t fset[2][32];
    uint8_t fisn[2][32];
    NaFast fast[kNaMaxPatterns];
    uint8_t b4[kNaMaxPatterns][32];
};
static_assert(sizeof(NaTables) <= kNaTableBytes, "pattern tables exceed their scratch slot");

// counters: [0] candidates, [1] candidate overflow, [2] rows, [3] row-count
// overflow (the 32-bit row counter came within 16 of wrapping)
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNaScratchBytes];

__device__ __forceinline__ uint32_t na_gather(uint32_t v) {
    v &= 0x11111111u;
    v = (v | (v >> 3)) & 0x03030303u;
    v = (v | (v >> 6)) & 0x000F000Fu;
    return (v | (v >> 12)) & 0xFFu;
}

// H / L / S plane words of nucleotides [32w, 32w + 32); bytes past n_bytes
// read as padding (S set).
__device__ void na_planes(const uint8_t *bit4, uint64_t n_bytes, uint64_t w, uint32_t &h,
                          uint32_t &l, uint32_t &s) {
    uint32_t x[4] = {0, 0, 0, 0};
    const uint64_t b0 = 16 * w;
    if (b0 + 16 <= n_bytes) {
        const uint4 q = *reinterpret_cast<const uint4 *>(bit4 + b0);
        x[0] = q.x; x[1] = q.y; x[2] = q.z; x[3] = q.w;
    } else {
        for (int i = 0; i < 16; ++i)
            if (b0 + i < n_bytes) x[i >> 2] |= (uint32_t)bit4[b0 + i] << (8 * (i & 3));
    }
    h = l = s = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t v = x[j];
        uint32_t pc = v - ((v >> 1) & 0x55555555u);
        pc = (pc & 0x33333333u) + ((pc >> 2) & 0x33333333u);
        const uint32_t t = pc ^ 0x11111111u;
        h |= na_gather((v >> 3) | v) << (8 * j);
        l |= na_gather((v >> 1) | v) << (8 * j);
        s |= na_gather(t | (t >> 1) | (t >> 2)) << (8 * j);
    }
}

// One warp per run of kNaRun consecutive 1024-start tiles (a 32-nt word per
// lane).  The words are converted to planes once: a tile's neighbour words are
// the next lane's and, for lane 31, lane 0's of the next tile, which is
// converted one tile ahead.  PAM-passing starts are compacted into a queue per
// strand and warp, and every 128 queued windows are compared with the strand's
// patterns (staged in shared memory), four per lane.  Bound by issue: 50 Mnt x 8
// guides 0.201 ms a call (0.1 of it the caller's sort); converting each word twice
// and comparing each lane's starts in a loop of its own, with a second wait for
// the candidates, took 0.351.
constexpr uint32_t kNaWarps = 4;
constexpr uint32_t kNaRun = 4;
constexpr uint32_t kNaQueue = 128 + 32;  // one step adds at most 32

struct NaQueue {
    uint4 e[kNaQueue];  // start, H, L, S of the window
};

__device__ __forceinline__ void na_flush(const NaQueue &q, uint32_t n, const NaFast *fast, uint32_t pb,
                                         uint32_t pe, uint32_t *ctr, uint2 *cand, uint32_t lane) {
    uint32_t h[4], l[4], s[4];
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) {
        const uint32_t i = lane + 32 * j;
        const uint4 e = i < n ? q.e[i] : make_uint4(0, 0, 0, 0xFFFFFFFFu);
        h[j] = e.y;
        l[j] = e.z;
        s[j] = e.w;
    }
    for (uint32_t p = pb; p < pe; ++p) {
        const NaFast f = fast[p];
        int m[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) m[j] = __popc(((h[j] ^ f.h) | (l[j] ^ f.l) | s[j]) & f.care);
        if (min(min(m[0], m[1]), min(m[2], m[3])) > f.k) continue;
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
            const uint32_t i = lane + 32 * j;
            if (i >= n || m[j] > f.k) continue;
            const uint32_t c = atomicAdd(&ctr[0], 1u);
            if (c < kNaMaxCandidates) cand[c] = make_uint2(q.e[i].x, p);
            else ctr[1] = 1;
        }
    }
}

__global__ void __launch_bounds__(kNaWarps * 32)
na_scan_kernel(const uint8_t *__restrict__ bit4, uint64_t n_bytes, uint32_t lo, uint32_t hi,
               unsigned char *scratch) {
    const NaTables &T = *reinterpret_cast<const NaTables *>(scratch + kNaCounterBytes);
    uint32_t *ctr = reinterpret_cast<uint32_t *>(scratch);
    uint2 *cand = reinterpret_cast<uint2 *>(scratch + kNaCandOffset);
    extern __shared__ __align__(16) unsigned char na_smem[];
    NaFast *fast = reinterpret_cast<NaFast *>(na_smem);
    const uint32_t n_pat = T.n_pat, n_fwd = T.n_fwd;
    NaQueue *queues = reinterpret_cast<NaQueue *>(fast + n_pat);
    __shared__ NaPam pam[2][32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, full = 0xFFFFFFFFu;
    const uint32_t lt_mask = (1u << lane) - 1u;
    for (uint32_t i = threadIdx.x; i < n_pat; i += blockDim.x) fast[i] = T.fast[i];
    if (threadIdx.x < 64) pam[threadIdx.x >> 5][lane] = T.pam[threadIdx.x >> 5][lane];
    __syncthreads();
    NaQueue *q = queues + 2 * warp;  // one per strand
    uint32_t qn[2] = {0, 0};
    const uint32_t np[2] = {T.n_pam[0], T.n_pam[1]};
    const uint64_t t_lo = lo / 1024, t_hi = ((uint64_t)hi + 1023) / 1024;
    const uint64_t warps = (uint64_t)gridDim.x * kNaWarps;
    for (uint64_t t0 = t_lo + (blockIdx.x * (uint64_t)kNaWarps + warp) * kNaRun; t0 < t_hi;
         t0 += warps * kNaRun) {
        const uint64_t t1 = min(t0 + kNaRun, t_hi);
        uint32_t nh, nl, ns;  // the tile ahead
        na_planes(bit4, n_bytes, 32 * t0 + lane, nh, nl, ns);
        for (uint64_t t = t0; t < t1; ++t) {
            const uint32_t h0 = nh, l0 = nl, s0 = ns;
            // (of the run's last tile only the first word of the next is needed)
            if (t + 1 < t1 || lane == 0) na_planes(bit4, n_bytes, 32 * (t + 1) + lane, nh, nl, ns);
            __syncwarp();
            uint32_t h1 = __shfl_down_sync(full, h0, 1), l1 = __shfl_down_sync(full, l0, 1),
                     s1 = __shfl_down_sync(full, s0, 1);
            const uint32_t fh = __shfl_sync(full, nh, 0), fl = __shfl_sync(full, nl, 0),
                           fs = __shfl_sync(full, ns, 0);
            if (lane == 31) {
                h1 = fh;
                l1 = fl;
                s1 = fs;
            }
            const uint64_t p0 = 1024 * t + 32 * lane;
            uint32_t range = full;
            if (p0 < lo) range = (lo - p0 >= 32) ? 0u : (range << (uint32_t)(lo - p0));
            if (p0 + 32 > hi) range = (hi <= p0) ? 0u : (range & (full >> (uint32_t)(32 - (hi - p0))));
#pragma unroll
            for (uint32_t st = 0; st < 2; ++st) {
                uint32_t m = range;
                for (uint32_t c = 0; c < np[st]; ++c) {
                    const NaPam pc = pam[st][c];
                    const uint32_t h = __funnelshift_r(h0, h1, pc.cell);
                    const uint32_t l = __funnelshift_r(l0, l1, pc.cell);
                    const uint32_t s = __funnelshift_r(s0, s1, pc.cell);
                    const uint32_t a = (l & pc.fc) | (~l & pc.fa);
                    const uint32_t b = (l & pc.ft) | (~l & pc.fg);
                    m &= ((h & b) | (~h & a)) & ~s;
                }
                for (;;) {
                    const uint32_t bal = __ballot_sync(full, m != 0);
                    if (!bal) break;
                    if (m) {
                        const uint32_t k = __ffs(m) - 1;
                        m &= m - 1;
                        q[st].e[qn[st] + __popc(bal & lt_mask)] =
                            make_uint4((uint32_t)(p0 + k), __funnelshift_r(h0, h1, k),
                                       __funnelshift_r(l0, l1, k), __funnelshift_r(s0, s1, k));
                    }
                    qn[st] += __popc(bal);
                    if (qn[st] >= 128) {
                        __syncwarp();
                        na_flush(q[st], 128, fast, st ? n_fwd : 0, st ? n_pat : n_fwd, ctr, cand, lane);
                        const uint32_t rest = qn[st] - 128;
                        uint4 e = make_uint4(0, 0, 0, 0);
                        if (lane < rest) e = q[st].e[128 + lane];
                        __syncwarp();
                        if (lane < rest) q[st].e[lane] = e;
                        __syncwarp();
                        qn[st] = rest;
                    }
                }
            }
        }
    }
    __syncwarp();
    for (uint32_t st = 0; st < 2; ++st)
        if (qn[st]) na_flush(q[st], qn[st], fast, st ? n_fwd : 0, st ? n_pat : n_fwd, ctr, cand, lane);
}
constexpr size_t na_scan_smem(size_t n_pat) {
    return n_pat * sizeof(NaFast) + 2 * kNaWarps * sizeof(NaQueue);
}

__device__ __forceinline__ uint8_t na_nib(const uint8_t *g, uint64_t i) {
    const uint8_t b = g[i >> 1];
    return (i & 1) ? (uint8_t)(b >> 4) : (uint8_t)(b & 0xF);
}

// (the scan's count is read here: the host waits once for both kernels; a
// list that overflowed has no rows, its range is split)
__global__ void na_verify_kernel(const uint8_t *__restrict__ bit4, uint64_t n_nucl,
                                 unsigned char *scratch, uint32_t *rows, uint32_t rows_cap) {
    const NaTables &T = *reinterpret_cast<const NaTables *>(scratch + kNaCounterBytes);
    uint32_t *ctr = reinterpret_cast<uint32_t *>(scratch);
    const uint32_t n_cand = ctr[0];
    if (ctr[1] || n_cand > kNaMaxCandidates) return;
    const uint2 *cand = reinterpret_cast<const uint2 *>(scratch + kNaCandOffset);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_cand;
         i += gridDim.x * blockDim.x) {
        const uint32_t s = cand[i].x, p = cand[i].y, L = T.L;
        if ((uint64_t)s + L > n_nucl) continue;  // record-end drop
        const uint32_t st = p >= T.n_fwd;
        int matches = 0;
        uint32_t actual = 0;
        bool pam_ok = true;
        for (uint32_t c = 0; c < L; ++c) {
            uint8_t g = na_nib(bit4, (uint64_t)s + c);
            if (g == 0xF) g = 0;  // N masked for the popcount count
            const uint8_t pb = T.b4[p][c];
            matches += __popc(g & pb);
            const bool single = g && !(g & (g - 1));
            if (!T.fisn[st][c] && !(single && (g & T.fset[st][c]))) pam_ok = false;
            if (pb != 0xF && !(single && (g & pb))) ++actual;
        }
        if ((int)L - matches > (int)T.max_mm || !pam_ok || actual > T.max_mm) continue;
        const uint32_t r = atomicAdd(&ctr[2], 1u);
        if (r >= kNaRowCountLimit) ctr[3] = 1;  // every value is returned once: none is missed
        if (r < rows_cap) {
            const uint64_t o = 3ull * r;  // rows_cap may exceed 2^32 / 3
            rows[o] = s;
            rows[o + 1] = p;
            rows[o + 2] = actual;
        }
    }
}

std::mutex g_na_mu;
void *g_na_ptr[64] = {};  // device address of g_noalloc_scratch, per device

int na_fail(int code, const std::string &m) { return cof::set_last_error(code, m); }

uint32_t na_code(uint8_t b4) { return b4 == 4 ? 0 : b4 == 2 ? 1 : b4 == 8 ? 2 : 3; }

}  // namespace

// See include/cof.h.
extern "C" COF_API int cof_search_seq_noalloc(const uint8_t *d_bit4, uint64_t n_nucl,
                                              const char *search_filter,
                                              const char *const *patterns, size_t n_patterns,
                                              uint32_t max_mismatches, uint32_t *d_rows,
                                              uint32_t rows_cap, uint32_t *n_rows,
                                              void *stream) {
    if (!d_bit4 || !search_filter || !patterns || !n_rows || (!d_rows && rows_cap))
        return na_fail(COF_E_BADINPUT, "null argument");
    if (reinterpret_cast<uintptr_t>(d_bit4) % 16)
        return na_fail(COF_E_BADINPUT, "d_bit4 must be 16-byte aligned");
    const size_t L = std::strlen(search_filter);
    if (L == 0 || L > 32)
        return na_fail(COF_E_UNSUPPORTED, "pattern length must be 1..32");
    if (n_patterns == 0 || n_patterns > kNaMaxPatterns)
        return na_fail(COF_E_UNSUPPORTED,
                       "n_patterns must be 1.." + std::to_string(kNaMaxPatterns) +
                           " (fwd + reverse) for the fixed scratch tables");
    if (n_patterns % 2)
        return na_fail(COF_E_BADINPUT,
                       "n_patterns must be even: the forward patterns, then their reverse "
                       "complements (search.rs:1455 takes index < n / 2 as '+')");
    if (n_nucl >= (1ull << 31))
        return na_fail(COF_E_UNSUPPORTED, "sequence longer than 2^31 - 1 nucleotides");
    if (max_mismatches >= L)
        return na_fail(COF_E_BADINPUT, "max_mismatches must be below the pattern length");
    const cof::Bit4Tables &t = cof::bit4();
    NaTables T;
    std::memset(&T, 0, sizeof T);
    T.L = (uint32_t)L;
    T.n_pat = (uint32_t)n_patterns;
    T.n_fwd = (uint32_t)(n_patterns / 2);
    T.max_mm = max_mismatches;
    for (size_t c = 0; c < L; ++c) {
        const char f = search_filter[c], fr = search_filter[L - 1 - c];
        if (!cof::is_mixed_base(f))
            return na_fail(COF_E_BADINPUT, "search filter must be a mixed base string");
        T.fset[0][c] = t.str2b4[1][(uint8_t)f];
        T.fisn[0][c] = f == 'N' || f == 'n';
        T.fset[1][c] = cof::comp4(t.str2b4[1][(uint8_t)fr]);
        T.fisn[1][c] = fr == 'N' || fr == 'n';
        for (int st = 0; st < 2; ++st) {
            if (T.fisn[st][c]) continue;
            const uint8_t fs = T.fset[st][c];
            T.pam[st][T.n_pam[st]++] = NaPam{(uint32_t)c, (fs & 4) ? ~0u : 0u, (fs & 2) ? ~0u : 0u,
                                              (fs & 8) ? ~0u : 0u, (fs & 1) ? ~0u : 0u};
        }
    }
    for (size_t p = 0; p < n_patterns; ++p) {
        if (!patterns[p] || std::strlen(patterns[p]) != L)
            return na_fail(COF_E_BADINPUT, "All patterns must have same length");
        NaFast f{0, 0, 0, (int32_t)max_mismatches};
        for (size_t c = 0; c < L; ++c) {
            const char ch = patterns[p][c];
            if (!cof::is_mixed_base(ch))
                return na_fail(COF_E_BADINPUT, "pattern must be a mixed base string");
            const uint8_t v = t.str2b4[1][(uint8_t)ch];
            T.b4[p][c] = v;
            if (!(v & (v - 1))) {
                const uint32_t cd = na_code(v);
                f.care |= 1u << c;
                f.h |= ((cd >> 1) & 1u) << c;
                f.l |= (cd & 1u) << c;
            }
        }
        T.fast[p] = f;
    }

    std::lock_guard<std::mutex> lk(g_na_mu);
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
        return na_fail(COF_E_CUDA, "no usable CUDA device");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (s) {
        // the scratch address below belongs to the current device: a stream
        // of another device would run the kernels against the wrong array
        int sdev = -1;
        const cudaError_t e = cudaStreamGetDevice(s, &sdev);
        if (e != cudaSuccess)
            return na_fail(COF_E_BADINPUT, std::string("stream: ") + cudaGetErrorString(e));
        if (sdev != dev)
            return na_fail(COF_E_BADINPUT, "stream belongs to device " + std::to_string(sdev) +
                                                ", the current device is " + std::to_string(dev));
    }
    if (!g_na_ptr[dev]) {
        // once per device, with that device current: the array's name is only
        // a host-side stand-in, the kernels need its device address.  The
        // address is kept for the process; a cudaDeviceReset of this device
        // by the caller invalidates it (and the array itself)
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p)
            return na_fail(COF_E_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
        g_na_ptr[dev] = p;
    }
    unsigned char *scratch = static_cast<unsigned char *>(g_na_ptr[dev]);
    auto cu = [&](cudaError_t e, const char *what) {
        if (e == cudaSuccess) return 0;
        na_fail(COF_E_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
        return 1;
    };
    // the tables in use: up to the last pattern's scan form, and the cells
    if (cu(cudaMemcpyAsync(scratch + kNaCounterBytes, &T, offsetof(NaTables, fast) + n_patterns * sizeof(NaFast),
                           cudaMemcpyHostToDevice, s),
           "table upload") ||
        cu(cudaMemcpyAsync(scratch + kNaCounterBytes + offsetof(NaTables, b4), T.b4,
                           n_patterns * sizeof(T.b4[0]), cudaMemcpyHostToDevice, s),
           "table upload") ||
        cu(cudaMemsetAsync(scratch, 0, kNaCounterBytes, s), "counter reset"))
        return COF_E_CUDA;
    const uint64_t n_bytes = (n_nucl + 1) / 2;
    // ranges still to scan; bisection keeps the stack below 2 x 31 + 1
    uint32_t pend_a[80], pend_b[80];
    int np = 0;
    if (n_nucl >= L) {
        pend_a[0] = 0;
        pend_b[0] = (uint32_t)(n_nucl - L + 1);
        np = 1;
    }
    uint32_t c4[4] = {0, 0, 0, 0};  // candidates, overflow, rows, row-count overflow
    while (np > 0) {
        --np;
        const uint32_t a = pend_a[np], b = pend_b[np];
        if (cu(cudaMemsetAsync(scratch, 0, 8, s), "counter reset")) return COF_E_CUDA;
        const uint64_t runs = (((uint64_t)b + 1023) / 1024 - a / 1024 + kNaRun - 1) / kNaRun;
        const unsigned blocks = (unsigned)std::min<uint64_t>((runs + kNaWarps - 1) / kNaWarps, 2048);
        na_scan_kernel<<<blocks, kNaWarps * 32, na_scan_smem(n_patterns), s>>>(d_bit4, n_bytes, a, b,
                                                                              scratch);
        if (cu(cudaGetLastError(), "scan launch")) return COF_E_CUDA;
        na_verify_kernel<<<512, 256, 0, s>>>(d_bit4, n_nucl, scratch, d_rows, rows_cap);
        if (cu(cudaGetLastError(), "verify launch") ||
            cu(cudaMemcpyAsync(c4, scratch, sizeof c4, cudaMemcpyDeviceToHost, s), "count readback") ||
            cu(cudaStreamSynchronize(s), "scan"))
            return COF_E_CUDA;
        if (c4[1] || c4[0] > kNaMaxCandidates) {
            // more candidates than the fixed list holds: split the range
            // (the reference bisects its Myers ranges the same way,
            // search.rs:1106-1153)
            if (b - a <= 64)
                return na_fail(COF_E_UNSUPPORTED, "candidate list overflow on a minimal range");
            const uint32_t mid = a + (b - a) / 2;
            pend_a[np] = mid;
            pend_b[np] = b;
            pend_a[np + 1] = a;
            pend_b[np + 1] = mid;
            np += 2;
        }
    }
    if (n_nucl < L && cu(cudaStreamSynchronize(s), "counter reset")) return COF_E_CUDA;
    if (c4[3]) {
        *n_rows = 0xFFFFFFFFu;
        return na_fail(COF_E_UNSUPPORTED,
                       "more than 2^32 - 16 rows: the row count does not fit its 32-bit counter");
    }
    const uint32_t nr = c4[2];
    *n_rows = nr;
    if (nr > rows_cap)
        return na_fail(COF_E_UNSUPPORTED, "rows_cap too small: " + std::to_string(nr) +
                                              " rows found, the first rows_cap were written");
    return COF_OK;
}
