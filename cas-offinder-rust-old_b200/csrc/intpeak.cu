// intpeak.cu -- peaks of this GPU for the scan's comparisons, its roofline
// denominators (libcof_peak.so, used by bench.py; not part of libcof).
//
//   popc : __popc results per second (8 independent chains per thread)
//   lop3 : 3-input logic results per second (8 independent chains)
//   pair : window x pattern comparisons per second of the scan's inner loop
//          (popc((H^pH)|(L^pL)|S) folded into a per-pattern minimum over 8
//          windows, one threshold test per pattern) on register-resident,
//          care-masked windows and shared-memory patterns, i.e. the scan with
//          no memory traffic and no hits.
//   product : window x pattern comparisons per second of the tensor cores: products
//          of 128 windows and 64, 128 or 256 patterns, K = 64 or 96 e4m3 columns,
//          f16 accumulators, back to back on operands in shared memory.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "mma_f8.cuh"

namespace {

__global__ void popc_kernel(uint32_t seed, int iters, uint32_t *out) {
    uint32_t x[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = seed * (threadIdx.x + 1 + j * 977) + blockIdx.x;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = __popc(x[j]) ^ (x[j] << 5);
    }
    uint32_t a = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) a ^= x[j];
    if (a == 0x12345678u) out[0] = a;
}

__global__ void lop3_kernel(uint32_t seed, int iters, uint32_t *out) {
    uint32_t x[8], y = seed ^ threadIdx.x, z = seed + blockIdx.x;
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = seed * (threadIdx.x + 1 + j * 977);
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = (x[j] ^ y) | (x[j] & z);
        y += 1;
    }
    uint32_t a = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) a ^= x[j];
    if (a == 0x12345678u) out[0] = a;
}

constexpr int kPats = 256;

__global__ void pair_kernel(uint32_t seed, int iters, uint32_t *out) {
    __shared__ uint4 pat[kPats];
    for (int i = threadIdx.x; i < kPats; i += blockDim.x)
        pat[i] = make_uint4(seed * (i + 3), seed ^ (i * 7919), 0x007FFFFFu, 0xFFFFFFFFu);
    __syncthreads();
    uint32_t h[8], l[8], s[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        h[j] = seed * (threadIdx.x + 11 + j);
        l[j] = seed ^ (threadIdx.x * 31 + j);
        s[j] = 0;
    }
    uint32_t hits = 0;
    for (int it = 0; it < iters; ++it) {
        for (int p = 0; p < kPats; ++p) {
            const uint4 q = pat[p];
            int mn = 64;
#pragma unroll
            for (int j = 0; j < 8; ++j) mn = min(mn, (int)__popc((h[j] ^ q.x) | (l[j] ^ q.y) | s[j]));
            if (mn <= (int)q.w) hits += mn + 1;  // q.w = -1: never
        }
    }
    if (hits) out[0] = hits;
}

// One CTA per SM of up to eight warps.  A thread of each issues products of 128
// windows, n patterns and 32 x steps columns, `iters` in all, in turn to the warp's
// share of the accumulators that 512 TMEM columns hold, and waits for them kBatch at
// a time.
constexpr uint32_t kIssuers = 8, kBatch = 16;
__global__ void __launch_bounds__(32 * kIssuers) product_kernel(uint32_t n, uint32_t steps,
                                                                uint32_t iters, uint32_t *out) {
    extern __shared__ __align__(128) unsigned char operands[];  // A (128 rows), then B (n rows)
    __shared__ __align__(8) uint64_t done[kIssuers];
    __shared__ uint32_t s_tmem;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const uint32_t mbar = (uint32_t)__cvta_generic_to_shared(&done[warp]);
    for (uint32_t i = threadIdx.x; i < (128 + n) * 32 * steps / 4; i += blockDim.x)
        reinterpret_cast<uint32_t *>(operands)[i] = 0x38B838B8u;  // +1 and -1
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(&s_tmem)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (lane == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t a0 = (uint32_t)__cvta_generic_to_shared(operands);
    const uint32_t da = cof::mma_desc(a0, 2048), db = cof::mma_desc(a0 + 128 * 32 * steps, n * 16),
                   idesc = cof::mma_f8_desc(n), slots = 512 / n / warps, tmem = s_tmem + warp * slots * n;
    uint32_t phase = 0;
    bool ok = true;
    for (uint32_t i = 0; i < iters / warps && ok; i += kBatch) {
        if (lane == 0) {
            for (uint32_t j = 0; j < kBatch; ++j) {
                const uint32_t d = tmem + (j % slots) * n;
                cof::mma_f8<false>(d, da, db, idesc);
                for (uint32_t s = 1; s < steps; ++s)
                    cof::mma_f8<true>(d, da + s * 256, db + s * 2 * n, idesc);
            }
            cof::mma_commit(mbar);
        }
        __syncwarp();
        ok = cof::mma_wait(mbar, phase, 1u << 20);
        phase ^= 1;
    }
    if (!ok) {  // once more before the TMEM goes back
        cof::mma_wait(mbar, phase ^ 1, 1u << 20);
        if (lane == 0) out[0] = 1;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(s_tmem), "r"(512));
    }
}

template <class K>
double time_kernel(K kernel, int blocks, int threads, int iters, uint32_t *d_out, double per) {
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    kernel<<<blocks, threads>>>(0x9E3779B1u, iters / 8 + 1, d_out);  // warm-up
    cudaEventRecord(a);
    kernel<<<blocks, threads>>>(0x9E3779B1u, iters, d_out);
    cudaEventRecord(b);
    cudaEventSynchronize(b);
    float ms = 0;
    cudaEventElapsedTime(&ms, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    return (double)blocks * threads * (double)iters * per / (ms * 1e-3);
}

}  // namespace

// out[0] = popc/s, out[1] = lop3/s, out[2] = scan pairs/s, out[3] = SM clock
// (kHz) reported by the driver.  Returns 0 or a CUDA error code.
extern "C" __attribute__((visibility("default"))) int cof_peak_measure(int device, double *out) {
    if (cudaSetDevice(device) != cudaSuccess) return -1;
    int n_sm = 0, clk = 0;
    cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, device);
    cudaDeviceGetAttribute(&clk, cudaDevAttrClockRate, device);
    uint32_t *d_out = nullptr;
    if (cudaMalloc(&d_out, 16) != cudaSuccess) return -2;
    const int blocks = n_sm * 8, threads = 256;
    out[0] = time_kernel(popc_kernel, blocks, threads, 4096, d_out, 8.0);
    out[1] = time_kernel(lop3_kernel, blocks, threads, 4096, d_out, 8.0);
    out[2] = time_kernel(pair_kernel, n_sm * 4, threads, 64, d_out, 8.0 * kPats);
    out[3] = clk;
    cudaError_t e = cudaDeviceSynchronize();
    cudaFree(d_out);
    return e == cudaSuccess ? 0 : (int)e;
}

// out[i], out[3 + i]: comparisons per second of products with 64, 128 and 256
// patterns, K = 64 and K = 96, from as many issuing warps as are fastest.  Returns 0 or a CUDA error code.
extern "C" __attribute__((visibility("default"))) int cof_peak_products(int device, double *out) {
    if (cudaSetDevice(device) != cudaSuccess) return -1;
    int n_sm = 0;
    cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, device);
    uint32_t *d_out = nullptr;
    if (cudaMalloc(&d_out, 16) != cudaSuccess) return -2;
    cudaMemset(d_out, 0, 16);
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    const uint32_t iters = 8192;
    for (uint32_t steps = 2; steps <= 3; ++steps)
        for (uint32_t i = 0; i < 3; ++i) {
            const uint32_t n = 64u << i, smem = (128 + n) * 32 * steps;
            float best = 0;
            for (uint32_t warps = 1; warps <= 512 / n && warps <= kIssuers; warps *= 2)
                for (int rep = 0; rep < 4; ++rep) {  // the first is a warm-up
                    cudaEventRecord(a);
                    product_kernel<<<n_sm, 32 * warps, smem>>>(n, steps, iters, d_out);
                    cudaEventRecord(b);
                    cudaEventSynchronize(b);
                    float ms = 0;
                    cudaEventElapsedTime(&ms, a, b);
                    if (rep) best = best > 0 ? std::min(best, ms) : ms;
                }
            out[3 * (steps - 2) + i] = 128.0 * n * iters * n_sm / (best * 1e-3);
        }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    uint32_t lost = 0;
    cudaMemcpy(&lost, d_out, 4, cudaMemcpyDeviceToHost);
    const cudaError_t e = cudaDeviceSynchronize();
    cudaFree(d_out);
    return e != cudaSuccess ? (int)e : lost ? -3 : 0;
}
