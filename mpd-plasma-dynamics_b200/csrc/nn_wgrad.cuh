// Weight and bias gradients of one linear layer in two launches (included by
// nn_gemm.cu):
//
//   dW(m, n) = sum over rows r of a(r, m) g(r, n),   db(n) = sum over r of g(r, n)
//
// nn_wgrad_kernel: a CTA per (sample, split of K) sums its span of rows in TMEM
// and leaves the FP32 partial sum; further CTAs of the same launch make the
// partial column sums of g meanwhile.  nn_wgrad_sum_kernel adds the partials:
// splits in order, then samples in order, and the 128 column slices in order --
// the partition and every order are those of the GEMM, sum and column-sum
// kernels that it stands for (five launches), so the values are the same.
// Both operands run along the rows (K), so a thread takes 8 rows of one column
// (whole lines per warp), rounds them and writes 16 bytes of the tensor core's
// layout; the rows of chunk i + 1 are in flight in registers while chunk i is
// multiplied.  A chunk is 64 rows, 32 KB: the kernel lives by the number of
// loads in flight (two to four CTAs per SM, 32 or more loads a thread).
// Measured (B200, each launch alone, 65600 rows): 64 x 64 51 -> 24 us, 64 x 128
// 63 -> 32, 128 x 8 50 -> 22, 6 x 64 (its rows of 24 bytes were fetched element
// by element) 86 -> 25.
#pragma once

namespace {

constexpr int kWgThreads = 256, kWgK = 64;
constexpr int kWgColSlices = 128;   // as mpd_nn_colsum
constexpr uint32_t kWgTmem = 128;

// 8-row units of a 64-row chunk of W columns per thread.
template <int W>
constexpr int kWgUnits = (W * (kWgK / 8) + kWgThreads - 1) / kWgThreads;

template <int W>
__device__ __forceinline__ void wg_load(float (&f)[kWgUnits<W>][8], const float *src, int left) {
#pragma unroll
    for (int j = 0; j < kWgUnits<W>; ++j) {
        const int u = threadIdx.x + j * kWgThreads, n = u % W, c = u / W;
#pragma unroll
        for (int e = 0; e < 8; ++e)
            f[j][e] = (c < kWgK / 8 && 8 * c + e < left) ? __ldg(src + (8 * c + e) * W + n) : 0.0f;
    }
}

// ROWS: rows of the operand's tile (64 or 128).
template <int W, int ROWS>
__device__ __forceinline__ void wg_store(unsigned char *dst, const float (&f)[kWgUnits<W>][8]) {
#pragma unroll
    for (int j = 0; j < kWgUnits<W>; ++j) {
        const int u = threadIdx.x + j * kWgThreads, n = u % W, c = u / W;
        if (c < kWgK / 8)
            *reinterpret_cast<uint4 *>(dst + (n / ROWS) * (ROWS * kWgK * 2) +
                                       (c * (ROWS / 8) + (n % ROWS >> 3)) * 128 + (n & 7) * 16) =
                make_uint4(pack_bf16(f[j][0], f[j][1]), pack_bf16(f[j][2], f[j][3]),
                           pack_bf16(f[j][4], f[j][5]), pack_bf16(f[j][6], f[j][7]));
    }
}

template <int KA, int N>
constexpr int wg_smem() {
    return 2 * (128 * kWgK * 2 + ((N + 63) / 64) * 64 * kWgK * 2);
}

struct WgradArgs {
    const float *a, *g;       // rows x KA, rows x N, dense
    int P, B, ksplit, kspan;  // rows of one sample, samples
    float *part;              // ksplit x B x KA x N
    float *colpart;           // kWgColSlices x N
    float *dw, *db;
};

// Column slice `by` of 32 columns: as colsum_partial_kernel.
template <int N>
__device__ void wg_colsum(const WgradArgs &a, int blk, float (*part)[33]) {
    constexpr int kCols = (N + 31) / 32;
    const int bx = blk % kCols, by = blk / kCols;
    const int c = bx * 32 + (threadIdx.x & 31), ry = threadIdx.x >> 5;
    const long long rows = (long long)a.B * a.P;
    float s = 0.0f;
    if (c < N) {
#pragma unroll 8
        for (long long r = (long long)by * 8 + ry; r < rows; r += 8LL * kWgColSlices)
            s += __ldg(a.g + r * N + c);
    }
    part[ry][threadIdx.x & 31] = s;
    __syncthreads();
    if (ry == 0 && c < N) {
        float t = 0.0f;
        for (int k = 0; k < 8; ++k) t += part[k][threadIdx.x & 31];
        a.colpart[by * N + c] = t;
    }
}

template <int KA, int N>
__global__ void __launch_bounds__(kWgThreads, 2) nn_wgrad_kernel(const WgradArgs a) {
    constexpr int NB = (N + 63) / 64;
    constexpr int kABuf = 128 * kWgK * 2, kGBuf = NB * 64 * kWgK * 2;
    extern __shared__ __align__(1024) unsigned char gemm_smem[];
    __shared__ __align__(8) uint64_t bar[2];
    __shared__ uint32_t tmem_slot;
    const int ncta = a.B * a.ksplit;
    if (blockIdx.x >= ncta) {
        wg_colsum<N>(a, blockIdx.x - ncta, reinterpret_cast<float (*)[33]>(gemm_smem));
        return;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int b = blockIdx.x % a.B, split = blockIdx.x / a.B;
    const int k_begin = split * a.kspan, k_end = min(a.P, k_begin + a.kspan);
    const int n_chunks = (k_end - k_begin + kWgK - 1) / kWgK;
    unsigned char *sA = gemm_smem, *sG = sA + 2 * kABuf;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_addr(&tmem_slot)),
                     "r"(kWgTmem)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x == 0) {
        mbar_init(smem_addr(&bar[0]), 1);
        mbar_init(smem_addr(&bar[1]), 1);
        mbar_init_fence();
    }
    // rows of the tiles past KA and N are zero throughout
    if (KA < 128 || N < 64)
        for (int u = threadIdx.x; u < 2 * (kABuf + kGBuf) / 16; u += kWgThreads)
            reinterpret_cast<uint4 *>(gemm_smem)[u] = make_uint4(0, 0, 0, 0);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;

    float fa[kWgUnits<KA>][8], fg[kWgUnits<N>][8];
    const float *pa = a.a + ((long long)b * a.P + k_begin) * KA;
    const float *pg = a.g + ((long long)b * a.P + k_begin) * N;
    wg_load<KA>(fa, pa, k_end - k_begin);
    wg_load<N>(fg, pg, k_end - k_begin);
    bool ok = true;
    int issued = 0;
    for (int i = 0; i < n_chunks; ++i) {
        const int buf = i & 1;
        // the products of chunk i - 2 read this buffer
        if (i >= 2) ok = mbar_wait_bounded(smem_addr(&bar[buf]), ((i - 2) >> 1) & 1);
        if (!__syncthreads_and(ok)) break;
        wg_store<KA, 128>(sA + buf * kABuf, fa);
        wg_store<N, 64>(sG + buf * kGBuf, fg);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (threadIdx.x == 0) {
            tc_fence_after();
#pragma unroll
            for (int s = 0; s < kWgK / 16; ++s)
#pragma unroll
                for (int nb = 0; nb < NB; ++nb)
                    mma_bf16(tmem + nb * 64,
                             smem_desc(smem_addr(sA + buf * kABuf) + s * 2 * 2048, 2048, 128),
                             smem_desc(smem_addr(sG + buf * kGBuf) + nb * (64 * kWgK * 2) +
                                           s * 2 * 1024,
                                       1024, 128),
                             (i > 0 || s > 0) ? 1u : 0u);
            mma_commit(smem_addr(&bar[buf]));
        }
        __syncwarp();
        issued = i + 1;
        if (i + 1 < n_chunks) {
            const int left = k_end - k_begin - (i + 1) * kWgK;
            wg_load<KA>(fa, pa + (long long)(i + 1) * kWgK * KA, left);
            wg_load<N>(fg, pg + (long long)(i + 1) * kWgK * N, left);
        }
    }
    if (issued) {
        const bool last =
            mbar_wait_bounded(smem_addr(&bar[(issued - 1) & 1]), ((issued - 1) >> 1) & 1);
        ok = __syncthreads_and(last && ok && issued == n_chunks);
    }
    if (ok) {
        tc_fence_after();
        // 16 rows x 32 columns per step: warp w has rows 32 (w & 3) .., column half w >> 2
        float *o = a.part + (long long)blockIdx.x * (KA * N);
        const int rw = (warp & 3) * 32;
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            if (rw + hf * 16 >= KA) continue;
#pragma unroll
            for (int nb = 0; nb < NB; ++nb) {
                const int col = nb * 64 + (warp >> 2) * 32;
                if (col >= N) continue;
                float v[16];
                tmem_ld_16x32(tmem + ((uint32_t)(rw + hf * 16) << 16) + (uint32_t)col, v);
                tmem_ld_wait(v);
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    const int row = rw + hf * 16 + t * 8 + (lane >> 2);
                    if (row >= KA) continue;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int n = col + 8 * j + 2 * (lane & 3);
                        if (n < N)
                            *reinterpret_cast<float2 *>(o + row * N + n) =
                                make_float2(v[4 * j + 2 * t], v[4 * j + 2 * t + 1]);
                    }
                }
            }
        }
    } else if (threadIdx.x == 0) {
        atomicExch(&g_gemm_wait_fail, 1);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(kWgTmem)
                     : "memory");
    }
}

// 32 elements of dW a block: a warp takes samples warp, warp + 16, ... and adds
// their splits (16 loads in flight at a time); the first warp adds the samples.
// The blocks after them finish db, a column a thread.
constexpr int kWgSumWarps = 16;
__global__ void __launch_bounds__(kWgSumWarps * 32) nn_wgrad_sum_kernel(const WgradArgs a,
                                                                        int n_dw, int N) {
    __shared__ float red[kWgSumWarps][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int dw_blocks = (n_dw + 31) / 32;
    if (blockIdx.x >= dw_blocks) {
        const int c = (blockIdx.x - dw_blocks) * (kWgSumWarps * 32) + threadIdx.x;
        if (c >= N) return;
        float t = 0.0f;
#pragma unroll 32
        for (int k = 0; k < kWgColSlices; ++k) t += a.colpart[k * N + c];
        a.db[c] = t;
        return;
    }
    const int e = blockIdx.x * 32 + lane;
    const long long plane = (long long)a.B * n_dw;
    float sum = 0.0f;
    for (int b0 = 0; b0 < a.B; b0 += kWgSumWarps) {
        const int b = b0 + warp;
        float s = 0.0f;
        if (b < a.B && e < n_dw) {
            const float *p = a.part + (long long)b * n_dw + e;
#pragma unroll 16
            for (int k = 0; k < a.ksplit; ++k) s += __ldg(p + k * plane);
        }
        red[warp][lane] = s;
        __syncthreads();
        if (warp == 0)
            for (int k = 0; k < kWgSumWarps && b0 + k < a.B; ++k) sum += red[k][lane];
        __syncthreads();
    }
    if (warp == 0 && e < n_dw) a.dw[e] = sum;
}

}  // namespace
