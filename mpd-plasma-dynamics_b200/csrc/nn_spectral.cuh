// The way into the spectral space and the mix there, as two kernels (included
// by nn_gemm.cu after nn_layer.cuh):
//
//   nn_project_kernel  V[b] = basis h[b]      256 x 64 sums over the P points
//   nn_mix_kernel      U[b, q] = V[b, q] R[q] 64 x 64 per coefficient, and the
//                      sums over the split of K before it
//
// nn_project_kernel: one CTA per (sample, split of K), both 128-row tiles of the
// basis as two TMEM accumulators (a CTA per tile where that many have an SM
// each), so a row of h is fetched and rounded once (the
// general kernel: once per tile, with the basis rounded again per sample, and
// 320 CTAs in two waves at two per SM).  The basis is an image of the tensor
// core's layout in blocks of 32 points (basis_image_kernel), so a stage of the
// four-stage ring is two bulk copies (16 KB of basis, 8 KB of h); two sets of
// four warps transpose and round h, one thread issues the products.  112 KB of
// shared memory: two CTAs per SM.  The split of K, the order of the products in an
// accumulator and the order of the partial sums are the general kernel's, so
// the values are too.  Both kernels together, measured against the general one
// (B200): 455 -> 104 us at 16 samples of 64400 points (the copies: 264 MB of h
// from memory and 530 MB of the basis from L2; with one set of converting warps
// 113), 53 -> 21 us at 16 of 4100 and 146 -> 51 us at 1 of 64400 (32 CTAs of one
// tile each, bound by what one SM takes in).
#pragma once

namespace {

constexpr int kPjK = 32;
constexpr int kPjCvtWarps = 8, kPjThreads = (kPjCvtWarps + 2) * 32;
constexpr int kPjFTile = 128 * kPjK * 2;         // 8 KB: a row tile of a block
constexpr int kPjHBytes = kPjK * kLyW * 4;       // 8 KB
constexpr int kPjHbBytes = kPjK * kLyW * 2;      // 4 KB
// TILES (row tiles of the basis per CTA): 2 with 4 stages, or 1 with 8.
template <int TILES>
constexpr int kPjStages = 8 / TILES;
template <int TILES>
constexpr int kPjSmem = kPjStages<TILES> * (TILES * kPjFTile + kPjHBytes + kPjHbBytes);
constexpr uint32_t kPjTmem = 128;

// out: ksplit == 1 ? V (B x 256 x 64) : the partial sums (ksplit x B x 256 x 64)
template <int TILES>
__global__ void __launch_bounds__(kPjThreads) nn_project_kernel(const unsigned char *f_img,
                                                                const float *h, int P, int B,
                                                                int kspan, float *out) {
    constexpr int STAGES = kPjStages<TILES>, kPjFBytes = TILES * kPjFTile;
    extern __shared__ __align__(1024) unsigned char gemm_smem[];
    __shared__ __align__(8) uint64_t full[STAGES], done[STAGES], hb_full[STAGES], all_done;
    __shared__ uint32_t tmem_slot;
    unsigned char *sF = gemm_smem, *sH = sF + STAGES * kPjFBytes,
                  *sHb = sH + STAGES * kPjHBytes;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int part = blockIdx.x / (2 / TILES), tile0 = blockIdx.x % (2 / TILES);
    const int b = part % B, split = part / B;
    const int k_begin = split * kspan, k_end = min(P, k_begin + kspan);
    const int n_chunks = (k_end - k_begin + kPjK - 1) / kPjK;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_addr(&tmem_slot)),
                     "r"(kPjTmem)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) {
            mbar_init(smem_addr(&full[i]), 1);
            mbar_init(smem_addr(&done[i]), 1);
            mbar_init(smem_addr(&hb_full[i]), 4);
        }
        mbar_init(smem_addr(&all_done), 1);
        mbar_init_fence();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    bool ok = true;

    if (warp < kPjCvtWarps) {
        // ---- h (points x columns) to its transpose in BF16, zero past K's end;
        // four warps take the even chunks, four the odd ones.  The copies of
        // chunk i were issued after the products of chunk i - STAGES, so its
        // buffer is free as well.
        const int n = threadIdx.x & 63, cb = (threadIdx.x >> 6) & 1;
        for (int i = warp >> 2; i < n_chunks; i += 2) {
            const int s = i % STAGES;
            ok = mbar_wait_bounded(smem_addr(&full[s]), (i / STAGES) & 1);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            const float *src = reinterpret_cast<const float *>(sH + s * kPjHBytes);
            unsigned char *dst = sHb + s * kPjHbBytes;
            const int left = k_end - k_begin - i * kPjK;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int c = cb + 2 * j;
                float f[8];
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    f[e] = 8 * c + e < left ? src[(8 * c + e) * kLyW + n] : 0.0f;
                *reinterpret_cast<uint4 *>(dst + (c * (kLyW / 8) + (n >> 3)) * 128 +
                                           (n & 7) * 16) =
                    make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]),
                               pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_addr(&hb_full[s]));
        }
        // A barrier of one phase.  The last chunk's done[] would not do: a set
        // knows how far that barrier has come only from the chunks it converts
        // itself, so the set that did not convert the last one could take the
        // phase two before (the same parity) for the last.
        if (ok) ok = mbar_wait_bounded(smem_addr(&all_done), 0);
        ok = __all_sync(0xffffffffu, ok);
        if (ok && (warp >> 2) < TILES) {
            tc_fence_after();
            const int mt = warp >> 2, r0 = (warp & 3) * 32;   // a tile per four warps
            float *o = out + ((long long)part * kLyQ + (tile0 + mt) * 128 + r0 + (lane >> 2)) * kLyW +
                       2 * (lane & 3);
#pragma unroll
            for (int q = 0; q < 4; ++q) {   // 16 rows x 32 columns each
                const int hf = q & 1, col = (q >> 1) * 32;
                float v[16];
                tmem_ld_16x32(tmem + ((uint32_t)(r0 + hf * 16) << 16) + (uint32_t)(mt * 64 + col),
                              v);
                tmem_ld_wait(v);
#pragma unroll
                for (int t = 0; t < 2; ++t)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        *reinterpret_cast<float2 *>(o + (hf * 16 + t * 8) * kLyW + col + 8 * j) =
                            make_float2(v[4 * j + 2 * t] + 0.0f, v[4 * j + 2 * t + 1] + 0.0f);
            }
        }
    } else if (warp == kPjCvtWarps) {
        // ---- copies
        if (lane == 0) {
            int n = 0;
            for (; n < n_chunks; ++n) {
                const int s = n % STAGES, k0 = k_begin + n * kPjK;
                if (n >= STAGES)
                    ok = mbar_wait_bounded(smem_addr(&done[s]), (n / STAGES - 1) & 1);
                if (!ok) break;
                const uint32_t hbytes = (uint32_t)min(kPjK, k_end - k0) * (kLyW * 4);
                mbar_expect_tx(smem_addr(&full[s]), kPjFBytes + hbytes);
                bulk_load(smem_addr(sF + s * kPjFBytes),
                          f_img + ((size_t)(k0 / kPjK) * 2 + tile0) * kPjFTile, kPjFBytes,
                          smem_addr(&full[s]));
                bulk_load(smem_addr(sH + s * kPjHBytes), h + ((long long)b * P + k0) * kLyW,
                          hbytes, smem_addr(&full[s]));
            }
            // no copy may still land after the CTA exits
            for (int k = max(0, n - STAGES); k < n; ++k)
                ok = mbar_wait_bounded(smem_addr(&full[k % STAGES]), (k / STAGES) & 1) && ok;
        }
    } else {
        // ---- products
        if (lane == 0) {
            int n = 0;
            for (; n < n_chunks; ++n) {
                const int s = n % STAGES;
                ok = mbar_wait_bounded(smem_addr(&full[s]), (n / STAGES) & 1) &&
                     mbar_wait_bounded(smem_addr(&hb_full[s]), (n / STAGES) & 1);
                if (!ok) break;
                tc_fence_after();
#pragma unroll
                for (int mt = 0; mt < TILES; ++mt)
#pragma unroll
                    for (int k = 0; k < kPjK / 16; ++k) {
                        const uint64_t ad = smem_desc(
                            smem_addr(sF + s * kPjFBytes) + mt * kPjFTile + k * 2 * 2048,
                            2048, 128);
                        const uint64_t bd = smem_desc(
                            smem_addr(sHb + s * kPjHbBytes) + k * 2 * 1024, 1024, 128);
                        mma_bf16(tmem + mt * 64, ad, bd, (n > 0 || k > 0) ? 1u : 0u);
                    }
                mma_commit(smem_addr(&done[s]));
            }
            // TMEM and shared memory are given back only after every product
            if (n == n_chunks) {
                mma_commit(smem_addr(&all_done));
                ok = mbar_wait_bounded(smem_addr(&all_done), 0) && ok;
            } else if (n)
                ok = mbar_wait_bounded(smem_addr(&done[(n - 1) % STAGES]),
                                       ((n - 1) / STAGES) & 1) && ok;
        }
    }
    if (!ok) atomicExch(&g_gemm_wait_fail, 1);
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(kPjTmem)
                     : "memory");
    }
}

// One CTA per coefficient q and 128 samples: the partial sums of V[b, q] in
// split order, V, and the product with R[q] (64 x 64).  The operands are tiny
// (16 KB of R, ksplit x 256 B a sample), so what it costs is one trip to memory
// for both, taken together, the product and the stores.  U also leaves as the
// image the layer kernel copies (element (q, n) of sample b: 16-byte unit q / 8).
// GRAD (one CTA of samples, at most 32: K of one block of the general kernel) adds
// the gradient of R[q] = V_fwd[., q]^T V[., q], whose second operand is at hand:
// as a launch of its own it took 13.6 us, here it is within the trip.
constexpr int kMixGradK = MPD_NN_MIX_GRAD_MAX_B;
constexpr uint32_t kMixTmem = 128;

template <bool GRAD>
__global__ void __launch_bounds__(128) nn_mix_kernel(const float *part, int ksplit, int B,
                                                     const float *R, long long r_sn,
                                                     long long r_sk, float *V, float *U,
                                                     __nv_bfloat16 *u_img, const float *V_fwd,
                                                     float *dR) {
    __shared__ __align__(1024) unsigned char sA2[GRAD ? 128 * kMixGradK * 2 : 16];
    __shared__ __align__(1024) unsigned char sB2[GRAD ? kLyW * kMixGradK * 2 : 16];
    __shared__ __align__(1024) unsigned char sA[128 * kLyW * 2];
    __shared__ __align__(1024) unsigned char sB[kLyW * kLyW * 2];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_slot;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q = blockIdx.x, b0 = blockIdx.y * 128, rows = min(128, B - b0);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_addr(&tmem_slot)),
                     "r"(kMixTmem)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x == 0) {
        mbar_init(smem_addr(&bar), 1);
        mbar_init_fence();
    }
    const float *Rq = R + (long long)q * (kLyW * kLyW);
    float r[4][8];
    const bool n_inner = r_sn == 1;   // which way a warp reads whole lines of R
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int u = threadIdx.x + 128 * j;
        const int n = n_inner ? u % kLyW : u / 8, c = n_inner ? u / kLyW : u % 8;
#pragma unroll
        for (int e = 0; e < 8; ++e) r[j][e] = __ldg(Rq + n * r_sn + (8 * c + e) * r_sk);
    }
    // the first operand of the gradient: 8 samples of one row k of V_fwd's transpose
    float vf[2][8];
    if (GRAD) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int u = threadIdx.x + 128 * j, k = u % kLyW, c = u / kLyW;
#pragma unroll
            for (int e = 0; e < 8; ++e)
                vf[j][e] = 8 * c + e < B
                               ? __ldg(V_fwd + ((long long)(8 * c + e) * kLyQ + q) * kLyW + k)
                               : 0.0f;
        }
        // samples past B are zero in both operands
        for (int u = threadIdx.x; u < (int)sizeof(sB2) / 16; u += 128)
            reinterpret_cast<uint4 *>(sB2)[u] = make_uint4(0, 0, 0, 0);
        __syncthreads();
    }
    const long long plane = (long long)B * kLyQ * kLyW;
    for (int u = threadIdx.x; u < rows * 8; u += 128) {
        const int row = u >> 3, c = u & 7;
        const long long at = ((long long)(b0 + row) * kLyQ + q) * kLyW + 8 * c;
        float f[8];
        if (ksplit > 1) {
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = 0.0f;
#pragma unroll 8
            for (int k = 0; k < ksplit; ++k) {
                const float4 x = __ldg(reinterpret_cast<const float4 *>(part + k * plane + at));
                const float4 y = __ldg(reinterpret_cast<const float4 *>(part + k * plane + at) + 1);
                f[0] += x.x; f[1] += x.y; f[2] += x.z; f[3] += x.w;
                f[4] += y.x; f[5] += y.y; f[6] += y.z; f[7] += y.w;
            }
            *reinterpret_cast<float4 *>(V + at) = make_float4(f[0], f[1], f[2], f[3]);
            *reinterpret_cast<float4 *>(V + at + 4) = make_float4(f[4], f[5], f[6], f[7]);
        } else {
            const float4 x = *reinterpret_cast<const float4 *>(V + at);
            const float4 y = *reinterpret_cast<const float4 *>(V + at + 4);
            f[0] = x.x; f[1] = x.y; f[2] = x.z; f[3] = x.w;
            f[4] = y.x; f[5] = y.y; f[6] = y.z; f[7] = y.w;
        }
        *reinterpret_cast<uint4 *>(sA + (c * 16 + (row >> 3)) * 128 + (row & 7) * 16) =
            make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]),
                       pack_bf16(f[6], f[7]));
        if (GRAD) {   // element (n, sample)
#pragma unroll
            for (int e = 0; e < 8; ++e)
                *reinterpret_cast<__nv_bfloat16 *>(sB2 + ((row >> 3) * 8 + c) * 128 + e * 16 +
                                                   (row & 7) * 2) = __float2bfloat16_rn(f[e]);
        }
    }
    if (GRAD) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int u = threadIdx.x + 128 * j, k = u % kLyW, c = u / kLyW;
            *reinterpret_cast<uint4 *>(sA2 + (c * 16 + (k >> 3)) * 128 + (k & 7) * 16) =
                make_uint4(pack_bf16(vf[j][0], vf[j][1]), pack_bf16(vf[j][2], vf[j][3]),
                           pack_bf16(vf[j][4], vf[j][5]), pack_bf16(vf[j][6], vf[j][7]));
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int u = threadIdx.x + 128 * j;
        const int n = n_inner ? u % kLyW : u / 8, c = n_inner ? u / kLyW : u % 8;
        *reinterpret_cast<uint4 *>(sB + (c * 8 + (n >> 3)) * 128 + (n & 7) * 16) =
            make_uint4(pack_bf16(r[j][0], r[j][1]), pack_bf16(r[j][2], r[j][3]),
                       pack_bf16(r[j][4], r[j][5]), pack_bf16(r[j][6], r[j][7]));
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < kLyW / 16; ++k)
            mma_bf16(tmem, smem_desc(smem_addr(sA) + k * 2 * 2048, 2048, 128),
                     smem_desc(smem_addr(sB) + k * 2 * 1024, 1024, 128), k > 0 ? 1u : 0u);
        if (GRAD) {
#pragma unroll
            for (int k = 0; k < kMixGradK / 16; ++k)
                mma_bf16(tmem + 64, smem_desc(smem_addr(sA2) + k * 2 * 2048, 2048, 128),
                         smem_desc(smem_addr(sB2) + k * 2 * 1024, 1024, 128), k > 0 ? 1u : 0u);
        }
        mma_commit(smem_addr(&bar));
    }
    __syncwarp();
    const bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(smem_addr(&bar), 0));
    if (ok) {
        tc_fence_after();
#pragma unroll
        for (int p = 0; p < 4; ++p) {   // 16 rows x 32 columns each
            const int hf = p & 1, col = (p >> 1) * 32;
            if (warp * 32 + hf * 16 >= rows) continue;
            float v[16];
            tmem_ld_16x32(tmem + ((uint32_t)(warp * 32 + hf * 16) << 16) + (uint32_t)col, v);
            tmem_ld_wait(v);
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const int row = warp * 32 + hf * 16 + t * 8 + (lane >> 2);
                if (row >= rows) continue;
                const long long b = b0 + row;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int n = col + 8 * j + 2 * (lane & 3);
                    const float2 s =
                        make_float2(v[4 * j + 2 * t] + 0.0f, v[4 * j + 2 * t + 1] + 0.0f);
                    *reinterpret_cast<float2 *>(U + (b * kLyQ + q) * kLyW + n) = s;
                    __nv_bfloat16 *im = u_img + b * (kLyQ * kLyW) + ((q >> 3) * kLyW + n) * 8 +
                                        (q & 7);
                    im[0] = __float2bfloat16_rn(s.x);
                    im[8] = __float2bfloat16_rn(s.y);
                }
            }
        }
        if (GRAD && warp < 2) {   // rows k of dR[q]
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                const int hf = p & 1, col = (p >> 1) * 32;
                float v[16];
                tmem_ld_16x32(tmem + ((uint32_t)(warp * 32 + hf * 16) << 16) +
                                  (uint32_t)(64 + col),
                              v);
                tmem_ld_wait(v);
                float *o = dR + (long long)q * (kLyW * kLyW) +
                           (warp * 32 + hf * 16 + (lane >> 2)) * kLyW + col + 2 * (lane & 3);
#pragma unroll
                for (int t = 0; t < 2; ++t)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        *reinterpret_cast<float2 *>(o + t * 8 * kLyW + 8 * j) =
                            make_float2(v[4 * j + 2 * t] + 0.0f, v[4 * j + 2 * t + 1] + 0.0f);
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
                     "r"(kMixTmem)
                     : "memory");
    }
}

}  // namespace
