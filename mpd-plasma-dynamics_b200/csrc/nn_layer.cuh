// The surrogate's layer product as one persistent kernel (included by
// nn_gemm.cu, whose tcgen05 helpers it uses):
//
//   s = h W  +  G U[b]                 rows = B samples x P grid points, width 64
//   forward:   z = s + bias;  out = GELU(z) (or out = z: one array)
//   backward:  s (W and G the transposed operands), or s * GELU'(z)
//
// As separate launches the layer moved each row 7 times (h in; z out; z in and
// out; z in and out, h' out) and read and rounded G once per sample: 1013 us at
// 16 x 64400 rows against a floor of 121 (h in, z and h' out).  Both products
// keep their own FP32 accumulator in TMEM and the epilogue adds them, so a
// value is rounded exactly as by the separate launches.
//   * one CTA per SM takes an even share of the (128-row tile, sample) items,
//     samples fastest, so the tile of G (64 KB of BF16) stays in shared memory
//     over its samples;
//   * G and U come as images of the tensor core's K-major core-matrix layout
//     (basis_image_kernel, once per network; the mix's epilogue), so they are
//     bulk copies without any work by the threads; h arrives as FP32
//     (a tile is 32 KB of contiguous memory) and four warps round it;
//   * warps 0-7 run the epilogue of item i while the tensor core works on item
//     i + 1 and the copies of item i + 2 are in flight (TMEM, h and U are
//     double-buffered).  tcgen05.ld in the 16x256b form gives four lanes a
//     whole 32-byte sector of a row, so the stores need no transposition.
// 216 KB of shared memory, 256 TMEM columns, 14 warps.  Measured (B200, both
// products, bias and GELU): 998 -> 145 us at 16 x 64400 rows (5.5 TB/s of the
// 792 MB it must move: bound by memory), 75 -> 20 us at 16 x 4100 rows (3 to 4
// items a CTA: the pipeline's fill and the tile of G are a third of it).
#pragma once

namespace {

constexpr int kLyW = MPD_NN_WIDTH;   // columns of h, K of the first product
constexpr int kLyQ = MPD_NN_BASIS;   // K of the second product
constexpr int kLyRows = 128;
constexpr int kLyEpiWarps = 8, kLyCvtWarps = 4;
constexpr int kLyThreads = (kLyEpiWarps + kLyCvtWarps + 2) * 32;
constexpr int kLyGBytes = kLyRows * kLyQ * 2;     // 64 KB
constexpr int kLyUBytes = kLyQ * kLyW * 2;        // 32 KB
constexpr int kLyHBytes = kLyRows * kLyW * 4;     // 32 KB
constexpr int kLyHbBytes = kLyRows * kLyW * 2;    // 16 KB
constexpr int kLyWBytes = kLyW * kLyW * 2;        // 8 KB per 64 output columns
constexpr uint32_t kLyTmem = 256;
// The 128-wide projection with another product after it (OUT2 columns):
constexpr int kLyYBytes = kLyRows * 128 * 2;      // 32 KB: GELU(z) in BF16
constexpr int kLyW2Bytes = 64 * 128 * 2;          // 16 KB: columns past OUT2 are zero

static_assert(kLyW == 64 && kLyQ == 256 && MPD_NN_HIDDEN == 128 && MPD_NN_OUTPUTS == 8 &&
                  MPD_NN_INPUTS <= 8,
              "tiles, accumulators and operand layouts below are laid out for these");

enum LayerEpilogue { kEpiForward = 0, kEpiActBwd = 1, kEpiPlain = 2 };

struct LayerArgs {
    const float *h;              // rows x 64
    const float *w;              // (n, k) at w[n * w_sn + k * w_sk]
    long long w_sn, w_sk;
    const unsigned char *g_img;  // tiles of kLyGBytes (K2 != 0)
    const unsigned char *u_img;  // B x kLyUBytes (K2 != 0): chunk of 8 k, column n, 16 bytes
    const float *bias;           // forward
    const float *z_in;           // kEpiActBwd: GELU' is taken at these
    float *out0, *out1;          // out1: GELU(out0), or NULL
    const float *w2, *bias2;     // OUT2: (n, k) at w2[n * w2_sn + k * w2_sk]
    long long w2_sn, w2_sk;
    float *out2;                 // rows x OUT2
    int P, B, tiles;             // rows of one sample, samples, 128-row tiles of one sample
};

// How items are dealt: CTA c of n takes [total c / n, total (c + 1) / n).
__device__ __forceinline__ long long layer_first(long long total, int c, int n) {
    return total * c / n;
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes,
                                          uint32_t bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(dst), "l"(src), "r"(bytes), "r"(bar)
        : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// 16 TMEM lanes x 32 columns: register 4 j + 2 i + e of lane l holds row
// l / 4 + 8 i, column 8 j + 2 (l % 4) + e.
__device__ __forceinline__ void tmem_ld_16x32(uint32_t taddr, float v[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, "
        "%11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
// The values of earlier tcgen05.ld may be used after this.
__device__ __forceinline__ void tmem_ld_wait(float v[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]),
                   "+f"(v[6]), "+f"(v[7]), "+f"(v[8]), "+f"(v[9]), "+f"(v[10]), "+f"(v[11]),
                   "+f"(v[12]), "+f"(v[13]), "+f"(v[14]), "+f"(v[15])
                 :
                 : "memory");
}

// The tanh-form GELU and its derivative (the same operations as nn_ops.cu's).
__device__ __forceinline__ float layer_gelu(float x) {
    const float c = 0.7978845608028654f;
    const float u = c * (x + 0.044715f * x * x * x);
    const float t = tanhf(u);
    return 0.5f * x * (1.0f + t);
}
__device__ __forceinline__ float layer_dgelu(float x) {
    const float c = 0.7978845608028654f;
    const float u = c * (x + 0.044715f * x * x * x);
    const float t = tanhf(u);
    return 0.5f * (1.0f + t) + 0.5f * x * (1.0f - t * t) * c * (1.0f + 3.0f * 0.044715f * x * x);
}

template <int K2, int NB, int OUT2>
constexpr int layer_smem() {
    return (K2 ? kLyGBytes + 2 * kLyUBytes : 0) + 2 * kLyHBytes + kLyHbBytes + NB * kLyWBytes +
           (OUT2 ? 2 * kLyYBytes + kLyW2Bytes : 0);
}

// OUT2 (with NB == 2) is the projection and what follows it, while its values are
// in registers: the epilogue also leaves them in BF16 as the A operand of a third
// product, whose result it stores one item later.
//   forward, OUT2 8:    out2 = GELU(z) W2 + bias2
//   backward, OUT2 64:  out0 = (h W) GELU'(z_in) with h of K1 = 8 columns (the
//                       gradient of the outputs), out2 = out0 W2
// As its own launches the forward form read the 528 MB of out1 back (16 x 64400
// rows: 230 + 340 us, here 268 where memory alone takes 207), the backward one
// moved its 128 columns five times (96 us at 65600 rows, here 33).  The
// epilogue's tanh and 32-byte stores bound both; 16 epilogue warps instead of 8
// gave 285 and 33.
template <int K1, int K2, int NB, int EPI, int OUT2>
__global__ void __launch_bounds__(kLyThreads, 1) nn_layer_kernel(const LayerArgs a) {
    static_assert(K2 == 0 || NB == 1, "one accumulator pair of 64 columns each");
    constexpr bool HEAD = OUT2 != 0;
    static_assert(!HEAD || (K2 == 0 && NB == 2 && EPI != kEpiPlain), "after the projection");
    static_assert(K1 == kLyW || K1 == 8, "whole chunks of h, one product of K 16 at least");
    constexpr int kHRow = K1 * 4;   // bytes of a row of h
    constexpr uint32_t kTmem = HEAD ? 512 : kLyTmem;
    extern __shared__ __align__(1024) unsigned char gemm_smem[];
    __shared__ __align__(8) uint64_t h_full[2], h_free[2], u_full[2], acc_full[2], acc_free[2],
        g_full, hb_full, hb_free, y_full[2], o_full[2];
    __shared__ uint32_t tmem_slot;
    unsigned char *sG = gemm_smem;
    unsigned char *sU = sG + (K2 ? kLyGBytes : 0);
    unsigned char *sH = sU + (K2 ? 2 * kLyUBytes : 0);
    unsigned char *sHb = sH + 2 * kLyHBytes;
    unsigned char *sW = sHb + kLyHbBytes;
    unsigned char *sY = sW + NB * kLyWBytes;
    unsigned char *sW2 = sY + 2 * kLyYBytes;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long total = (long long)a.tiles * a.B;
    const long long first = layer_first(total, blockIdx.x, gridDim.x);
    const int items = (int)(layer_first(total, blockIdx.x + 1, gridDim.x) - first);

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_addr(&tmem_slot)),
                     "r"(kTmem)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(smem_addr(&h_full[i]), 1);
            mbar_init(smem_addr(&h_free[i]), kLyCvtWarps);
            mbar_init(smem_addr(&u_full[i]), 1);
            mbar_init(smem_addr(&acc_full[i]), 1);
            mbar_init(smem_addr(&acc_free[i]), kLyEpiWarps);
            mbar_init(smem_addr(&y_full[i]), kLyEpiWarps);
            mbar_init(smem_addr(&o_full[i]), 1);
        }
        mbar_init(smem_addr(&g_full), 1);
        mbar_init(smem_addr(&hb_full), kLyCvtWarps);
        mbar_init(smem_addr(&hb_free), 1);
        mbar_init_fence();
    }
    // W rounded once: (n, k) of 64-column block n / 64
    constexpr int kK1 = K1 < 16 ? 16 : K1;   // zero past K1
    for (int u = threadIdx.x; u < NB * kLyW * (kK1 / 8); u += kLyThreads) {
        const int n = u % (NB * kLyW), c = u / (NB * kLyW), nl = n % kLyW;
        float f[8];
#pragma unroll
        for (int e = 0; e < 8; ++e)
            f[e] = 8 * c + e < K1 ? __ldg(a.w + n * a.w_sn + (8 * c + e) * a.w_sk) : 0.0f;
        *reinterpret_cast<uint4 *>(sW + (n / kLyW) * kLyWBytes + (c * (kLyW / 8) + (nl >> 3)) * 128 +
                                   (nl & 7) * 16) =
            make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]),
                       pack_bf16(f[6], f[7]));
    }
    if (K1 < 16)   // the second chunk of K
        for (int u = threadIdx.x; u < kLyRows; u += kLyThreads)
            reinterpret_cast<uint4 *>(sHb + 2048)[u] = make_uint4(0, 0, 0, 0);
    if (HEAD) {
        for (int u = threadIdx.x; u < 64 * (128 / 8); u += kLyThreads) {
            const int n = u % 64, c = u / 64;
            float f[8];
#pragma unroll
            for (int e = 0; e < 8; ++e)
                f[e] = n < OUT2 ? __ldg(a.w2 + n * a.w2_sn + (8 * c + e) * a.w2_sk) : 0.0f;
            *reinterpret_cast<uint4 *>(sW2 + (c * 8 + (n >> 3)) * 128 + (n & 7) * 16) =
                make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]),
                           pack_bf16(f[6], f[7]));
        }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    bool ok = true;

    if (warp < kLyEpiWarps) {
        // ---- epilogue: rows 32 (warp & 3) .. + 31, columns 32 (warp >> 2) .. + 31 of 64
        const int quad = warp & 3, col0 = (warp >> 2) * 32;
        float2 bias[NB][4];
        if (EPI == kEpiForward) {
#pragma unroll
            for (int nb = 0; nb < NB; ++nb)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float *bp = a.bias + nb * 64 + col0 + 8 * j + 2 * (lane & 3);
                    bias[nb][j] = make_float2(bp[0], bp[1]);
                }
        }
        // the third product of item k: 16 rows a warp
        auto head_out = [&](int k) {
            if (!mbar_wait_bounded(smem_addr(&o_full[k & 1]), (k >> 1) & 1)) return false;
            tc_fence_after();
            const int rw = quad * 32 + (warp >> 2) * 16;
            const uint32_t ta = tmem + ((uint32_t)rw << 16) + (uint32_t)(256 + (k & 1) * 64);
            const long long it = first + k;
            const int tile = (int)(it / a.B), b = (int)(it % a.B);
            const int nrows = min(kLyRows, a.P - tile * kLyRows);
            float *o = a.out2 + ((long long)b * a.P + (long long)tile * kLyRows) * OUT2;
            if constexpr (OUT2 == 8) {
                uint32_t r[4];
                asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0, %1, %2, %3}, [%4];"
                             : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                             : "r"(ta));
                asm volatile("tcgen05.wait::ld.sync.aligned;"
                             : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3])
                             :
                             : "memory");
                const int n = 2 * (lane & 3);
                const float2 bias2 = make_float2(__ldg(a.bias2 + n), __ldg(a.bias2 + n + 1));
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    const int row = rw + t * 8 + (lane >> 2);
                    if (row < nrows)
                        *reinterpret_cast<float2 *>(o + row * OUT2 + n) =
                            make_float2(__uint_as_float(r[2 * t]) + bias2.x,
                                        __uint_as_float(r[2 * t + 1]) + bias2.y);
                }
            } else if constexpr (OUT2 == 64) {
#pragma unroll
                for (int col = 0; col < 64; col += 32) {
                    float v[16];
                    tmem_ld_16x32(ta + col, v);
                    tmem_ld_wait(v);
#pragma unroll
                    for (int t = 0; t < 2; ++t) {
                        const int row = rw + t * 8 + (lane >> 2);
                        if (row >= nrows) continue;
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            *reinterpret_cast<float2 *>(o + row * OUT2 + col + 8 * j +
                                                        2 * (lane & 3)) =
                                make_float2(v[4 * j + 2 * t] + 0.0f, v[4 * j + 2 * t + 1] + 0.0f);
                    }
                }
            }
            tc_fence_before();
            return true;
        };
        for (int i = 0; i < items; ++i) {
            const long long it = first + i;
            const int tile = (int)(it / a.B), b = (int)(it % a.B), buf = i & 1;
            const int nrows = min(kLyRows, a.P - tile * kLyRows);
            const int r0 = quad * 32 + (lane >> 2);           // + 8 t, t = 0..3
            const long long at =
                ((long long)b * a.P + (long long)tile * kLyRows + r0) * (NB * 64) + col0 +
                2 * (lane & 3);
            float2 zin[4][4];
            auto load_z = [&](int nb) {
#pragma unroll
                for (int t = 0; t < 4; ++t)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        zin[t][j] = r0 + 8 * t < nrows
                                        ? __ldg(reinterpret_cast<const float2 *>(
                                              a.z_in + at + t * 8 * (NB * 64) + nb * 64 + 8 * j))
                                        : make_float2(0.0f, 0.0f);
            };
            if (EPI == kEpiActBwd) load_z(0);
            ok = mbar_wait_bounded(smem_addr(&acc_full[buf]), (i >> 1) & 1);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int nb = 0; nb < NB; ++nb) {
                if (EPI == kEpiActBwd && nb > 0) load_z(nb);
                float s[2][16];
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    const uint32_t ta = tmem + ((uint32_t)(quad * 32 + hf * 16) << 16) +
                                        (uint32_t)(buf * 128 + nb * 64 + col0);
                    tmem_ld_16x32(ta, s[hf]);
                    if (K2) {
                        float g[16];
                        tmem_ld_16x32(ta + 64, g);
                        tmem_ld_wait(s[hf]);
                        tmem_ld_wait(g);
#pragma unroll
                        for (int k = 0; k < 16; ++k) s[hf][k] = g[k] + s[hf][k];
                    } else {
                        tmem_ld_wait(s[hf]);
                    }
                }
                if (nb == NB - 1) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_addr(&acc_free[buf]));
                }
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    const bool in = r0 + 8 * t < nrows;
                    if (!HEAD && !in) continue;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        float2 v = make_float2(s[t >> 1][4 * j + 2 * (t & 1)],
                                               s[t >> 1][4 * j + 2 * (t & 1) + 1]);
                        const long long e = at + t * 8 * (NB * 64) + nb * 64 + 8 * j;
                        if (EPI == kEpiForward) {
                            v.x += bias[nb][j].x;
                            v.y += bias[nb][j].y;
                        } else if (EPI == kEpiActBwd) {
                            v.x *= layer_dgelu(zin[t][j].x);
                            v.y *= layer_dgelu(zin[t][j].y);
                        }
                        if (in) *reinterpret_cast<float2 *>(a.out0 + e) = v;
                        if (HEAD || (EPI == kEpiForward && a.out1)) {
                            float2 y = v;
                            if (EPI == kEpiForward) {
                                y = make_float2(layer_gelu(v.x), layer_gelu(v.y));
                                if (in) *reinterpret_cast<float2 *>(a.out1 + e) = y;
                            }
                            if (HEAD) {   // 8 rows x 4 lanes: 128 bytes in a row
                                const int c = (nb * 64 + col0) / 8 + j, row = r0 + 8 * t;
                                *reinterpret_cast<uint32_t *>(
                                    sY + buf * kLyYBytes + (c * (kLyRows / 8) + (row >> 3)) * 128 +
                                    (row & 7) * 16 + 4 * (lane & 3)) = pack_bf16(y.x, y.y);
                            }
                        }
                    }
                }
            }
            if (HEAD) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_addr(&y_full[buf]));
                if (i >= 1) {
                    ok = __all_sync(0xffffffffu, head_out(i - 1));
                    if (!ok) break;
                }
            }
        }
        if (HEAD && ok && items > 0) ok = __all_sync(0xffffffffu, head_out(items - 1));
    } else if (warp < kLyEpiWarps + kLyCvtWarps) {
        // ---- round h: 8 rows x 8 chunks of 8 columns per step of a warp; the
        // chunk and the half read first rotate with the row, so the 16-byte
        // reads (256-byte rows) and writes both fall on all banks
        const int cw = warp - kLyEpiWarps, rl = lane & 7, cg = lane >> 3;
        for (int i = 0; i < items; ++i) {
            const int buf = i & 1;
            ok = mbar_wait_bounded(smem_addr(&h_full[buf]), (i >> 1) & 1);
            if (ok && i >= 1) ok = mbar_wait_bounded(smem_addr(&hb_free), (i - 1) & 1);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            const unsigned char *src = sH + buf * kLyHBytes;
            if (K1 < 16) {
                const int row = cw * 32 + lane;
                const float4 x = *reinterpret_cast<const float4 *>(src + row * kHRow);
                const float4 y = *reinterpret_cast<const float4 *>(src + row * kHRow + 16);
                *reinterpret_cast<uint4 *>(sHb + row * 16) =
                    make_uint4(pack_bf16(x.x, x.y), pack_bf16(x.z, x.w), pack_bf16(y.x, y.y),
                               pack_bf16(y.z, y.w));
            }
#pragma unroll
            for (int st = 0; st < (K1 < 16 ? 0 : 8); ++st) {
                const int row = cw * 32 + (st >> 1) * 8 + rl;
                const int c = ((st & 1) * 4 + cg + rl) & 7;
                const int swap = (rl >> 2) & 1;
                const float4 x = *reinterpret_cast<const float4 *>(src + row * 256 + c * 32 +
                                                                   swap * 16);
                const float4 y = *reinterpret_cast<const float4 *>(src + row * 256 + c * 32 +
                                                                   (swap ^ 1) * 16);
                const float4 lo = swap ? y : x, hi = swap ? x : y;
                *reinterpret_cast<uint4 *>(sHb + (c * (kLyRows / 8) + (row >> 3)) * 128 +
                                           (row & 7) * 16) =
                    make_uint4(pack_bf16(lo.x, lo.y), pack_bf16(lo.z, lo.w),
                               pack_bf16(hi.x, hi.y), pack_bf16(hi.z, hi.w));
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(smem_addr(&h_free[buf]));
                mbar_arrive(smem_addr(&hb_full));
            }
        }
    } else if (warp == kLyEpiWarps + kLyCvtWarps) {
        // ---- copies
        if (lane == 0) {
            int nh = 0, nu = 0, ng = 0, tile_now = -1;   // copies issued of h, U, G
            for (int i = 0; i < items; ++i) {
                const long long it = first + i;
                const int tile = (int)(it / a.B), b = (int)(it % a.B), buf = i & 1;
                const uint32_t hbytes =
                    (uint32_t)min(kLyRows, a.P - tile * kLyRows) * kHRow;
                if (i >= 2) ok = mbar_wait_bounded(smem_addr(&h_free[buf]), ((i - 2) >> 1) & 1);
                if (!ok) break;
                mbar_expect_tx(smem_addr(&h_full[buf]), hbytes);
                bulk_load(smem_addr(sH + buf * kLyHBytes),
                          a.h + ((long long)b * a.P + (long long)tile * kLyRows) * K1, hbytes,
                          smem_addr(&h_full[buf]));
                ++nh;
                if (!K2) continue;
                if (i >= 2) ok = mbar_wait_bounded(smem_addr(&acc_full[buf]), ((i - 2) >> 1) & 1);
                if (!ok) break;
                mbar_expect_tx(smem_addr(&u_full[buf]), kLyUBytes);
                bulk_load(smem_addr(sU + buf * kLyUBytes), a.u_img + (size_t)b * kLyUBytes,
                          kLyUBytes, smem_addr(&u_full[buf]));
                ++nu;
                if (tile == tile_now) continue;
                // the products of the item before read the old tile of G
                if (i >= 1)
                    ok = mbar_wait_bounded(smem_addr(&acc_full[(i - 1) & 1]), ((i - 1) >> 1) & 1);
                if (!ok) break;
                mbar_expect_tx(smem_addr(&g_full), kLyGBytes);
                bulk_load(smem_addr(sG), a.g_img + (size_t)tile * kLyGBytes, kLyGBytes,
                          smem_addr(&g_full));
                tile_now = tile;
                ++ng;
            }
            // no copy may still land after the CTA exits
            for (int k = max(0, nh - 2); k < nh; ++k)
                ok = mbar_wait_bounded(smem_addr(&h_full[k & 1]), (k >> 1) & 1) && ok;
            for (int k = max(0, nu - 2); k < nu; ++k)
                ok = mbar_wait_bounded(smem_addr(&u_full[k & 1]), (k >> 1) & 1) && ok;
            if (ng) ok = mbar_wait_bounded(smem_addr(&g_full), (ng - 1) & 1) && ok;
        }
    } else {
        // ---- products
        if (lane == 0) {
            int tile_now = -1, gloads = 0, done = 0, heads = 0;
            auto head = [&](int k) {   // the third product of item k
                if (!mbar_wait_bounded(smem_addr(&y_full[k & 1]), (k >> 1) & 1)) return false;
                tc_fence_after();
#pragma unroll
                for (int s = 0; s < 128 / 16; ++s)
                    mma_bf16(tmem + 256 + (k & 1) * 64,
                             smem_desc(smem_addr(sY + (k & 1) * kLyYBytes) + s * 2 * 2048, 2048,
                                       128),
                             smem_desc(smem_addr(sW2) + s * 2 * 1024, 1024, 128), s > 0 ? 1u : 0u);
                mma_commit(smem_addr(&o_full[k & 1]));
                ++heads;
                return true;
            };
            for (int i = 0; i < items; ++i) {
                const int tile = (int)((first + i) / a.B), buf = i & 1;
                if (i >= 2)
                    ok = mbar_wait_bounded(smem_addr(&acc_free[buf]), ((i - 2) >> 1) & 1);
                ok = ok && mbar_wait_bounded(smem_addr(&hb_full), i & 1);
                if (!ok) break;
                tc_fence_after();
                const uint32_t d1 = tmem + (uint32_t)(buf * 128);
#pragma unroll
                for (int s = 0; s < kK1 / 16; ++s) {
                    const uint64_t ad = smem_desc(smem_addr(sHb) + s * 2 * (kLyRows / 8) * 128,
                                                  (kLyRows / 8) * 128, 128);
#pragma unroll
                    for (int nb = 0; nb < NB; ++nb) {
                        const uint64_t bd =
                            smem_desc(smem_addr(sW) + nb * kLyWBytes + s * 2 * (kLyW / 8) * 128,
                                      (kLyW / 8) * 128, 128);
                        mma_bf16(d1 + nb * 64, ad, bd, s > 0 ? 1u : 0u);
                    }
                }
                mma_commit(smem_addr(&hb_free));
                if (K2) {
                    ok = mbar_wait_bounded(smem_addr(&u_full[buf]), (i >> 1) & 1);
                    if (ok && tile != tile_now) {
                        ok = mbar_wait_bounded(smem_addr(&g_full), gloads & 1);
                        ++gloads;
                        tile_now = tile;
                    }
                    if (!ok) {   // cover what was issued
                        mma_commit(smem_addr(&acc_full[buf]));
                        ++done;
                        break;
                    }
                    const uint32_t ua = smem_addr(sU + buf * kLyUBytes);
#pragma unroll
                    for (int s = 0; s < K2 / 16; ++s) {
                        const uint64_t ad = smem_desc(smem_addr(sG) + s * 2 * (kLyRows / 8) * 128,
                                                      (kLyRows / 8) * 128, 128);
                        const uint64_t bd =
                            smem_desc(ua + s * 2 * (kLyW / 8) * 128, (kLyW / 8) * 128, 128);
                        mma_bf16(d1 + 64, ad, bd, s > 0 ? 1u : 0u);
                    }
                }
                mma_commit(smem_addr(&acc_full[buf]));
                ++done;
                if (HEAD && i >= 1) {
                    ok = head(i - 1);
                    if (!ok) break;
                }
            }
            if (HEAD && ok && items > 0) ok = head(items - 1);
            // TMEM and shared memory are given back only after every product
            if (done)
                ok = mbar_wait_bounded(smem_addr(&acc_full[(done - 1) & 1]),
                                       ((done - 1) >> 1) & 1) && ok;
            if (heads)
                ok = mbar_wait_bounded(smem_addr(&o_full[(heads - 1) & 1]),
                                       ((heads - 1) >> 1) & 1) && ok;
        }
    }
    if (!ok) atomicExch(&g_gemm_wait_fail, 1);
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(kTmem)
                     : "memory");
    }
}

// A (rows x K) operand in FP32 as BF16 images of the K-major core-matrix
// layout, tile by tile: `mt` 128-row tiles next to each other for each block of
// kc columns of K.  Unit (block kb, row tile t, chunk c of 8 k, row r) is 16
// bytes; rows past `rows` and k past K are zero.
__global__ void basis_image_kernel(const float *src, long long s_row, long long s_k, int rows,
                                   int K, int mt, int kc, int nkb, uint4 *img) {
    const long long units = (long long)nkb * mt * (kc / 8) * 128;
    for (long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x; u < units;
         u += (long long)gridDim.x * blockDim.x) {
        const int rl = (int)(u % 128);
        const long long v = u / 128;
        const int c = (int)(v % (kc / 8));
        const int t = (int)(v / (kc / 8) % mt);
        const int kb = (int)(v / (kc / 8) / mt);
        const int row = t * 128 + rl;
        float f[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int k = kb * kc + 8 * c + e;
            f[e] = row < rows && k < K ? src[row * s_row + k * s_k] : 0.0f;
        }
        img[u] = make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]),
                            pack_bf16(f[6], f[7]));
    }
}

}  // namespace

namespace {

// The lift z = x W + bias (x: rows x 6, 64 columns).  One MMA of K 16 a tile and
// 24 bytes a row in for 256 out: bound by the stores.  Four CTAs of 128 threads
// per SM (their TMEM is 2 x 64 columns each) take even shares of the 128-row
// tiles; the rows of tile i + 1 are fetched into registers and the product of
// tile i runs while tile i - 1 is stored.
constexpr int kLiftK = MPD_NN_INPUTS;

__global__ void __launch_bounds__(128, 4) nn_lift_kernel(const float *x, const float *w,
                                                         const float *bias, long long rows,
                                                         float *z) {
    __shared__ __align__(1024) unsigned char sA[2][kLyRows * 16 * 2];
    __shared__ __align__(1024) unsigned char sB[kLyW * 16 * 2];
    __shared__ __align__(8) uint64_t bar[2];
    __shared__ uint32_t tmem_slot;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long total = (rows + kLyRows - 1) / kLyRows;
    const long long first = layer_first(total, blockIdx.x, gridDim.x);
    const int items = (int)(layer_first(total, blockIdx.x + 1, gridDim.x) - first);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_addr(&tmem_slot)),
                     "r"(128)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x == 0) {
        mbar_init(smem_addr(&bar[0]), 1);
        mbar_init(smem_addr(&bar[1]), 1);
        mbar_init_fence();
    }
    // K 6 .. 15 of both operands stay zero
    for (int u = threadIdx.x; u < 2 * kLyRows * 2; u += 128)
        reinterpret_cast<uint4 *>(sA)[u] = make_uint4(0, 0, 0, 0);
    {
        const int n = threadIdx.x & 63, c = threadIdx.x >> 6;
        float f[8];
#pragma unroll
        for (int e = 0; e < 8; ++e)
            f[e] = 8 * c + e < kLiftK ? __ldg(w + (8 * c + e) * kLyW + n) : 0.0f;
        *reinterpret_cast<uint4 *>(sB + (c * 8 + (n >> 3)) * 128 + (n & 7) * 16) =
            make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]),
                       pack_bf16(f[6], f[7]));
    }
    float2 bs[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
        bs[j] = make_float2(__ldg(bias + 8 * j + 2 * (lane & 3)),
                            __ldg(bias + 8 * j + 2 * (lane & 3) + 1));
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    // element e = thread + 128 j of a tile's 768: row e / 6, k e % 6
    float v[kLiftK];
    auto load = [&](int i) {
        const long long base = (first + i) * (kLyRows * kLiftK);
#pragma unroll
        for (int j = 0; j < kLiftK; ++j) {
            const long long e = base + threadIdx.x + 128 * j;
            v[j] = e < rows * kLiftK ? __ldg(x + e) : 0.0f;
        }
    };
    auto store = [&](int i) {
        if (!mbar_wait_bounded(smem_addr(&bar[i & 1]), (i >> 1) & 1)) return false;
        tc_fence_after();
        const long long r0 = (first + i) * kLyRows + warp * 32 + (lane >> 2);
#pragma unroll
        for (int p = 0; p < 4; ++p) {   // 16 rows x 32 columns each
            const int hf = p >> 1, col = (p & 1) * 32;
            float s[16];
            tmem_ld_16x32(tmem + ((uint32_t)(warp * 32 + hf * 16) << 16) +
                              (uint32_t)((i & 1) * 64 + col),
                          s);
            tmem_ld_wait(s);
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const long long row = r0 + hf * 16 + t * 8;
                if (row >= rows) continue;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 b = bs[col / 8 + j];
                    *reinterpret_cast<float2 *>(z + row * kLyW + col + 8 * j + 2 * (lane & 3)) =
                        make_float2(s[4 * j + 2 * t] + b.x, s[4 * j + 2 * t + 1] + b.y);
                }
            }
        }
        tc_fence_before();
        return true;
    };
    bool ok = true;
    int issued = 0;
    if (items > 0) load(0);
    for (int i = 0; i < items; ++i) {
#pragma unroll
        for (int j = 0; j < kLiftK; ++j) {
            const int e = threadIdx.x + 128 * j, row = e / kLiftK, k = e % kLiftK;
            *reinterpret_cast<__nv_bfloat16 *>(sA[i & 1] + (row >> 3) * 128 + (row & 7) * 16 +
                                               2 * k) = __float2bfloat16_rn(v[j]);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tc_fence_before();
        if (!__syncthreads_and(ok)) break;
        if (threadIdx.x == 0) {
            tc_fence_after();
            mma_bf16(tmem + (i & 1) * 64, smem_desc(smem_addr(sA[i & 1]), 2048, 128),
                     smem_desc(smem_addr(sB), 1024, 128), 0u);
            mma_commit(smem_addr(&bar[i & 1]));
        }
        issued = i + 1;
        __syncwarp();
        if (i + 1 < items) load(i + 1);
        if (i >= 1) ok = __all_sync(0xffffffffu, store(i - 1));
    }
    if (issued == items && ok) {
        if (items > 0) ok = __all_sync(0xffffffffu, store(items - 1));
    } else if (issued) {   // a wait gave up: TMEM goes back only after every product
        ok = false;
        mbar_wait_bounded(smem_addr(&bar[(issued - 1) & 1]), ((issued - 1) >> 1) & 1);
    }
    if (!ok && lane == 0) atomicExch(&g_gemm_wait_fail, 1);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(128)
                     : "memory");
    }
}

}  // namespace
