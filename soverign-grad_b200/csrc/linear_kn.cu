// Decode-shape forward (M <= 16) for weights stored [K, N] — the reference module's own layout
// (nn::QuantizedLinear / QuantizedLinear4Bit keep W as [in, out], include/sovereigngrad/nn.hpp:
// 935-1001) — so that a drop-in user who keeps that layout does not fall onto the any-shape kernel.
//
//   INT4: groups of G consecutive elements of the FLAT tensor, i.e. along N inside a row k when
//         N % G == 0: scale[k][n / G].  The scale depends on k, so the k-sum cannot be taken in
//         integers first (as the [N,K] kernels do); every code is turned into fp32 and multiplied by
//         (x[m,k] * scale): y[m,n] = sum_k (x[m,k] * s[k, n/G]) * code[k,n].
//   INT8: one scale per row k of the stored tensor (per "channel" = input feature) or per tensor:
//         y[m,n] = sum_k (x[m,k] * s[k]) * code[k,n].
//
// kn_mma_kernel: codes are exact in bf16, and the fp32 factor x * s splits into three bf16 numbers without loss
// (24 significant bits), so the products run on the tensor cores (mma.sync m16n8k16) at fp32 precision: codes are the A
// operand (16 output features per tile), the three parts of every batch row the columns of B.  The factor is formed and
// split per (k, 32 output features), 20 instructions for 16 k and 8 rows (INT8: once per k, by a warp of its own), instead of
// five per weight and row.  What bounds
// it is W itself up to ~8 rows (INT4; INT8 throughout): W[4096,11008] INT4 with four rows 6x, INT8 with one row 3x faster
// than the fp32 kernel below.
//   * A CTA owns 256 (or 128) output features and a slice of K; a cluster of up to eight CTAs covers K and adds its partial
//     sums through distributed shared memory in ascending order (no scratch, no second kernel, the same bits every run).
//     How many features and slices: kn_split(), which fills whole waves of two CTAs per SM.
//   * A stage is 64 k: a TMA box of codes, two of activations (fp32, 128-byte swizzle) and the scales (cp.async).  A warp
//     owns 32 features (one scale column); lane (g, t) reads the 4 (INT4: a halfword) codes of features 4g .. 4g + 3 in four
//     rows of k, which is exactly what its fragments of two A tiles need, so nothing is transposed.
//
// kn_partial_kernel / kn_reduce_kernel: what the tensor-core form cannot take (INT4 groups of 16, N % 32, K % 4): a thread
// owns 16 consecutive output features, K is split into slices over the second grid dimension, codes become fp32 by a magic
// number and one subtraction; a second kernel adds the slices in ascending order and the bias.
//
// fp32 throughout in either form; the summation order differs from the reference's single chain, the result is inside the
// 1e-3 contract.  The split holds away from the ends of the exponent range only: the remainders of an Inf, and of a finite
// factor above bf16's largest value, are Inf - Inf, and those of a factor below about 2^-110 end under bf16's smallest.  The
// first makes every output of its row NaN, the second leaves outputs near zero, so the epilogue recognises both by the sum
// itself and, behind its last store, forms such an output again as the plain chain of fp32 multiply-adds (kn_chain4): +-Inf and NaN per output as
// in the reference, and no loss for vanishing rows.
#include "sgq_common.cuh"
#include "sm100_ptx.cuh"

#include <cooperative_groups.h>

namespace sgq {
namespace {

// ---------------------------------------------------------------------------------------------------------------------
// tensor-core form
// ---------------------------------------------------------------------------------------------------------------------
constexpr int kStageK = 64;
constexpr int kMmaWarps = 8;
constexpr int kMmaThreads = (kMmaWarps + 2) * 32;      // + producer warp, + a warp that splits the activations (INT8)
constexpr int kMmaMaxStages = 8;
constexpr int kMmaSmem = 108 * 1024;                    // two CTAs per SM
constexpr int kMaxCluster = 8;

__device__ uint32_t g_status_kn = 0;
__device__ __forceinline__ void report(uint32_t code, uint32_t detail) {
    atomicCAS(&g_status_kn, 0u, (code << 24) | (detail & 0xFFFFFFu));
}

// T: B tiles of eight columns per 16 k.  1: up to two rows (columns 2 * part + row); 2: up to four (columns row | 4 + row of the
// first tile hold parts 0 and 1, the second tile part 2); 3: up to eight (a tile per part); 6: up to sixteen (three per half).
template <int BITS, int T, int NBW>
struct KnCfg {
    static constexpr int kRowsX = T == 1 ? 2 : (T == 2 ? 4 : (T == 3 ? 8 : 16));
    static constexpr int kChains = T == 6 ? 2 : 1;               // sets of eight rows
    static constexpr int kAcc = T == 6 ? 4 : (T == 1 ? 1 : 2);    // accumulator tiles per A tile
    static constexpr int kFeatures = 32 * NBW;
    static constexpr int kKWays = kMmaWarps / NBW;               // warps that share a feature block take alternate 16 k
    static constexpr int kW = kStageK * kFeatures * BITS / 8;
    static constexpr int kXBox = kRowsX * 128 < 1024 ? 1024 : kRowsX * 128;
    static constexpr int kSBytes = BITS == 4 ? kStageK * NBW * 4 : 1024;
    // INT8: the factors do not depend on the feature: B fragments of a stage [16-k step][tile][lane] uint2, in two slots
    static constexpr int kFrag = BITS == 8 ? 4 * T * 256 : 0;
    static constexpr int kStage = (kW + 2 * kXBox + kSBytes + 1023) / 1024 * 1024;
    static constexpr int kPitch = kFeatures + 8;
    static constexpr int kPart = kKWays * kRowsX * kPitch * 4;
    static constexpr int kStages0 = (kMmaSmem - 1024 - kPart - 2 * kFrag - 2 * kMmaMaxStages * 8 - 32) / kStage;
    static constexpr int kStages = kStages0 < kMmaMaxStages ? kStages0 : kMmaMaxStages;
    static constexpr int kSmem = kStages * kStage + kPart + 2 * kFrag + 2 * kMmaMaxStages * 8 + 32 + 1024;
};

struct KnMmaParams {
    const float* scales;
    int scale_mode;          // 0: INT4 groups, 1: one per k, 2: one
    int64_t group;           // INT4: a multiple of 32 that divides N
    int64_t per_row;         // INT4: scales per k (N / group; a division per stage in the producer cost 4096 x 5792 10 %)
    int group_shift;         // log2(group / 32), or -1
    int pitch;               // INT4: scales per k in a stage (groups that a CTA's features span)
    int vec_scales;          // INT4: a stage's scales can be copied 16 bytes at a time
    const float* bias;
    float* y;
    int64_t ldy;
    int vec_y;
    int M;
    int64_t K, N;
    int early;               // weights may be requested before the dependency wait (overlapped launches)
    const float* x;          // the operands by address, for kn_chain4
    const uint8_t* wq;
};

__device__ __forceinline__ void kn_cp_async_16(uint32_t dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void kn_cp_async_4(uint32_t dst, const void* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ uint32_t bf16_fma(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}

// (p0, p1) = sum of three bf16 pairs, exactly (for finite values away from the ends of the exponent range)
__device__ __forceinline__ void split3(float p0, float p1, uint32_t (&part)[3]) {
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        part[j] = bf16_pair(p0, p1);
        p0 -= __uint_as_float(part[j] << 16);
        p1 -= __uint_as_float(part[j] & 0xFFFF0000u);
    }
}

// Whether one of four sums (without the bias) may come from factors that the split does not hold exactly: not finite, or
// below 2^-90 and not zero.  (Factors below 2^-110, or 2^-117 where remainders under 2^-126 count as zero, are wrong by at most 2^-126: 2^13
// of them times a code of 8 are 2^-110, a millionth of the smallest sum that passes.  A row of zeros is exact.)
__device__ __forceinline__ bool kn_sums_suspect(const float4& v) {
    constexpr uint32_t kLow = 0x12800000u, kHigh = 0x7F7FFFFFu;          // 2^-90 and the largest finite value, as bits
    const uint32_t a[4] = {__float_as_uint(v.x) & 0x7FFFFFFFu, __float_as_uint(v.y) & 0x7FFFFFFFu, __float_as_uint(v.z) & 0x7FFFFFFFu,
                           __float_as_uint(v.w) & 0x7FFFFFFFu};
    uint32_t far = 0;                                        // an unsigned difference is one compare for both ends
#pragma unroll
    for (int j = 0; j < 4; ++j) far |= (a[j] - kLow > kHigh - kLow && a[j] != 0u) ? 1u : 0u;
    return far != 0u;
}

// Four neighbouring outputs as one chain of fp32 multiply-adds each, in ascending k; x: the row of activations, w and s: the
// codes and the scale at k = 0.  A call of its own (not inlined) with its arguments by value: it runs for rows at the ends of the
// exponent range only, its registers are not the kernel's, and the parameter block keeps no address.
template <int BITS>
__device__ __noinline__ float4 kn_chain4(const float* x, const uint8_t* w, const float* s, int64_t K, int64_t row_bytes, int64_t scale_step) {
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 4
    for (int64_t k = 0; k < K; ++k) {
        const float f = x[k] * s[k * scale_step];
        const uint32_t c = BITS == 4 ? *reinterpret_cast<const uint16_t*>(w + k * row_bytes) : *reinterpret_cast<const uint32_t*>(w + k * row_bytes);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            acc[j] = fmaf(f, static_cast<float>(static_cast<int>(c << (32 - BITS - BITS * j)) >> (32 - BITS)), acc[j]);
    }
    return make_float4(acc[0], acc[1], acc[2], acc[3]);
}

template <int BITS, int T, int NBW>
__global__ void __launch_bounds__(kMmaThreads, 2)
kn_mma_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const KnMmaParams p) {
    using C = KnCfg<BITS, T, NBW>;
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    float* part = reinterpret_cast<float*>(smem + C::kStages * C::kStage);
    uint8_t* frags = smem + C::kStages * C::kStage + C::kPart;
    uint64_t* full = reinterpret_cast<uint64_t*>(frags + 2 * C::kFrag);
    uint64_t* empty = full + kMmaMaxStages;
    uint64_t* frag_full = empty + kMmaMaxStages;             // [2] INT8: the stage's fragments are written
    uint64_t* frag_empty = frag_full + 2;                    // [2] and read

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int rank = blockIdx.y, ranks = gridDim.y;
    const int nst = static_cast<int>((p.K + kStageK - 1) / kStageK);
    const int s0 = nst * rank / ranks, s1 = nst * (rank + 1) / ranks;
    const int64_t n0 = static_cast<int64_t>(blockIdx.x) * C::kFeatures;

    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int i = 0; i < C::kStages; ++i) {
            mbar_init(&full[i], 1 + 32);
            mbar_init(&empty[i], kMmaWarps + (BITS == 8 ? 1 : 0));
        }
        for (int i = 0; i < 2; ++i) { mbar_init(&frag_full[i], 1); mbar_init(&frag_empty[i], kMmaWarps); }
        mbar_fence_init();
        fence_proxy_async_smem();
    }
    __syncthreads();

    if (warp == kMmaWarps + 1) {
        // ------------------------------- INT8: factors x * s of a stage, split and laid out as B fragments --------------
        if (BITS == 8) {
            pdl_wait();
            const int g = lane >> 2, t = lane & 3;
            const int m0 = T == 1 ? (g & 1) : (T == 2 ? (g & 3) : g);
            const float s_all = p.scale_mode == 2 ? __ldg(p.scales) : 1.0f;
            int slot = 0;
            uint32_t ph = 0;
            for (int s = s0; s < s1; ++s) {
                const int fs = (s - s0) & 1;
                const uint32_t fph = ((s - s0) >> 1) & 1u;
                if (!mbar_wait(&full[slot], ph) || !mbar_wait(&frag_empty[fs], fph ^ 1u)) {
                    if (lane == 0) report(kDevErrFullWait, 0x800000u | s);
                    break;
                }
                const uint8_t* sx = smem + slot * C::kStage + C::kW;
                const float* ss = reinterpret_cast<const float*>(sx + 2 * C::kXBox);
                uint2* dst = reinterpret_cast<uint2*>(frags + fs * C::kFrag) + lane;
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
#pragma unroll
                    for (int c = 0; c < C::kChains; ++c) {
                        float f[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {        // k = 2t + (i & 1) + 8 (i >> 1) of the step
                            const int chunk = 4 * (kk & 1) + (t >> 1) + 2 * (i >> 1);
                            f[i] = *reinterpret_cast<const float*>(sx + (kk >> 1) * C::kXBox + c * 1024 + m0 * 128 + ((chunk ^ (m0 & 7)) << 4) +
                                                                   8 * (t & 1) + 4 * (i & 1)) *
                                   (p.scale_mode == 1 ? ss[16 * kk + 2 * t + (i & 1) + 8 * (i >> 1)] : s_all);
                        }
                        uint32_t b0[3], b1[3];
                        split3(f[0], f[1], b0);
                        split3(f[2], f[3], b1);
                        uint2* d = dst + (kk * T + 3 * c) * 32;
                        if (T == 1) {
                            d[0] = g < 2 ? make_uint2(b0[0], b1[0]) : (g < 4 ? make_uint2(b0[1], b1[1]) : (g < 6 ? make_uint2(b0[2], b1[2]) : make_uint2(0u, 0u)));
                        } else if (T == 2) {
                            d[0] = g < 4 ? make_uint2(b0[0], b1[0]) : make_uint2(b0[1], b1[1]);
                            d[32] = g < 4 ? make_uint2(b0[2], b1[2]) : make_uint2(0u, 0u);
                        } else {
#pragma unroll
                            for (int j = 0; j < 3; ++j) d[32 * j] = make_uint2(b0[j], b1[j]);
                        }
                    }
                }
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&frag_full[fs]);
                    mbar_arrive(&empty[slot]);
                }
                if (++slot == C::kStages) { slot = 0; ph ^= 1u; }
            }
        }
    } else if (warp == kMmaWarps) {
        // ------------------------------- producer ------------------------------------
        const bool leader = elect_one();
        auto codes = [&](int slot, int s) {
            mbar_arrive_expect_tx(&full[slot], C::kW + 2 * C::kRowsX * 128);
            uint8_t* sw = smem + slot * C::kStage;
            if (BITS == 4) {
                tma_load_2d(sw, &map_w, &full[slot], static_cast<int32_t>(n0 / 2), s * kStageK);
            } else {
#pragma unroll
                for (int h = 0; h < C::kFeatures / 128; ++h)
                    tma_load_2d(sw + h * (kStageK * 128), &map_w, &full[slot], static_cast<int32_t>(n0) + 128 * h, s * kStageK);
            }
        };
        auto rest = [&](int slot, int s) {
            uint8_t* sx = smem + slot * C::kStage + C::kW;
            if (leader) {
                tma_load_2d(sx, &map_x, &full[slot], s * kStageK, 0);
                tma_load_2d(sx + C::kXBox, &map_x, &full[slot], s * kStageK + 32, 0);
            }
            const uint32_t dst = smem_u32(sx + 2 * C::kXBox);
            const int64_t k0 = static_cast<int64_t>(s) * kStageK;
            if (BITS == 4 && p.group_shift >= 0) {
                const int64_t per_row = p.per_row, g0 = (n0 / 32) >> p.group_shift;
                if (p.vec_scales) {
                    const int quads = p.pitch / 4;                              // 1 or 2
                    for (int c = lane; c < kStageK * quads; c += 32) {
                        const int row = quads == 2 ? c >> 1 : c, c4 = quads == 2 ? c & 1 : 0;
                        const int64_t k = k0 + row, g = g0 + 4 * c4;
                        const bool in = k < p.K && g < per_row;
                        kn_cp_async_16(dst + c * 16, p.scales + (in ? k * per_row + g : 0), in ? 16 : 0);
                    }
                } else {
                    const int sh = p.pitch == 8 ? 3 : (p.pitch == 4 ? 2 : (p.pitch == 2 ? 1 : 0));
                    for (int e = lane; e < kStageK << sh; e += 32) {
                        const int64_t k = k0 + (e >> sh), g = g0 + (e & (p.pitch - 1));
                        const bool in = k < p.K && g < per_row;
                        kn_cp_async_4(dst + e * 4, p.scales + (in ? k * per_row + g : 0), in ? 4 : 0);
                    }
                }
            } else if (BITS == 4) {
                const int64_t per_row = p.per_row;
                for (int q = 0; q < kStageK * NBW / 32; ++q) {
                    const int e = lane + 32 * q, row = e / NBW, w = e % NBW;
                    const int64_t k = k0 + row, n = n0 + 32 * w;
                    const bool in = k < p.K && n < p.N;
                    kn_cp_async_4(dst + e * 4, p.scales + (in ? k * per_row + n / p.group : 0), in ? 4 : 0);
                }
            } else if (p.scale_mode == 1) {
#pragma unroll
                for (int q = 0; q < kStageK / 32; ++q) {
                    const int64_t k = k0 + lane + 32 * q;
                    kn_cp_async_4(dst + (lane + 32 * q) * 4, p.scales + (k < p.K ? k : 0), k < p.K ? 4 : 0);
                }
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&full[slot])) : "memory");
        };
        if (leader) {
            tma_prefetch_descriptor(&map_w);
            tma_prefetch_descriptor(&map_x);
        }
        const int head = s1 - s0 < C::kStages ? s1 - s0 : C::kStages;
        if (!p.early) pdl_wait();
        if (leader)
            for (int i = 0; i < head; ++i) codes(i, s0 + i);
        if (p.early) pdl_wait();
        for (int i = 0; i < head; ++i) rest(i, s0 + i);
        int slot = 0;
        uint32_t ph = 0;
        for (int s = s0 + head; s < s1; ++s) {
            if (!mbar_wait(&empty[slot], ph)) {
                if (leader) report(kDevErrEmptyWait, s);
                break;
            }
            if (leader) codes(slot, s);
            rest(slot, s);
            if (++slot == C::kStages) { slot = 0; ph ^= 1u; }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
        // ------------------------------- consumers -----------------------------------
        pdl_wait();
        const int g = lane >> 2, t = lane & 3;
        const int nb = warp % NBW, kh = warp / NBW;
        const int scol = p.group_shift >= 0 ? static_cast<int>(((n0 / 32 + nb) >> p.group_shift) - ((n0 / 32) >> p.group_shift)) : nb;
        float acc[2][C::kAcc][4];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < C::kAcc; ++j)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[i][j][c] = 0.0f;
        const int m0 = T == 1 ? (g & 1) : (T == 2 ? (g & 3) : g);
        const int soff = t * p.pitch + scol;
        // byte offsets of this lane's codes inside a 16-k step, rows (t, i): INT4 t + 4i, INT8 2t + (i & 1) + 8 (i >> 1)
        uint32_t woff[4], xoff = m0 * 128 + t * 4;           // xoff (INT4): + ((chunk i ^ row) << 4) below
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (BITS == 4) {
                const int r = t + 4 * i;
                woff[i] = NBW == 8 ? r * 128 + ((nb ^ (r & 7)) << 4) + 2 * g : r * 64 + ((nb ^ ((r >> 1) & 3)) << 4) + 2 * g;
            } else {
                const int r = 2 * t + (i & 1) + 8 * (i >> 1);
                woff[i] = (nb >> 2) * (kStageK * 128) + r * 128 + (((2 * (nb & 3) + (g >> 2)) ^ (r & 7)) << 4) + (g & 3) * 4;
            }
        }
        int slot = 0;
        uint32_t ph = 0;
        for (int s = s0; s < s1; ++s) {
            // One answer for the warp.  A warp that gives up hands nothing back, so the producer requests no more, and what it
            // did request is as old as this wait when the CTA ends.
            const bool ready = mbar_wait(&full[slot], ph) && (BITS == 4 || mbar_wait(&frag_full[(s - s0) & 1], ((s - s0) >> 1) & 1u));
            if (!__all_sync(0xffffffffu, ready)) {
                if (lane == 0) report(kDevErrFullWait, s);
                break;
            }
            const uint8_t* sw = smem + slot * C::kStage;
            const uint8_t* sx = sw + C::kW;
            const float* ss = reinterpret_cast<const float*>(sx + 2 * C::kXBox);
#pragma unroll
            for (int q = 0; q < 4 / C::kKWays; ++q) {
                const int kk = kh + q * C::kKWays;
                // ---- factors x * s of this lane's column, split into three bf16 parts (INT8: by the splitting warp) ----
                uint32_t b[C::kChains][2][3];                // [rows][k pair][part]
                uint2 frag[T];
                if (BITS == 4) {
                    float sc[4];
                    const float* sk = ss + 16 * kk * p.pitch + soff;
#pragma unroll
                    for (int i = 0; i < 4; ++i) sc[i] = sk[4 * i * p.pitch];
#pragma unroll
                    for (int c = 0; c < C::kChains; ++c) {
                        float f[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            f[i] = *reinterpret_cast<const float*>(sx + (kk >> 1) * C::kXBox + xoff + c * 1024 + (((4 * (kk & 1) + i) ^ (m0 & 7)) << 4)) * sc[i];
                        split3(f[0], f[1], b[c][0]);
                        split3(f[2], f[3], b[c][1]);
                    }
                    if (T == 1) {
                        frag[0].x = g < 2 ? b[0][0][0] : (g < 4 ? b[0][0][1] : (g < 6 ? b[0][0][2] : 0u));
                        frag[0].y = g < 2 ? b[0][1][0] : (g < 4 ? b[0][1][1] : (g < 6 ? b[0][1][2] : 0u));
                    } else if (T == 2) {
                        frag[0] = g < 4 ? make_uint2(b[0][0][0], b[0][1][0]) : make_uint2(b[0][0][1], b[0][1][1]);
                        frag[T - 1] = g < 4 ? make_uint2(b[0][0][2], b[0][1][2]) : make_uint2(0u, 0u);
                    } else {
#pragma unroll
                        for (int j = 0; j < T; ++j) frag[j] = make_uint2(b[j / 3][0][j % 3], b[j / 3][1][j % 3]);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < T; ++j) frag[j] = *(reinterpret_cast<const uint2*>(frags + ((s - s0) & 1) * C::kFrag) + (kk * T + j) * 32 + lane);
                }
                // ---- codes of features 4g .. 4g + 3 in four rows of k -> A fragments of two tiles ----
                uint32_t a[2][4];                            // tile i: features 4g + 2i (row g) and 4g + 2i + 1 (row g + 8)
                if (BITS == 4) {
                    uint32_t h[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) h[i] = *reinterpret_cast<const uint16_t*>(sw + kk * (16 * C::kFeatures / 2) + woff[i]);
                    const uint32_t u[2] = {h[0] | (h[1] << 16), h[2] | (h[3] << 16)};
#pragma unroll
                    for (int hl = 0; hl < 2; ++hl)
#pragma unroll
                        for (int j = 0; j < 4; ++j)          // 136 + code, minus 136: exact
                            a[j >> 1][2 * hl + (j & 1)] = bf16_fma(((u[hl] >> (4 * j)) & 0x000F000Fu) ^ 0x43084308u, 0x3F803F80u, 0xC308C308u);
                } else {
                    uint32_t w[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) w[i] = *reinterpret_cast<const uint32_t*>(sw + kk * (16 * 128) + woff[i]);
#pragma unroll
                    for (int hl = 0; hl < 2; ++hl)
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            // byte j of both rows; 128 + low seven bits, plus -128 or (sign bit) -256: exact
                            const uint32_t u = __byte_perm(w[2 * hl], w[2 * hl + 1], 0x0400 + 0x1111 * j);
                            a[j >> 1][2 * hl + (j & 1)] = bf16_fma((u & 0x007F007Fu) | 0x43004300u, 0x3F803F80u, (u & 0x00800080u) | 0xC300C300u);
                        }
                }
                // ---- products: parts 1 and 2 of a row in a tile of their own share an accumulator ----
#pragma unroll
                for (int j = 0; j < T; ++j)
#pragma unroll
                    for (int i = 0; i < 2; ++i)
                        mma_bf16_16816(acc[i][T <= 2 ? j : 2 * (j / 3) + (j % 3 ? 1 : 0)], a[i], frag[j].x, frag[j].y);
            }
            uint32_t fold = 0;
#pragma unroll
            for (int j = 0; j < C::kAcc; ++j) fold ^= __float_as_uint(acc[0][j][0]) ^ __float_as_uint(acc[1][j][3]);
            const uint32_t landed = loads_landed(fold);
            if (lane == 0) {
                mbar_arrive_after(&empty[slot], landed);
                if (BITS == 8) mbar_arrive_after(&frag_empty[(s - s0) & 1], landed);
            }
            if (++slot == C::kStages) { slot = 0; ph ^= 1u; }
        }
        // ---- this warp's sums: smallest parts first, then [K ways][row][feature] in shared memory ----
#pragma unroll
        for (int c = 0; c < C::kChains; ++c) {
            float v[2][4];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    if (T == 1) {                           // parts sit in the columns of lanes t = 0, 1, 2
                        const float d = acc[i][0][e];
                        const float mid = __shfl_sync(0xffffffffu, d, (lane & ~3) | 1), low = __shfl_sync(0xffffffffu, d, (lane & ~3) | 2);
                        v[i][e] = (low + mid) + d;
                    } else if (T == 2) {                    // part 1 two lanes up, part 2 in the other tile
                        const float mid = __shfl_sync(0xffffffffu, acc[i][0][e], (lane & ~3) | ((t + 2) & 3));
                        v[i][e] = (acc[i][C::kAcc - 1][e] + mid) + acc[i][0][e];
                    } else {
                        v[i][e] = acc[i][(2 * c + 1) % C::kAcc][e] + acc[i][2 * c % C::kAcc][e];
                    }
                }
            const int m = 8 * c + 2 * t;                     // columns 2t, 2t + 1
            if (m + 1 < C::kRowsX + 1 && m < C::kRowsX) {
                float* dst = part + (kh * C::kRowsX + m) * C::kPitch + 32 * nb + 4 * g;
                *reinterpret_cast<float4*>(dst) = make_float4(v[0][0], v[0][2], v[1][0], v[1][2]);
                *reinterpret_cast<float4*>(dst + C::kPitch) = make_float4(v[0][1], v[0][3], v[1][1], v[1][3]);
            }
        }
    }
    cluster.sync();                                          // every CTA's sums are in its shared memory
    const int quads = C::kFeatures / 4, step = ranks * kMmaThreads;
    uint32_t suspect = 0;                                    // bit per quad of this thread (at most 16 * 64 / 320 = 4)
    auto store = [&](float4 v, int m, int64_t n) {
        if (p.bias) { v.x += p.bias[n]; v.y += p.bias[n + 1]; v.z += p.bias[n + 2]; v.w += p.bias[n + 3]; }
        float* dst = p.y + static_cast<int64_t>(m) * p.ldy + n;
        if (p.vec_y) {
            *reinterpret_cast<float4*>(dst) = v;
        } else {
            dst[0] = v.x; dst[1] = v.y; dst[2] = v.z; dst[3] = v.w;
        }
    };
    uint32_t bit = 1;
    for (int e = rank * kMmaThreads + threadIdx.x; e < p.M * quads; e += step, bit <<= 1) {
        const int m = e / quads, c = (e - m * quads) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int r = 0; r < ranks; ++r) {
            const float* src = cluster.map_shared_rank(part, r);
#pragma unroll
            for (int kw = 0; kw < C::kKWays; ++kw) {
                const float4 q = *reinterpret_cast<const float4*>(src + (kw * C::kRowsX + m) * C::kPitch + c);
                v.x += q.x; v.y += q.y; v.z += q.z; v.w += q.w;
            }
        }
        if (n0 + c < p.N) {                                  // N % 4 == 0
            store(v, m, n0 + c);
            if (kn_sums_suspect(v)) suspect |= bit;
        }
    }
    cluster.sync();                                          // shared memory stays until the others have read it
    if (suspect != 0) {
        for (int e = rank * kMmaThreads + threadIdx.x; suspect != 0; e += step, suspect >>= 1) {
            if ((suspect & 1u) == 0) continue;
            const int m = e / quads, c = (e - m * quads) * 4;
            const int64_t n = n0 + c;
            store(kn_chain4<BITS>(p.x + static_cast<int64_t>(m) * p.K, p.wq + (BITS == 4 ? n / 2 : n), p.scales + (BITS == 4 ? n / p.group : 0), p.K,
                                  BITS == 4 ? p.N / 2 : p.N, BITS == 4 ? p.per_row : (p.scale_mode == 1 ? 1 : 0)), m, n);
        }
    }
}

// Features per CTA (256 or 128) and slices of K (the cluster size): the split with the shortest longest CTA, in stages of 64 k
// and 256 features plus a fixed cost of starting and of adding up, times the waves of two CTAs per SM that it takes.
struct KnSplit {
    int nbw, slices;
};
KnSplit kn_split(int64_t K, int64_t N) {
    const int64_t nst = ceil_div(K, kStageK), slots = 2LL * sm_count();
    KnSplit best{8, 1};
    double cost = 1e300;
    for (int nbw = 8; nbw >= 4; nbw /= 2)
        for (int c = 1; c <= kMaxCluster && c <= nst; ++c) {
            const int64_t ctas = ceil_div(N, 32 * nbw) * c;
            const double w = static_cast<double>(ceil_div(ctas, slots)) * (static_cast<double>(ceil_div(nst, c)) * nbw / 8 + 4.0);
            if (w < cost) { cost = w; best = KnSplit{nbw, c}; }
        }
    return best;
}

template <int BITS, int T, int NBW>
int launch_mma(const LinearArgs& a, int slices) {
    using C = KnCfg<BITS, T, NBW>;
    static SmemOptIn optin;
    SGQ_CUDA_TRY(optin.ensure(kn_mma_kernel<BITS, T, NBW>, C::kSmem));
    CUtensorMap map_w, map_x;
    const uint64_t row_bytes = static_cast<uint64_t>(BITS == 4 ? a.N / 2 : a.N);
    if (!make_tensor_map_2d(&map_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, a.wq, row_bytes, static_cast<uint64_t>(a.K), row_bytes,
                            BITS == 4 ? 16 * NBW : 128, kStageK, BITS == 4 && NBW == 4 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B) ||
        !make_tensor_map_2d(&map_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, a.x, static_cast<uint64_t>(a.K), static_cast<uint64_t>(a.M),
                            static_cast<uint64_t>(a.K) * 4, 32, C::kRowsX, CU_TENSOR_MAP_SWIZZLE_128B))
        return SGQ_ERR_CUDA;
    KnMmaParams p{};
    p.scales = a.scales;
    p.scale_mode = BITS == 4 ? 0 : (a.scheme == SGQ_PER_ROW ? 1 : 2);
    p.group = a.group;
    p.per_row = BITS == 4 ? a.N / a.group : 1;
    p.group_shift = -1;
    p.pitch = NBW;
    if (BITS == 4) {
        for (int sh = 0; sh < 20; ++sh)
            if (a.group == 32LL << sh) p.group_shift = sh;
        // (a CTA starts at a multiple of NBW features of 32, so groups of up to as many never straddle its edge)
        if (p.group_shift >= 0) p.pitch = NBW >> p.group_shift ? NBW >> p.group_shift : 1;
        p.vec_scales = p.group_shift >= 0 && p.pitch % 4 == 0 && (a.N / a.group) % 4 == 0 && aligned(a.scales, 16) ? 1 : 0;
    }
    p.bias = a.bias; p.y = a.y; p.ldy = a.ldy; p.M = static_cast<int>(a.M); p.K = a.K; p.N = a.N;
    p.vec_y = aligned(a.y, 16) && (a.ldy % 4) == 0 ? 1 : 0;
    p.early = stream_overlap_enabled() ? 1 : 0;
    p.x = a.x; p.wq = static_cast<const uint8_t*>(a.wq);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(ceil_div(a.N, C::kFeatures)), static_cast<unsigned>(slices));
    cfg.blockDim = dim3(kMmaThreads);
    cfg.dynamicSmemBytes = C::kSmem;
    cfg.stream = a.stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = static_cast<unsigned>(slices);
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    SGQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kn_mma_kernel<BITS, T, NBW>, map_w, map_x, p));
    return SGQ_OK;
}

template <int BITS, int T>
int launch_mma_nb(const LinearArgs& a, const KnSplit& sp) {
    return sp.nbw == 8 ? launch_mma<BITS, T, 8>(a, sp.slices) : launch_mma<BITS, T, 4>(a, sp.slices);
}

template <int BITS>
int launch_mma_rows(const LinearArgs& a, const KnSplit& sp) {
    if (a.M <= 2) return launch_mma_nb<BITS, 1>(a, sp);
    if (a.M <= 4) return launch_mma_nb<BITS, 2>(a, sp);
    if (a.M <= 8) return launch_mma_nb<BITS, 3>(a, sp);
    return launch_mma_nb<BITS, 6>(a, sp);
}

// Whether the output rows and x share memory (a caller that multiplies in place, K == N).
bool output_overlaps_x(const LinearArgs& a) {
    const uintptr_t x0 = reinterpret_cast<uintptr_t>(a.x), y0 = reinterpret_cast<uintptr_t>(a.y);
    const uintptr_t x1 = x0 + static_cast<uintptr_t>(a.M * a.K) * 4, y1 = y0 + static_cast<uintptr_t>((a.M - 1) * a.ldy + a.N) * 4;
    return x0 < y1 && y0 < x1;
}

// TMA needs rows that are multiples of 16 bytes; a warp's 32 features must lie in one INT4 group.  One launch reads x and
// stores y, a cluster storing its columns while others still load x: an output that overlaps x goes to the any-shape form,
// whose first launch reads the rows of a pass and whose second stores them.
bool kn_mma_supported(const LinearArgs& a) {
    return !output_overlaps_x(a) && (a.K % 4) == 0 && aligned(a.x, 16) && (a.bits == 8 || ((a.N % 32) == 0 && (a.group % 32) == 0)) && a.K < (1LL << 24);
}

// ---------------------------------------------------------------------------------------------------------------------
// any-shape form
// ---------------------------------------------------------------------------------------------------------------------

constexpr int kThreads = 128;
constexpr int kColsPerThread = 16;
constexpr int kColsPerBlock = kThreads * kColsPerThread;   // 2048
constexpr int kMaxSliceK = 256;                            // k per slice (x slice of MB rows sits in shared memory)
constexpr int kMaxM = 16;

template <int BITS>
struct Word;
template <>
struct Word<4> {
    using T = uint2;   // 16 nibbles
};
template <>
struct Word<8> {
    using T = uint4;   // 16 bytes
};

// 16 codes of one k as fp32
template <int BITS>
__device__ __forceinline__ void codes_to_float(const typename Word<BITS>::T& w, float (&c)[16]) {
    if constexpr (BITS == 4) {
        const uint32_t words[2] = {w.x, w.y};
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int j = 0; j < 8; ++j)
                c[8 * h + j] = __uint_as_float(0x4B000000u | (((words[h] >> (4 * j)) & 0xFu) ^ 8u)) - 8388616.0f;
    } else {
        const uint32_t words[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int h = 0; h < 4; ++h)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                c[4 * h + j] = __uint_as_float(0x4B000000u | (((words[h] >> (8 * j)) & 0xFFu) ^ 0x80u)) - 8388736.0f;
    }
}

// scale_mode: 0 = INT4 groups (scales[(k * N + n) / group]), 1 = one scale per k, 2 = one scale
template <int BITS, int MB>
__global__ void __launch_bounds__(kThreads) kn_partial_kernel(const float* __restrict__ x, int64_t K, int64_t N,
                                                              const uint8_t* __restrict__ wq, const float* __restrict__ scales,
                                                              int scale_mode, int64_t group, int slice_k, float* __restrict__ part) {
    __shared__ float xs[MB][kMaxSliceK];
    pdl_launch_dependents();
    pdl_wait();
    const int64_t k0 = static_cast<int64_t>(blockIdx.y) * slice_k;
    const int kn = static_cast<int>((K - k0 < slice_k) ? K - k0 : slice_k);
    for (int i = threadIdx.x; i < MB * kn; i += kThreads) {
        const int m = i / kn, kk = i - m * kn;
        xs[m][kk] = x[static_cast<int64_t>(m) * K + k0 + kk];
    }
    __syncthreads();
    const int64_t n0 = (static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x) * kColsPerThread;
    if (n0 >= N) return;                                     // N % 16 == 0: a thread is in or out as a whole
    float acc[MB][16];
#pragma unroll
    for (int m = 0; m < MB; ++m)
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[m][j] = 0.0f;

    using W = typename Word<BITS>::T;
    const int64_t row_bytes = (BITS == 4) ? N / 2 : N;
    const uint8_t* wp = wq + k0 * row_bytes + ((BITS == 4) ? n0 / 2 : n0);
    const float s_all = (scale_mode == 2) ? __ldg(scales) : 1.0f;
    constexpr int U = 4;                                     // k rows in flight per thread
    for (int kk = 0; kk < kn; kk += U) {
        W w[U];
        float s[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = (kk + u < kn) ? kk + u : kn - 1;   // clamped: the tail reloads a valid row, its x is zeroed below
            w[u] = __ldcs(reinterpret_cast<const W*>(wp + static_cast<int64_t>(k) * row_bytes));
            if (scale_mode == 0)
                s[u] = __ldg(scales + ((k0 + k) * N + n0) / group);
            else if (scale_mode == 1)
                s[u] = __ldg(scales + k0 + k);
            else
                s[u] = s_all;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            float c[16];
            codes_to_float<BITS>(w[u], c);
            const bool live = kk + u < kn;
#pragma unroll
            for (int m = 0; m < MB; ++m) {
                const float xsv = live ? xs[m][kk + u] * s[u] : 0.0f;
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[m][j] = fmaf(xsv, c[j], acc[m][j]);
            }
        }
    }
    float* out = part + (static_cast<int64_t>(blockIdx.y) * MB) * N + n0;
#pragma unroll
    for (int m = 0; m < MB; ++m)
#pragma unroll
        for (int j = 0; j < 16; j += 4)
            *reinterpret_cast<float4*>(out + static_cast<int64_t>(m) * N + j) =
                make_float4(acc[m][j], acc[m][j + 1], acc[m][j + 2], acc[m][j + 3]);
}

// y[m, n] = sum over slices (ascending) + bias
__global__ void __launch_bounds__(256) kn_reduce_kernel(const float* __restrict__ part, int slices, int mb, int64_t N,
                                                        const float* __restrict__ bias, float* __restrict__ y, int64_t ldy) {
    pdl_launch_dependents();
    pdl_wait();
    const int64_t total = static_cast<int64_t>(mb) * N;
    for (int64_t i = blockIdx.x * 256ll + threadIdx.x; i < total; i += gridDim.x * 256ll) {
        const int64_t m = i / N, n = i - m * N;
        float v = 0.0f;
        for (int s = 0; s < slices; ++s) v += __ldcg(part + (static_cast<int64_t>(s) * mb + m) * N + n);
        if (bias) v += bias[n];
        y[m * ldy + n] = v;
    }
}

struct KnPlan {
    int mb;          // batch rows per pass (1, 2 or 4)
    int slice_k;     // k per slice
    int slices;
    int nblocks;
};

KnPlan kn_plan(int64_t M, int64_t K, int64_t N) {
    KnPlan p;
    p.mb = M >= 4 ? 4 : (M >= 2 ? 2 : 1);
    p.nblocks = static_cast<int>(ceil_div(N, kColsPerBlock));
    int64_t want_slices = ceil_div(static_cast<int64_t>(6) * sm_count(), p.nblocks);   // ~6 CTAs of 128 threads per SM
    int64_t sk = ceil_div(K, want_slices);
    sk = (sk + 7) / 8 * 8;
    if (sk < 16) sk = 16;
    if (sk > kMaxSliceK) sk = kMaxSliceK;
    p.slice_k = static_cast<int>(sk);
    p.slices = static_cast<int>(ceil_div(K, sk));
    return p;
}

template <int BITS, int MB>
int launch_pass(const LinearArgs& a, const KnPlan& p, int scale_mode, const float* x, float* y, int rows, float* part) {
    SGQ_CUDA_TRY(launch_kernel(kn_partial_kernel<BITS, MB>, dim3(static_cast<unsigned>(p.nblocks), static_cast<unsigned>(p.slices)),
                               dim3(kThreads), 0, a.stream, true, x, a.K, a.N, static_cast<const uint8_t*>(a.wq), a.scales,
                               scale_mode, a.group, p.slice_k, part));
    int64_t blocks = ceil_div(static_cast<int64_t>(rows) * a.N, 256);
    const int64_t cap = static_cast<int64_t>(sm_count()) * 8;
    if (blocks > cap) blocks = cap;
    SGQ_CUDA_TRY(launch_kernel(kn_reduce_kernel, dim3(static_cast<unsigned>(blocks)), dim3(256), 0, a.stream, true,
                               static_cast<const float*>(part), p.slices, MB, a.N, a.bias, y, a.ldy));
    (void)rows;
    return SGQ_OK;
}

}  // namespace

cudaError_t read_status_kn(uint32_t* v, bool clear) {
    cudaError_t e = cudaMemcpyFromSymbol(v, g_status_kn, sizeof(uint32_t));
    if (e == cudaSuccess && clear && *v != 0) {
        const uint32_t zero = 0;
        e = cudaMemcpyToSymbol(g_status_kn, &zero, sizeof(zero));
    }
    return e;
}

bool kn_decode_supported(const LinearArgs& a) {
    if (a.layout != SGQ_LAYOUT_KN || a.M < 1 || a.M > kMaxM || a.K < 1 || a.N < 16 || (a.N % 16) != 0) return false;
    if (a.K >= (1LL << 31) || a.N >= (1LL << 31)) return false;
    if (!aligned(a.wq, 16) || !aligned(a.x, 4)) return false;
    if (a.bits == 4) return a.group >= 16 && (a.group % 16) == 0 && (a.N % a.group) == 0;
    return a.bits == 8;
}

size_t kn_decode_workspace_bytes(int bits, int64_t M, int64_t K, int64_t N) {
    (void)bits;
    if (M < 1 || M > kMaxM || K < 1 || N < 16 || (N % 16) != 0) return 0;
    const KnPlan p = kn_plan(M, K, N);
    return (static_cast<size_t>(p.slices) * p.mb * N * sizeof(float) + 255) / 256 * 256;
}

int launch_linear_kn_decode(const LinearArgs& a) {
    if (!kn_decode_supported(a)) {
        set_error("[K,N] decode path needs M<=16, N%%16==0, INT4 groups that are a multiple of 16 and divide N, 16-byte aligned codes");
        return SGQ_ERR_UNSUPPORTED;
    }
    const size_t need = kn_decode_workspace_bytes(a.bits, a.M, a.K, a.N);
    if (!a.workspace || a.workspace_bytes < need || !aligned(a.workspace, 256)) {
        set_error("[K,N] decode path needs %zu bytes of 256-byte aligned workspace", need);
        return SGQ_ERR_WORKSPACE;
    }
    if (kn_mma_supported(a)) {
        const KnSplit sp = kn_split(a.K, a.N);
        return a.bits == 4 ? launch_mma_rows<4>(a, sp) : launch_mma_rows<8>(a, sp);
    }
    const KnPlan p = kn_plan(a.M, a.K, a.N);
    const int scale_mode = a.bits == 4 ? 0 : (a.scheme == SGQ_PER_ROW ? 1 : 2);
    float* part = static_cast<float*>(a.workspace);
    // batches larger than the pass width run as several passes over row blocks (weights streamed again)
    for (int64_t m0 = 0; m0 < a.M;) {
        const int64_t left = a.M - m0;
        const int mb = (p.mb == 4 && left >= 4) ? 4 : (left >= 2 && p.mb >= 2 ? 2 : 1);
        const float* x = a.x + m0 * a.K;
        float* y = a.y + m0 * a.ldy;
        int rc;
        if (a.bits == 4)
            rc = mb == 4 ? launch_pass<4, 4>(a, p, scale_mode, x, y, mb, part)
                         : (mb == 2 ? launch_pass<4, 2>(a, p, scale_mode, x, y, mb, part) : launch_pass<4, 1>(a, p, scale_mode, x, y, mb, part));
        else
            rc = mb == 4 ? launch_pass<8, 4>(a, p, scale_mode, x, y, mb, part)
                         : (mb == 2 ? launch_pass<8, 2>(a, p, scale_mode, x, y, mb, part) : launch_pass<8, 1>(a, p, scale_mode, x, y, mb, part));
        if (rc != SGQ_OK) return rc;
        m0 += mb;
    }
    return SGQ_OK;
}

}  // namespace sgq
