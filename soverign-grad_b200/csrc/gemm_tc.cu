// Prefill-shape forward on the 5th-generation tensor cores (tcgen05.mma, accumulators in TMEM):
// y[M,N] = x[M,K] * deq(W) + bias, weights stored [N,K] or [K,N].
//
// Two persistent, warp-specialised kernels:
//   linear_pair_kernel  both operands arrive by TMA in the form the MMA reads.  Two CTAs (cta_group::2) share a tile
//         of 256 rows and up to 256 columns: INT8 codes x INT8 activations (kind::i8, exact int32 sums, the epilogue
//         applies sx[m] * sw[n]), or bf16 activations x a weight that expand_ordered_kernel has expanded to bf16.
//   linear_tc_kernel    weights stored [N,K] dequantized in shared memory, for callers whose scratch has no room for
//         the expanded weight: activations are pre-converted to bf16; packed INT4 weights arrive by TMA as raw
//         nibbles and dequant warps expand them in shared memory to bf16 (exact integer from one LOP3 per pair, times
//         the bf16-rounded group scale) directly in the swizzled K-major layout the MMA reads; INT8 codes likewise,
//         with their scale in the epilogue.  One CTA per 256 x 256 tile (two 128-row halves, each with its own
//         256-column accumulator, sharing every B tile).  Warps: 0 = TMA producer of A, 1 = MMA issuer (one thread),
//         2..5 = epilogue (TMEM lane quarter = warp % 4), 6 = TMA producer of the raw codes, 7..22 = dequant (512
//         threads, two per weight row).
// All waits are bounded; a wait that runs out records a code in the device status word and the role winds down to the
// common exit.
#include <cuda_bf16.h>

#include <cstring>

#include "sgq_common.cuh"
#include "sm100_ptx.cuh"

namespace sgq {

__device__ uint32_t g_status_gemm = 0;

cudaError_t read_status_gemm(uint32_t* v, bool clear) {
    cudaError_t e = cudaMemcpyFromSymbol(v, g_status_gemm, sizeof(uint32_t));
    if (e == cudaSuccess && clear && *v != 0) {
        const uint32_t zero = 0;
        e = cudaMemcpyToSymbol(g_status_gemm, &zero, sizeof(zero));
    }
    return e;
}

namespace {

// bf16 x INT4 g=32 | bf16 x INT8 codes (scale in the epilogue)
enum Mode { kBF16 = 1, kBF16W8 = 2 };

constexpr int BM = 256, BN = 256;     // two UMMA_M = 128 halves per tile
constexpr int kHalfM = 128;
constexpr int kABytes = BM * 128;     // 256 rows x 128 B (rows 128.. are the second half)
constexpr int kBBytes = BN * 128;     // 256 rows x 128 B
constexpr int kRawBytes = BN * 32;    // 256 rows x 64 nibbles (kBF16); the INT8 form is twice that, Cfg::kRawStageBytes
constexpr int kDequantWarps = 16;     // two threads per row of the 256-row weight tile (one 32-k group each)
constexpr int kEpilogueWarp0 = 2;
constexpr int kBProducerWarp = 6;     // loads the raw codes
constexpr int kDequantWarp0 = 7;
constexpr int kTmemCols = 512;

// Three rings with their own depth, so that the latency of a TMA load never sits in the chain
// "MMA frees a slot -> slot refilled -> MMA": A tiles and raw nibbles are requested several
// k-blocks ahead; the (large) bf16 B tiles only need to cover the dequant time.
template <int MODE>
struct Cfg {
    static constexpr int kBlockK = 64;                               // elements per k-block
    static constexpr int kUmmaK = 16;                                // elements per instruction (32 bytes)
    static constexpr int kAStages = MODE == kBF16W8 ? 2 : 3;         // the INT8 raw ring takes the room of one A stage
    static constexpr int kBStages = 3;
    static constexpr int kRawStages = 3;
    static constexpr int kRawStageBytes = MODE == kBF16W8 ? BN * 64 : kRawBytes;
    static constexpr int kWarps = 7 + kDequantWarps;
    static constexpr int kThreads = kWarps * 32;
    static constexpr int kAOff = 0;
    static constexpr int kBOff = kAStages * kABytes;
    static constexpr int kRawOff = kBOff + kBStages * kBBytes;
    static constexpr int kOutOff = kRawOff + kRawStages * kRawStageBytes;   // 4 epilogue warps x [16 rows x 32 fp32], swizzled
    static constexpr int kBarOffset = kOutOff + 4 * 2048;
    static constexpr int kNumBars = 2 * kAStages + 2 * kBStages + 2 * kRawStages + 4;
    static constexpr int kSmemBytes = kBarOffset + kNumBars * 8 + 16 + 1024;   // barriers + tmem slot + alignment slack
};

struct Params {
    const float* bias;      // [N] or null
    float* y;               // [M, ldy]
    int64_t ldy;
    int64_t M, N, K;
    const float* sx;        // W8A8: [M] activation scales
    const float* sw;        // weight scales of the epilogue: [1] or [N], or null
    int sw_per_row;
    int32_t* acc_out;       // W8A8: optional [M,N]
    const float* wscales;   // kBF16: [N, K/32]
    int vec_store;          // y is 16-byte aligned with ldy % 4 == 0: 128-bit stores
    // linear_pair_kernel
    int bn;                 // columns of a tile: a multiple of 32, at most 256
    int b_mn;               // B is stored [K,N] (the MMA reads it MN-major), else [N,K]
    // The operands may still be being written when the kernel starts (see expand_ordered_kernel).  They become
    // complete slice of K by slice of K; ready[q] counts the expansion CTAs that have finished slice q of x and of W.
    const uint32_t* ready;      // null: both operands are complete before the launch
    uint32_t ready_target;      // CTAs of the expansion launch
    int ready_part_kblocks;     // k-blocks per slice
    // Column-sharded layer: the output tile goes into every GPU's full-width output (plain peer stores from the
    // epilogue), so the all-gather needs no pass of its own.  n_peers == 0: y only.
    float* peer_y[kMaxPeers];
    int n_peers;
};

__device__ __forceinline__ void report(uint32_t code, uint32_t detail) {
    atomicCAS(&g_status_gemm, 0u, (code << 24) | (detail & 0xFFFFFFu));
}

// Waits (bounded: about a second) until `target` CTAs of the expansion launch have counted themselves into *cnt,
// then orders the TMA loads that follow behind what those CTAs wrote.  false = gave up.
__device__ __forceinline__ bool wait_expanded(const uint32_t* cnt, uint32_t target) {
    for (uint32_t n = 0; n < (1u << 22); ++n) {
        uint32_t v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(cnt) : "memory");
        if (v >= target) {
            fence_proxy_async_all();
            return true;
        }
        __nanosleep(200);
    }
    return false;
}

// Position in a ring of N slots and the mbarrier phase that goes with it, advanced by steps of
// `stride` without any division (these loops run in single threads that feed the tensor core).
template <int N>
struct Ring {
    int slot = 0;
    uint32_t phase = 0;
    __device__ __forceinline__ void advance(int stride = 1) {
        slot += stride;
        while (slot >= N) {
            slot -= N;
            phase ^= 1u;
        }
    }
};

// Walks this CTA's (tile, k-block) sequence: tiles blockIdx.x, +gridDim.x, ...; kb = 0..kblocks-1.
struct Walk {
    int64_t tile;
    int kb = 0;
    uint32_t tcount = 0;   // tiles completed so far
    __device__ __forceinline__ explicit Walk(int64_t first_tile) : tile(first_tile) {}
    __device__ __forceinline__ void advance(int stride, int kblocks, int64_t tile_stride) {
        kb += stride;
        while (kb >= kblocks) {
            kb -= kblocks;
            tile += tile_stride;
            ++tcount;
        }
    }
};

// The epilogue of one warp.  TMEM hands lane i row i of a [32 x 32] block; stored like that each store instruction would
// touch 32 different 128-byte lines.  The block goes through shared memory instead, 16 rows at a time (16-byte chunk j of
// row i at position j ^ (i & 7): conflict free both ways), and leaves with every instruction writing 4 complete 128-byte
// row segments.
// PEERS: every tile goes into p.n_peers outputs (a column-sharded layer; a form of its own so that the single-output
// epilogue keeps its straight-line stores).
template <bool I8, bool PEERS>
struct Epilogue {
    const Params& p;
    uint8_t* stage_out;
    const int lane, cq, rq;        // after the transpose: columns 4cq..4cq+3, rows rq + 4i
    const bool scale_n;            // weight scale applied per output column here
    const float sw_all;
    __device__ __forceinline__ Epilogue(const Params& p_, uint8_t* stage, int lane_)
        : p(p_), stage_out(stage), lane(lane_), cq(lane_ & 7), rq(lane_ >> 3), scale_n(p_.sw != nullptr),
          sw_all((p_.sw != nullptr && !p_.sw_per_row) ? p_.sw[0] : 1.0f) {}

    __device__ __forceinline__ void store4(float* dst, bool vec, const float4& o, int64_t n4) const {
        if (vec) {
            *reinterpret_cast<float4*>(dst) = o;
        } else {
            if (n4 + 0 < p.N) dst[0] = o.x;
            if (n4 + 1 < p.N) dst[1] = o.y;
            if (n4 + 2 < p.N) dst[2] = o.z;
            if (n4 + 3 < p.N) dst[3] = o.w;
        }
    }

    // 32 rows from mrow0 on (one TMEM lane each), `cols` columns (a multiple of 32) from n0 on
    __device__ __forceinline__ void rows32(uint32_t taddr, int64_t mrow0, int64_t n0, int cols) const {
        const int64_t m = mrow0 + lane;
        if (mrow0 >= p.M) return;                                  // uniform across the warp
        float sxm = 1.0f;
        if (I8 && m < p.M) sxm = p.sx[m];
        for (int c = 0; c < cols / 32; ++c) {
            const int64_t nb = n0 + c * 32;
            if (nb >= p.N) break;                                  // uniform across the warp
            uint32_t v[32];
            tmem_ld_32x32b_x32(taddr + c * 32, v);
            // column-dependent factors of this lane's 4 columns after the transpose
            const int64_t n4 = nb + 4 * cq;
            float swv[4] = {sw_all, sw_all, sw_all, sw_all}, bv[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (n4 + e < p.N) {
                    if (scale_n && p.sw_per_row) swv[e] = p.sw[n4 + e];
                    if (p.bias) bv[e] = p.bias[n4 + e];
                }
            }
            tmem_ld_wait();
            if (I8 && p.acc_out && m < p.M) {
#pragma unroll
                for (int j = 0; j < 32; ++j)
                    if (nb + j < p.N) p.acc_out[m * p.N + nb + j] = static_cast<int32_t>(v[j]);
            }
            const bool vec = p.vec_store && n4 + 4 <= p.N;
#pragma unroll
            for (int part = 0; part < 2; ++part) {                 // rows 0..15, then 16..31 of the block
                __syncwarp();                                       // the previous part has been read out
                if ((lane >> 4) == part) {
                    const int lr = lane & 15;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        float4 o;
                        if (I8) {                              // row scale first: y = ((float)acc * sx[m]) * sw[n] + bias[n]
                            o.x = __fmul_rn(static_cast<float>(static_cast<int32_t>(v[4 * j + 0])), sxm);
                            o.y = __fmul_rn(static_cast<float>(static_cast<int32_t>(v[4 * j + 1])), sxm);
                            o.z = __fmul_rn(static_cast<float>(static_cast<int32_t>(v[4 * j + 2])), sxm);
                            o.w = __fmul_rn(static_cast<float>(static_cast<int32_t>(v[4 * j + 3])), sxm);
                        } else {
                            o = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]),
                                            __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
                        }
                        *reinterpret_cast<float4*>(stage_out + lr * 128 + ((j ^ (lr & 7)) << 4)) = o;
                    }
                }
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int row = rq + 4 * i;                     // 0..15 inside the part
                    const int64_t mm = mrow0 + part * 16 + row;
                    float4 o = *reinterpret_cast<const float4*>(stage_out + row * 128 + ((cq ^ (row & 7)) << 4));
                    if (scale_n) {
                        o.x = __fmul_rn(o.x, swv[0]); o.y = __fmul_rn(o.y, swv[1]); o.z = __fmul_rn(o.z, swv[2]); o.w = __fmul_rn(o.w, swv[3]);
                    }
                    if (p.bias) {
                        o.x = __fadd_rn(o.x, bv[0]); o.y = __fadd_rn(o.y, bv[1]); o.z = __fadd_rn(o.z, bv[2]); o.w = __fadd_rn(o.w, bv[3]);
                    }
                    if (mm < p.M) {
                        if constexpr (PEERS) {
#pragma unroll 1
                            for (int r = 0; r < p.n_peers; ++r) store4(p.peer_y[r] + mm * p.ldy + n4, vec, o, n4);
                        } else {
                            store4(p.y + mm * p.ldy + n4, vec, o, n4);
                        }
                    }
                }
            }
        }
    }
};
template <int MODE>
__global__ void __launch_bounds__(Cfg<MODE>::kThreads, 1)
linear_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, Params p) {
    using C = Cfg<MODE>;
    constexpr int NA = C::kAStages, NB = C::kBStages, NR = C::kRawStages;
    extern __shared__ uint8_t smem_raw[];
    // aligned by pointer arithmetic on the shared array itself: a round trip through an integer would make the
    // compiler lose the address space and emit generic loads for every shared-memory access below
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kBarOffset);
    uint64_t* a_full = bars;                 // [NA] A tile landed
    uint64_t* a_empty = a_full + NA;         // [NA] the MMAs reading it completed
    uint64_t* b_full = a_empty + NA;         // [NB] B tile ready (TMA landed, or dequant warps done)
    uint64_t* b_empty = b_full + NB;         // [NB] the MMAs reading it completed
    uint64_t* raw_full = b_empty + NB;       // [NR] packed nibbles landed (kBF16)
    uint64_t* raw_empty = raw_full + NR;     // [NR] packed nibbles are in registers (kBF16)
    uint64_t* tmem_full = raw_empty + NR;    // [2] (one used) both accumulators of the tile complete
    uint64_t* tmem_empty = tmem_full + 2;    // [2] (one used) both accumulators drained
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int64_t m_tiles = (p.M + BM - 1) / BM, n_tiles = (p.N + BN - 1) / BN;
    const int64_t tiles = m_tiles * n_tiles;
    const int kblocks = static_cast<int>((p.K + C::kBlockK - 1) / C::kBlockK);
    // this CTA's tiles: blockIdx.x, blockIdx.x + gridDim.x, ...; `it` counts its k-blocks across tiles
    const int64_t my_tiles = (tiles > blockIdx.x) ? (tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
    const int64_t total_its = my_tiles * kblocks;

    if (threadIdx.x == 0) {
        for (int i = 0; i < NA; ++i) { mbar_init(&a_full[i], 1); mbar_init(&a_empty[i], 1); }
        for (int i = 0; i < NB; ++i) { mbar_init(&b_full[i], kDequantWarps); mbar_init(&b_empty[i], 1); }
        for (int i = 0; i < NR; ++i) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], kDequantWarps); }
        for (int i = 0; i < 2; ++i) { mbar_init(&tmem_full[i], 1); mbar_init(&tmem_empty[i], 4); }
        mbar_fence_init();
        fence_proxy_async_smem();
    }
    if (warp == kEpilogueWarp0) {
        tmem_alloc(tmem_slot, kTmemCols);
        tmem_relinquish();
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ------------------------------- A producer ---------------------------------
        if (elect_one()) {
            tma_prefetch_descriptor(&map_a);
            Ring<NA> ra;
            Walk w(blockIdx.x);
            for (int64_t it = 0; it < total_its; ++it, ra.advance(), w.advance(1, kblocks, gridDim.x)) {
                const int s = ra.slot;
                if (!mbar_wait(&a_empty[s], ra.phase ^ 1u)) { report(kDevErrEmptyWait, static_cast<uint32_t>(it)); break; }
                mbar_arrive_expect_tx(&a_full[s], kABytes);
                tma_load_2d(smem + C::kAOff + s * kABytes, &map_a, &a_full[s], w.kb * C::kBlockK, static_cast<int32_t>((w.tile % m_tiles) * BM));
            }
        }
        __syncwarp();
    } else if (warp == kBProducerWarp) {
        // ------------------------------- raw producer -------------------------------
        if (elect_one()) {
            tma_prefetch_descriptor(&map_b);
            Ring<NR> rr;
            Walk w(blockIdx.x);
            for (int64_t it = 0; it < total_its; ++it, rr.advance(), w.advance(1, kblocks, gridDim.x)) {
                const int s = rr.slot;
                if (!mbar_wait(&raw_empty[s], rr.phase ^ 1u)) { report(kDevErrEmptyWait, 0x800000u | static_cast<uint32_t>(it)); break; }
                mbar_arrive_expect_tx(&raw_full[s], C::kRawStageBytes);
                tma_load_2d(smem + C::kRawOff + s * C::kRawStageBytes, &map_b, &raw_full[s],
                            w.kb * (MODE == kBF16W8 ? C::kBlockK : C::kBlockK / 2), static_cast<int32_t>((w.tile / m_tiles) * BN));
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------- MMA issuer ---------------------------------
        if (elect_one()) {
            const uint32_t idesc = umma_idesc(1u, 1u, kHalfM, BN);
            Ring<NA> ra;
            Ring<NB> rb;
            Walk w(blockIdx.x);
            for (int64_t it = 0; it < total_its; ++it, ra.advance(), rb.advance(), w.advance(1, kblocks, gridDim.x)) {
                const int kb = w.kb;
                const uint32_t tcount = w.tcount;
                if (kb == 0) {
                    // both accumulators are reused by every tile: wait until the epilogue has drained them
                    if (!mbar_wait(&tmem_empty[0], (tcount & 1u) ^ 1u)) { report(kDevErrMmaWait, tcount); break; }
                    tcgen05_fence_after();
                }
                const int sa = ra.slot, sb = rb.slot;
                if (!mbar_wait(&a_full[sa], ra.phase)) { report(kDevErrFullWait, static_cast<uint32_t>(it)); break; }
                if (!mbar_wait(&b_full[sb], rb.phase)) { report(kDevErrFullWait, 0x800000u | static_cast<uint32_t>(it)); break; }
                tcgen05_fence_after();
                const uint64_t bdesc = umma_desc_sw128(smem_u32(smem + C::kBOff + sb * kBBytes));
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const uint32_t tmem_d = tmem_base + half * BN;
                    const uint64_t adesc = umma_desc_sw128(smem_u32(smem + C::kAOff + sa * kABytes + half * (kHalfM * 128)));
#pragma unroll
                    for (int k = 0; k < C::kBlockK / C::kUmmaK; ++k)
                        // +32 bytes per instruction inside the 128-byte swizzle row: +2 in the address field
                        tcgen05_mma_f16(tmem_d, adesc + 2 * k, bdesc + 2 * k, idesc, (kb | k) != 0 ? 1u : 0u);
                }
                tcgen05_commit(&a_empty[sa]);
                tcgen05_commit(&b_empty[sb]);
                if (kb == kblocks - 1) tcgen05_commit(&tmem_full[0]);
            }
        }
        __syncwarp();
    } else if (warp >= kEpilogueWarp0 && warp < kEpilogueWarp0 + 4) {
        // ------------------------------- epilogue -----------------------------------
        const int quarter = warp & 3;
        Epilogue<false, false> epi(p, smem + C::kOutOff + (warp - kEpilogueWarp0) * 2048, lane);
        for (uint32_t tcount = 0; static_cast<int64_t>(tcount) < my_tiles; ++tcount) {
            const int64_t tile = blockIdx.x + static_cast<int64_t>(tcount) * gridDim.x;
            const int64_t m0 = (tile % m_tiles) * BM, n0 = (tile / m_tiles) * BN;
            if (!mbar_wait(&tmem_full[0], tcount & 1u)) { report(kDevErrMmaWait, 0x800000u | tcount); break; }
            tcgen05_fence_after();
            for (int half = 0; half < 2; ++half)
                epi.rows32(tmem_base + half * BN + (static_cast<uint32_t>(quarter * 32) << 16), m0 + half * kHalfM + quarter * 32, n0, BN);
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tmem_empty[0]);
        }
    } else if (MODE == kBF16W8 && warp >= kDequantWarp0) {
        // ------------------------------- int8 -> bf16 --------------------------------
        // Thread (r, h) owns 32 consecutive codes of row r (32 bytes in, 64 bytes of bf16 out).  A code
        // c = 16*hi + lo (hi signed, lo unsigned nibble) is built exactly from two magic numbers:
        // 0x4300|lo = 128 + lo, 0x4300|(hi^8) = 136 + hi, t = fma(136 + hi, 16, -2304) = 16 hi - 128,
        // c = fma(128 + lo, 1, t).  The weight scale is applied in fp32 by the epilogue, so the only
        // rounding of this path is x -> bf16.  Bytes (0,2) and (1,3) of a word leave as pairs: inside
        // every 4 codes the order is k+{0,2,1,3}, which is the order the activations were stored in.
        const int tid = threadIdx.x - kDequantWarp0 * 32;
        const int r = tid >> 1, h = tid & 1;
        Ring<NR> rr;
        Ring<NB> rb;
        bool alive = true;
        for (int64_t it = 0; it < total_its && alive; ++it) {
            const int sr = rr.slot, sb = rb.slot;
            if (!mbar_wait(&raw_full[sr], rr.phase)) { report(kDevErrFullWait, 0x400000u | static_cast<uint32_t>(it)); alive = false; break; }
            const uint8_t* src = smem + C::kRawOff + sr * C::kRawStageBytes + r * 64 + h * 32;
            const uint4 w0 = *reinterpret_cast<const uint4*>(src);
            const uint4 w1 = *reinterpret_cast<const uint4*>(src + 16);
            // the slot is handed back only once the codes really are in registers
            const uint32_t landed = loads_landed(w0.x ^ w0.y ^ w0.z ^ w0.w ^ w1.x ^ w1.y ^ w1.z ^ w1.w);
            if (lane == 0) mbar_arrive_after(&raw_empty[sr], landed);
            if (!mbar_wait(&b_empty[sb], rb.phase ^ 1u)) { report(kDevErrEmptyWait, 0x400000u | static_cast<uint32_t>(it)); alive = false; break; }
            const uint32_t words[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
            uint8_t* brow = smem + C::kBOff + sb * kBBytes + r * 128;
#pragma unroll
            for (int w = 0; w < 4; ++w) {                           // output chunk w: words 2w and 2w+1
                uint32_t o[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t word = words[2 * w + (j >> 1)] >> (8 * (j & 1));     // bytes (0,2), then (1,3)
                    const uint32_t lo = (word & 0x000F000Fu) | 0x43004300u;            // 128 + lo
                    const uint32_t hi = ((word >> 4) & 0x000F000Fu) ^ 0x43084308u;     // 136 + hi
                    uint32_t t;
                    asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(t) : "r"(hi), "r"(0x41804180u), "r"(0xC510C510u));   // 16 hi - 128
                    asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(o[j]) : "r"(lo), "r"(0x3F803F80u), "r"(t));
                }
                *reinterpret_cast<uint4*>(brow + (((4 * h + w) ^ (r & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&b_full[sb]);
            rr.advance();
            rb.advance();
        }
    } else if (MODE == kBF16 && warp >= kDequantWarp0) {
        // ------------------------------- dequant ------------------------------------
        // Thread (r, h) owns half h (one 32-k group: 16 packed bytes in, 64 bytes of bf16 out) of row r of
        // the 256-row weight tile.  The group's scale is requested one k-block ahead so that its L2
        // latency is never waited for.
        const int tid = threadIdx.x - kDequantWarp0 * 32;
        const int r = tid >> 1, h = tid & 1;
        const int64_t sgroups = p.K / 32;
        Walk wn(blockIdx.x);                      // walks one k-block ahead, for the scale prefetch
        auto load_scale = [&](int64_t it, const Walk& w) {
            float sc = 0.0f;
            if (it < total_its) {
                const int64_t n = (w.tile / m_tiles) * BN + r;
                if (n < p.N) sc = __ldg(p.wscales + n * sgroups + 2 * w.kb + h);
            }
            return sc;
        };
        // scales are requested kAhead k-blocks before they are used (an L2 round trip is several
        // k-blocks long at full speed)
        constexpr int kAhead = 4;
        float scq[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            scq[u] = load_scale(u, wn);
            wn.advance(1, kblocks, gridDim.x);
        }
        Ring<NR> rr;
        Ring<NB> rb;
        bool alive = true;
        for (int64_t it0 = 0; it0 < total_its && alive; it0 += kAhead) {
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                const int64_t it = it0 + u;
                if (it >= total_its || !alive) break;
                const float sc = scq[u];
                scq[u] = load_scale(it + kAhead, wn);
                wn.advance(1, kblocks, gridDim.x);
                const int sr = rr.slot, sb = rb.slot;
                if (!mbar_wait(&raw_full[sr], rr.phase)) { report(kDevErrFullWait, 0x400000u | static_cast<uint32_t>(it)); alive = false; break; }
                const uint4 w0 = *reinterpret_cast<const uint4*>(smem + C::kRawOff + sr * kRawBytes + r * 32 + h * 16);
                // make sure the load has returned before the slot is handed back to the TMA producer
                // the slot is handed back only once the nibbles really are in registers
                const uint32_t landed = loads_landed(w0.x ^ w0.y ^ w0.z ^ w0.w);
                if (lane == 0) mbar_arrive_after(&raw_empty[sr], landed);
                if (!mbar_wait(&b_empty[sb], rb.phase ^ 1u)) { report(kDevErrEmptyWait, 0x400000u | static_cast<uint32_t>(it)); alive = false; break; }
                const uint32_t words[4] = {w0.x, w0.y, w0.z, w0.w};
                const uint32_t sx2 = static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(sc))) * 0x00010001u;
                uint8_t* brow = smem + C::kBOff + sb * kBBytes + r * 128;
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    uint32_t o[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint32_t v = ((words[w] >> (4 * j)) & 0x000F000Fu) ^ 0x43084308u;  // 136 + code
                        // (v - 136) is exact in bf16, then one rounding for code * scale; both as fused
                        // multiply-adds, which the half-precision pipe executes natively
                        uint32_t c;
                        asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(c) : "r"(v), "r"(0x3F803F80u), "r"(0xC308C308u));
                        asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(o[j]) : "r"(c), "r"(sx2), "r"(0x80008000u));
                    }
                    // chunk (4h + w) of the row goes to chunk ((4h + w) ^ (r & 7)): the 128-byte swizzle the MMA expects
                    *reinterpret_cast<uint4*>(brow + (((4 * h + w) ^ (r & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&b_full[sb]);
                rr.advance();
                rb.advance();
            }
        }
    }

    tcgen05_fence_before();
    __syncthreads();
    if (warp == kEpilogueWarp0) {
        tcgen05_fence_after();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

// ---- both operands by TMA: CTA pairs ------------------------------------------------------------------------------------
// Two CTAs of a cluster (one SM each) share a tile of 256 rows x bn columns: each loads its 128 rows of A and its bn/2
// rows of B, and the even CTA issues tcgen05.mma.cta_group::2, which reads both halves of B and gives each CTA the
// accumulators of its own 128 rows.  A k-block is 128 bytes of K: 32 KB per CTA, so six of them fit, and an accumulator
// takes at most 256 of the 512 TMEM columns, so that the epilogue of one tile runs under the MMAs of the next.
// B: [N,K] (K-major, the loads are bn/2 rows of 128 bytes) or, bf16 only, [K,N] (MN-major, blocks of 64 columns x 64 k).
constexpr int kPairM = 256;
constexpr int kPairStages = 6;
constexpr int kPairABytes = 128 * 128, kPairBBytes = 128 * 128;
constexpr int kPairStageBytes = kPairABytes + kPairBBytes;
constexpr int kPairOutOff = kPairStages * kPairStageBytes;           // 4 epilogue warps x [16 rows x 32 fp32], swizzled
constexpr int kPairBarOff = kPairOutOff + 4 * 2048;
constexpr int kPairSmemBytes = kPairBarOff + (2 * kPairStages + 4) * 8 + 16 + 1024;
constexpr int kPairThreads = 6 * 32;      // 0 = TMA producer, 1 = MMA issuer, 2..5 = epilogue (TMEM lane quarter = warp % 4)
constexpr int kPairGroupM = 8;            // row tiles that are walked together, see PairTiles

// Order of the tiles: bands of kPairGroupM row tiles, inside a band column by column.  The 74 tiles in flight then cover
// about 8 row tiles x 9 column tiles, and the operands that they read (17 strips of 256 rows) stay in L2 between tiles;
// with whole columns of a tall problem (32 row tiles of 8192 rows) every round read all of x again.
struct PairTiles {
    uint32_t m_tiles, n_tiles, tiles;
    __device__ __forceinline__ PairTiles(const Params& p)
        : m_tiles(static_cast<uint32_t>((p.M + kPairM - 1) / kPairM)), n_tiles(static_cast<uint32_t>((p.N + p.bn - 1) / p.bn)),
          tiles(m_tiles * n_tiles) {}
    __device__ __forceinline__ void locate(uint32_t t, int32_t& m, int32_t& n) const {
        const uint32_t band = kPairGroupM * n_tiles, g = t / band, r = t - g * band;
        const uint32_t left = m_tiles - g * kPairGroupM, rows = left < kPairGroupM ? left : kPairGroupM;
        m = static_cast<int32_t>(g * kPairGroupM + r % rows);
        n = static_cast<int32_t>(r / rows);
    }
};

template <bool I8, bool PEERS = false>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
linear_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ Params p) {
    constexpr int NS = kPairStages;
    constexpr int kBlockK = I8 ? 128 : 64;                  // elements per k-block (128 bytes)
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);     // the same offset in both CTAs
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + kPairBarOff);   // [NS] both CTAs' tiles landed (the even CTA's is used)
    uint64_t* empty = full + NS;             // [NS] the MMAs reading the slot completed (arrives in both CTAs)
    uint64_t* tmem_full = empty + NS;        // [2] the accumulator is complete (arrives in both CTAs)
    uint64_t* tmem_empty = tmem_full + 2;    // [2] all 8 epilogue warps of the pair have drained it (the even CTA's is used)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_cta_rank();
    const uint32_t pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const PairTiles tl(p);
    const int kblocks = static_cast<int>((p.K + kBlockK - 1) / kBlockK);

    if (threadIdx.x == 0) {
        for (int i = 0; i < NS; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&tmem_full[i], 1); mbar_init(&tmem_empty[i], 8); }
        mbar_fence_init();
        fence_proxy_async_smem();
    }
    if (warp == 2) tmem_alloc_pair(tmem_slot, kTmemCols);
    tcgen05_fence_before();
    __syncthreads();
    cluster_sync_all();                      // the other CTA's barriers are initialised
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (p.ready == nullptr) pdl_wait();      // operands from the kernel in front; with `ready` it is waited for slice by slice

    if (warp == 0) {
        // ------------------------------- producer: this CTA's halves of A and B ---------------------------------
        if (elect_one()) {
            tma_prefetch_descriptor(&map_a);
            tma_prefetch_descriptor(&map_b);
            const int half_n = p.bn / 2;
            const int b_loads = p.b_mn ? (half_n + 63) / 64 : 1;
            const uint32_t tx = 2u * (kPairABytes + (p.b_mn ? b_loads * 8192u : half_n * 128u));
            Ring<NS> r;
            int parts_seen = 0;                             // slices of K known to be complete (they fill in order)
            uint32_t issued = 0;
            bool alive = true;
            for (uint32_t t = pair; t < tl.tiles && alive; t += pairs) {
                int32_t mt, nt;
                tl.locate(t, mt, nt);
                const int32_t m0 = mt * kPairM + static_cast<int32_t>(rank) * 128, n0 = nt * p.bn + static_cast<int32_t>(rank) * half_n;
                for (int kb = 0; kb < kblocks; ++kb, r.advance()) {
                    if (p.ready != nullptr && kb >= parts_seen * p.ready_part_kblocks) {
                        const int q = kb / p.ready_part_kblocks;
                        if (!wait_expanded(p.ready + q, p.ready_target)) { report(kDevErrFullWait, 0x400000u | q); alive = false; break; }
                        parts_seen = q + 1;
                    }
                    const int s = r.slot;
                    if (!mbar_wait(&empty[s], r.phase ^ 1u)) { report(kDevErrEmptyWait, static_cast<uint32_t>(kb)); alive = false; break; }
                    const uint32_t bar = map_to_rank(&full[s], 0);
                    if (rank == 0) mbar_arrive_expect_tx(&full[s], tx);
                    uint8_t* dst = smem + s * kPairStageBytes;
                    tma_load_2d_pair(dst, &map_a, bar, kb * kBlockK, m0);
                    if (!I8 && p.b_mn) {
                        for (int j = 0; j < b_loads; ++j) tma_load_2d_pair(dst + kPairABytes + j * 8192, &map_b, bar, n0 + j * 64, kb * kBlockK);
                    } else {
                        tma_load_2d_pair(dst + kPairABytes, &map_b, bar, kb * kBlockK, n0);
                    }
                    ++issued;
                }
            }
            // Neither CTA may leave while the other's MMAs, loads or commits still refer to its shared memory: every slot
            // that was filled is waited for once more.  (After a wait that ran out: a millisecond for the loads in flight.)
            for (int i = 0; i < NS && alive; ++i, r.advance())
                if (issued >= static_cast<uint32_t>(NS - i) && !mbar_wait(&empty[r.slot], r.phase ^ 1u)) {
                    report(kDevErrEmptyWait, 0x800000u);
                    alive = false;
                }
            for (int i = 0; i < 1000 && !alive; ++i) __nanosleep(1000);
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------- MMA issuer (even CTA) ---------------------------------------------------
        if (rank == 0 && elect_one()) {
            const uint32_t idesc = umma_idesc(I8 ? 2u : 1u, 1u, kPairM, static_cast<uint32_t>(p.bn)) | (p.b_mn ? kIdescBMajorMN : 0u);
            // an instruction takes 32 bytes of K: +2 in the address field inside the swizzled row, or 16 rows of 128 bytes
            const uint64_t bstep = p.b_mn ? 128 : 2;
            const uint64_t a0 = umma_desc_sw128(smem_u32(smem));
            const uint64_t b0 = p.b_mn ? umma_desc_sw128_mn(smem_u32(smem + kPairABytes)) : umma_desc_sw128(smem_u32(smem + kPairABytes));
            Ring<NS> r;
            bool alive = true;
            uint32_t n = 0;                                 // tiles done by this pair
            for (uint32_t t = pair; t < tl.tiles && alive; t += pairs, ++n) {
                const uint32_t acc = n & 1u;
                if (!mbar_wait(&tmem_empty[acc], ((n >> 1) & 1u) ^ 1u)) { report(kDevErrMmaWait, n); break; }
                tcgen05_fence_after();
                const uint32_t tmem_d = tmem_base + acc * 256;
                for (int kb = 0; kb < kblocks; ++kb, r.advance()) {
                    const int s = r.slot;
                    if (!mbar_wait(&full[s], r.phase)) { report(kDevErrFullWait, static_cast<uint32_t>(kb)); alive = false; break; }
                    tcgen05_fence_after();
                    const uint64_t adesc = a0 + static_cast<uint64_t>(s) * (kPairStageBytes >> 4);
                    const uint64_t bdesc = b0 + static_cast<uint64_t>(s) * (kPairStageBytes >> 4);
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        tcgen05_mma_pair<I8>(tmem_d, adesc + 2 * k, bdesc + bstep * k, idesc, (kb | k) != 0 ? 1u : 0u);
                    tcgen05_commit_pair(&empty[s]);
                }
                if (alive) tcgen05_commit_pair(&tmem_full[acc]);
            }
        }
        __syncwarp();
    } else {
        // ------------------------------- epilogue: this CTA's 128 rows -------------------------------------------
        const int quarter = warp & 3;
        Epilogue<I8, PEERS> epi(p, smem + kPairOutOff + (warp - 2) * 2048, lane);
        uint32_t n = 0;
        for (uint32_t t = pair; t < tl.tiles; t += pairs, ++n) {
            const uint32_t acc = n & 1u;
            int32_t mt, nt;
            tl.locate(t, mt, nt);
            if (!mbar_wait(&tmem_full[acc], (n >> 1) & 1u)) { report(kDevErrMmaWait, 0x800000u | n); break; }
            tcgen05_fence_after();
            epi.rows32(tmem_base + acc * 256 + (static_cast<uint32_t>(quarter * 32) << 16),
                       static_cast<int64_t>(mt) * kPairM + rank * 128 + quarter * 32, static_cast<int64_t>(nt) * p.bn, p.bn);
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_remote(map_to_rank(&tmem_empty[acc], 0));
        }
        __syncwarp();
    }

    tcgen05_fence_before();
    __syncthreads();
    cluster_sync_all();
    if (warp == 2) {
        tcgen05_fence_after();
        tmem_dealloc_pair(tmem_base, kTmemCols);
    }
}

// x fp32 [M,K] -> bf16 [M,K].  ORDER 0: inside every aligned group of 8 the order is k+{0,4,1,5,2,6,3,7},
// the order in which the dequant warps emit the 8 nibbles of a packed word.  ORDER 1 (INT8 weights):
// k+{0,2,1,3,4,6,5,7}.
template <int ORDER>
__global__ void __launch_bounds__(256) convert_x_bf16_kernel(const float* __restrict__ x, uint4* __restrict__ out,
                                                             int64_t chunks) {
    int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * 256;
    for (; i < chunks; i += stride) {
        const float4 a = reinterpret_cast<const float4*>(x)[2 * i];
        const float4 b = reinterpret_cast<const float4*>(x)[2 * i + 1];
        auto pk = [](float lo, float hi) {
            return static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(lo))) |
                   (static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(hi))) << 16);
        };
        out[i] = ORDER == 1   ? make_uint4(pk(a.x, a.z), pk(a.y, a.w), pk(b.x, b.z), pk(b.y, b.w))
                              : make_uint4(pk(a.x, b.x), pk(a.y, b.y), pk(a.z, b.z), pk(a.w, b.w));
    }
}

// Weights -> bf16 in global memory in the order in which they are stored ([N,K], or KN: [K,N]; the MMA reads either),
// eight elements per step (one packed word, or eight code bytes).  INT4: code * scale in fp32, rounded once.  INT8: the
// codes themselves (exact in bf16), their scale is applied by the GEMM's epilogue in fp32; stored [K,N], where the scale
// may run along K (one per stored row), code * scale in fp32, rounded once.  The same launch converts the
// activations (x fp32 [M,K] -> bf16), and the GEMM starts while it runs: the grid is one resident wave that leaves room
// for the GEMM's CTA on every SM, and the work is ordered by `parts` equal slices of K: slice 0 of x, slice 0 of W,
// slice 1 of x, ...  ready[q] counts the CTAs that have finished slice q of both; a CTA counts itself after a fence
// behind all of its stores, so a reader that sees gridDim.x in ready[q] (acquire load) may read slices 0 .. q.  The
// counters must be zero at launch.  Indices are 32-bit with FastDiv; a [K,N] weight or its activations of 2^31 steps or more
// (2^34 elements) take the 64-bit form, WideDiv.
constexpr int kExpandCtasPerSm = 2;
constexpr int kReadyParts = 8;            // at most
constexpr size_t kReadyBytes = 256;       // reserved behind the expanded weight for the counters

// n / d for n < 2^31 by one multiplication: with 2^(s-1) < d <= 2^s and m = floor(2^(31+s) / d) + 1, m exceeds the exact
// quotient by at most 1, and n * 1 / 2^(31+s) < 2^-s <= 1/d, too little to reach the next integer.  (The compiler's
// division by a variable is about twenty instructions, and the kernel below needs two per eight elements: INT4
// [28672,8192] with 128 rows 283 us, 265 so; INT8 [4096,11008] with 1000 rows 96.3, 95.8 so.)
struct FastDiv {
    using Index = uint32_t;
    uint32_t d, m, s;
    explicit FastDiv(uint32_t d_) : d(d_), m(0), s(0) {
        while ((1ull << s) < d) ++s;
        m = static_cast<uint32_t>((1ull << (31 + s)) / d + 1);          // at most 2^32 - 1 (d > 2^(s-1)), 2^31 + 1 for powers of two
    }
    __device__ __forceinline__ uint32_t operator()(uint32_t n) const {
        return static_cast<uint32_t>((static_cast<uint64_t>(n) * m) >> (31 + s));
    }
};

struct WideDiv {
    using Index = uint64_t;
    uint64_t d;
    explicit WideDiv(uint64_t d_) : d(d_) {}
    __device__ __forceinline__ uint64_t operator()(uint64_t n) const { return n / d; }
};

template <int BITS, bool KN, typename Div>
__global__ void __maxnreg__(64)            // per SM quarter: 4 of these warps (4 x 64 x 32) beside 2 of the GEMM (2 x 128 x 32)
expand_ordered_kernel(const uint8_t* __restrict__ wq, const float* __restrict__ scales, Div per_scale, Div per_slice, uint32_t N,
                      uint32_t K, uint32_t parts, uint4* __restrict__ out, const float* __restrict__ x, uint32_t M, uint4* __restrict__ xout,
                      uint32_t* __restrict__ ready) {
    pdl_launch_dependents();             // the GEMM behind this launch may take its places now; it waits on `ready`
    auto pk = [](float lo, float hi) {
        return static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(lo))) |
               (static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(hi))) << 16);
    };
    using Index = typename Div::Index;
    const Index first = blockIdx.x * 256u + threadIdx.x, stride = gridDim.x * 256u;
    const Index row = K / 8, slice = per_slice.d;                        // steps per row of x (and of W [N,K]) / per row and slice
    const Index wslice = KN ? (K / parts) * static_cast<Index>(N / 8) : N * slice;      // steps of W per slice
    constexpr bool scaled = BITS == 4 || KN;                             // multiply here (else the epilogue does)
    auto step_of = [&](Index v, uint32_t part) {                      // v-th step of the slice -> index in the whole tensor
        const Index r = per_slice(v);
        return r * row + part * slice + (v - r * slice);
    };
    auto expand = [&](Index i, uint32_t lo, uint32_t hi, float sc) {
        float v[8];
        if (BITS == 4) {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = __fmul_rn(static_cast<float>(static_cast<int>(lo << (28 - 4 * j)) >> 28), sc);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                v[j] = static_cast<float>(static_cast<int>(lo << (24 - 8 * j)) >> 24);
                v[4 + j] = static_cast<float>(static_cast<int>(hi << (24 - 8 * j)) >> 24);
            }
            if (scaled) {
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = __fmul_rn(v[j], sc);
            }
        }
        out[i] = make_uint4(pk(v[0], v[1]), pk(v[2], v[3]), pk(v[4], v[5]), pk(v[6], v[7]));
    };
    // Called by whole CTAs only.  The barrier orders the CTA's stores before thread 0's fence, which makes all of them
    // visible to the GPU before the count; the other threads go on to the next slice instead of waiting for their stores
    // (a fence in every thread: 0.5 us of 50 to 96).
    auto signal = [&](uint32_t part) {
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            atomicAdd(ready + part, 1u);
        }
    };
    // Four words and their scales per thread and pass, and the loads of the next pass, be it in this slice or the next,
    // are issued before the current one is converted (before the slice's activations for the first): with two CTAs per SM
    // the loads have to overlap the arithmetic inside a thread, and a slice that began with nothing on its way waited for
    // memory twice (INT8 [4096,11008], 1000 rows: 47 us, now 37; INT4 [6144,2048], 4096 rows: 39, now 31).
    Index i[4], in[4];
    uint32_t lo[4], hi[4], lon[4], hin[4];
    float sc[4], scn[4];
    auto fetch = [&](Index v, uint32_t part, Index (&ii)[4], uint32_t (&l)[4], uint32_t (&h)[4], float (&f)[4]) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const Index vq = v + q * stride, vv = vq < wslice ? vq : v;
            ii[q] = KN ? part * wslice + vv : step_of(vv, part);
            if (BITS == 4) {
                l[q] = reinterpret_cast<const uint32_t*>(wq)[ii[q]];
                h[q] = 0;
            } else {
                const uint2 w = reinterpret_cast<const uint2*>(wq)[ii[q]];
                l[q] = w.x;
                h[q] = w.y;
            }
            f[q] = scaled ? scales[per_scale(ii[q])] : 1.0f;              // a step never straddles groups or rows
        }
    };
    if (first < wslice) fetch(first, 0, i, lo, hi, sc);
    for (uint32_t part = 0; part < parts; ++part) {
        const Index xtotal = M * slice;
        for (Index v = first; v < xtotal; v += 2 * stride) {                     // two chunks in flight per thread
            const bool two = v + stride < xtotal;
            const Index j0 = step_of(v, part), j1 = two ? step_of(v + stride, part) : j0;
            const float4 a0 = reinterpret_cast<const float4*>(x)[2 * static_cast<size_t>(j0)], b0 = reinterpret_cast<const float4*>(x)[2 * static_cast<size_t>(j0) + 1];
            const float4 a1 = reinterpret_cast<const float4*>(x)[2 * static_cast<size_t>(j1)], b1 = reinterpret_cast<const float4*>(x)[2 * static_cast<size_t>(j1) + 1];
            xout[j0] = make_uint4(pk(a0.x, a0.y), pk(a0.z, a0.w), pk(b0.x, b0.y), pk(b0.z, b0.w));
            if (two) xout[j1] = make_uint4(pk(a1.x, a1.y), pk(a1.z, a1.w), pk(b1.x, b1.y), pk(b1.z, b1.w));
        }
        for (Index v = first; v < wslice; v += 4 * stride) {
            const Index vn = v + 4 * stride;
            if (vn < wslice) fetch(vn, part, in, lon, hin, scn);
            else if (part + 1 < parts) fetch(first, part + 1, in, lon, hin, scn);
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (q == 0 || v + q * stride < wslice) expand(i[q], lo[q], hi[q], sc[q]);
#pragma unroll
            for (int q = 0; q < 4; ++q) { i[q] = in[q]; lo[q] = lon[q]; hi[q] = hin[q]; sc[q] = scn[q]; }
        }
        signal(part);
    }
}

size_t round_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

template <int MODE>
int launch_tc(const CUtensorMap& ma, const CUtensorMap& mb, Params p, cudaStream_t stream) {
    using C = Cfg<MODE>;
    if (p.n_peers > 0) {
        set_error("the fused all-gather of the tensor-core path needs the scratch for the expanded weight");
        return SGQ_ERR_WORKSPACE;
    }
    p.vec_store = (aligned(p.y, 16) && (p.ldy % 4) == 0) ? 1 : 0;
    const int64_t tiles = ceil_div(p.M, BM) * ceil_div(p.N, BN);
    const int grid = static_cast<int>(tiles < sm_count() ? tiles : sm_count());
    static SmemOptIn optin;   // one per MODE instantiation
    SGQ_CUDA_TRY(optin.ensure(linear_tc_kernel<MODE>, C::kSmemBytes));
    linear_tc_kernel<MODE><<<grid, C::kThreads, C::kSmemBytes, stream>>>(ma, mb, p);
    SGQ_LAUNCH_CHECK("linear_tc_kernel");
    return SGQ_OK;
}

// Columns of a pair's tile.  256 does the least work per byte loaded; a narrower tile is taken where it fills the rounds
// of the persistent grid better.  Cycles of a k-block: the MMAs take 2 * bn, and the loads of a CTA, 16 KB of A and
// bn * 64 bytes of B, about one cycle per 64 bytes from L2.
int pair_columns(int64_t M, int64_t N, int64_t kblocks, int64_t pairs) {
    const int64_t m_tiles = ceil_div(M, kPairM);
    int best = 256;
    int64_t best_cost = INT64_MAX;
    for (int bn = 256; bn >= 64; bn -= 32) {
        const int64_t rounds = ceil_div(m_tiles * ceil_div(N, bn), pairs);
        const int64_t cycles = 2 * bn > 256 + bn ? 2 * bn : 256 + bn;
        const int64_t cost = rounds * cycles * kblocks + 16 * bn;          // ... and the last tile's epilogue
        if (cost < best_cost) { best_cost = cost; best = bn; }
    }
    return best;
}

// act: activations [M,K], codes or bf16; w: weights [N,K], or [K,N] with p.b_mn
template <bool I8>
int launch_pair(Params p, const void* act, const void* w, cudaStream_t stream) {
    const int64_t elem = I8 ? 1 : 2, block_k = 128 / elem;
    const int64_t pairs = sm_count() / 2;
    p.bn = pair_columns(p.M, p.N, ceil_div(p.K, block_k), pairs);
    const int64_t tiles = ceil_div(p.M, kPairM) * ceil_div(p.N, p.bn);
    if (tiles >= (1LL << 31)) {
        set_error("tensor-core path: more than 2^31 tiles");
        return SGQ_ERR_UNSUPPORTED;
    }
    const CUtensorMapDataType type = I8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    const uint64_t K = static_cast<uint64_t>(p.K), N = static_cast<uint64_t>(p.N);
    CUtensorMap ma, mb;
    if (!make_tensor_map_2d(&ma, type, act, K, static_cast<uint64_t>(p.M), K * elem, static_cast<uint32_t>(block_k), 128, CU_TENSOR_MAP_SWIZZLE_128B))
        return SGQ_ERR_CUDA;
    const bool ok = p.b_mn ? make_tensor_map_2d(&mb, type, w, N, K, N * elem, 64, 64, CU_TENSOR_MAP_SWIZZLE_128B)
                           : make_tensor_map_2d(&mb, type, w, K, N, K * elem, static_cast<uint32_t>(block_k), static_cast<uint32_t>(p.bn / 2),
                                                CU_TENSOR_MAP_SWIZZLE_128B);
    if (!ok) return SGQ_ERR_CUDA;
    p.vec_store = (aligned(p.y, 16) && (p.ldy % 4) == 0) ? 1 : 0;
    for (int r = 0; r < p.n_peers; ++r)
        if (!aligned(p.peer_y[r], 16)) p.vec_store = 0;
    const dim3 grid(static_cast<unsigned>(2 * (tiles < pairs ? tiles : pairs)));
    // always overlapped with the kernel in front: the operands are waited for in the kernel
    if (!I8 && p.n_peers > 0) {
        static SmemOptIn optin_peers;
        SGQ_CUDA_TRY(optin_peers.ensure(linear_pair_kernel<false, true>, kPairSmemBytes));
        SGQ_CUDA_TRY(launch_kernel(linear_pair_kernel<false, true>, grid, dim3(kPairThreads), kPairSmemBytes, stream, true, ma, mb, p));
        return SGQ_OK;
    }
    static SmemOptIn optin;
    SGQ_CUDA_TRY(optin.ensure(linear_pair_kernel<I8>, kPairSmemBytes));
    SGQ_CUDA_TRY(launch_kernel(linear_pair_kernel<I8>, grid, dim3(kPairThreads), kPairSmemBytes, stream, true, ma, mb, p));
    return SGQ_OK;
}

}  // namespace

bool tc_bf16_supported(int bits, int64_t M, int64_t K, int64_t N, int layout, int64_t group) {
    // INT4: any group that is a multiple of 8 (the weight is expanded word by word); 32 also has the form that
    // dequantizes in shared memory
    if (!(((bits == 4 && group >= 8 && (group % 8) == 0) || bits == 8) && M >= 1 && N >= 1 && K >= 64 && (K % 64) == 0 &&
          M < (1LL << 31) && N < (1LL << 31) && K < (1LL << 31)))
        return false;
    // [K,N]: quantization groups run along N and must not straddle rows of the stored tensor
    return layout == SGQ_LAYOUT_NK || (layout == SGQ_LAYOUT_KN && (N % 32) == 0);
}

// bf16 activations plus the whole weight expanded to bf16 [N,K]: the faster form (a GEMM whose operands both
// arrive by TMA), and the only one for weights stored [K,N]
size_t tc_bf16_workspace_bytes(int bits, int64_t M, int64_t K, int64_t N, int layout) {
    (void)bits; (void)layout;
    return round_up(static_cast<size_t>(M) * static_cast<size_t>(K) * 2, 256) +
           round_up(static_cast<size_t>(N) * static_cast<size_t>(K) * 2, 256) + kReadyBytes;
}

// the least the path runs with: weights stored [N,K] can be dequantized tile by tile in shared memory instead
size_t tc_bf16_min_workspace_bytes(int bits, int64_t M, int64_t K, int64_t N, int layout, int64_t group) {
    if (layout == SGQ_LAYOUT_KN || (bits == 4 && group != 32)) return tc_bf16_workspace_bytes(bits, M, K, N, layout);
    return round_up(static_cast<size_t>(M) * static_cast<size_t>(K) * 2, 256);
}

int launch_linear_tc_bf16(const LinearArgs& a) {
    if (!tc_bf16_supported(a.bits, a.M, a.K, a.N, a.layout, a.group)) {
        set_error("bf16 tensor-core path needs INT4 (group a multiple of 8) or INT8 weights, K%%64==0, and N%%32==0 when stored [K,N]");
        return SGQ_ERR_UNSUPPORTED;
    }
    if (!aligned(a.x, 16) || !aligned(a.wq, 16) || !aligned(a.scales, 8)) {
        set_error("bf16 tensor-core path needs 16-byte aligned x and packed weights, 8-byte aligned scales");
        return SGQ_ERR_ALIGNMENT;
    }
    const size_t need = tc_bf16_min_workspace_bytes(a.bits, a.M, a.K, a.N, a.layout, a.group);
    const bool expand = a.workspace && a.workspace_bytes >= tc_bf16_workspace_bytes(a.bits, a.M, a.K, a.N, a.layout);
    if (!a.workspace || a.workspace_bytes < need) {
        set_error("bf16 tensor-core path needs %zu workspace bytes, got %zu", need, a.workspace ? a.workspace_bytes : 0);
        return SGQ_ERR_WORKSPACE;
    }
    const int64_t chunks = a.M * a.K / 8;
    Params p{};
    p.bias = a.bias; p.y = a.y; p.ldy = a.ldy; p.M = a.M; p.N = a.N; p.K = a.K;
    p.n_peers = a.peers.n;
    for (int r = 0; r < a.peers.n; ++r) p.peer_y[r] = a.peers.p[r];
    if (expand) {
        // Expand the stored weight to bf16 behind the activations in the workspace, then a GEMM whose operands both
        // arrive by TMA.  One resident wave converts x and the weight slice of K by slice of K, counting finished
        // slices into `ready`; the GEMM is launched behind it with programmatic serialization and starts on the first
        // slice while the rest is still being expanded.  (The expansion itself is an ordinary launch: when it starts,
        // everything older is complete, so the GEMM that starts beside it finds the outputs free whatever
        // sgq_set_stream_overlap says.)
        const bool kn = a.layout == SGQ_LAYOUT_KN;
        uint8_t* xb = static_cast<uint8_t*>(a.workspace);
        uint8_t* wt = xb + round_up(static_cast<size_t>(a.M) * static_cast<size_t>(a.K) * 2, 256);
        const int64_t wsteps = a.N * a.K / 8;
        const int64_t most = wsteps > chunks ? wsteps : chunks;
        // Beside the GEMM only while the register budget of an SM quarter holds: 2 GEMM warps of at most 128
        // registers a thread next to 4 expansion warps of 64 (16384 in all); a compiler that needs more for
        // the GEMM gets the serial form instead of a silent loss of the overlap.
        static const bool fits = [] {
            cudaFuncAttributes fa{};
            return cudaFuncGetAttributes(&fa, linear_pair_kernel<false>) == cudaSuccess && fa.numRegs <= 128;
        }();
        const bool beside = fits && a.peers.n == 0;
        const int64_t wave = static_cast<int64_t>(sm_count()) * (beside ? kExpandCtasPerSm : 16);
        const int egrid = static_cast<int>(ceil_div(most, 1024) < wave ? ceil_div(most, 1024) : wave);
        const int64_t kblocks = a.K / 64;
        // Few slices where a thread has few passes: every slice ends in a pass that is partly empty.  Four against eight:
        // [4096,11008] 256 rows 49.8 / 54.0 us, 1000 rows 95.8 / 97.9, [14336,4096] 512 rows 88 / 96; from the line (48
        // passes, 116 M weights) on eight are level or ahead: [32768,4096] 256 rows 148 / 147, [14336,8192] 1024 rows 255 / 240.
        int parts = !beside ? 1 : (wsteps >= 48LL * 4 * 256 * egrid ? kReadyParts : kReadyParts / 2);
        while (kblocks % parts) parts /= 2;
        // 32-bit indices hold up to 2^31 steps and what the last pass adds to them; weights stored [N,K] end there
        const bool wide = most >= (1LL << 31) - 4LL * egrid * 256;
        if (wide && !kn) {
            set_error("bf16 tensor-core path: more than 2^31 expansion steps");
            return SGQ_ERR_UNSUPPORTED;
        }
        uint32_t* ready = reinterpret_cast<uint32_t*>(wt + round_up(static_cast<size_t>(a.N) * static_cast<size_t>(a.K) * 2, 256));
        SGQ_CUDA_TRY(cudaMemsetAsync(ready, 0, kReadyBytes, a.stream));
        // INT8 codes stored [N,K] are exact in bf16 and their scale goes to the epilogue; stored [K,N] it may run along K
        if (a.bits == 8 && !kn) {
            p.sw = a.scales;
            p.sw_per_row = (a.scheme == SGQ_PER_ROW) ? 1 : 0;
        }
        // (one scale for all: more steps per scale than there are)
        const int64_t scale_steps = a.bits == 4 ? a.group / 8 : (a.scheme == SGQ_PER_ROW && kn ? a.N / 8 : most + 1);
        const int64_t slice_steps = a.K / 8 / parts;
        auto run = [&](auto kernel, auto per_scale, auto per_slice) {
            // the GEMM's CTA can only join an SM that runs under the same memory split
            prefer_max_shared(reinterpret_cast<const void*>(kernel));
            kernel<<<egrid, 256, 0, a.stream>>>(static_cast<const uint8_t*>(a.wq), a.scales, per_scale, per_slice, static_cast<uint32_t>(a.N),
                                                static_cast<uint32_t>(a.K), static_cast<uint32_t>(parts), reinterpret_cast<uint4*>(wt), a.x,
                                                static_cast<uint32_t>(a.M), reinterpret_cast<uint4*>(xb), ready);
        };
        if (wide) {
            const WideDiv per_scale(static_cast<uint64_t>(scale_steps)), per_slice(static_cast<uint64_t>(slice_steps));
            if (a.bits == 4) run(expand_ordered_kernel<4, true, WideDiv>, per_scale, per_slice);
            else run(expand_ordered_kernel<8, true, WideDiv>, per_scale, per_slice);
        } else {
            const FastDiv per_scale(static_cast<uint32_t>(scale_steps < (1LL << 31) ? scale_steps : (1LL << 31)));
            const FastDiv per_slice(static_cast<uint32_t>(slice_steps));
            if (a.bits == 4) run(kn ? expand_ordered_kernel<4, true, FastDiv> : expand_ordered_kernel<4, false, FastDiv>, per_scale, per_slice);
            else run(kn ? expand_ordered_kernel<8, true, FastDiv> : expand_ordered_kernel<8, false, FastDiv>, per_scale, per_slice);
        }
        SGQ_LAUNCH_CHECK("expand_ordered_kernel");
        p.b_mn = kn ? 1 : 0;
        p.ready = ready;
        p.ready_target = static_cast<uint32_t>(egrid);
        p.ready_part_kblocks = static_cast<int>(kblocks / parts);
        return launch_pair<false>(p, xb, wt, a.stream);
    }
    const int64_t blocks = ceil_div(chunks, 256), cap = static_cast<int64_t>(sm_count()) * 16;
    const int cgrid = static_cast<int>(blocks < cap ? blocks : cap);
    if (a.bits == 8)
        convert_x_bf16_kernel<1><<<cgrid, 256, 0, a.stream>>>(a.x, static_cast<uint4*>(a.workspace), chunks);
    else
        convert_x_bf16_kernel<0><<<cgrid, 256, 0, a.stream>>>(a.x, static_cast<uint4*>(a.workspace), chunks);
    SGQ_LAUNCH_CHECK("convert_x_bf16_kernel");
    CUtensorMap ma, mb;
    if (!make_tensor_map_2d(&ma, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, a.workspace, static_cast<uint64_t>(a.K),
                            static_cast<uint64_t>(a.M), static_cast<uint64_t>(a.K) * 2, 64, BM, CU_TENSOR_MAP_SWIZZLE_128B))
        return SGQ_ERR_CUDA;
    if (a.bits == 8) {
        if (!make_tensor_map_2d(&mb, CU_TENSOR_MAP_DATA_TYPE_UINT8, a.wq, static_cast<uint64_t>(a.K), static_cast<uint64_t>(a.N),
                                static_cast<uint64_t>(a.K), 64, BN, CU_TENSOR_MAP_SWIZZLE_NONE))
            return SGQ_ERR_CUDA;
        p.sw = a.scales;
        p.sw_per_row = (a.scheme == SGQ_PER_ROW) ? 1 : 0;
        return launch_tc<kBF16W8>(ma, mb, p, a.stream);
    }
    if (!make_tensor_map_2d(&mb, CU_TENSOR_MAP_DATA_TYPE_UINT8, a.wq, static_cast<uint64_t>(a.K / 2),
                            static_cast<uint64_t>(a.N), static_cast<uint64_t>(a.K / 2), 32, BN, CU_TENSOR_MAP_SWIZZLE_NONE))
        return SGQ_ERR_CUDA;
    p.wscales = a.scales;
    return launch_tc<kBF16>(ma, mb, p, a.stream);
}

bool tc_i8_supported(int64_t M, int64_t K, int64_t N) {
    return M >= 1 && N >= 1 && K >= 16 && (K % 16) == 0 && M < (1LL << 31) && N < (1LL << 31) && K < (1LL << 31);
}

size_t tc_i8_workspace_bytes(int64_t M, int64_t K, int64_t N) {
    (void)N;
    return round_up(static_cast<size_t>(M) * static_cast<size_t>(K), 256) + round_up(static_cast<size_t>(M) * 4, 256);
}

int launch_linear_w8a8(const LinearArgs& a, int8_t* xq_out, float* sx_out, int32_t* acc_out) {
    if (!tc_i8_supported(a.M, a.K, a.N)) {
        set_error("kind::i8 path needs K%%16==0");
        return SGQ_ERR_UNSUPPORTED;
    }
    int8_t* xq = xq_out;
    float* sx = sx_out;
    uint8_t* ws = static_cast<uint8_t*>(a.workspace);
    size_t off = 0;
    if (!xq) {
        const size_t need = round_up(static_cast<size_t>(a.M) * a.K, 256);
        if (!ws || a.workspace_bytes < off + need) { set_error("kind::i8 path: workspace too small"); return SGQ_ERR_WORKSPACE; }
        xq = reinterpret_cast<int8_t*>(ws + off);
        off += need;
    }
    if (!sx) {
        const size_t need = round_up(static_cast<size_t>(a.M) * 4, 256);
        if (!ws || a.workspace_bytes < off + need) { set_error("kind::i8 path: workspace too small"); return SGQ_ERR_WORKSPACE; }
        sx = reinterpret_cast<float*>(ws + off);
        off += need;
    }
    if (!aligned(xq, 16) || !aligned(a.wq, 16)) {
        set_error("kind::i8 path needs 16-byte aligned code buffers");
        return SGQ_ERR_ALIGNMENT;
    }
    // activations: the reference's per-row rule (src/quantization.cpp:42-75) applied to x
    int rc = launch_quantize_int8(a.x, a.M, a.K, SGQ_PER_ROW, xq, sx, a.stream);
    if (rc != SGQ_OK) return rc;
    Params p{};
    p.bias = a.bias; p.y = a.y; p.ldy = a.ldy; p.M = a.M; p.N = a.N; p.K = a.K;
    p.sx = sx; p.sw = a.scales; p.sw_per_row = (a.scheme == SGQ_PER_ROW) ? 1 : 0; p.acc_out = acc_out;
    return launch_pair<true>(p, xq, a.wq, a.stream);
}

}  // namespace sgq
