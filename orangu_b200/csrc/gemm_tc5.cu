// Many-token products on the fifth-generation tensor cores: tcgen05.mma with accumulators in tensor memory, operands brought into shared
// memory by TMA (cp.async.bulk.tensor, no multicast: every tensor map covers this GPU's own memory and every CTA fetches its own tiles).
// Q8_0 as int8 products, Q4_K as f16 products of whole numbers; the arithmetic is the reference's, so the results equal the CPU's bit for
// bit at any batch size.
//
// Stages and accumulators are handed over through mbarriers; every wait is bounded -- a wait that runs out sets a status word, all roles
// end, nothing more is stored, and the CTA frees its tensor memory and returns.
#include "common.cuh"
#include "kernels.h"
#include "packed.cuh"
#include "pdl.cuh"
#include "tc5_common.cuh"

namespace ob {

namespace {

constexpr int TC_M = 128, TC_N = 64;
constexpr int TC_EPI_WARPS = 8;
constexpr int TC_TMA_WARP = 8, TC_MMA_WARP = 9;
constexpr int TC_THREADS = 10 * 32;
// D (tensor memory, int32, 128 lanes x N columns) [+]= A (128 x 32 int8, K-major) * B (N x 32 int8, K-major)^T
__device__ __forceinline__ void umma_i8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Instruction descriptor: int32 accumulator, A and B signed (1) or unsigned (0) 8-bit, both K-major, N columns, M = 128.
__host__ __device__ constexpr uint32_t umma_idesc_i8(uint32_t a_signed, uint32_t b_signed, uint32_t n) {
    return (2u << 4) | (a_signed << 7) | (b_signed << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}

// ---- Q8_0 ------------------------------------------------------------------------------------------------------------
// engine/vecdot.rs:2598-2629 (flat GEMM), :2829-2838 (decode): acc += (ad_b * s_b) * (f32)dot32_b per block of 32, in block order.  The int8
// codes of a row are already a K-major int8 matrix, so TMA loads them straight into the 128-byte-swizzled operand layout.  One fp32 rounding
// per 32 elements means every K = 32 step needs its own integer result: each tcgen05.mma kind::i8 (M = 128 rows, N = 64 tokens, K = 32) writes
// a fresh accumulator, four per pipeline step in one half of tensor memory while the epilogue warps drain the other half (tcgen05.ld), scale
// and accumulate in fp32.
//
// Roles in a CTA of ten warps: warps 0-7 epilogue (warp w reads the 32 tensor-memory lanes of quadrant w % 4, token columns 32 * (w / 4) ..),
// warp 8 lane 0 issues the TMA loads, warp 9 allocates tensor memory and its lane 0 issues the MMAs.
constexpr int Q8_STAGES = 4;
constexpr uint32_t Q8_A_BYTES = TC_M * 128, Q8_B_BYTES = TC_N * 128, Q8_XD_BYTES = TC_N * 16;
struct Q8Smem {  // offsets from the 1024-byte aligned base
    static constexpr uint32_t A = 0, B = A + Q8_STAGES * Q8_A_BYTES, XD = B + Q8_STAGES * Q8_B_BYTES, BAR = XD + Q8_STAGES * Q8_XD_BYTES;
    static constexpr uint32_t FULL = BAR, EMPTY = FULL + 8 * Q8_STAGES, ACC_FULL = EMPTY + 8 * Q8_STAGES, ACC_EMPTY = ACC_FULL + 16, SLOT = ACC_EMPTY + 16, ABORT = SLOT + 8;
    static constexpr uint32_t BYTES = ABORT + 8, ALLOC = BYTES + 1024;
};

struct TcQ8Args {
    GemvSegment seg;
    uint32_t n_tokens, n_steps;  // steps of four blocks (128 elements)
};

__global__ void __launch_bounds__(TC_THREADS, 1)
gemm_tc5_q8_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_xd, TcQ8Args a) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *smem = smem_raw + (sbase - smem_u32(smem_raw));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t row0 = blockIdx.x * TC_M, tok0 = blockIdx.y * TC_N;
    volatile uint32_t *abort = reinterpret_cast<volatile uint32_t *>(smem + Q8Smem::ABORT);
    const uint32_t n_steps = a.n_steps;

    if (threadIdx.x == 0) {
        for (int s = 0; s < Q8_STAGES; ++s) {
            mbar_init(sbase + Q8Smem::FULL + 8 * s, 1);                  // the producer's expect_tx arrival
            mbar_init(sbase + Q8Smem::EMPTY + 8 * s, 1 + TC_EPI_WARPS);  // MMA completion + the epilogue warps (they read the token scales)
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(sbase + Q8Smem::ACC_FULL + 8 * b, 1);
            mbar_init(sbase + Q8Smem::ACC_EMPTY + 8 * b, TC_EPI_WARPS);
        }
        *abort = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == TC_MMA_WARP) tmem_alloc(sbase + Q8Smem::SLOT, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(smem + Q8Smem::SLOT);

    if (warp == TC_TMA_WARP) {
        if (lane == 0) {
            for (uint32_t it = 0; it < n_steps; ++it) {
                const uint32_t s = it % Q8_STAGES;
                if (it >= Q8_STAGES && !mbar_wait(sbase + Q8Smem::EMPTY + 8 * s, ((it / Q8_STAGES) & 1u) ^ 1u, abort)) break;
                const uint32_t full = sbase + Q8Smem::FULL + 8 * s;
                mbar_expect_tx(full, Q8_A_BYTES + Q8_B_BYTES + Q8_XD_BYTES);
                tma_load_2d(sbase + Q8Smem::A + s * Q8_A_BYTES, &tm_w, (int32_t)(it * 128), (int32_t)row0, full);
                tma_load_2d(sbase + Q8Smem::B + s * Q8_B_BYTES, &tm_x, (int32_t)(it * 128), (int32_t)tok0, full);
                tma_load_2d(sbase + Q8Smem::XD + s * Q8_XD_BYTES, &tm_xd, (int32_t)(it * 4), (int32_t)tok0, full);
            }
        }
    } else if (warp == TC_MMA_WARP) {
        if (lane == 0) {
            constexpr uint32_t idesc = umma_idesc_i8(1, 1, TC_N);
            for (uint32_t it = 0; it < n_steps; ++it) {
                const uint32_t s = it % Q8_STAGES, buf = it & 1u;
                if (!mbar_wait(sbase + Q8Smem::FULL + 8 * s, (it / Q8_STAGES) & 1u, abort)) break;
                if (it >= 2 && !mbar_wait(sbase + Q8Smem::ACC_EMPTY + 8 * buf, ((it / 2) & 1u) ^ 1u, abort)) break;
                tc_fence_after();
                const uint64_t da = umma_desc_sw128(sbase + Q8Smem::A + s * Q8_A_BYTES), db = umma_desc_sw128(sbase + Q8Smem::B + s * Q8_B_BYTES);
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j)  // block j of the step: its own accumulator, nothing is added up on the tensor core
                    umma_i8(tmem + buf * 256 + j * TC_N, da + 2 * j, db + 2 * j, idesc, 0u);
                umma_commit(sbase + Q8Smem::EMPTY + 8 * s);
                umma_commit(sbase + Q8Smem::ACC_FULL + 8 * buf);
            }
        }
    } else {
        // ---- epilogue: thread = one row x 32 tokens
        const uint32_t quad = warp & 3u, half = warp >> 2;
        const uint32_t row = row0 + quad * 32 + lane;
        const bool row_ok = row < a.seg.w.out_dim;
        const uint8_t *wrow = a.seg.w.data + (uint64_t)min(row, a.seg.w.out_dim - 1) * a.seg.w.row_stride + a.seg.w.d_off;
        float acc[32];
#pragma unroll
        for (int t = 0; t < 32; ++t) acc[t] = 0.0f;
        uint2 sw_next = __ldg(reinterpret_cast<const uint2 *>(wrow));  // the row's four f16 block scales of step 0
        for (uint32_t it = 0; it < n_steps; ++it) {
            const uint32_t s = it % Q8_STAGES, buf = it & 1u;
            const uint2 swb = sw_next;
            if (it + 1 < n_steps) sw_next = __ldg(reinterpret_cast<const uint2 *>(wrow + 8 * (it + 1)));
            mbar_wait_on(sbase + Q8Smem::ACC_FULL + 8 * buf, (it / 2) & 1u, abort);
            tc_fence_after();
            const float sw[4] = {f16_bits_to_f32(swb.x & 0xffffu), f16_bits_to_f32(swb.x >> 16), f16_bits_to_f32(swb.y & 0xffffu), f16_bits_to_f32(swb.y >> 16)};
            const float4 *xd = reinterpret_cast<const float4 *>(smem + Q8Smem::XD + s * Q8_XD_BYTES) + half * 32;  // [token] the four block scales
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                uint32_t r[32];
                tmem_ld32(tmem + ((quad * 32) << 16) + buf * 256 + j * TC_N + half * 32, r);
                tmem_ld_wait();
#pragma unroll
                for (int t = 0; t < 32; ++t) {
                    const float4 d4 = xd[t];
                    const float ad = j == 0 ? d4.x : j == 1 ? d4.y : j == 2 ? d4.z : d4.w;
                    acc[t] = __fadd_rn(acc[t], __fmul_rn(__fmul_rn(ad, sw[j]), (float)(int)r[t]));  // (ad_b * s_b) * dot32_b, vecdot.rs:2620
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(sbase + Q8Smem::ACC_EMPTY + 8 * buf);
                mbar_arrive(sbase + Q8Smem::EMPTY + 8 * s);
            }
        }
        if (!*abort && row_ok) {
#pragma unroll
            for (int t = 0; t < 32; ++t) {
                const uint32_t tok = tok0 + half * 32 + t;
                if (tok < a.n_tokens) {
                    const uint64_t o = (uint64_t)tok * a.seg.y_stride + row;
                    float v = acc[t];
                    if (a.seg.epilogue == EPI_ADD_RESIDUAL) v = __fadd_rn(a.seg.residual[o], v);
                    a.seg.y[o] = v;
                }
            }
        }
    }
    if (*abort) {  // let copies that are still in flight land before the shared memory goes away
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == TC_MMA_WARP) tmem_dealloc(tmem, 512);
}

// ---- Q4_K -----------------------------------------------------------------------------------------------------------
// The codes cannot go to the tensor core as they are: every 32-element sub-block has its own 6-bit scale, and
// isum = sum_j sc_j * dot32_j has to be exact.  So the scale goes into the operand: sc * code <= 63 * 15 = 945 is a whole number that
// f16 holds exactly, and so is every 8-bit activation code; fp32 accumulators add whole numbers exactly below 2^24.  Where the scales
// times codes of every block of a row add up to no more than Q4K_SUM24, 256 products stay below that whatever the activations are, and the
// accumulator is (float)isum.  The few rows with a larger block (two or three in a matrix of 14336; found at registration) are left to a
// kernel of their own (gemm_few.cu); a matrix with many keeps the halves of a super-block in two accumulators, whose rounded sum is
// (float)isum.  The min term imin = sum_j m_j * bsum_j is one K = 16 step: with bsum = lo + 64 hi, weights [m | 64 m] against [lo | hi],
// all whole numbers that f16 holds.  The epilogue forms the super-block's fp32 term in the CPU's association and order:
//   decode order   acc += ad * (d * isum - dmin * imin)                          (engine/vecdot.rs:3152-3178)
//   prefill order  first for every super-block acc -= (ad * dmin) * imin, then acc += ad * (d * isum)
//                  (engine/vecdot.rs:2119-2143, 2213-2255): two sweeps over K, the first over the block headers only.
//
// A CTA is persistent over tiles of 128 rows x N tokens.  Its warps: 0-7 epilogue (thread = one row x N / 2 tokens, two at a time in
// packed fp32), 8-15 expanders (thread = half a super-block of one row), 16 loads (TMA), 17 and 18 issue products.  An expander turns its half
// into 64 words of two f16 -- codes enter a mantissa by a mask, one packed multiply-add takes the offset off and the scale on -- and writes
// them to tensor memory, where the products read their A operand: expanded weights never touch shared memory, whose bandwidth the
// activations (B, f16 from the quantizer) already take.  The order of elements within a group of four is the one the mask leaves
// (0, 2, 1, 3); the quantizer writes activations in that order.
//
// The form before had byte planes of the weights' scale digits in shared memory, int8 products and two or three accumulators to read
// back: 14336 x 4096 with 509 tokens 213 us in prefill order (now 130), 4096 x 14336 with 64 tokens 70 us in decode order on mma.sync
// tiles (now 52).  What bounds this form is the chain of its warps, five to a scheduler: 53 % of the issue slots are used and the tensor pipe
// is busy for 29 % of the time, at 320 instructions a warp and super-block, both sweeps of the prefill order together.
constexpr int KQ_EPI_WARPS = 8, KQ_EXP_WARPS = 8, KQ_TMA_WARP = 16, KQ_MMA_WARP = 17, KQ_THREADS = 19 * 32;
constexpr uint32_t KQ_RAW_BYTES = TC_M * 144, KQ_A_COLS = 128;
// TWO: the halves of a super-block have accumulators of their own (matrices with many wide rows).
template <bool GEMM, int N>
struct KqPlan {
    static constexpr uint32_t A_COL = GEMM ? 256 : 240, MIN_COL = A_COL + 2 * KQ_A_COLS;  // tensor memory: accumulators, then the two A buffers (decode order: and their mins)
    static constexpr uint32_t SLOT_COLS = (GEMM ? 1 : 2) * N;  // accumulators of a super-block (decode order: and of its mins), or of half of a wide one
    static_assert(2 * SLOT_COLS <= A_COL, "products of a super-block run while the epilogue reads the one before");
    static constexpr uint32_t B_BYTES = N * 512, B_STAGE = B_BYTES + (GEMM ? 0 : N * 128);  // decode order: and the sums of four super-blocks
    static constexpr uint32_t B_STAGES = N > 64 ? 2 : 3, RAW_STAGES = N > 64 ? 3 : 4;
    static constexpr uint32_t RAW = 0, B = RAW + RAW_STAGES * KQ_RAW_BYTES, BAR = B + B_STAGES * B_STAGE;
    static constexpr uint32_t RAW_FULL = BAR, RAW_EMPTY = RAW_FULL + 8 * RAW_STAGES, B_FULL = RAW_EMPTY + 8 * RAW_STAGES, B_EMPTY = B_FULL + 8 * B_STAGES, A_FULL = B_EMPTY + 8 * B_STAGES,
                              A_EMPTY = A_FULL + 16, XD_FULL = A_EMPTY + 16, XD_EMPTY = XD_FULL + 16, ACC_FULL = XD_EMPTY + 16, ACC_EMPTY = ACC_FULL + 16, SLOT = ACC_EMPTY + 16, ABORT = SLOT + 8;
    static constexpr uint32_t XD = (ABORT + 8 + 127) / 128 * 128;  // token scales of a tile, [nb][N] floats; twice when there is room
    __host__ __device__ static constexpr uint32_t xd_bytes(uint32_t nb) { return (nb * N * 4 + 127) / 128 * 128; }
    static constexpr uint32_t bytes(uint32_t nb, uint32_t n_xd) { return XD + n_xd * xd_bytes(nb) + 1024; }
};

struct KqMaps {
    CUtensorMap raw[3], x, bs, xd;
};
struct KqArgs {
    GemvSegment seg[3];  // matrices of one width that read the same activations
    const uint8_t *wide[3];
    uint32_t tiles[3];   // running sums of their row tiles
    uint32_t n_tokens, nb, tok_tiles, n_tiles, n_xd;
    uint64_t ones;       // F2_ONES
};

__device__ __forceinline__ uint32_t h2_fma(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t v;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(v) : "r"(a), "r"(b), "r"(c));
    return v;
}
__device__ __forceinline__ uint32_t h2_mul(uint32_t a, uint32_t b) {
    uint32_t v;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(v) : "r"(a), "r"(b));
    return v;
}
__device__ __forceinline__ uint32_t h2_sub(uint32_t a, uint32_t b) {
    uint32_t v;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(v) : "r"(a), "r"(b));
    return v;
}
constexpr uint32_t H2_1024 = 0x64006400u, H2_M1024 = 0xe400e400u, H2_M64 = 0xd400d400u, H2_64 = 0x54005400u, H2_16TH = 0x2c002c00u;

// STEPS products of K = 16 in a row: A in tensor memory (128 lanes, two f16 of K a column, 8 columns a step), B in shared memory in boxes of
// four steps, box_step (16-byte units) apart.  One lane of a converged warp issues all of them.
__device__ __forceinline__ void umma_f16_ta_8(uint32_t d, uint32_t a, uint64_t b, uint32_t box_step, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q, t;\n\t.reg .b64 b1, b2, b3, b4, b5, b6, b7, bs;\n\t.reg .b32 a1, a2, a3, a4, a5, a6, a7;\n\t"
        "elect.sync _|q, 0xffffffff;\n\tsetp.ne.b32 p, %5, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
        "cvt.u64.u32 bs, %3;\n\tadd.s64 b1, %2, 2;\n\tadd.s64 b2, %2, 4;\n\tadd.s64 b3, %2, 6;\n\tadd.s64 b4, %2, bs;\n\tadd.s64 b5, b4, 2;\n\tadd.s64 b6, b4, 4;\n\tadd.s64 b7, b4, 6;\n\t"
        "add.s32 a1, %1, 8;\n\tadd.s32 a2, %1, 16;\n\tadd.s32 a3, %1, 24;\n\tadd.s32 a4, %1, 32;\n\tadd.s32 a5, %1, 40;\n\tadd.s32 a6, %1, 48;\n\tadd.s32 a7, %1, 56;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %4, p;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %4, t;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b2, %4, t;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], b3, %4, t;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a4], b4, %4, t;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a5], b5, %4, t;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a6], b6, %4, t;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a7], b7, %4, t;\n\t}" ::"r"(d),
        "r"(a), "l"(b), "r"(box_step), "r"(idesc), "r"(accumulate)
        : "memory");
}
__host__ __device__ constexpr uint32_t umma_idesc_f16(uint32_t n) { return (1u << 4) | ((n >> 3) << 17) | ((128u >> 4) << 24); }  // fp32 accumulator, A and B f16, both K-major

// A counter through a ring of S places: the place and the parity of its current round.
template <uint32_t S>
struct Ring {
    uint32_t at = 0, round = 0;
    __device__ __forceinline__ void next() {
        if (++at == S) {
            at = 0;
            ++round;
        }
    }
    __device__ __forceinline__ void skip(uint32_t n) {
        at += n;
        round += at / S;
        at %= S;
    }
    __device__ __forceinline__ uint32_t full_parity() const { return round & 1u; }
    __device__ __forceinline__ uint32_t empty_parity() const { return (round & 1u) ^ 1u; }  // of the round before
};

// 8 words: the mins of a super-block, m_j in pairs, then 64 m_j.
__device__ __forceinline__ void kq_mins(const uint4 &hd, uint32_t *out) {
    const uint32_t ml = hd.z & 0x3f3f3f3fu, mh = ((hd.w >> 4) & 0x0f0f0f0fu) | ((hd.z >> 2) & 0x30303030u);
    out[0] = h2_sub(__byte_perm(ml, 0x64646464u, 0x4140), H2_1024);
    out[1] = h2_sub(__byte_perm(ml, 0x64646464u, 0x4342), H2_1024);
    out[2] = h2_sub(__byte_perm(mh, 0x64646464u, 0x4140), H2_1024);
    out[3] = h2_sub(__byte_perm(mh, 0x64646464u, 0x4342), H2_1024);
#pragma unroll
    for (int i = 0; i < 4; ++i) out[4 + i] = h2_mul(out[i], H2_64);
}

template <bool GEMM, bool TWO, int N>
__global__ void __launch_bounds__(KQ_THREADS, 1) gemm_tc5_q4k_kernel(const __grid_constant__ KqMaps maps, const __grid_constant__ KqArgs a) {
    using P = KqPlan<GEMM, N>;
    constexpr int TPT = N / 2;                   // tokens per epilogue thread
    constexpr int CH = TPT % 16 || TPT >= 48 ? 8 : 16;         // tokens at a time
    extern __shared__ uint8_t smem_raw[];
    const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *smem = smem_raw + (sbase - smem_u32(smem_raw));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    volatile uint32_t *abort = reinterpret_cast<volatile uint32_t *>(smem + P::ABORT);
    const uint32_t nb = a.nb, n_min = GEMM ? (nb + 15) / 16 : 0;  // prefill order: sixteen super-blocks of mins fill an A buffer

    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < P::RAW_STAGES; ++i) {
            mbar_init(sbase + P::RAW_FULL + 8 * i, 1);
            mbar_init(sbase + P::RAW_EMPTY + 8 * i, KQ_EXP_WARPS);
        }
        for (uint32_t i = 0; i < P::B_STAGES; ++i) {
            mbar_init(sbase + P::B_FULL + 8 * i, 1);
            mbar_init(sbase + P::B_EMPTY + 8 * i, 1);
        }
        for (uint32_t i = 0; i < 2; ++i) {
            mbar_init(sbase + P::A_FULL + 8 * i, KQ_EXP_WARPS);
            mbar_init(sbase + P::A_EMPTY + 8 * i, 1);
            mbar_init(sbase + P::XD_FULL + 8 * i, 1);
            mbar_init(sbase + P::XD_EMPTY + 8 * i, KQ_EPI_WARPS);
            mbar_init(sbase + P::ACC_FULL + 8 * i, 1);
            mbar_init(sbase + P::ACC_EMPTY + 8 * i, KQ_EPI_WARPS);
        }
        *abort = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == KQ_MMA_WARP) tmem_alloc(sbase + P::SLOT, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(smem + P::SLOT);

    // tile -> matrix, first row, first token; tokens change fastest, so that CTAs side by side read the same weights
    auto locate = [&](uint32_t tile, uint32_t &row0, uint32_t &tok0) -> uint32_t {
        const uint32_t rt = tile / a.tok_tiles;
        tok0 = (tile - rt * a.tok_tiles) * N;
        const uint32_t si = rt < a.tiles[0] ? 0u : rt < a.tiles[1] ? 1u : 2u;
        row0 = (rt - (si ? a.tiles[si - 1] : 0u)) * TC_M;
        return si;
    };

    if (warp == KQ_TMA_WARP) {
        if (lane == 0) {
            Ring<P::RAW_STAGES> raw;
            Ring<P::B_STAGES> bs;
            uint32_t it = 0;
            bool ok = true;
            auto load_b = [&](const CUtensorMap *tm, uint32_t x, uint32_t tok0, uint32_t sums) {
                if (bs.round && !mbar_wait(sbase + P::B_EMPTY + 8 * bs.at, bs.empty_parity(), abort)) return false;
                const uint32_t full = sbase + P::B_FULL + 8 * bs.at, dst = sbase + P::B + bs.at * P::B_STAGE;
                mbar_expect_tx(full, P::B_STAGE);
#pragma unroll
                for (uint32_t i = 0; i < 4; ++i) tma_load_2d(dst + i * N * 128, tm, (int32_t)(x + 64 * i), (int32_t)tok0, full);
                if (!GEMM) tma_load_2d(dst + N * 512, &maps.bs, (int32_t)sums, (int32_t)tok0, full);
                bs.next();
                return true;
            };
            for (uint32_t tile = blockIdx.x; tile < a.n_tiles && ok; tile += gridDim.x, ++it) {
                uint32_t row0, tok0;
                const uint32_t si = locate(tile, row0, tok0);
                {   // token scales of the tile
                    const uint32_t xs = it % a.n_xd, xr = it / a.n_xd;
                    if (xr && !(ok = mbar_wait(sbase + P::XD_EMPTY + 8 * xs, (xr & 1u) ^ 1u, abort))) break;
                    mbar_expect_tx(sbase + P::XD_FULL + 8 * xs, nb * N * 4);
                    tma_load_2d(sbase + P::XD + xs * P::xd_bytes(nb), &maps.xd, (int32_t)tok0, 0, sbase + P::XD_FULL + 8 * xs);
                }
                for (uint32_t j = 0; j < n_min && ok; ++j) ok = load_b(&maps.bs, j * 256, tok0, 0);
                for (uint32_t s = 0; s < nb && ok; ++s) {
                    if (raw.round && !(ok = mbar_wait(sbase + P::RAW_EMPTY + 8 * raw.at, raw.empty_parity(), abort))) break;
                    mbar_expect_tx(sbase + P::RAW_FULL + 8 * raw.at, KQ_RAW_BYTES);
                    tma_load_2d(sbase + P::RAW + raw.at * KQ_RAW_BYTES, &maps.raw[si], (int32_t)(s * 144), (int32_t)row0, sbase + P::RAW_FULL + 8 * raw.at);
                    raw.next();
                    ok = load_b(&maps.x, s * 256, tok0, (s & ~3u) * 16);
                }
            }
        }
    } else if (warp >= KQ_MMA_WARP) {
        // Two warps issue, on schedulers of their own: the first all mins, then each every other super-block.  A warp goes through the phases
        // of its barriers one by one: it waits for a slot's, a buffer's or a stage's n-th use only when the one before is known to be over
        // (by its own waits, by the epilogue's order, or by the meeting points before and after the mins).
        const uint32_t which = warp - KQ_MMA_WARP;
        auto meet = [] { asm volatile("bar.sync 1, 64;" ::: "memory"); };
        constexpr uint32_t idesc = umma_idesc_f16(N), BOX = N * 128 / 16;
        Ring<P::B_STAGES> bs;
        Ring<2> ab, ac;
        bool ok = true;
        auto wait_operands = [&] {
            const uint32_t b = sbase + P::B_FULL + 8 * bs.at, x = sbase + P::A_FULL + 8 * ab.at;
            if (__all_sync(0xffffffffu, mbar_try2(x, ab.full_parity(), b, bs.full_parity()))) return true;
            return mbar_wait_warp(b, bs.full_parity(), abort) && mbar_wait_warp(x, ab.full_parity(), abort);
        };
        auto wait_slot = [&] { return !ac.round || mbar_wait_ready_warp(sbase + P::ACC_EMPTY + 8 * ac.at, ac.empty_parity(), abort); };
        auto stage_done = [&] {
            umma_commit_warp(sbase + P::A_EMPTY + 8 * ab.at);
            umma_commit_warp(sbase + P::B_EMPTY + 8 * bs.at);
            ab.next();
            bs.next();
        };
        for (uint32_t tile = blockIdx.x; tile < a.n_tiles; tile += gridDim.x) {  // (after a failed wait too: both warps come to every meeting)
            if (GEMM) {
                if (which == 0) {
                    for (uint32_t j = 0; j < n_min && ok; ++j) {  // sixteen super-blocks of mins
                        if (!(ok = wait_operands())) break;
                        const uint64_t db = umma_desc_sw128(sbase + P::B + bs.at * P::B_STAGE);
                        const uint32_t ta = tmem + P::A_COL + ab.at * KQ_A_COLS;
                        for (uint32_t i = 0; i < 16 && 16 * j + i < nb; ++i) {
                            if (!(ok = wait_slot())) break;
                            tc_fence_after();
                            umma_bf16_ta_warp(tmem + ac.at * P::SLOT_COLS, ta + 8 * i, db + (i >> 2) * BOX + (i & 3u) * 2, idesc, 0u);
                            umma_commit_warp(sbase + P::ACC_FULL + 8 * ac.at);
                            ac.next();
                        }
                        if (ok) stage_done();
                    }
                } else {
                    ab.skip(n_min);
                    bs.skip(n_min);
                    ac.skip(nb);
                }
                meet();
            }
            for (uint32_t s = 0; s < nb && ok; ++s) {
                if (TWO ? which == 1 : (s & 1u) != which) {  // (halves apart take both slots: one warp issues them all)
                    ab.next();
                    bs.next();
                    ac.skip(TWO ? 2 : 1);
                    continue;
                }
                const uint32_t ta = tmem + P::A_COL + ab.at * KQ_A_COLS;
                const uint64_t db = umma_desc_sw128(sbase + P::B + bs.at * P::B_STAGE);
                if (!(ok = wait_slot() && wait_operands())) break;
                tc_fence_after();
                uint32_t td = tmem + ac.at * P::SLOT_COLS;
                umma_f16_ta_8(td, ta, db, BOX, idesc, 0u);
                if (TWO) {  // the halves' sums apart
                    umma_commit_warp(sbase + P::ACC_FULL + 8 * ac.at);
                    ac.next();
                    if (!(ok = wait_slot())) break;
                    tc_fence_after();
                    td = tmem + ac.at * P::SLOT_COLS;
                }
                umma_f16_ta_8(td, ta + 64, db + 2 * BOX, BOX, idesc, TWO ? 0u : 1u);
                if (!GEMM) umma_bf16_ta_warp(td + N, tmem + P::MIN_COL + 8 * ab.at, db + 4 * BOX + (s & 3u) * 2, idesc, 0u);
                umma_commit_warp(sbase + P::ACC_FULL + 8 * ac.at);
                stage_done();
                ac.next();
            }
            meet();
        }
    } else if (warp >= KQ_EPI_WARPS) {
        // ---- expanders: thread = half a super-block of one row
        const uint32_t quad = warp & 3u, h = (warp >> 2) & 1u, r = quad * 32 + lane;
        const uint32_t ta = tmem + ((quad * 32) << 16) + P::A_COL;
        Ring<P::RAW_STAGES> raw;
        Ring<2> ab;
        auto wait_a = [&] { if (ab.round) mbar_wait_on(sbase + P::A_EMPTY + 8 * ab.at, ab.empty_parity(), abort); };
        auto store = [&](uint32_t (&w)[64]) {
            const uint32_t to = ta + ab.at * KQ_A_COLS + 64 * h;
            tmem_st32(to, *reinterpret_cast<uint32_t(*)[32]>(w));
            tmem_st32(to + 32, *reinterpret_cast<uint32_t(*)[32]>(w + 32));
        };
        auto done_a = [&] {
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(sbase + P::A_FULL + 8 * ab.at);
            ab.next();
        };
        for (uint32_t tile = blockIdx.x; tile < a.n_tiles; tile += gridDim.x) {
            uint32_t row0, tok0;
            const GemvSegment &seg = a.seg[locate(tile, row0, tok0)];
            const uint8_t *wrow = seg.w.data + (uint64_t)min(row0 + r, seg.w.out_dim - 1) * seg.w.row_stride;
            for (uint32_t j = 0; j < n_min; ++j) {
                uint32_t w[64];
#pragma unroll
                for (uint32_t i = 0; i < 8; ++i) {
                    const uint4 hd = __ldg(reinterpret_cast<const uint4 *>(wrow + (uint64_t)min(16 * j + 8 * h + i, nb - 1) * 144));
                    kq_mins(hd, w + 8 * i);
                }
                wait_a();
                tc_fence_after();
                store(w);
                done_a();
            }
            for (uint32_t s = 0; s < nb; ++s, raw.next()) {
                mbar_wait_on(sbase + P::RAW_FULL + 8 * raw.at, raw.full_parity(), abort);
                const uint8_t *blk = smem + P::RAW + raw.at * KQ_RAW_BYTES + r * 144u;
                const uint4 hd = *reinterpret_cast<const uint4 *>(blk);
                // the half's four 6-bit scales (engine/quant.rs:653-662) as bytes of a word, then each twice as f16
                const uint32_t scw = h == 0 ? hd.y & 0x3f3f3f3fu : (hd.w & 0x0f0f0f0fu) | ((hd.y >> 2) & 0x30303030u);
                uint32_t out[64];
#pragma unroll
                for (uint32_t g = 0; g < 2; ++g) {  // 64 elements: 32 low nibbles, 32 high ones
                    const uint4 qa = *reinterpret_cast<const uint4 *>(blk + 16 + 64 * h + 32 * g), qb = *reinterpret_cast<const uint4 *>(blk + 32 + 64 * h + 32 * g);
                    const uint32_t sa = h2_sub(__byte_perm(scw, 0x64646464u, g ? 0x4242 : 0x4040), H2_1024), sb = h2_sub(__byte_perm(scw, 0x64646464u, g ? 0x4343 : 0x4141), H2_1024);
                    const uint32_t oa = h2_mul(sa, H2_M1024), sb16 = h2_mul(sb, H2_16TH), ob = h2_mul(sb, H2_M64);
                    const uint32_t w[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
#pragma unroll
                    for (int i = 0; i < 8; ++i) {  // 1024 + code and 1024 + 16 code as f16 mantissas; times the scale, less 1024 times it: exact
                        const uint32_t v = w[i] >> 8;
                        out[32 * g + 2 * i] = h2_fma((w[i] & 0x000f000fu) | H2_1024, sa, oa);
                        out[32 * g + 2 * i + 1] = h2_fma((v & 0x000f000fu) | H2_1024, sa, oa);
                        out[32 * g + 16 + 2 * i] = h2_fma((w[i] & 0x00f000f0u) | H2_1024, sb16, ob);
                        out[32 * g + 16 + 2 * i + 1] = h2_fma((v & 0x00f000f0u) | H2_1024, sb16, ob);
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(sbase + P::RAW_EMPTY + 8 * raw.at);
                wait_a();
                tc_fence_after();
                store(out);
                if (!GEMM && h == 1) {
                    uint32_t w[8];
                    kq_mins(hd, w);
                    tmem_st8(tmem + ((quad * 32) << 16) + P::MIN_COL + 8 * ab.at, w);
                }
                done_a();
            }
        }
    } else {
        // ---- epilogue: thread = one row x N / 2 tokens
        const uint32_t quad = warp & 3u, half = warp >> 2, rl = quad * 32 + lane;
        const uint32_t tbase = tmem + ((quad * 32) << 16) + half * TPT;
        const uint64_t ones = a.ones;
        Ring<2> ac;
        uint32_t it = 0;
        for (uint32_t tile = blockIdx.x; tile < a.n_tiles; tile += gridDim.x, ++it) {
            uint32_t row0, tok0;
            const uint32_t si = locate(tile, row0, tok0);
            const GemvSegment &seg = a.seg[si];
            const uint32_t row = row0 + rl;
            const uint8_t *wrow = seg.w.data + (uint64_t)min(row, seg.w.out_dim - 1) * seg.w.row_stride;
            const uint32_t xs = it % a.n_xd, xr = it / a.n_xd;
            mbar_wait_on(sbase + P::XD_FULL + 8 * xs, xr & 1u, abort);
            const float *xd = reinterpret_cast<const float *>(smem + P::XD + xs * P::xd_bytes(nb)) + half * TPT;
            uint64_t acc[TPT / 2];
#pragma unroll
            for (int t = 0; t < TPT / 2; ++t) acc[t] = 0ull;
            auto header = [&](uint32_t s) { return __ldg(reinterpret_cast<const uint32_t *>(wrow + (uint64_t)min(s, nb - 1) * 144)); };  // d | dmin << 16
            uint32_t dw0 = header(0), dw1 = header(1);
            if (GEMM) {
                for (uint32_t s = 0; s < nb; ++s) {
                    const uint32_t dw2 = header(s + 2);
                    mbar_wait_on(sbase + P::ACC_FULL + 8 * ac.at, ac.full_parity(), abort);
                    tc_fence_after();
                    const uint64_t dmin2 = f2_both(-f16_bits_to_f32(dw0 >> 16));
                    const float4 *ad4 = reinterpret_cast<const float4 *>(xd + s * N);
#pragma unroll
                    for (int c = 0; c < TPT / CH; ++c) {
                        uint32_t p[CH];
                        tmem_ldn<CH>(tbase + ac.at * P::SLOT_COLS + c * CH, p);
                        tmem_ld_wait();
#pragma unroll
                        for (int t = 0; t < CH / 4; ++t) {
                            const float4 v = ad4[c * (CH / 4) + t];
                            const uint64_t ad[2] = {f2_pack(v.x, v.y), f2_pack(v.z, v.w)};
#pragma unroll
                            for (int k = 0; k < 2; ++k) {
                                uint64_t &o = acc[c * (CH / 2) + 2 * t + k];
                                o = f2_add(f2_mul(f2_mul(ad[k], dmin2), f2_pack(p[4 * t + 2 * k], p[4 * t + 2 * k + 1])), o, ones);  // x - y = x + (-y), the sign taken with dmin
                            }
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(sbase + P::ACC_EMPTY + 8 * ac.at);
                    ac.next();
                    dw0 = dw1;
                    dw1 = dw2;
                }
                dw0 = header(0);
                dw1 = header(1);
            }
            auto sweep = [&] {
                for (uint32_t s = 0; s < nb; ++s) {
                    const uint32_t dw2 = header(s + 2);
                    const uint64_t d2 = f2_both(f16_bits_to_f32(dw0 & 0xffffu)), dmin2 = f2_both(-f16_bits_to_f32(dw0 >> 16));
                    const uint32_t first = ac.at;
                    mbar_wait_on(sbase + P::ACC_FULL + 8 * ac.at, ac.full_parity(), abort);
                    if (TWO) {
                        ac.next();
                        mbar_wait_on(sbase + P::ACC_FULL + 8 * ac.at, ac.full_parity(), abort);
                    }
                    tc_fence_after();
                    const float4 *ad4 = reinterpret_cast<const float4 *>(xd + s * N);
                    const uint32_t tslot = tbase + ac.at * P::SLOT_COLS;
#pragma unroll
                    for (int c = 0; c < TPT / CH; ++c) {
                        uint32_t p0[CH], p1[CH], p2[CH];
                        tmem_ldn<CH>(tslot + c * CH, p0);
                        if (TWO) tmem_ldn<CH>(tbase + first * P::SLOT_COLS + c * CH, p1);
                        if (!GEMM) tmem_ldn<CH>(tslot + N + c * CH, p2);
                        tmem_ld_wait();
#pragma unroll
                        for (int t = 0; t < CH / 4; ++t) {
                            const float4 v = ad4[c * (CH / 4) + t];
                            const uint64_t ad[2] = {f2_pack(v.x, v.y), f2_pack(v.z, v.w)};
#pragma unroll
                            for (int k = 0; k < 2; ++k) {
                                const int i = 4 * t + 2 * k;
                                uint64_t &o = acc[c * (CH / 2) + 2 * t + k];
                                uint64_t m = f2_pack(p0[i], p0[i + 1]);
                                if (TWO) m = f2_add(m, f2_pack(p1[i], p1[i + 1]), ones);  // both are whole numbers: their rounded sum is (float)isum
                                m = f2_mul(d2, m);
                                if (!GEMM) m = f2_add(f2_mul(dmin2, f2_pack(p2[i], p2[i + 1])), m, ones);
                                o = f2_add(f2_mul(ad[k], m), o, ones);
                            }
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(sbase + P::ACC_EMPTY + 8 * ac.at);
                        if (TWO) mbar_arrive(sbase + P::ACC_EMPTY + 8 * first);
                    }
                    ac.next();
                    dw0 = dw1;
                    dw1 = dw2;
                }
            };
            sweep();
            __syncwarp();
            if (lane == 0) mbar_arrive(sbase + P::XD_EMPTY + 8 * xs);
            if (!*abort && row < seg.w.out_dim && (TWO || !__ldg(a.wide[si] + row))) {  // (wide rows are left to the kernel that follows)
                const uint32_t t0 = tok0 + half * TPT, n = a.n_tokens > t0 ? min((uint32_t)TPT, a.n_tokens - t0) : 0u;
                float *y = seg.y + (uint64_t)t0 * seg.y_stride + row;
                const float *res = seg.epilogue == EPI_ADD_RESIDUAL ? seg.residual + (uint64_t)t0 * seg.y_stride + row : nullptr;
#pragma unroll
                for (int c = 0; c < TPT; c += 8) {
                    float v[8];
#pragma unroll
                    for (int t = 0; t < 8; ++t) v[t] = res && c + t < (int)n ? res[(uint64_t)(c + t) * seg.y_stride] : 0.0f;
#pragma unroll
                    for (int t = 0; t < 8; ++t) {
                        const float o = t & 1 ? f2_hi(acc[(c + t) / 2]) : f2_lo(acc[(c + t) / 2]);
                        if (c + t < (int)n) y[(uint64_t)(c + t) * seg.y_stride] = res ? __fadd_rn(v[t], o) : o;
                    }
                }
            }
        }
    }
    pdl_wait();  // started beside the kernel of the wide rows (launch_q4k_instance), this one does not end before it
    if (*abort) {  // let copies that are still in flight land before the shared memory goes away
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == KQ_MMA_WARP) tmem_dealloc(tmem, 512);
}

}  // namespace

bool gemm_tc5_supported(const GemvArgs &a) {
    static const bool enabled = [] { const char *e = getenv("OB_TC5"); return !(e && e[0] == '0' && e[1] == 0); }();
    if (!enabled || a.n_seg < 1 || a.n_tokens < (a.seg[0].w.type == TYPE_Q4_K ? ACT_H_ROWS : 16u) || a.isum_out || !encode_fn()) return false;
    const uint32_t type = a.seg[0].w.type, in_dim = a.seg[0].w.in_dim;
    if (type == TYPE_Q8_0) {
        if (in_dim % 128 || a.act.dim_cap % 128) return false;
    } else if (type == TYPE_Q4_K) {
        if (in_dim % 256 || in_dim / 256 > 256 || a.act.dim_cap % 256) return false;
        for (int s = 0; s < a.n_seg; ++s)
            if (!a.seg[s].wide || !a.seg[s].wide->flags) return false;
    } else {
        return false;  // Q6_K stays on the mma.sync tiles (gemm_mma.cu)
    }
    for (int s = 0; s < a.n_seg; ++s)
        if (a.seg[s].w.type != type || a.seg[s].w.in_dim != in_dim || (a.seg[s].w.row_stride & 15) || (type == TYPE_Q8_0 && (a.seg[s].w.d_off & 7))) return false;
    return true;
}

template <bool GEMM, bool TWO, int N>
static uint32_t launch_q4k_instance(const GemvArgs &a, int sm_count, cudaStream_t st) {
    using P = KqPlan<GEMM, N>;
    static PerDeviceOnce once;
    if (once.run([] { return cudaFuncSetAttribute(gemm_tc5_q4k_kernel<GEMM, TWO, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024); }) != cudaSuccess) return 0;
    const uint32_t in_dim = a.seg[0].w.in_dim, nb = in_dim / 256;
    KqArgs k{};
    KqMaps m;
    k.n_xd = P::bytes(nb, 2) <= 227 * 1024 ? 2 : 1;
    if (P::bytes(nb, k.n_xd) > 227 * 1024) return 0;
    if (!make_map_2d(&m.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, a.act.h, in_dim, a.n_tokens, (uint64_t)a.act.dim_cap * 2, 64, N, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !make_map_2d(&m.bs, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, a.act.hs, in_dim / 16, a.n_tokens, a.act.dim_cap / 16 * 2, 64, N, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !make_map_2d(&m.xd, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, a.act.dt, a.n_tokens, nb, (uint64_t)a.act.dt_pitch * 4, N, nb, CU_TENSOR_MAP_SWIZZLE_NONE))
        return 0;
    uint32_t row_tiles = 0;
    for (int s = 0; s < 3; ++s) {
        const int used = std::min(s, a.n_seg - 1);
        k.seg[s] = a.seg[used];
        k.wide[s] = a.seg[used].wide->flags;
        const DevWeight &w = k.seg[s].w;
        if (!make_map_2d(&m.raw[s], CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, w.data, (uint64_t)nb * 144, w.out_dim, w.row_stride, 144, TC_M, CU_TENSOR_MAP_SWIZZLE_NONE)) return 0;
        if (s < a.n_seg) row_tiles += (w.out_dim + TC_M - 1) / TC_M;
        k.tiles[s] = row_tiles;
    }
    k.ones = F2_ONES;
    k.n_tokens = a.n_tokens;
    k.nb = nb;
    k.tok_tiles = (a.n_tokens + N - 1) / N;
    k.n_tiles = row_tiles * k.tok_tiles;
    // Wide rows first, in a kernel that lets this one start beside it: neither reads what the other writes, and both read what was complete
    // before the first of them started.
    uint32_t beside = 0;
    for (int s = 0; s < a.n_seg && !TWO; ++s) {
        if (!a.seg[s].wide->n) continue;
        if (!launch_gemm_few_rows(a, s, sm_count, st)) return 0;
        ++beside;
    }
    const uint32_t grid = std::min(k.n_tiles, (uint32_t)std::max(1, sm_count));
    if (beside) launch_pdl(gemm_tc5_q4k_kernel<GEMM, TWO, N>, grid, KQ_THREADS, P::bytes(nb, k.n_xd), st, m, k);
    else gemm_tc5_q4k_kernel<GEMM, TWO, N><<<grid, KQ_THREADS, P::bytes(nb, k.n_xd), st>>>(m, k);
    g_tc5_launched.store(true, std::memory_order_relaxed);
    return 1 + beside;
}

// How the product of Q4_K matrices is cut: tokens per tile, whether halves are kept apart, and about how long it takes.
struct KqChoice {
    uint32_t n = 0;
    bool two = false;
    double us = 1e30;
};
static KqChoice choose_q4k(const GemvArgs &a, int sm_count) {
    KqChoice best;
    // A few wide rows are computed apart; a matrix with one in 128 or more keeps all halves apart, which is slower for all of its rows.
    bool wide = false;
    for (int s = 0; s < a.n_seg; ++s) {
        const DevWeight &w = a.seg[s].w;
        wide = wide || a.seg[s].wide->n;
        best.two = best.two || a.seg[s].wide->n > (gemm_few_rows_supported(a) ? w.out_dim / 128 : 0u);
    }
    uint32_t rows = 0;
    for (int s = 0; s < a.n_seg; ++s) rows += (a.seg[s].w.out_dim + TC_M - 1) / TC_M;
    // Microseconds that a tile takes per super-block (4096 x 14336 and 14336 x 4096, 64 to 512 tokens).  Wider tiles lose their registers.
    struct Width {
        uint32_t n;
        double prefill, decode;  // 0: not built
    };
    for (const Width &w : {Width{96, 1.57, 0}, Width{64, 1.45, 0}, Width{48, 0, 0.95}, Width{32, 1.15, 0.88}, Width{16, 1.08, 0.83}}) {
        const double each = a.gemm_order ? w.prefill : w.decode;
        if (each == 0 || (best.two && w.n > (a.gemm_order ? 64u : 32u))) continue;
        const uint32_t nb = a.seg[0].w.nb, raw = (w.n > 64 ? 3u : 4u) * KQ_RAW_BYTES, b = (w.n > 64 ? 2u : 3u) * w.n * (a.gemm_order ? 512u : 640u);
        if (raw + b + nb * w.n * 4 + 2048 > 227 * 1024) continue;
        const uint32_t tiles = rows * ((a.n_tokens + w.n - 1) / w.n), waves = (tiles + sm_count - 1) / sm_count;
        // (with the quantizer, without wide rows, with a few, with halves apart: 4096 x 14336 with 64 tokens in prefill order 67.0, 66.3 and 74.1 us,
        // 37838 x 2304 39.1, 40.0 and 43.2; 32 tokens in decode order 26.8, 28.8 and 28.8)
        const double us = 4.0 + (wide ? 3.0 : 0.0) + (best.two ? 1.15 : 1.0) * waves * nb * each;
        if (us < best.us) best.us = us, best.n = w.n;
    }
    return best;
}
double gemm_tc5_q4k_us(const GemvArgs &a, int sm_count) { return choose_q4k(a, std::max(1, sm_count)).us; }

static uint32_t launch_q4k(const GemvArgs &a, int sm_count, cudaStream_t st) {
    if (!a.act.h) return 0;
    const KqChoice c = choose_q4k(a, std::max(1, sm_count));
    if (a.gemm_order && !c.two) {
        switch (c.n) {
        case 96: return launch_q4k_instance<true, false, 96>(a, sm_count, st);
        case 64: return launch_q4k_instance<true, false, 64>(a, sm_count, st);
        case 32: return launch_q4k_instance<true, false, 32>(a, sm_count, st);
        case 16: return launch_q4k_instance<true, false, 16>(a, sm_count, st);
        }
    } else if (a.gemm_order) {
        switch (c.n) {
        case 64: return launch_q4k_instance<true, true, 64>(a, sm_count, st);
        case 32: return launch_q4k_instance<true, true, 32>(a, sm_count, st);
        case 16: return launch_q4k_instance<true, true, 16>(a, sm_count, st);
        }
    } else if (!c.two) {
        switch (c.n) {
        case 48: return launch_q4k_instance<false, false, 48>(a, sm_count, st);
        case 32: return launch_q4k_instance<false, false, 32>(a, sm_count, st);
        case 16: return launch_q4k_instance<false, false, 16>(a, sm_count, st);
        }
    } else {
        switch (c.n) {
        case 32: return launch_q4k_instance<false, true, 32>(a, sm_count, st);
        case 16: return launch_q4k_instance<false, true, 16>(a, sm_count, st);
        }
    }
    return 0;  // a row too long for any tile
}

uint32_t launch_gemm_tc5(const GemvArgs &a, int sm_count, cudaStream_t st) {
    if (a.seg[0].w.type == TYPE_Q4_K) return launch_q4k(a, sm_count, st);
    static PerDeviceOnce once;
    if (once.run([] { return cudaFuncSetAttribute(gemm_tc5_q8_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Q8Smem::ALLOC); }) != cudaSuccess) return 0;
    const uint32_t in_dim = a.seg[0].w.in_dim;
    CUtensorMap tm_x, tm_xd;
    if (!make_map_2d(&tm_x, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a.act.q, in_dim, a.n_tokens, a.act.dim_cap, 128, TC_N, CU_TENSOR_MAP_SWIZZLE_128B)) return 0;
    if (!make_map_2d(&tm_xd, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, a.act.d, in_dim / 32, a.n_tokens, (uint64_t)(a.act.dim_cap / 32) * 4, 4, TC_N, CU_TENSOR_MAP_SWIZZLE_NONE))
        return 0;
    for (int s = 0; s < a.n_seg; ++s) {
        const GemvSegment &g = a.seg[s];
        CUtensorMap tm_w;
        if (!make_map_2d(&tm_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, g.w.data, in_dim, g.w.out_dim, g.w.row_stride, 128, TC_M, CU_TENSOR_MAP_SWIZZLE_128B)) return 0;
        TcQ8Args k{};
        k.seg = g;
        k.n_tokens = a.n_tokens;
        k.n_steps = in_dim / 128;
        const dim3 grid((g.w.out_dim + TC_M - 1) / TC_M, (a.n_tokens + TC_N - 1) / TC_N);
        gemm_tc5_q8_kernel<<<grid, TC_THREADS, Q8Smem::ALLOC, st>>>(tm_w, tm_x, tm_xd, k);
        g_tc5_launched.store(true, std::memory_order_relaxed);
    }
    return (uint32_t)a.n_seg;
}

int gemm_tc5_take_status() { return tc5_take_status(); }
void gemm_tc5_mark_launched() { g_tc5_launched.store(true, std::memory_order_relaxed); }

namespace {
// A barrier that nothing arrives at, waited for by every lane of a warp with a short limit of its own, then words through tensor memory, which
// takes all lanes together: *lanes counts the lanes that got theirs back, and the status word is what a product whose wait ran out leaves.
__global__ void __launch_bounds__(32) wait_selftest_kernel(uint32_t *lanes) {
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t abort, slot;
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&bar), 1);
        abort = 0u;
    }
    __syncwarp();
    tmem_alloc(smem_u32(&slot), 32);
    __syncwarp();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(&slot);
    for (uint32_t i = 0; i < 2; ++i) mbar_wait_on(smem_u32(&bar), 0u, &abort, 256 + threadIdx.x);
    uint32_t w[8], r[8];
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) w[i] = threadIdx.x * 8 + i;
    tmem_st8(tmem, w);
    tmem_st_wait();
    tmem_ld8(tmem, r);
    tmem_ld_wait();
    bool same = true;
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) same = same && r[i] == w[i];
    atomicAdd(lanes, same ? 1u : 0u);
    __syncwarp();
    tmem_dealloc(tmem, 32);
}
}  // namespace

void launch_tc5_wait_selftest(uint32_t *lanes, cudaStream_t st) { wait_selftest_kernel<<<1, 32, 0, st>>>(lanes); }

}  // namespace ob
