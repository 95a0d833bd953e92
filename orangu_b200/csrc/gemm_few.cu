// Products of K-quant matrices with a few tokens (decode batches, short portions) on mma.sync.
//
// A few tokens leave a product bound by reading the weights, so what counts is how many bytes are on their way.  A CTA takes tiles of 16
// rows x 8 NT tokens, and its eight warps split the super-blocks of the rows among them: every warp copies blocks into a ring of its own,
// some super-blocks ahead and across tiles, without a barrier.  The fp32 order forbids splitting a sum, not its terms: each warp leaves
// the fp32 terms of its super-blocks in shared memory and at a tile's end one thread per (row, token) adds them in block order, so the
// results are the single-token kernels' bit for bit.
//
// Q4_K: a 32-byte group holds two sub-blocks as low and high nibbles.  Lane t of a row's four takes bytes 8t .. 8t + 7 of it: its first
// word is the lane's share of k 0-15 of an m16n8k32 product, its second of k 16-31, and activations are read in the same order (a sum does
// not care which k is which).  Q6_K: sub-blocks of 16 elements, m16n8k16.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "pdl.cuh"

namespace ob {

namespace {

constexpr int FW_WARPS = 8, FW_ROWS = 16;

// c = a b (the accumulator goes in as zeros, which costs no registers)
__device__ __forceinline__ void mma_u8s8_k32(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ void mma_s8s8_k16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
                 : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
                 : "r"(a0), "r"(a1), "r"(b0), "r"(0));
}
__device__ __forceinline__ int dp2a_lo_su(uint32_t a, uint32_t b, int c) {  // c + a.lo16 * b.byte0 + a.hi16 * b.byte1 (a signed, b unsigned)
    int d;
    asm("dp2a.lo.s32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ int dp2a_hi_su(uint32_t a, uint32_t b, int c) {  // c + a.lo16 * b.byte2 + a.hi16 * b.byte3
    int d;
    asm("dp2a.hi.s32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ uint32_t word(const uint8_t *p) { return *reinterpret_cast<const uint32_t *>(p); }

// A stage of a warp's ring: blocks of 16 rows | activations of 8 NT tokens, 16-byte pieces exchanged by the token's number so that fragment
// reads meet no bank twice | (Q4_K) sums of 16 | token scales
template <uint32_t TYPE, int NT>
struct FewPlan {
    static constexpr uint32_t BLK = TYPE == TYPE_Q4_K ? 144 : 208, PIECES = BLK / 16, TOK = 8 * NT;
    static constexpr uint32_t X = FW_ROWS * BLK, S16 = X + TOK * 256, AD = S16 + (TYPE == TYPE_Q4_K ? TOK * 32 : 0), STAGE = AD + TOK * 4;
    static constexpr uint32_t STAGES = NT == 1 && TYPE == TYPE_Q4_K ? 3 : 2, RING = FW_WARPS * STAGES * STAGE;
    static constexpr uint32_t COPIES = (FW_ROWS * PIECES + 31) / 32;  // 16-byte copies of a lane per super-block
};

// GEMM: the prefill association; otherwise every (row, token) is the single-token product.  NT: n-tiles of 8 tokens.  rows: the numbers of
// the n_rows rows to compute (one matrix), or null for all.
template <uint32_t TYPE, bool GEMM, int NT>
__global__ void __launch_bounds__(FW_WARPS * 32, 2) gemm_few_kernel(const __grid_constant__ GemvArgs a, uint32_t row_tiles, uint32_t n_tiles, const uint32_t *rows, uint32_t n_rows) {
    using P = FewPlan<TYPE, NT>;
    constexpr uint32_t TOK = 8 * NT, PAIRS = FW_ROWS * TOK;
    constexpr bool TWO = GEMM && TYPE == TYPE_Q4_K;  // min terms apart
    extern __shared__ __align__(16) uint8_t smem[];
    float *terms = reinterpret_cast<float *>(smem + P::RING);  // [nb][row][token], then the min terms
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
    const uint32_t nb = a.seg[0].w.nb, last = a.n_tokens - 1;
    uint8_t *ring = smem + warp * P::STAGES * P::STAGE;

    // tile -> matrix and first row; a matrix's tiles for one group of tokens lie side by side
    auto locate = [&](uint32_t tile, uint32_t &row0, uint32_t &tok0) -> const GemvSegment & {
        uint32_t t = tile % row_tiles;
        tok0 = tile / row_tiles * TOK;
        int si = 0;
        while (si + 1 < a.n_seg && t >= (a.seg[si].w.out_dim + FW_ROWS - 1) / FW_ROWS) {
            t -= (a.seg[si].w.out_dim + FW_ROWS - 1) / FW_ROWS;
            ++si;
        }
        row0 = t * FW_ROWS;
        return a.seg[si];
    };
    pdl_release();  // (a product that leaves these rows out may start beside this one)
    auto row_of = [&](const DevWeight &w, uint32_t i) { return rows ? __ldg(rows + min(i, n_rows - 1)) : min(i, w.out_dim - 1); };
    // ---- the copies: where this warp's ring is being filled
    uint32_t c_tile = blockIdx.x, c_b = warp, c_stage = 0, c_tok0 = 0;
    const uint8_t *src[P::COPIES];
    const int8_t *x_src[4 * NT];  // two tokens a round
    const int16_t *s_src = nullptr;
    const float *d_src = nullptr;
    auto aim = [&] {
        if (c_tile >= n_tiles) return;
        uint32_t row0;
        const DevWeight &w = locate(c_tile, row0, c_tok0).w;
#pragma unroll
        for (uint32_t i = 0; i < P::COPIES; ++i) {
            const uint32_t c = min(32 * i + lane, FW_ROWS * P::PIECES - 1), r = c / P::PIECES;
            src[i] = w.data + (uint64_t)row_of(w, row0 + r) * w.row_stride + (c - r * P::PIECES) * 16;
        }
#pragma unroll
        for (uint32_t i = 0; i < 4 * NT; ++i) x_src[i] = a.act.q + (uint64_t)min(c_tok0 + 2 * i + (lane >> 4), last) * a.act.dim_cap + (lane & 15) * 16;
        s_src = a.act.sums + (uint64_t)min(c_tok0 + lane / 2, last) * (a.act.dim_cap / 16) + (lane & 1) * 8;  // (tokens 0-15: two pieces each)
        d_src = a.act.d + (uint64_t)min(c_tok0 + lane, last) * (a.act.dim_cap / 256);
    };
    auto cp16 = [](uint32_t dst, const void *from) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(from) : "memory"); };
    // (Places of tokens past the end hold anything: what comes of them is not stored.  Copies of the last token instead made 2 tokens slower
    // than 8, every CTA asking for the same lines seven times over.)
    auto copy = [&] {  // the next super-block of this warp, or an empty group
        if (c_tile < n_tiles && c_b < nb) {
            const uint32_t st = (uint32_t)__cvta_generic_to_shared(ring + c_stage * P::STAGE), dst = st + lane * 16;
#pragma unroll
            for (uint32_t i = 0; i < 4 * NT; ++i) {
                const uint32_t t = 2 * i + (lane >> 4), k = lane & 15;
                if (c_tok0 + t <= last) cp16(st + P::X + t * 256 + ((k ^ (t & 7u)) * 16), x_src[i] + c_b * 256);
            }
            if (TYPE == TYPE_Q4_K && lane < 2 * TOK && c_tok0 + lane / 2 <= last) cp16(st + P::S16 + lane * 16, s_src + c_b * 16);
            if (lane < TOK && c_tok0 + lane <= last) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(st + P::AD + lane * 4), "l"(d_src + c_b) : "memory");
#pragma unroll
            for (uint32_t i = 0; i < P::COPIES; ++i)
                if (32 * i + lane < FW_ROWS * P::PIECES) cp16(dst + i * 512, src[i] + (uint64_t)c_b * P::BLK);
            c_stage = c_stage + 1 == P::STAGES ? 0 : c_stage + 1;
            c_b += FW_WARPS;
            if (c_b >= nb) {
                c_b = warp;
                c_tile += gridDim.x;
                aim();
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if ((uint32_t)warp < nb) aim();
#pragma unroll
    for (uint32_t i = 0; i + 1 < P::STAGES; ++i) copy();

    uint32_t stage = 0;
    for (uint32_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    uint32_t row0, tok0;
    const GemvSegment &seg = locate(tile, row0, tok0);
    const DevWeight &w = seg.w;
    const uint8_t *d_row[2];  // Q6_K
#pragma unroll
    for (int r = 0; r < 2; ++r) d_row[r] = w.data + (uint64_t)row_of(w, row0 + gid + 8 * r) * w.row_stride + w.d_off;

    for (uint32_t b = warp; b < nb; b += FW_WARPS) {
        copy();
        int isum[NT][4];
#pragma unroll
        for (int n = 0; n < NT; ++n) isum[n][0] = isum[n][1] = isum[n][2] = isum[n][3] = 0;
        float *out = terms + (uint64_t)b * PAIRS;
        const uint8_t *base = ring + stage * P::STAGE, *blk[2] = {base + gid * P::BLK, base + (gid + 8) * P::BLK};
        // bytes e .. of the lane's token of a B fragment (within a 16-byte piece)
        auto x_at = [&](int n, uint32_t e) { return base + P::X + (8 * n + gid) * 256 + (((e >> 4) ^ gid) * 16) + (e & 15u); };
        stage = stage + 1 == P::STAGES ? 0 : stage + 1;

        asm volatile("cp.async.wait_group %0;" ::"n"(P::STAGES - 1) : "memory");  // this super-block's copies, every lane's
        __syncwarp();
        float2 ad[NT];  // the lane's two tokens of an accumulator
#pragma unroll
        for (int n = 0; n < NT; ++n) ad[n] = *reinterpret_cast<const float2 *>(base + P::AD + (8 * n + 2 * tig) * 4);
        if constexpr (TYPE == TYPE_Q4_K) {
            uint2 q[2][4];
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int g = 0; g < 4; ++g) q[r][g] = *reinterpret_cast<const uint2 *>(blk[r] + 16 + 32 * g + 8 * tig);
            uint32_t scw[2][2], mw[2][2];  // the eight 6-bit scales and mins (engine/quant.rs:653-662) as bytes
            float dd[2], dmin[2];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const uint4 hd = *reinterpret_cast<const uint4 *>(blk[r]);
                dd[r] = f16_bits_to_f32(hd.x & 0xffffu);
                dmin[r] = f16_bits_to_f32(hd.x >> 16);
                scw[r][0] = hd.y & 0x3f3f3f3fu;
                mw[r][0] = hd.z & 0x3f3f3f3fu;
                scw[r][1] = (hd.w & 0x0f0f0f0fu) | ((hd.y >> 2) & 0x30303030u);
                mw[r][1] = ((hd.w >> 4) & 0x0f0f0f0fu) | ((hd.z >> 2) & 0x30303030u);
            }
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                const uint32_t M = 0x0f0f0f0fu;
                const int g = s >> 1, sh = s & 1 ? 4 : 0;
                const uint32_t a0 = (q[0][g].x >> sh) & M, a1 = (q[1][g].x >> sh) & M, a2 = (q[0][g].y >> sh) & M, a3 = (q[1][g].y >> sh) & M;
                const int s0 = (int)__byte_perm(scw[0][s >> 2], 0, 0x4440 + (s & 3)), s1 = (int)__byte_perm(scw[1][s >> 2], 0, 0x4440 + (s & 3));
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    int c[4];
                    const uint2 x = *reinterpret_cast<const uint2 *>(x_at(n, 32 * s + 8 * tig));
                    mma_u8s8_k32(c, a0, a1, a2, a3, x.x, x.y);
                    isum[n][0] += s0 * c[0];
                    isum[n][1] += s0 * c[1];
                    isum[n][2] += s1 * c[2];
                    isum[n][3] += s1 * c[3];
                }
            }
            // mins against the sums of 16: each min twice
            uint32_t m2[2][4];
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int i = 0; i < 4; ++i) m2[r][i] = __byte_perm(mw[r][i >> 1], 0, i & 1 ? 0x3322 : 0x1100);
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                float t[2][2], tm[2][2];  // [row][token]
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const uint4 *sp = reinterpret_cast<const uint4 *>(base + P::S16 + (8 * n + 2 * tig + k) * 32), u = sp[0], v = sp[1];
                    const float adk = k ? ad[n].y : ad[n].x;
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        int im = dp2a_lo_su(u.x, m2[r][0], 0);
                        im = dp2a_hi_su(u.y, m2[r][0], im);
                        im = dp2a_lo_su(u.z, m2[r][1], im);
                        im = dp2a_hi_su(u.w, m2[r][1], im);
                        im = dp2a_lo_su(v.x, m2[r][2], im);
                        im = dp2a_hi_su(v.y, m2[r][2], im);
                        im = dp2a_lo_su(v.z, m2[r][3], im);
                        im = dp2a_hi_su(v.w, m2[r][3], im);
                        const float fi = (float)isum[n][2 * r + k], fm = (float)im;
                        if (GEMM) {
                            t[r][k] = __fmul_rn(adk, __fmul_rn(dd[r], fi));
                            tm[r][k] = __fmul_rn(__fmul_rn(adk, dmin[r]), fm);
                        } else {
                            t[r][k] = __fmul_rn(adk, __fsub_rn(__fmul_rn(dd[r], fi), __fmul_rn(dmin[r], fm)));
                        }
                    }
                }
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const uint32_t at = (gid + 8 * r) * TOK + 8 * n + 2 * tig;
                    *reinterpret_cast<float2 *>(out + at) = make_float2(t[r][0], t[r][1]);
                    if (TWO) *reinterpret_cast<float2 *>(out + (uint64_t)nb * PAIRS + at) = make_float2(tm[r][0], tm[r][1]);
                }
            }
        } else {
            uint32_t d[2];
#pragma unroll
            for (int r = 0; r < 2; ++r) d[r] = __ldg(reinterpret_cast<const uint16_t *>(d_row[r] + 2 * b));
            const uint4 sc[2] = {*reinterpret_cast<const uint4 *>(blk[0] + 192), *reinterpret_cast<const uint4 *>(blk[1] + 192)};
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int is = 0; is < 2; ++is) {
                    uint32_t v[2][4];
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const uint8_t *at = blk[r] + 16 * is + 4 * tig;
                        const uint32_t qa = word(at + 64 * h), qb = word(at + 64 * h + 32), qh = word(at + 128 + 32 * h);
                        v[r][0] = __vsub4((qa & 0x0f0f0f0fu) | ((qh << 4) & 0x30303030u), 0x20202020u);  // q - 32 as signed bytes
                        v[r][1] = __vsub4((qb & 0x0f0f0f0fu) | ((qh << 2) & 0x30303030u), 0x20202020u);
                        v[r][2] = __vsub4(((qa >> 4) & 0x0f0f0f0fu) | (qh & 0x30303030u), 0x20202020u);
                        v[r][3] = __vsub4(((qb >> 4) & 0x0f0f0f0fu) | ((qh >> 2) & 0x30303030u), 0x20202020u);
                    }
#pragma unroll
                    for (int run = 0; run < 4; ++run) {
                        const int sidx = 8 * h + 2 * run + is;  // scale of elements 128 h + 32 run + 16 is ..
                        const uint32_t w0 = reinterpret_cast<const uint32_t *>(&sc[0])[sidx >> 2], w1 = reinterpret_cast<const uint32_t *>(&sc[1])[sidx >> 2];
                        const int s0 = (int)(int8_t)((w0 >> (8 * (sidx & 3))) & 0xff), s1 = (int)(int8_t)((w1 >> (8 * (sidx & 3))) & 0xff);
#pragma unroll
                        for (int n = 0; n < NT; ++n) {
                            int c[4];
                            mma_s8s8_k16(c, v[0][run], v[1][run], word(x_at(n, 128 * h + 32 * run + 16 * is + 4 * tig)));
                            isum[n][0] += s0 * c[0];
                            isum[n][1] += s0 * c[1];
                            isum[n][2] += s1 * c[2];
                            isum[n][3] += s1 * c[3];
                        }
                    }
                }
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const float dw = f16_bits_to_f32(d[r]);
                    float t[2];
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const float fi = (float)isum[n][2 * r + k], adk = k ? ad[n].y : ad[n].x;
                        t[k] = GEMM ? __fmul_rn(adk, __fmul_rn(dw, fi)) : __fmul_rn(__fmul_rn(adk, dw), fi);
                    }
                    *reinterpret_cast<float2 *>(out + (gid + 8 * r) * TOK + 8 * n + 2 * tig) = make_float2(t[0], t[1]);
                }
        }
        __syncwarp();  // the next copy goes into the stage that was read first
    }
    __syncthreads();

    // block order, one thread per (row, token)
    for (uint32_t i = threadIdx.x; i < PAIRS; i += FW_WARPS * 32) {
        const uint32_t r = row0 + i / TOK, t = tok0 + i % TOK;
        float total = 0.0f;
        if (TWO) {
            const float *tm = terms + (uint64_t)nb * PAIRS + i;
#pragma unroll 8
            for (uint32_t b = 0; b < nb; ++b) total = __fsub_rn(total, tm[(uint64_t)b * PAIRS]);
        }
#pragma unroll 8
        for (uint32_t b = 0; b < nb; ++b) total = __fadd_rn(total, terms[(uint64_t)b * PAIRS + i]);
        if (r < (rows ? n_rows : w.out_dim) && t < a.n_tokens) {
            const uint64_t o = (uint64_t)t * seg.y_stride + row_of(w, r);
            seg.y[o] = seg.epilogue == EPI_ADD_RESIDUAL ? __fadd_rn(seg.residual[o], total) : total;
        }
    }
    __syncthreads();
    }
}

size_t few_smem(uint32_t type, uint32_t nb, bool gemm, int nt) {
    const uint32_t ring = type == TYPE_Q4_K ? (nt == 1 ? FewPlan<TYPE_Q4_K, 1>::RING : FewPlan<TYPE_Q4_K, 2>::RING) : nt == 1 ? FewPlan<TYPE_Q6_K, 1>::RING : FewPlan<TYPE_Q6_K, 2>::RING;
    return ring + (size_t)nb * FW_ROWS * 8 * nt * 4 * (gemm && type == TYPE_Q4_K ? 2 : 1);
}

// n-tiles of a CTA: 16 tokens where there are more than 8 and the terms of a tile fit beside its ring, else 8
int few_n_tiles(const GemvArgs &a) { return a.n_tokens > 8 && few_smem(a.seg[0].w.type, a.seg[0].w.nb, a.gemm_order, 2) <= 226 * 1024 ? 2 : 1; }

template <uint32_t TYPE, bool GEMM, int NT>
bool launch_few(const GemvArgs &a, int sm_count, cudaStream_t st, const uint32_t *rows = nullptr, uint32_t n_rows = 0) {
    static PerDeviceOnce once;
    if (once.run([] { return cudaFuncSetAttribute(gemm_few_kernel<TYPE, GEMM, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024); }) != cudaSuccess) return false;
    uint32_t tiles = 0;
    for (int s = 0; s < a.n_seg; ++s) tiles += ((rows ? n_rows : a.seg[s].w.out_dim) + FW_ROWS - 1) / FW_ROWS;
    const size_t smem = few_smem(TYPE, a.seg[0].w.nb, GEMM, NT);
    const uint32_t all = tiles * ((a.n_tokens + 8 * NT - 1) / (8 * NT)), slots = (2 * smem <= 226 * 1024 ? 2u : 1u) * (uint32_t)std::max(1, sm_count);
    gemm_few_kernel<TYPE, GEMM, NT><<<std::min(all, slots), FW_WARPS * 32, smem, st>>>(a, tiles, all, rows, n_rows);
    return true;
}
template <uint32_t TYPE, bool GEMM>
bool launch_few_nt(const GemvArgs &a, int nt, int sm_count, cudaStream_t st) {
    return nt == 1 ? launch_few<TYPE, GEMM, 1>(a, sm_count, st) : launch_few<TYPE, GEMM, 2>(a, sm_count, st);
}

}  // namespace

bool gemm_few_supported(const GemvArgs &a) {
    if (a.n_seg < 1 || a.n_tokens < 2 || a.isum_out) return false;
    const uint32_t type = a.seg[0].w.type;
    if ((type != TYPE_Q4_K && type != TYPE_Q6_K) || few_smem(type, a.seg[0].w.nb, a.gemm_order, 1) > 226 * 1024) return false;
    for (int s = 0; s < a.n_seg; ++s)
        if (a.seg[s].w.type != type || a.seg[s].w.in_dim != a.seg[0].w.in_dim || (a.seg[s].w.row_stride & 15)) return false;
    return true;
}

bool launch_gemm_few(const GemvArgs &a, int sm_count, cudaStream_t st) {
    const uint32_t type = a.seg[0].w.type;
    const int nt = few_n_tiles(a);
    if (type == TYPE_Q4_K) return a.gemm_order ? launch_few_nt<TYPE_Q4_K, true>(a, nt, sm_count, st) : launch_few_nt<TYPE_Q4_K, false>(a, nt, sm_count, st);
    return a.gemm_order ? launch_few_nt<TYPE_Q6_K, true>(a, nt, sm_count, st) : launch_few_nt<TYPE_Q6_K, false>(a, nt, sm_count, st);
}

// Microseconds: a tile's super-block costs 1.05e-3 with 8 tokens and 1.3e-3 with 16 (4096 x 14336, 8 tokens: 18 us; 14336 x 4096, 16: 24).
// Rows whose terms allow 8 tokens only are twice the tiles (4096 x 28672, 48 tokens, prefill order: 151 us, the tcgen05 tiles 133).
double gemm_few_us(const GemvArgs &a) {
    const uint32_t nt = few_n_tiles(a);
    double tiles = 0;
    for (int s = 0; s < a.n_seg; ++s) tiles += (a.seg[s].w.out_dim + FW_ROWS - 1) / FW_ROWS;
    return 5.0 + tiles * ((a.n_tokens + 8 * nt - 1) / (8 * nt)) * a.seg[0].w.nb * (nt == 1 ? 1.05e-3 : 1.3e-3);
}

bool gemm_few_rows_supported(const GemvArgs &a) { return few_smem(TYPE_Q4_K, a.seg[0].w.nb, a.gemm_order, 1) <= 226 * 1024; }

bool launch_gemm_few_rows(const GemvArgs &a, int segment, int sm_count, cudaStream_t st) {
    GemvArgs one = a;
    one.n_seg = 1;
    one.seg[0] = a.seg[segment];
    const WideRows &wide = *one.seg[0].wide;
    const bool two = few_smem(TYPE_Q4_K, one.seg[0].w.nb, a.gemm_order, 2) <= 226 * 1024;
    if (a.gemm_order) return two ? launch_few<TYPE_Q4_K, true, 2>(one, sm_count, st, wide.rows, wide.n) : launch_few<TYPE_Q4_K, true, 1>(one, sm_count, st, wide.rows, wide.n);
    return two ? launch_few<TYPE_Q4_K, false, 2>(one, sm_count, st, wide.rows, wide.n) : launch_few<TYPE_Q4_K, false, 1>(one, sm_count, st, wide.rows, wide.n);
}

}  // namespace ob
