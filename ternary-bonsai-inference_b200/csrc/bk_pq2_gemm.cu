// PQ2_0 ternary rows times a block of activations (prompt or speculative tokens) on the 5th-generation
// tensor cores: y[t][r] = sum_j x[t][j] * W[base_row + r][j] for n_tok tokens at once
// (src/kernels.rs:333-420 `pq2_matmul_n`; row format src/kernels.rs:204-229).  bk_pq2.cu is the form for
// one or two tokens, where the weight stream is the cost and every launch reads it once per pair of tokens.
//
// What bounds it: with hundreds of tokens the multiply-adds, 2 tensor-core terms each; with a few tokens the
// unpacking of the weights.  The layout follows from three numbers:
//   * Weights are the A operand, IN TENSOR MEMORY: M = 128 rows, a thread's tensor-memory lane is a row, so
//     unpacking is register work (a mask and an f16 FMA give two weights -1, 0, 1, 2) and a tcgen05.st; no shared-memory pass, and the MMA reads only B from shared memory.
//   * Activations are the B operand, as f16 hi + mid parts of x scaled by a power of two per token (at least
//     22 bits of every element, and 2^-40 of the token's largest one as the floor, so no less than the
//     25-bit fixed point per block of the one-token form gives: its grid is 2^-24 of a block's largest element).
//     A first kernel writes them once, already permuted (the order of the K slots is free and is chosen so that the
//     unpacking needs no shuffles) and swizzled, one contiguous piece per (token tile, block of 128): the
//     main kernel fetches a block with ONE bulk copy.
//   * The block scale is the row's, so the accumulator is drained after every block of 128 and added up in f32 as
//     scale * block sum, grouped as the reference's scalar path does it (src/kernels.rs:633-650); the tensor
//     core never accumulates more than 16 MMAs, which keeps its truncating f32 adds from building up a bias.
//     Two D buffers alternate: the drain of one step runs under the MMAs of the next.
// Measured (q, k, v and output projection of a layer, 14336 x 5120 and 5120 x 6144): 512 tokens 290 us = 370
// TFLOP/s of useful work (two passes of it on the tensor cores), 5760 us as pairs of tokens; 5 tokens 58 us against 64
// (where the line lies: 4 tokens as pairs take 46), 16 tokens 59 against 180, 128 tokens 129 against 1440.  Rounding against float64: 1.0e-7 of the result's 2-norm, as one token at a time (with x20 outliers in x 1.0e-7 against
// 2.6e-7); 1.4e-7, and 240 us, with one running sum over all blocks.
// A step is (row tile of 128, block of 128); a CTA works on one or two row tiles (two share every B block: 32
// instead of 64 bytes per clock and SM from L2, which is what the L2 delivers) and one token tile of 16..128.
// The sum over blocks takes the same order and groups whatever the tiling, so a result does not depend on it bit for bit.
#include <algorithm>
#include <atomic>
#include <cuda_fp16.h>

#include "bk_device.cuh"
#include "bk_internal.h"
#include "bk_mma_common.cuh"
#include "bk_umma.cuh"

namespace bk {

namespace {

constexpr int kGemmThreads = 320;                 // 8 warps that unpack and drain, one that issues MMAs, one that loads B
constexpr int kGemmBlock = 128, kGemmBlockBytes = 34;
constexpr int kGemmSegBlocks = 4;                 // blocks of a row staged together
constexpr int kGemmRowWords = 36;                 // words of a staged row: nine 16-byte pieces hold any four blocks of an aligned row
constexpr int kGemmMaxSegs = 4;
constexpr int kGemmGroup = 8;                     // blocks that are added up before their sum goes to y
constexpr uint32_t kColsD = 128, kColA = 256, kColsA = 64;  // tensor-memory columns: D0 | D1 | four A stages

struct GemmArgs {
    const uint8_t *rows[kGemmMaxSegs];
    float *y[kGemmMaxSegs];
    int seg_rows[kGemmMaxSegs], seg_tile0[kGemmMaxSegs + 1];
    const uint8_t *xb;        // [token tile][block][hi|mid][2 slabs of 64 slots][n][128 B, swizzled]
    const float *tok_scale;   // [token tile * n]: what a token's sums are multiplied by
    int nb, row_bytes, n_tok, n_stages_b;
    int vec;                  // bit s: the rows of range s all start on 16-byte boundaries
    int *err_flag;
};

// x -> scaled hi and mid parts in the order and swizzle of the B operand.  One CTA per (padded) token.
// Slot k = 16 i + 2 p + h of a block holds weight 16 i + p + 8 h (see unpack16()), so the eight slots of a
// 16-byte chunk are four consecutive elements and the four that lie eight further on, alternating.
__global__ void __launch_bounds__(256) pq2_split_x_kernel(const float *x, int ne0, int nb, int n_tok, int n, uint8_t *xb, float *tok_scale) {
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    __shared__ float wmax[8];
    const int tok = blockIdx.x, tile = tok / n, r = tok - tile * n, tid = threadIdx.x;
    const float *xr = x + (size_t)tok * ne0;
    const bool real = tok < n_tok;
    const bool vec = (ne0 & 3) == 0 && ((uintptr_t)x & 15) == 0;
    const int chunks = nb * 16;
    auto load = [&](int c, float (&v)[8]) {
        const int j = (c >> 1) * 16 + (c & 1) * 4;  // and j + 8
        if (real && vec && j + 12 <= ne0) {
            const float4 a = __ldg(reinterpret_cast<const float4 *>(xr + j)), b = __ldg(reinterpret_cast<const float4 *>(xr + j + 8));
            v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
        } else {
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = (real && j + i + (i & 4) < ne0) ? xr[j + i + (i & 4)] : 0.f;
        }
    };
    float v[8], am = 0.f;
    for (int c = tid; c < chunks; c += 256) {
        load(c, v);
#pragma unroll
        for (int i = 0; i < 8; i++) am = fmaxf(am, fabsf(v[i]));
    }
    for (int o = 16; o > 0; o >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
    if ((tid & 31) == 0) wmax[tid >> 5] = am;
    __syncthreads();
    am = wmax[0];
#pragma unroll
    for (int i = 1; i < 8; i++) am = fmaxf(am, wmax[i]);
    int e = 0;
    if (am > 0.f && am < INFINITY) frexpf(am, &e);  // am = f * 2^e, f in [0.5, 1)
    const int up = max(-126, min(15 - e, 127));     // the largest element lands in [2^14, 2^15)
    const float s = ldexpf(1.0f, up);
    if (tid == 0) tok_scale[tok] = ldexpf(1.0f, -up);
    for (int c = tid; c < chunks; c += 256) {
        load(c, v);
        uint32_t hi[4], mid[4];
#pragma unroll
        for (int p = 0; p < 4; p++) {
            const float a = v[p] * s, b = v[p + 4] * s;
            const __half ha = __float2half_rn(a), hb = __float2half_rn(b);
            const __half2 h2 = __halves2half2(ha, hb);
            const __half2 m2 = __halves2half2(__float2half_rn(a - __half2float(ha)), __float2half_rn(b - __half2float(hb)));
            hi[p] = *reinterpret_cast<const uint32_t *>(&h2);
            mid[p] = *reinterpret_cast<const uint32_t *>(&m2);
        }
        const int blk = c >> 4, slab = (c >> 3) & 1, ch = c & 7;
        uint8_t *dst = xb + ((size_t)tile * nb + blk) * (size_t)n * 512 + (size_t)slab * n * 128 + (size_t)r * 128 + ((ch ^ (r & 7)) << 4);
        *reinterpret_cast<uint4 *>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4 *>(dst + (size_t)n * 256) = make_uint4(mid[0], mid[1], mid[2], mid[3]);
    }
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t *r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}

// Sixteen 2-bit codes -> eight registers of two f16 weights (code - 1): register p = codes p and p + 8.  A code that
// is masked where it lies and put under the exponent of 1024 is the f16 number 1024 + 4^i code; one f16 FMA brings
// it to code - 1 exactly.  (Nine integer operations for sixteen weights; shift, mask and byte permute took 23 and, at half
// the issue rate of the FMA pipe, were most of a step.)
__device__ __forceinline__ void unpack16(uint32_t w, uint32_t *out) {
    const uint32_t w2 = w >> 10;
#pragma unroll
    for (int p = 0; p < 8; p++) {
        const int i = p < 5 ? p : p - 5;
        const uint32_t u = ((p < 5 ? w : w2) & (0x00030003u << (2 * i))) | 0x64006400u;
        const float f = 1.0f / (float)(1 << (2 * i));
        const __half2 r = __hfma2(*reinterpret_cast<const __half2 *>(&u), __float2half2_rn(f), __float2half2_rn(-(1024.0f * f + 1.0f)));
        out[p] = *reinterpret_cast<const uint32_t *>(&r);
    }
}

// MT row tiles per CTA, N = 16 NC tokens.
template <int MT, int NC>
__global__ void __launch_bounds__(kGemmThreads, 1) pq2_gemm_kernel(const GemmArgs a) {
    extern __shared__ __align__(1024) uint8_t sm[];
    constexpr int N = 16 * NC, NH = 8 * NC;  // tokens of the tile, and of one warpgroup
    constexpr uint32_t kBlockB = (uint32_t)N * 512u;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(sm);
    // barriers: B full [4] | B free [4] | A full [4] | D full [2] | D free [2]; then the tensor-memory address and a give-up flag
    const uint32_t bar_bf = sbase, bar_be = sbase + 32, bar_af = sbase + 64, bar_df = sbase + 96, bar_de = sbase + 112, slot = sbase + 128;
    volatile int *gave_up = reinterpret_cast<volatile int *>(sm + 132);
    const int nst = a.n_stages_b, nb = a.nb, n_steps = nb * MT;
    const uint32_t off_b = 1024u, off_w = off_b + (uint32_t)nst * kBlockB;

    if (tid == 0) {
        for (int i = 0; i < 4; i++) {
            mbar_init(bar_bf + 8 * i, 1);
            mbar_init(bar_be + 8 * i, 1);
            mbar_init(bar_af + 8 * i, 8);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(bar_df + 8 * i, 1);
            mbar_init(bar_de + 8 * i, 8);
        }
        *gave_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 8) tmem_alloc(slot, 512);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t *>(sm + 128), 0);

    // bounded wait; after one has run out (never expected) the others of the CTA do not start to wait
    auto wait = [&](uint32_t bar, uint32_t parity) -> bool {
        int polls = 0;
        while (!mbar_try_wait(bar, parity)) {
            if (*gave_up) return false;
            if (++polls > kWaitPolls) {
                *gave_up = 1;
                raise_error(a.err_flag, 5);
                return false;
            }
        }
        return true;
    };

    const int row_tile = blockIdx.x, tok_tile = blockIdx.y;
    int sg = 0;
#pragma unroll
    for (int i = 1; i < kGemmMaxSegs; i++) sg += (row_tile >= a.seg_tile0[i]) ? 1 : 0;
    const int row0 = (row_tile - a.seg_tile0[sg]) * (128 * MT), seg_rows = a.seg_rows[sg];
    const uint8_t *wrows = a.rows[sg];

    if (warp == 9) {
        // B blocks, in order through the ring of stages
        const uint8_t *xb = a.xb + (size_t)tok_tile * nb * kBlockB;
        asm volatile("griddepcontrol.wait;\n" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
        int b = 0;
        for (uint32_t st = 0, use = 0; b < nb; b++) {
            if (use > 0 && !wait(bar_be + 8 * st, (use - 1) & 1u)) break;
            if (elect_one()) {
                mbar_expect_tx(bar_bf + 8 * st, kBlockB);
                tma_bulk(sbase + off_b + st * kBlockB, xb + (size_t)b * kBlockB, kBlockB, bar_bf + 8 * st);
            }
            __syncwarp();
            if (++st == (uint32_t)nst) st = 0, use++;
        }
        for (int c = max(0, b - nst); c < b && b < nb; c++) {  // gave up: leave no copy in flight behind
            int polls = 0;
            while (!mbar_try_wait(bar_bf + 8 * (c % nst), (uint32_t)(c / nst) & 1u) && ++polls < kWaitPolls) {}
        }
    } else if (warp == 8) {
        const uint32_t idesc = umma_idesc_f16(128, N, 0, 0);
        uint32_t st = 0, b_par = 0;
        for (int s = 0; s < n_steps; s++) {
            bool ok = true;
            if (s % MT == 0) ok = wait(bar_bf + 8 * st, b_par);
            ok = ok && wait(bar_af + 8 * (s & 3), (uint32_t)(s >> 2) & 1u);
            if (s >= 2) ok = ok && wait(bar_de + 8 * (s & 1), (uint32_t)((s >> 1) - 1) & 1u);
            if (!__all_sync(0xffffffffu, ok)) break;
            tc_fence_after_sync();
            const uint32_t d = tmem + (s & 1) * kColsD, am = tmem + kColA + (s & 3) * kColsA;
            const uint64_t bd = umma_smem_desc(sbase + off_b + st * kBlockB, 16, 1024, kUmmaSwizzle128);
            if (elect_one()) {
#pragma unroll
                for (int term = 1; term >= 0; term--)  // the small parts first
#pragma unroll
                    for (int k = 0; k < 8; k++)  // (the address field of a descriptor counts 16-byte units)
                        umma_f16_ts(d, am + 8 * k, bd + (uint64_t)((term * (N * 256) + (k >> 2) * (N * 128) + (k & 3) * 32) >> 4), idesc,
                                    !(term == 1 && k == 0));
                umma_commit(bar_df + 8 * (s & 1));
                if (s % MT == MT - 1) umma_commit(bar_be + 8 * st);
            }
            __syncwarp();
            if (s % MT == MT - 1 && ++st == (uint32_t)nst) st = 0, b_par ^= 1u;
        }
    } else {
        const int quad = warp & 3, half = warp >> 2, r = quad * 32 + lane;  // tensor-memory lane = row of the tile
        uint32_t *wst = reinterpret_cast<uint32_t *>(sm + off_w);           // [2][MT * 128][kGemmRowWords]
        const int n_seg = (nb + kGemmSegBlocks - 1) / kGemmSegBlocks;
        // The two warps of a quadrant stage its 32 rows.  Rows on 16-byte boundaries (their length is then a multiple of
        // eight blocks): the nine 16-byte pieces around four blocks, which start at the segment's first byte or, every other
        // segment, 8 bytes before it.  Other rows: the words that overlap the blocks.
        const bool vec = (a.vec >> sg) & 1;
        const int t64 = half * 32 + lane;
        uint32_t src[5];
#pragma unroll
        for (int i = 0; i < 5; i++) {
            const int idx = t64 + 64 * i, rr = idx / 9;
            src[i] = (uint32_t)rr * a.row_bytes + (uint32_t)(idx - rr * 9) * 16u;
        }
        auto stage_w = [&](int k) {
            const int blocks = min(kGemmSegBlocks, nb - k * kGemmSegBlocks), bytes = blocks * kGemmBlockBytes;
#pragma unroll
            for (int m = 0; m < MT; m++) {
                const int rb = m * 128 + quad * 32;
                const uint32_t dst = sbase + off_w + (uint32_t)(((k & 1) * MT * 128 + rb) * kGemmRowWords) * 4u;
                const uint8_t *p0 = wrows + (size_t)(row0 + rb) * a.row_bytes + (size_t)k * (kGemmSegBlocks * kGemmBlockBytes);
                const int rows = min(32, seg_rows - row0 - rb);
                if (vec) {
                    p0 -= (k & 1) * 8;
#pragma unroll
                    for (int i = 0; i < 5; i++)
                        if (t64 + 64 * i < rows * 9)
                            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + (uint32_t)(t64 + 64 * i) * 16u), "l"(p0 + src[i]) : "memory");
                } else {
                    for (int rr = half; rr < rows; rr += 2) {
                        const uint8_t *p = p0 + (size_t)rr * a.row_bytes;
                        const uint32_t sh = (uint32_t)((uintptr_t)p & 2u);
                        for (int wd = lane; wd * 4 < (int)sh + bytes; wd += 32)
                            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst + (uint32_t)(rr * kGemmRowWords + wd) * 4u), "l"(p - sh + 4 * wd)
                                         : "memory");
                    }
                }
            }
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        };
        auto quad_sync = [&]() { asm volatile("bar.sync %0, 64;\n" ::"r"(1 + quad) : "memory"); };
        stage_w(0);

        float acc[MT][NH];
#pragma unroll
        for (int m = 0; m < MT; m++)
#pragma unroll
            for (int j = 0; j < NH; j++) acc[m][j] = 0.f;
        const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16);
        // where a segment starts in the staged row, in bytes: see stage_w (rows start on even addresses; a row's
        // misalignment is the same in every segment, 136 bytes on)
        uint32_t row_sh[MT];
#pragma unroll
        for (int m = 0; m < MT; m++) row_sh[m] = vec ? 0u : (uint32_t)((uintptr_t)(wrows + (size_t)(row0 + m * 128 + r) * a.row_bytes) & 2u);

        // this warp's half of block b of the thread's rows, from the staged words, and the block scales
        uint32_t w[MT][4];
        float sc0[MT];
        auto fetch = [&](int b) {
            const int k = b / kGemmSegBlocks;
            if (b % kGemmSegBlocks == 0) {
                asm volatile("cp.async.wait_group 0;\n" ::: "memory");
                quad_sync();  // both warps' pieces are in, and both have left the segment before
                if (k + 1 < n_seg) stage_w(k + 1);
            }
#pragma unroll
            for (int m = 0; m < MT; m++) {
                const uint32_t *row = wst + (size_t)((k & 1) * MT * 128 + m * 128 + r) * kGemmRowWords;
                const uint32_t byte = (vec ? (uint32_t)(k & 1) * 8u : row_sh[m]) + (uint32_t)(b - k * kGemmSegBlocks) * kGemmBlockBytes;
                sc0[m] = __half2float(__ushort_as_half(*reinterpret_cast<const unsigned short *>(reinterpret_cast<const uint8_t *>(row) + byte)));
                const uint32_t cb = byte + 2u + (uint32_t)half * 16u, cs = (cb & 2u) * 8u;
                const uint32_t *cw = row + (cb >> 2);
                uint32_t v[5];
#pragma unroll
                for (int i = 0; i < 4; i++) v[i] = cw[i];
                v[4] = cs ? cw[4] : 0u;
#pragma unroll
                for (int i = 0; i < 4; i++) w[m][i] = __funnelshift_r(v[i], v[i + 1], cs);
            }
        };
        // ... unpacked into the A stage of step s
        auto unpack = [&](int s, int m) {
            uint32_t regs[32];
#pragma unroll
            for (int i = 0; i < 4; i++) unpack16(w[m][i], regs + 8 * i);
            tmem_st32(lane_base + kColA + (uint32_t)(s & 3) * kColsA + (uint32_t)half * 32u, regs);
            tmem_wait_st();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_af + 8 * (s & 3));
        };
        bool ok = true;
        auto drain = [&](int s, float (&ac)[NH], float sc) {
            ok = ok && wait(bar_df + 8 * (s & 1), (uint32_t)(s >> 1) & 1u);
            __syncwarp();
            tc_fence_after_sync();
            const uint32_t d = lane_base + (uint32_t)(s & 1) * kColsD + (uint32_t)half * NH;
#pragma unroll
            for (int c0 = 0; c0 < NC; c0 += 4) {
                uint32_t v[32];
#pragma unroll
                for (int c = 0; c < 4; c++)
                    if (c0 + c < NC) tmem_ld8(d + 8u * (c0 + c), v + 8 * c);
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                if (c0 + 4 >= NC) {
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_de + 8 * (s & 1));
                }
#pragma unroll
                for (int c = 0; c < 4; c++)
                    if (c0 + c < NC)
#pragma unroll
                        for (int j = 0; j < 8; j++) ac[(c0 + c) * 8 + j] = fmaf(sc, __uint_as_float(v[8 * c + j]), ac[(c0 + c) * 8 + j]);
            }
        };
        // The sums so far join y and start again at zero: one running f32 sum over all blocks rounds at the size of the whole
        // result forty times (1.4e-7 of the 2-norm against 1.0e-7).  Eight elements at a time are read back, which are the registers
        // there are; an element belongs to one thread.  (red.add instead of the read was slower: 28 clocks a warp.)
        // kLag iterations on, a group's last block is drained; a rest of fewer than three blocks joins the last group, with either MT.
        constexpr int kLag = MT == 1 ? 2 : 1;
        int next_flush = kGemmGroup + kLag;
        bool first = true;
        auto flush = [&](int b) {
            if (first) asm volatile("griddepcontrol.wait;\n" ::: "memory");  // what came before on the stream may still read y until here
            const int t0 = tok_tile * N + half * NH, left = a.n_tok - t0;
#pragma unroll
            for (int m = 0; m < MT; m++) {
                const int row = row0 + m * 128 + r;
                if (row < seg_rows) {
                    float *yp = a.y[sg] + (size_t)t0 * seg_rows + row;
#pragma unroll
                    for (int j0 = 0; j0 < NH; j0 += 8) {
                        float old[8];
#pragma unroll
                        for (int j = 0; j < 8; j++) old[j] = (!first && j0 + j < left) ? __ldcg(yp + (size_t)(j0 + j) * seg_rows) : 0.f;
#pragma unroll
                        for (int j = 0; j < 8; j++)  // (the scale is a power of two)
                            if (j0 + j < left) __stcg(yp + (size_t)(j0 + j) * seg_rows, fmaf(acc[m][j0 + j], __ldg(a.tok_scale + t0 + j0 + j), old[j]));
                    }
                }
#pragma unroll
                for (int j = 0; j < NH; j++) acc[m][j] = 0.f;
            }
            first = false;
            next_flush = b + kGemmGroup;
        };
        // one iteration per block: unpack the block's steps, drain the steps of two steps ago.  An A stage is reused
        // four steps on, after the drain of its step, which waited for its MMAs.
        float sc1[MT] = {}, sc2 = 0.f;  // block scales of the steps that are unpacked and not yet drained
        fetch(0);
        for (int b = 0; b < nb; b++) {
            if (b == next_flush && b - kLag + 3 <= nb) flush(b);
            float now[MT];
#pragma unroll
            for (int m = 0; m < MT; m++) now[m] = sc0[m];
            unpack(MT * b, 0);
            if constexpr (MT == 2) {
                if (b > 0) drain(2 * b - 2, acc[0], sc1[0]);
                unpack(2 * b + 1, 1);
                if (b + 1 < nb) fetch(b + 1);
                if (b > 0) drain(2 * b - 1, acc[1], sc1[1]);
                sc1[1] = now[1];
            } else {
                if (b + 1 < nb) fetch(b + 1);
                if (b > 1) drain(b - 2, acc[0], sc2);
                sc2 = sc1[0];
            }
            sc1[0] = now[0];
        }
        if constexpr (MT == 2) {
            drain(2 * nb - 2, acc[0], sc1[0]);
            drain(2 * nb - 1, acc[1], sc1[1]);
        } else {
            if (nb > 1) drain(nb - 2, acc[0], sc2);
            drain(nb - 1, acc[0], sc1[0]);
        }
        flush(nb);
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 8) tmem_dealloc(tmem, 512);
}

template <int MT, int NC>
bk_status launch_gemm(bk_ctx *ctx, const GemmArgs &a, dim3 grid, size_t smem) {
    static std::atomic<bool> opted_in[64] = {};
    const int dev = ctx->device;
    if (dev < 0 || dev >= 64) return fail(ctx, BK_ERR_UNSUPPORTED, "pq2 matmul: device index above 63");
    if (!opted_in[dev].load()) {
        BK_CUDA(ctx, cudaFuncSetAttribute(pq2_gemm_kernel<MT, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
        opted_in[dev].store(true);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    BK_CUDA(ctx, cudaLaunchKernelEx(&cfg, pq2_gemm_kernel<MT, NC>, a));
    ctx->launches++;
    BK_CUDA(ctx, cudaGetLastError());
    return BK_OK;
}

template <int MT>
bk_status launch_gemm_nc(bk_ctx *ctx, int nc, const GemmArgs &a, dim3 grid, size_t smem) {
    switch (nc) {
        case 1: return launch_gemm<MT, 1>(ctx, a, grid, smem);
        case 2: return launch_gemm<MT, 2>(ctx, a, grid, smem);
        case 3: return launch_gemm<MT, 3>(ctx, a, grid, smem);
        case 4: return launch_gemm<MT, 4>(ctx, a, grid, smem);
        case 5: return launch_gemm<MT, 5>(ctx, a, grid, smem);
        case 6: return launch_gemm<MT, 6>(ctx, a, grid, smem);
        case 7: return launch_gemm<MT, 7>(ctx, a, grid, smem);
        default: return launch_gemm<MT, 8>(ctx, a, grid, smem);
    }
}

}  // namespace

// Row tiles per CTA and token-tile width for a product: the pair with the least estimated time.  A step (row tile,
// block) costs 8 clocks a token on the tensor cores, 16 with one row tile per CTA (its B blocks then come from L2 at
// twice the rate the L2 delivers), but never less than unpacking and draining take; work goes out in rounds of one
// CTA per SM.
static void plan_gemm(int n_sms, int n_seg, const int *n_rows, int nb, int n_tok, int *mt_out, int *nc_out) {
    double best = 1e300;
    for (int mt = 1; mt <= 2; mt++)
        for (int nc = 1; nc <= 8; nc++) {
            const int n = 16 * nc;
            if (nc > 1 && n - 16 >= n_tok) break;
            int64_t tiles = 0;
            for (int i = 0; i < n_seg; i++) tiles += (n_rows[i] + 128 * mt - 1) / (128 * mt);
            const int64_t items = tiles * ((n_tok + n - 1) / n);
            const double rounds = (double)((items + n_sms - 1) / n_sms);
            const double step = std::max((mt == 1 ? 16.0 : 8.0) * n, 260.0 + 1.3 * n);
            const double cost = rounds * (step * mt * nb + 4000.0);
            if (cost < best) {
                best = cost;
                *mt_out = mt;
                *nc_out = nc;
            }
        }
}

// Up to four row ranges with the same ne0 against n_tok activations (n_tok <= kPq2GemmTokens).
bk_status launch_pq2_gemm(bk_ctx *ctx, int n_seg, const uint8_t *const *rows, const int *n_rows, float *const *y, int ne0, const float *x,
                          int n_tok) {
    GemmArgs a{};
    a.nb = (ne0 + kGemmBlock - 1) / kGemmBlock;
    a.row_bytes = a.nb * kGemmBlockBytes;
    a.n_tok = n_tok;
    a.err_flag = ctx->d_err;
    int used = 0, rows_used[kGemmMaxSegs];
    for (int i = 0; i < n_seg && used < kGemmMaxSegs; i++) {
        if (n_rows[i] <= 0) continue;
        a.rows[used] = rows[i];
        a.y[used] = y[i];
        rows_used[used] = a.seg_rows[used] = n_rows[i];
        if (((uintptr_t)rows[i] | (uintptr_t)a.row_bytes) % 16 == 0) a.vec |= 1 << used;
        used++;
    }
    if (used == 0) return BK_OK;
    const bk_status fit = pq2_rows_fit(ctx, ne0, n_tok);  // one limit for every number of tokens from two on
    if (fit != BK_OK) return fit;
    int mt = 1, nc = 1;
    plan_gemm(ctx->n_sms, used, rows_used, a.nb, n_tok, &mt, &nc);
    const int n = 16 * nc, tok_tiles = (n_tok + n - 1) / n;
    int tiles = 0;
    for (int i = 0; i < kGemmMaxSegs; i++) {
        a.seg_tile0[i] = tiles;
        if (i < used) tiles += (a.seg_rows[i] + 128 * mt - 1) / (128 * mt);
        else a.seg_tile0[i] = INT32_MAX;
    }
    const size_t w_bytes = (size_t)2 * mt * 128 * kGemmRowWords * 4, b_bytes = (size_t)n * 512;
    const size_t limit = 227 * 1024;
    a.n_stages_b = (int)std::min<size_t>(4, (limit - 1024 - w_bytes) / b_bytes);
    // the activations' parts, one scale per padded token
    const size_t xb_bytes = (size_t)tok_tiles * a.nb * b_bytes, need = xb_bytes + (size_t)tok_tiles * n * sizeof(float);
    if (ctx->pq2_x_bytes < need) {
        BK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        if (ctx->d_pq2_x) cudaFree(ctx->d_pq2_x);
        ctx->d_pq2_x = nullptr;
        ctx->pq2_x_bytes = 0;
        BK_CUDA(ctx, cudaMalloc((void **)&ctx->d_pq2_x, need));
        ctx->pq2_x_bytes = need;
    }
    float *tok_scale = reinterpret_cast<float *>(ctx->d_pq2_x + xb_bytes);
    a.xb = ctx->d_pq2_x;
    a.tok_scale = tok_scale;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tok_tiles * n));
    cfg.blockDim = dim3(256);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    BK_CUDA(ctx, cudaLaunchKernelEx(&cfg, pq2_split_x_kernel, x, ne0, a.nb, n_tok, n, ctx->d_pq2_x, tok_scale));
    ctx->launches++;
    const size_t smem = 1024 + (size_t)a.n_stages_b * b_bytes + w_bytes;
    const dim3 grid((unsigned)tiles, (unsigned)tok_tiles);
    return mt == 1 ? launch_gemm_nc<1>(ctx, nc, a, grid, smem) : launch_gemm_nc<2>(ctx, nc, a, grid, smem);
}

}  // namespace bk
