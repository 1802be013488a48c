// PQ2_0 ternary rows times a block of activations (prompt or speculative tokens) on the 5th-generation
// tensor cores: y[t][r] = sum_j x[t][j] * W[base_row + r][j] for n_tok tokens at once
// (src/kernels.rs:333-420 `pq2_matmul_n`; row format src/kernels.rs:204-229).  bk_pq2.cu is the form for
// one to four tokens, where the weight stream is the cost and every launch reads it once per pair of tokens.
//
// The block sums are exact integers, as there: x is fixed point, X = round(x * 2^(27 - e)) with 2^e the power of two
// above the largest |x| of the token's block of 128 (three bits more than the form for few tokens keeps).
//
// What bounds it: what the sixteen warps that unpack weights and drain sums have to issue (two thirds of all issue slots with
// 512 tokens, the tensor cores 0.4 busy with four 8-bit products per weight and token); with a few tokens the round trips of a
// step.  The layout:
//   * X has 28 bits and an operand has 8, so X is cut into four digits, X = d0 - 64 d1 + 2^14 (d2 - 64 d3), each within
//     -128..127.  The weights are unpacked twice, as -1, 0, 1, 2 and times -64 (which fits 8 bits): d0 and d1 then meet in one
//     accumulator, d2 and d3 in another, and both stay within 2^21, exact in s32 and in f32.
//   * Weights are the A operand, IN TENSOR MEMORY: M = 128 rows, a thread's tensor-memory lane is a row, so unpacking is
//     register work (four codes in a byte permute's selector give four weights) and a tcgen05.st; no shared-memory pass, and
//     the MMA reads only B from shared memory.
//   * X is the B operand.  A first kernel writes the digits once, already permuted (the order of the K slots is free and is
//     chosen so that the unpacking needs no shuffles) and swizzled, one contiguous piece per (token tile, block of 128): the
//     main kernel fetches a block with ONE bulk copy, and a tile's block scales (2^(e - 27)) with one more.
//   * Both scales are the block's, so the accumulators are drained after every block of 128: the two sums become one f32
//     (one rounding) that is added up as scale * sum, as the reference's scalar path groups it (src/kernels.rs:633-650).
//     Two pairs of accumulators alternate: the drain of one step runs under the MMAs of the other's next.  128 columns a
//     pair are what the operand stages leave, hence at most 64 tokens a tile.
//   * The two digits that meet the same weights are one B operand of 2 N columns, into both sums of a pair at once: half as many
//     products as one digit each, and up to 32 tokens each costs the same 32 clocks (512 tokens: 298 us a layer before, 281 so).
// Measured (q, k, v and output projection of a layer, 14336 x 5120 and 5120 x 6144): 5 tokens 39 us, 16 tokens 41 (62 and
// 176 as pairs of tokens; 4 tokens 41.0 as pairs and 39.1 here, 3 tokens 37.4 and 39.1, so the line could lie at 4), 64 tokens 61 (702),
// 128 tokens 93 (1410), 512 tokens 281 (5750).  The form before, x as two f16 parts scaled per token and truncated f32 block sums, took
// 57, 86, 129, 287 and 574.  Error against float64, 2-norm: 7.4e-8 on normal data, 8.0e-8 with x20 outliers in x, 4.5e-8 without
// a bias on products of one sign; 1.02e-7, 2.4e-7 and 5.0e-8 as pairs of tokens; 1.01e-7, 1.0e-7 and 6.5e-8 (bias -5e-8) in the
// form before, which also lost blocks that lie 2^40 below the token's largest element.
// A step is (row tile of 128, block of 128); a CTA works on one or two row tiles (two share every B block: 32
// instead of 64 bytes per clock and SM from L2, which is what the L2 delivers) and one token tile of 16..64.
// The sum over blocks takes the same order and groups whatever the tiling, so a result does not depend on it bit for bit.
#include <algorithm>
#include <atomic>
#include <cuda_fp16.h>
#include <math_constants.h>

#include "bk_device.cuh"
#include "bk_internal.h"
#include "bk_mma_common.cuh"
#include "bk_umma.cuh"

namespace bk {

namespace {

constexpr int kWorkWarps = 16;                    // unpack and drain
constexpr int kMmaWarp = kWorkWarps, kLoadWarp = kWorkWarps + 1, kGemmThreads = (kWorkWarps + 2) * 32;
constexpr int kGemmBlock = 128, kGemmBlockBytes = 34;
constexpr int kGemmSegBlocks = 4;                 // blocks of a row staged together
constexpr int kGemmRowWords = 36;                 // words of a staged row: nine 16-byte pieces hold any four blocks of an aligned row
constexpr int kGemmMaxSegs = 4;
constexpr int kGemmMaxSegments = 64;              // of four blocks in a row (the length limit leaves 36)
constexpr uint32_t kGemmStageW = 2 * 2 * 128 * kGemmRowWords * 4;  // staged weights of the two owners
// Shared memory of the sums of the segments done, [row tile][token][row]; of a split tile every unit's, [unit of the CTA][token][row].
__host__ __device__ constexpr uint32_t gemm_sum_bytes(int places, int n) { return (uint32_t)(places * n) * 512u; }
// Pairs of units of a row of nb blocks, see the kernel.
__host__ __device__ constexpr int gemm_halves(int nb) { return ((nb + kGemmSegBlocks - 1) / kGemmSegBlocks + 1) / 2; }
__host__ __device__ constexpr int gemm_pairs(int nb) { return (gemm_halves(nb) + 1) / 2; }
__host__ __device__ constexpr int gemm_places(int mt, int nb, int split) { return split > 1 ? 2 * ((gemm_pairs(nb) + split - 1) / split) : mt; }
constexpr int kGemmFrac = 27;                     // X = round(x * 2^(kGemmFrac - e))
// tensor-memory columns: per owner one or two pairs of sums (low | high, N columns each), then per owner two A stages (weights | times -64)
constexpr uint32_t kColsD = 128, kColA = 256, kColsA = 64;

struct GemmArgs {
    const uint8_t *rows[kGemmMaxSegs];
    float *y[kGemmMaxSegs];
    int seg_rows[kGemmMaxSegs], seg_tile0[kGemmMaxSegs];
    int y_stride[kGemmMaxSegs];  // rows of a token in y (the range may be a part of them)
    const uint8_t *xb;        // [token tile][block][digit 0 2 1 3][n][128 B, swizzled]
    const float *x_scale;     // [token tile][block][n]: 2^(e - kGemmFrac), NaN for a block with an infinity or a NaN in it
    int nb, row_bytes, n_tok, n_stages_b;
    int split;                // CTAs, a cluster, that share the blocks of a tile (one row tile a CTA); 1: none do
    int vec;                  // bit s: the rows of range s all start on 16-byte boundaries
    int *err_flag;
};

// x -> digits in the order and swizzle of the B operand, and the block scales.  One thread per 16 elements of a (padded) token,
// eight per block.  Slots 16 i + 4 p .. + 3 of a block hold the elements 16 i + o, 16 i + o + 2, .. + 4, .. + 6 with
// o = 0, 8, 1, 9 for p = 0..3 (see unpack16()), so the sixteen elements of a thread are one 16-byte chunk of each digit.
__global__ void __launch_bounds__(256) pq2_split_x_kernel(const float *x, int ne0, int nb, int n_tok, int n, int n_pad, uint8_t *xb, float *x_scale) {
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    const int idx = blockIdx.x * 256 + threadIdx.x, tok = idx / (nb * 8), c = idx - tok * (nb * 8), blk = c >> 3, i = c & 7;
    const int tile = tok / n, r = tok - tile * n, j0 = 16 * c;
    float v[16];
    if (tok < n_tok && (ne0 & 3) == 0 && ((uintptr_t)x & 15) == 0 && j0 + 16 <= ne0) {
        const float4 *p = reinterpret_cast<const float4 *>(x + (size_t)tok * ne0 + j0);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float4 f = p[k];
            v[4 * k] = f.x, v[4 * k + 1] = f.y, v[4 * k + 2] = f.z, v[4 * k + 3] = f.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < 16; k++) v[k] = (tok < n_tok && j0 + k < ne0) ? x[(size_t)tok * ne0 + j0 + k] : 0.f;
    }
    float am = 0.f;
#pragma unroll
    for (int k = 0; k < 16; k++) am = fabsf(v[k]) <= am ? am : (fabsf(v[k]) < CUDART_INF_F ? fabsf(v[k]) : CUDART_INF_F);
    for (int o = 4; o > 0; o >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));  // the block's eight threads
    if (tok >= n_pad) return;
    int e = 0;
    if (am > 0.f && am < CUDART_INF_F) frexpf(am, &e);  // am = f * 2^e, f in [0.5, 1)
    const int up = min(kGemmFrac - e, 127);             // (blocks below 2^-100: the grid stays at 2^-127)
    const float s = ldexpf(1.0f, up);
    if (i == 0) x_scale[((size_t)tile * nb + blk) * n + r] = am < CUDART_INF_F ? ldexpf(1.0f, -up) : CUDART_NAN_F;
    uint32_t d[4][4] = {};
#pragma unroll
    for (int p = 0; p < 4; p++)
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int X = __float2int_rn(v[(p & 1) * 8 + (p >> 1) + 2 * q] * s);      // |X| < 2^27
            const int h = (X + 8192) >> 14, l = X - h * 16384;                        // -8192..8192, -8192..8191
            const int d1 = min(-((l + 32) >> 6), 127), d3 = min(-((h + 32) >> 6), 127);  // what 127 cuts off fits the digit below
            d[0][p] |= (uint32_t)((l + 64 * d1) & 255) << (8 * q);
            d[1][p] |= (uint32_t)(d1 & 255) << (8 * q);
            d[2][p] |= (uint32_t)((h + 64 * d3) & 255) << (8 * q);
            d[3][p] |= (uint32_t)(d3 & 255) << (8 * q);
        }
    uint8_t *dst = xb + ((size_t)tile * nb + blk) * (size_t)n * 512 + (size_t)r * 128 + ((i ^ (r & 7)) << 4);
#pragma unroll
    for (int k = 0; k < 4; k++)  // (in the order 0 2 1 3: what meets the same weights lies side by side)
        *reinterpret_cast<uint4 *>(dst + (size_t)((k & 1) * 2 + (k >> 1)) * n * 128) = make_uint4(d[k][0], d[k][1], d[k][2], d[k][3]);
}

// A tensor-memory load without the wait.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t *r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}

__device__ __forceinline__ uint32_t pick_bytes(uint32_t table, uint32_t nibbles) {  // (every nibble 0..3)
    uint32_t r;
    asm("prmt.b32 %0, %1, 0, %2;\n" : "=r"(r) : "r"(table), "r"(nibbles));
    return r;
}

// Sixteen 2-bit codes -> four registers of four 8-bit weights (code - 1) and four of the same times -64.  The codes are
// the selectors of a byte permute of the four weights: a nibble with one code in it picks a byte.  Registers in order:
// codes 0 2 4 6, 8 10 12 14, 1 3 5 7, 9 11 13 15.
__device__ __forceinline__ void unpack16(uint32_t w, uint32_t *one, uint32_t *wide) {
    const uint32_t even = w & 0x33333333u, odd = (w >> 2) & 0x33333333u;
    const uint32_t sel[4] = {even, even >> 16, odd, odd >> 16};
#pragma unroll
    for (int p = 0; p < 4; p++) {
        one[p] = pick_bytes(0x020100ffu, sel[p]);
        wide[p] = pick_bytes(0x80c00040u, sel[p]);
    }
}

// (Two f32 operations in one instruction: the draining warps are bound by what they issue.)
__device__ __forceinline__ uint64_t int2_to_f2(uint32_t a, uint32_t b) { return pack2(__int2float_rn((int)a), __int2float_rn((int)b)); }

// MT row tiles per CTA, N = 16 NC tokens.  Sixteen warps in two halves of eight ("owners") work on alternate steps, each with
// its own sums and operand stages, so that the round trips of a step (operand stores, the MMAs, reading the sums back) are under
// the other half's step: sixteen warps that share every step took 465 us for 512 tokens, two owners 340.
// With two row tiles an owner has one of them; with one, the owners take every other unit of up to eight blocks.
// SPLIT: a cluster of a.split CTAs shares a row tile's blocks.
template <int MT, int NC, bool SPLIT>
__global__ void __launch_bounds__(kGemmThreads, 1) pq2_gemm_kernel(const GemmArgs a) {
    extern __shared__ __align__(1024) uint8_t sm[];
    constexpr int N = 16 * NC, NH = 8 * NC;  // tokens of the tile, and of one warp
    constexpr uint32_t kBlockB = (uint32_t)N * 512u;
    constexpr int kBufs = 4 * N <= (int)kColsD ? 2 : 1;  // pairs of sums an owner has room for: with two, a step's products need not wait for the step before to be drained
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(sm);
    // barriers: B full [4] | B free [4] | A full [owner][2] | turn [2] | block scales | drain; then the tensor-memory address, a give-up flag,
    // the order of the segments, D full [owner][2] | D free [owner][2]
    const uint32_t bar_bf = sbase, bar_be = sbase + 32, bar_af = sbase + 64, bar_turn = sbase + 128, bar_sc = sbase + 144, bar_drain = sbase + 152,
                   slot = sbase + 160, bar_df = sbase + 384, bar_de = sbase + 416;
    static_assert(168 + 3 * kGemmMaxSegments <= 384, "the segments' order ends before the barriers behind it");
    volatile int *gave_up = reinterpret_cast<volatile int *>(sm + 164);
    const int nst = a.n_stages_b, nb = a.nb, n_seg = (nb + kGemmSegBlocks - 1) / kGemmSegBlocks;
    const uint32_t off_b = 1024u, off_w = off_b + (uint32_t)nst * kBlockB, off_t = off_w + kGemmStageW, off_s = off_t + gemm_sum_bytes(SPLIT ? gemm_places(MT, nb, a.split) : MT, N);
    // The segments form units of one or two, whose sums are kept apart; a pair of units has the same size as far as the row
    // goes.  Neither depends on the tiling.  The steps go in rounds of one per owner: round q is block q of both row tiles, or,
    // with one row tile, block q % 4 of the (q / 4)-th segment of the owner's units, which are every other one.
    // A split tile's CTAs take every split-th pair each.
    const int n_half = (n_seg + 1) / 2, n_pairs = (n_half + 1) / 2, split = SPLIT ? a.split : 1, rank = SPLIT ? blockIdx.x % split : 0;
    int n_mine = n_half;  // the CTA's segments of one owner
    if constexpr (SPLIT) {
        n_mine = 0;
        for (int p = rank; p < n_pairs; p += split) n_mine += (p + 1) * n_half / n_pairs - p * n_half / n_pairs;
    }
    volatile uint8_t *seg_order = sm + 168, *unit_end = sm + 168 + 2 * kGemmMaxSegments;  // [owner][i]: i-th segment (one row tile); [segment]
    if (tid < n_half) {
        // pair p has the segments 2 f .. 2 f + 2 h - 1
        const int p = ((tid + 1) * n_pairs - 1) / n_half, f = p * n_half / n_pairs, h = (p + 1) * n_half / n_pairs - f;
        int at = tid;
        if constexpr (SPLIT) {
            at -= f;
            for (int p2 = rank; p2 < p; p2 += split) at += (p2 + 1) * n_half / n_pairs - p2 * n_half / n_pairs;
        }
        for (int o = 0; o < 2; o++) {
            const int seg = 2 * f + o * h + tid - f;
            if (!SPLIT || p % split == rank) seg_order[o * kGemmMaxSegments + at] = (uint8_t)seg;
            unit_end[seg] = tid - f == h - 1 || seg == n_seg - 1;
        }
    }
    const int n_rounds = MT == 2 ? nb : n_mine * kGemmSegBlocks;
    auto segment = [&](int i, int owner) { return MT == 2 ? i : (int)seg_order[owner * kGemmMaxSegments + i]; };
    auto block_of = [&](int q, int owner) { return MT == 2 ? q : segment(q >> 2, owner) * kGemmSegBlocks + (q & 3); };

    if (tid == 0) {
        for (int i = 0; i < 4; i++) {
            mbar_init(bar_bf + 8 * i, 1);
            mbar_init(bar_be + 8 * i, 1);
            mbar_init(bar_af + 8 * i, 8);
            mbar_init(bar_df + 8 * i, 1);
            mbar_init(bar_de + 8 * i, 8);
        }
        for (int i = 0; i < 2; i++) mbar_init(bar_turn + 8 * i, 8);
        mbar_init(bar_sc, 1);
        mbar_init(bar_drain, 1);
        *gave_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == kMmaWarp) tmem_alloc(slot, 512);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t *>(sm + 160), 0);

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
    auto wait_all = [&](uint32_t bar, uint32_t parity) -> bool { return __all_sync(0xffffffffu, wait(bar, parity)); };  // one answer for the warp

    const int row_tile = SPLIT ? blockIdx.x / split : blockIdx.x, tok_tile = blockIdx.y;
    int sg = 0;
#pragma unroll
    for (int i = 1; i < kGemmMaxSegs; i++) sg += (row_tile >= a.seg_tile0[i]) ? 1 : 0;
    const int row0 = (row_tile - a.seg_tile0[sg]) * (128 * MT), seg_rows = a.seg_rows[sg];
    const uint8_t *wrows = a.rows[sg];

    if (warp == kLoadWarp) {
        // the tile's block scales, then its B blocks, in order of use through the ring of stages
        const uint8_t *xb = a.xb + (size_t)tok_tile * nb * kBlockB;
        asm volatile("griddepcontrol.wait;\n" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
        if (elect_one()) {
            const uint32_t bytes = (uint32_t)nb * N * 4u;
            mbar_expect_tx(bar_sc, bytes);
            tma_bulk(sbase + off_s, a.x_scale + (size_t)tok_tile * nb * N, bytes, bar_sc);
        }
        __syncwarp();
        uint32_t st = 0, use = 0;
        bool ok = true;
        for (int q = 0; q < n_rounds && ok; q++)
#pragma unroll
            for (int o = 0; o < 3 - MT; o++) {
                const int b = block_of(q, o);
                if (b >= nb) continue;
                if (use > 0) ok = ok && wait_all(bar_be + 8 * st, (use - 1) & 1u);
                if (!ok) break;
                if (elect_one()) {
                    mbar_expect_tx(bar_bf + 8 * st, kBlockB);
                    tma_bulk(sbase + off_b + st * kBlockB, xb + (size_t)b * kBlockB, kBlockB, bar_bf + 8 * st);
                }
                __syncwarp();
                if (++st == (uint32_t)nst) st = 0, use++;
            }
        // no copy in flight is left behind, whatever happened above
        const int filled = (int)use * nst + (int)st;
        for (int c = max(0, filled - nst); c < filled; c++)
            for (int polls = 0; !mbar_try_wait(bar_bf + 8 * (c % nst), (uint32_t)(c / nst) & 1u) && polls < kWaitPolls; polls++) {}
        for (int polls = 0; !mbar_try_wait(bar_sc, 0) && polls < kWaitPolls; polls++) {}
    } else if (warp == kMmaWarp) {
        const uint32_t idesc = umma_idesc_s8(128, 2 * N);
        uint32_t st = 0, b_par = 0;
        bool ok = true;
        for (int q = 0; q < n_rounds && ok; q++)
#pragma unroll
            for (int o = 0; o < 2; o++) {  // round q is every owner's q-th step
                if (block_of(q, o) >= nb) continue;
                if (MT == 1 || o == 0) ok = ok && wait_all(bar_bf + 8 * st, b_par);
                ok = ok && wait_all(bar_af + 16 * o + 8 * (q & 1), (uint32_t)(q >> 1) & 1u);
                const uint32_t buf = (uint32_t)q % kBufs, turn = (uint32_t)q / kBufs;
                if (turn > 0) ok = ok && wait_all(bar_de + 16 * o + 8 * buf, (turn - 1) & 1u);
                if (!ok) break;
                tc_fence_after_sync();
                const uint32_t d = tmem + o * kColsD + buf * (2 * N), am = tmem + kColA + o * (2 * kColsA) + (q & 1) * kColsA;
                const uint64_t bd = umma_smem_desc(sbase + off_b + st * kBlockB, 16, 1024, kUmmaSwizzle128);
                const bool last_use = MT == 1 || o == 1;
                if (elect_one()) {
#pragma unroll
                    // digits 0 and 2 side by side into low and high sums, then 1 and 3, which meet the weights times -64: a product of
                    // up to 64 columns takes the same 32 clocks
                    for (int odd = 0; odd < 2; odd++)
#pragma unroll
                        for (int k = 0; k < 4; k++)  // (the address field of a descriptor counts 16-byte units)
                            umma_i8_ts(d, am + odd * 32 + 8 * k, bd + (uint64_t)((odd * (2 * N * 128) + k * 32) >> 4), idesc, odd + k > 0);
                    umma_commit(bar_df + 16 * o + 8 * buf);
                    if (last_use) umma_commit(bar_be + 8 * st);
                }
                __syncwarp();
                if (last_use && ++st == (uint32_t)nst) st = 0, b_par ^= 1u;
            }
        // no product in flight is left behind, whatever happened above
        if (elect_one()) umma_commit(bar_drain);
        __syncwarp();
        for (int polls = 0; !mbar_try_wait(bar_drain, 0) && polls < kWaitPolls; polls++) {}
    } else {
        const int owner = warp >> 3, quad = warp & 3, half = (warp >> 2) & 1, r = quad * 32 + lane;  // tensor-memory lane = row of the tile
        const int trow0 = row0 + (MT == 2 ? owner * 128 : 0);                                        // first row of the owner's tile
        auto seg_of = [&](int k) { return segment(k, owner); };
        const int n_local = MT == 2 ? n_seg : (seg_of(n_mine - 1) < n_seg ? n_mine : n_mine - 1);    // segments of the owner
        uint32_t *wst = reinterpret_cast<uint32_t *>(sm + off_w) + owner * (2 * 128 * kGemmRowWords);  // [2][128][kGemmRowWords]
        // The two warps of a quadrant stage its 32 rows, a segment of four blocks at a time.  Rows on 16-byte boundaries (their
        // length is then a multiple of eight blocks): the nine 16-byte pieces around the blocks, which start at the segment's
        // first byte or, every other segment, 8 bytes before it.  Other rows: the words that overlap the blocks.
        const bool vec = (a.vec >> sg) & 1;
        const int t64 = half * 32 + lane;
        uint32_t src[5];
#pragma unroll
        for (int i = 0; i < 5; i++) {
            const int idx = t64 + 64 * i, rr = idx / 9;
            src[i] = (uint32_t)rr * a.row_bytes + (uint32_t)(idx - rr * 9) * 16u;
        }
        auto stage_w = [&](int k) {
            const int seg = seg_of(k), blocks = min(kGemmSegBlocks, nb - seg * kGemmSegBlocks), bytes = blocks * kGemmBlockBytes;
            const int rb = quad * 32;
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(wst) + (uint32_t)(((k & 1) * 128 + rb) * kGemmRowWords) * 4u;
            const uint8_t *p0 = wrows + (size_t)(trow0 + rb) * a.row_bytes + (size_t)seg * (kGemmSegBlocks * kGemmBlockBytes);
            const int rows = min(32, seg_rows - trow0 - rb);
            if (vec) {
                p0 -= (seg & 1) * 8;
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
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        };
        auto quad_sync = [&]() { asm volatile("bar.sync %0, 64;\n" ::"r"(1 + owner * 4 + quad) : "memory"); };
        if (n_local > 0) stage_w(0);

        uint64_t acc[NH / 2];  // pairs of tokens
#pragma unroll
        for (int j = 0; j < NH / 2; j++) acc[j] = 0;
        const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16);
        // where a segment starts in the staged row, in bytes: see stage_w (rows start on even addresses; a row's
        // misalignment is the same in every segment, 136 bytes on)
        const uint32_t row_sh = vec ? 0u : (uint32_t)((uintptr_t)(wrows + (size_t)(trow0 + r) * a.row_bytes) & 2u);

        // this warp's half of block i of the owner's segment k, from the staged words, and the block's weight scale
        uint32_t w[4];
        float sc_next;
        auto fetch = [&](int k, int i) {
            if (i == 0) {
                asm volatile("cp.async.wait_group 0;\n" ::: "memory");
                quad_sync();  // both warps' pieces are in, and both have left the segment before
                if (k + 1 < n_local) stage_w(k + 1);
            }
            const uint32_t *row = wst + (size_t)((k & 1) * 128 + r) * kGemmRowWords;
            const uint32_t byte = (vec ? (uint32_t)(seg_of(k) & 1) * 8u : row_sh) + (uint32_t)i * kGemmBlockBytes;
            sc_next = __half2float(__ushort_as_half(*reinterpret_cast<const unsigned short *>(reinterpret_cast<const uint8_t *>(row) + byte)));
            const uint32_t cb = byte + 2u + (uint32_t)half * 16u, cs = (cb & 2u) * 8u;
            const uint32_t *cw = row + (cb >> 2);
            uint32_t v[5];
#pragma unroll
            for (int j = 0; j < 4; j++) v[j] = cw[j];
            v[4] = cs ? cw[4] : 0u;
#pragma unroll
            for (int j = 0; j < 4; j++) w[j] = __funnelshift_r(v[j], v[j + 1], cs);
        };
        // ... unpacked into the operand stage of the owner's step t.  The stage's last user is step t - 2, whose sums have been drained.
        auto unpack = [&](int t) {
            const uint32_t at = lane_base + kColA + (uint32_t)owner * (2 * kColsA) + (uint32_t)(t & 1) * kColsA + (uint32_t)half * 16u;
            uint32_t one[16], wide[16];
#pragma unroll
            for (int i = 0; i < 4; i++) unpack16(w[i], one + 4 * i, wide + 4 * i);
            tmem_st16(at, one);
            tmem_st16(at + 32u, wide);
            tmem_wait_st();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_af + 16 * owner + 8 * (t & 1));
        };
        bool ok = wait(bar_sc, 0);
        auto drain = [&](int t, int b, float sc) {
            const uint32_t buf = (uint32_t)t % kBufs;
            ok = ok && wait(bar_df + 16 * owner + 8 * buf, ((uint32_t)t / kBufs) & 1u);
            __syncwarp();
            tc_fence_after_sync();
            const uint32_t d = lane_base + (uint32_t)owner * kColsD + buf * (2 * N) + (uint32_t)half * NH;
            const uint32_t xs = sbase + off_s + (uint32_t)(b * N + half * NH) * 4u;
            // eight tokens at a time, the next eight on their way meanwhile (sixteen at a time spill: 308 us for 512 tokens, 299 so)
            uint32_t lo[2][8], hi[2][8];
            tmem_ld8(d, lo[0]);
            tmem_ld8(d + N, hi[0]);
#pragma unroll
            for (int c = 0; c < NC; c++) {
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                if (c + 1 < NC) {
                    tmem_ld8(d + 8u * (c + 1), lo[(c + 1) & 1]);
                    tmem_ld8(d + N + 8u * (c + 1), hi[(c + 1) & 1]);
                } else {
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_de + 16 * owner + 8 * buf);
                }
#pragma unroll
                for (int c4 = 0; c4 < 2; c4++) {
                    const uint4 x4 = lds128(xs + 16u * (2 * c + c4));
                    const uint64_t xv[2] = {(uint64_t)x4.x | (uint64_t)x4.y << 32, (uint64_t)x4.z | (uint64_t)x4.w << 32};
#pragma unroll
                    for (int j = 0; j < 2; j++) {
                        const int k = 4 * c4 + 2 * j;
                        const uint64_t sum = fma2(int2_to_f2(hi[c & 1][k], hi[c & 1][k + 1]), pack2(16384.0f, 16384.0f),
                                                  int2_to_f2(lo[c & 1][k], lo[c & 1][k + 1]));
                        acc[4 * c + k / 2] = fma2(mul2(pack2(sc, sc), xv[j]), sum, acc[4 * c + k / 2]);
                    }
                }
            }
        };
        // A unit's sums join the ones before it in shared memory, in the order of the units, and leave for y after the last: one running
        // f32 sum over all blocks would round at the size of the whole result forty times.  With one row tile the owners take turns.
        float *tot = reinterpret_cast<float *>(sm + off_t) + (size_t)((MT == 2 ? owner * N : 0) + half * NH) * 128 + r;
        // Of a split tile every unit's sums stay apart until all are there.
        auto flush = [&](int unit, bool last) {
            if constexpr (SPLIT) {
                float *own = reinterpret_cast<float *>(sm + off_t) + (size_t)(unit * N + half * NH) * 128 + r;
#pragma unroll
                for (int j = 0; j < NH / 2; j++) {
                    const float2 v = unpack2(acc[j]);
                    own[2 * j * 128] = v.x, own[(2 * j + 1) * 128] = v.y;
                    acc[j] = 0;
                }
                return;
            }
            if (MT == 1 && unit > 0) {
                ok = ok && wait(bar_turn + 8 * (1 - owner), (uint32_t)((unit - 1) >> 1) & 1u);
                __syncwarp();
            }
            float2 v[NH / 2];
#pragma unroll
            for (int j = 0; j < NH / 2; j++) {
                v[j] = unpack2(acc[j]);
                acc[j] = 0;
                if (unit > 0) v[j].x += tot[2 * j * 128], v[j].y += tot[(2 * j + 1) * 128];
            }
            if (!last) {
#pragma unroll
                for (int j = 0; j < NH / 2; j++) tot[2 * j * 128] = v[j].x, tot[(2 * j + 1) * 128] = v[j].y;
                if (MT == 1) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_turn + 8 * owner);
                }
                return;
            }
            asm volatile("griddepcontrol.wait;\n" ::: "memory");  // what came before on the stream may still read y until here
            const int t0 = tok_tile * N + half * NH, left = a.n_tok - t0, row = trow0 + r, stride = a.y_stride[sg];
            if (row < seg_rows) {
                float *yp = a.y[sg] + (size_t)t0 * stride + row;
#pragma unroll
                for (int j = 0; j < NH; j++)
                    if (j < left) yp[(size_t)j * stride] = j & 1 ? v[j / 2].y : v[j / 2].x;
            }
        };
        // one iteration per step: the next step's operand goes out before this step's sums are awaited
        if (n_local > 0) {
            fetch(0, 0);
            unpack(0);
        }
        float sc = n_local > 0 ? sc_next : 0.f;
        int unit = MT == 2 ? 0 : owner;
        for (int k = 0; k < n_local; k++) {
            const int seg = seg_of(k), blocks = min(kGemmSegBlocks, nb - seg * kGemmSegBlocks);
            for (int i = 0; i < blocks; i++) {
                const int t = k * kGemmSegBlocks + i;
                const bool more = i + 1 < blocks;
                if (more || k + 1 < n_local) {
                    fetch(more ? k : k + 1, more ? i + 1 : 0);
                    unpack(t + 1);
                }
                drain(t, seg * kGemmSegBlocks + i, sc);
                sc = sc_next;
            }
            if (unit_end[seg]) {
                flush(unit, seg == n_seg - 1);
                unit += 3 - MT;
            }
        }
    }
    tc_fence_before_sync();
    __syncthreads();  // (every product and every copy has come to its end)
    if (warp == kMmaWarp) tmem_dealloc(tmem, 512);
    if constexpr (SPLIT) {
        // The units' sums join in the order of the units, as flush() does it, every CTA for its share of the tokens.
        asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
        asm volatile("griddepcontrol.wait;\n" ::: "memory");  // as in flush()
        const int r = tid & 127, row = row0 + r, left = a.n_tok - tok_tile * N;
        const int n_units = 2 * n_pairs;  // (none is empty where there are two pairs or more)
        if (tid < 512)
            for (int j = rank + split * (tid >> 7); j < N && j < left; j += split * 4) {
                float sum = 0.f;
                for (int u = 0; u < n_units; u++) {
                    const int p = u >> 1;
                    const uint32_t own = sbase + off_t + (uint32_t)(((p / split * 2 + (u & 1)) * N + j) * 128 + r) * 4u;
                    uint32_t at;
                    float v;
                    asm("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(at) : "r"(own), "r"(p % split));
                    asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(at) : "memory");
                    sum = u ? v + sum : v;
                }
                if (row < seg_rows) a.y[sg][(size_t)(tok_tile * N + j) * a.y_stride[sg] + row] = sum;
            }
        asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");  // nobody leaves while its sums are read
    }
}

template <int MT, int NC, bool SPLIT>
bk_status launch_gemm(bk_ctx *ctx, const GemmArgs &a, dim3 grid, size_t smem) {  // grid: tiles; their CTAs beside one another
    static std::atomic<bool> opted_in[64] = {};
    const int dev = ctx->device;
    if (dev < 0 || dev >= 64) return fail(ctx, BK_ERR_UNSUPPORTED, "pq2 matmul: device index above 63");
    if (!opted_in[dev].load()) {
        BK_CUDA(ctx, cudaFuncSetAttribute(pq2_gemm_kernel<MT, NC, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
        opted_in[dev].store(true);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid.x * a.split, grid.y);
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)a.split;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = SPLIT ? 2 : 1;
    BK_CUDA(ctx, cudaLaunchKernelEx(&cfg, pq2_gemm_kernel<MT, NC, SPLIT>, a));
    ctx->launches++;
    BK_CUDA(ctx, cudaGetLastError());
    return BK_OK;
}

template <int MT, bool SPLIT = false>
bk_status launch_gemm_nc(bk_ctx *ctx, int nc, const GemmArgs &a, dim3 grid, size_t smem) {
    switch (nc) {
        case 1: return launch_gemm<MT, 1, SPLIT>(ctx, a, grid, smem);
        case 2: return launch_gemm<MT, 2, SPLIT>(ctx, a, grid, smem);
        case 3: return launch_gemm<MT, 3, SPLIT>(ctx, a, grid, smem);
        default: return launch_gemm<MT, 4, SPLIT>(ctx, a, grid, smem);
    }
}

}  // namespace

static size_t gemm_smem(int mt, int n, int nb, int stages, int split) {
    return 1024 + (size_t)stages * n * 512 + kGemmStageW + gemm_sum_bytes(gemm_places(mt, nb, split), n) + (size_t)nb * n * sizeof(float);
}
static int gemm_stages(int mt, int n, int nb, int split = 1) {  // of B that shared memory has room for: four at most, two at least or the tile is not used
    int stages = 4;
    while (stages > 0 && gemm_smem(mt, n, nb, stages, split) > 227 * 1024) stages--;
    return stages;
}

struct GemmPlan {
    int mt = 1, nc = 1;
    int split = 1;           // CTAs that share the blocks of a tile, with one row tile a CTA
    int64_t main_tiles = 0;  // how many of the launch's tiles of 128 mt rows; the rows of the others go to a second launch with one row tile per CTA
};
// Row tiles per CTA and token-tile width for a product: what has the least estimated time.  Work goes out in rounds of one CTA per SM.  A step
// (row tile, block) takes what unpacking and draining issue, about 480 + 12 n clocks, or 700 + 11 n when two row tiles do not share a B block (L2).
// Where two row tiles a CTA leave a last round nearly empty, its rows go out as tiles of half the size: q, k and v of 512 tokens are
// 448 items for 148 SMs: 219 us in four rounds, 204 us as three rounds and one of half the length.
static GemmPlan plan_gemm(int n_sms, const int *clusters, int n_seg, const int *n_rows, int nb, int n_tok) {
    GemmPlan plan;
    double best = 1e300;
    const int n_pairs = gemm_pairs(nb), n_half = gemm_halves(nb);
    int most[kGemmMaxSplit + 1] = {};  // segments of an owner of a cluster's busiest CTA: the pairs differ
    for (int split = 2; split <= std::min(n_pairs, kGemmMaxSplit); split++)
        for (int rank = 0; rank < split; rank++) {
            int mine = 0;
            for (int p = rank; p < n_pairs; p += split) mine += (p + 1) * n_half / n_pairs - p * n_half / n_pairs;
            most[split] = std::max(most[split], mine);
        }
    for (int nc = 1; nc <= 4; nc++) {
        const int n = 16 * nc;
        if (nc > 1 && n - 16 >= n_tok) break;
        int64_t tiles[3] = {};
        for (int i = 0; i < n_seg; i++)
            for (int mt = 1; mt <= 2; mt++) tiles[mt] += (n_rows[i] + 128 * mt - 1) / (128 * mt);
        const int64_t tok_tiles = (n_tok + n - 1) / n;
        const double round[3] = {0.0, (700.0 + 11.0 * n) * nb + 6000.0, (480.0 + 12.0 * n) * 2 * nb + 6000.0};
        auto rounds = [&](int64_t row_tiles) { return (double)((row_tiles * tok_tiles + n_sms - 1) / n_sms); };
        auto take = [&](int mt, int64_t main_tiles, double cost, int split = 1) {
            if (cost >= best) return;
            best = cost;
            plan = GemmPlan{mt, nc, split, main_tiles};
        };
        for (int mt = 1; mt <= 2; mt++)
            if (gemm_stages(mt, n, nb) >= 2) take(mt, tiles[mt], rounds(tiles[mt]) * round[mt]);
        // Where the tiles leave SMs without work, clusters of up to eight share a tile's pairs of units, as long as all of them fit on the device at
        // once: the output projection of up to 64 tokens is 40 tiles of three pairs, 27 us on 40 SMs and 16 us on 120 for 16 tokens, 32 and 25 for
        // 64.  A cluster lies within a group of SMs, so of 148 SMs 74 clusters of two find room, but 45 of three, 33, 26, 22, 15 and 15 of
        // eight; one more is a second round: 24 tiles as 48 clusters of three 29 us, as 24 of wider tiles 18 (3072 rows, 32 tokens).  A cluster
        // costs about 3000 clocks beside its steps, and the last places are dear (the CTAs of a cluster start together): 72 clusters of two 31.7
        // us where 96 CTAs of their own take 29.7 (3072 rows, 100 tokens), 56 of them 27 against 29 (7168 rows, 40 tokens).
        for (int split = 2; split <= std::min(n_pairs, kGemmMaxSplit); split++)
            if (tiles[1] * tok_tiles <= clusters[split] && gemm_stages(1, n, nb, split) >= 2) {
                const double last_places = std::max(0.0, (double)(tiles[1] * tok_tiles * split) / n_sms - 0.9);
                take(1, tiles[1], (700.0 + 11.0 * n) * nb * most[split] / n_half + 9000.0 + 160000.0 * last_places, split);
            }
        const int64_t whole = tiles[2] * tok_tiles / n_sms, main_tiles = whole * n_sms / tok_tiles;
        if (whole > 0 && main_tiles < tiles[2] && gemm_stages(2, n, nb) >= 2)
            take(2, main_tiles, (double)whole * round[2] + rounds(2 * (tiles[2] - main_tiles)) * round[1]);
    }
    return plan;
}

// How many clusters of 2, 3 .. kGemmMaxSplit CTAs the device takes at once (a CTA fills an SM); none where it does not say.
static void pq2_gemm_clusters(int *clusters) {
    const int smem = 227 * 1024;
    std::fill(clusters, clusters + kGemmMaxSplit + 1, 0);
    bool ok = cudaFuncSetAttribute(pq2_gemm_kernel<1, 1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess;
    for (int split = 2; ok && split <= kGemmMaxSplit; split++) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)split);
        cfg.blockDim = dim3(kGemmThreads);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)split;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        ok = cudaOccupancyMaxActiveClusters(&n, pq2_gemm_kernel<1, 1, true>, &cfg) == cudaSuccess;
        clusters[split] = ok ? n : 0;
    }
    if (!ok) cudaGetLastError();
    clusters[0] = 1;  // asked
}

// A token has 512 bytes of digits and a scale a block; a tile is filled up with up to 63 tokens of zeros.
static constexpr size_t kXBytes = 512 + sizeof(float);
int pq2_gemm_tokens(int ne0) {
    const int64_t nb = ((int64_t)ne0 + kGemmBlock - 1) / kGemmBlock, room = (int64_t)(kPq2ScratchBytes / (nb * kXBytes)) - 63;
    return (int)std::max<int64_t>(64, std::min<int64_t>(kPq2GemmTokens, room / 64 * 64));  // (rows that leave fewer are refused)
}

// Up to four row ranges with the same ne0 against n_tok activations (n_tok <= pq2_gemm_tokens(ne0)).
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
        rows_used[used] = n_rows[i];
        if (((uintptr_t)rows[i] | (uintptr_t)a.row_bytes) % 16 == 0) a.vec |= 1 << used;
        used++;
    }
    if (used == 0) return BK_OK;
    const bk_status fit = pq2_rows_fit(ctx, ne0, n_tok);  // one limit for every number of tokens from two on
    if (fit != BK_OK) return fit;
    if (!ctx->gemm_clusters[0]) pq2_gemm_clusters(ctx->gemm_clusters);
    const GemmPlan plan = plan_gemm(ctx->n_sms, ctx->gemm_clusters, used, rows_used, a.nb, n_tok);
    const int n = 16 * plan.nc, tok_tiles = (n_tok + n - 1) / n;
    const size_t b_bytes = (size_t)n * 512, s_bytes = (size_t)a.nb * n * sizeof(float);
    // the digits, then one scale per block of every padded token
    const size_t xb_bytes = (size_t)tok_tiles * a.nb * b_bytes;
    if (xb_bytes + (size_t)tok_tiles * s_bytes > kPq2ScratchBytes) return fail(ctx, BK_ERR_UNSUPPORTED, "pq2_matvec: more tokens than a pass takes");
    float *x_scale = reinterpret_cast<float *>(ctx->d_pq2_x + xb_bytes);
    a.xb = ctx->d_pq2_x;
    a.x_scale = x_scale;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(((size_t)tok_tiles * n * a.nb * 8 + 255) / 256));
    cfg.blockDim = dim3(256);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    BK_CUDA(ctx, cudaLaunchKernelEx(&cfg, pq2_split_x_kernel, x, ne0, a.nb, n_tok, n, tok_tiles * n, ctx->d_pq2_x, x_scale));
    ctx->launches++;
    // the ranges' first main_tiles tiles, then what is left of them
    GemmArgs part[2] = {a, a};
    int tiles[2] = {0, 0};
    const int part_mt[2] = {plan.mt, 1};
    int64_t left = plan.main_tiles;
    for (int i = 0; i < kGemmMaxSegs; i++) {
        int done = 0;
        for (int h = 0; h < 2; h++) {
            GemmArgs &g = part[h];
            g.seg_tile0[i] = i < used ? tiles[h] : INT32_MAX;
            if (i >= used) continue;
            const int per = 128 * part_mt[h], want = rows_used[i] - done;
            const int64_t take = h == 0 ? std::min<int64_t>((want + per - 1) / per, left) : (want + per - 1) / per;
            g.rows[i] = a.rows[i] + (size_t)done * a.row_bytes;
            g.y[i] = a.y[i] + done;
            g.seg_rows[i] = (int)std::min<int64_t>(want, take * per);
            g.y_stride[i] = rows_used[i];
            tiles[h] += (int)take;
            if (h == 0) left -= take;
            done += g.seg_rows[i];
        }
    }
    for (int h = 0; h < 2; h++) {
        if (tiles[h] == 0) continue;
        GemmArgs &g = part[h];
        g.split = h == 0 ? plan.split : 1;
        g.n_stages_b = gemm_stages(part_mt[h], n, a.nb, g.split);
        const size_t smem = gemm_smem(part_mt[h], n, a.nb, g.n_stages_b, g.split);
        const dim3 grid((unsigned)tiles[h], (unsigned)tok_tiles);
        const bk_status st = g.split > 1          ? launch_gemm_nc<1, true>(ctx, plan.nc, g, grid, smem)
                             : part_mt[h] == 1 ? launch_gemm_nc<1>(ctx, plan.nc, g, grid, smem) : launch_gemm_nc<2>(ctx, plan.nc, g, grid, smem);
        if (st != BK_OK) return st;
    }
    return BK_OK;
}

}  // namespace bk

const int32_t *bk_hook_pq2_clusters(bk_ctx *ctx) {
    if (!ctx->gemm_clusters[0]) bk::pq2_gemm_clusters(ctx->gemm_clusters);
    return ctx->gemm_clusters;
}

int32_t bk_hook_pq2_plan(int32_t n_sms, const int32_t *clusters, int32_t n_rows, int32_t n_blocks, int32_t n_tok, int32_t *plan) {
    const bk::GemmPlan p = bk::plan_gemm(n_sms, clusters, 1, &n_rows, n_blocks, n_tok);
    plan[0] = p.mt, plan[1] = p.nc, plan[2] = p.split, plan[3] = (int32_t)p.main_tiles;
    return 4;
}
