// Batched (prefill) attention over a 4-, 3- or 2-bit planar cache, or an f16 or f32 cache, on the
// 5th-generation tensor cores: the same work split and operands as bk_prefill.cu (which documents them and
// stays as the mma.sync form), with both contractions issued as tcgen05.mma and the accumulators in tensor memory.
//
// One CTA = 128 query rows (M = 128) of one kv head over one context chunk, tile by tile of 32 positions.  What
// bounds it: for 4-bit and f32 rows six 128 x 32 x 256 products per tile (hi.hi, hi.lo, lo.hi twice), 1536 clocks of
// the tensor cores, and about as much traffic of shared memory; so nothing may wait for anything else, and shared
// memory has to be spared.  Thirteen warps in three roles, coupled by mbarriers only:
//   * warps 4-11 (producers) turn packed rows into f16 operand tiles (for 4 bit with the rounding remainders, for
//     f32 rows hi + lo parts) in a ring of four slots, in the order of use: K0, K1, V0, K2, V1, ...  A thread's four
//     16-byte pieces of a row go out in an order that depends on its lane, or the eight lanes of a row would meet on
//     two of eight bank groups.  f16 rows are operands as stored and are dropped in by the TMA engine.
//   * warp 12 issues the products: S(t + 1) = Q . K^T goes ahead of O += P(t) . V, so the tensor cores work on S(t + 1)
//     under the softmax of tile t.  The small terms of S have columns of their own: the accumulator truncates, and does
//     so at the size of what it holds.
//   * warps 0-3 (thread = query row = tensor-memory lane) read S, scale by ||k||, apply the causal limit, move the
//     running reference R of s + log2 ||v|| LAZILY (only when the row maximum exceeds R by more than 8: the weights
//     p = 2^(t - R) * 64 then stay below 2^14 in f16; their row of O is then rescaled in place) and write the
//     weights as f16 hi + lo.
// Tensor memory (all 512 columns): O 256 | half of q_hi 64 | S 2 x (32 + 32) | P (hi, lo) 2 x 32.  A product with N = 32 costs as
// much as one with N = 64 (32 clocks), so q_hi meets k_hi and k_lo side by side; P and as much of q_hi as there are columns for
// are A operands from tensor memory, which spares shared memory 4 KiB a product.
// Measured (4 layers, append included): a 4608-token planar4 prompt in blocks of 512 11.3 -> 5.9 ms, a 777-token f32 prompt in
// one block 741 -> 309 us.  Before, one role after the other per tile with every MMA operand moved to uniform registers.  Without
// the runs of collect_o 5.5 ms and 287 us.
// Every mbarrier wait is bounded: one that runs out raises the context's error flag, the others of the CTA stop
// waiting, and the kernel runs on to its end, where the tensor memory is always released.
#include <cuda_fp16.h>
#include <math_constants.h>

#include <algorithm>
#include <atomic>
#include <cmath>

#include "bk_device.cuh"
#include "bk_internal.h"
#include "bk_mma_common.cuh"
#include "bk_umma.cuh"

namespace bk {

namespace {

constexpr int kSoftWarps = 4, kProdWarps = 8, kMmaWarp = kSoftWarps + kProdWarps, kUWarps = kMmaWarp + 1, kUT = kUWarps * 32;
constexpr int kRows = 128;  // query rows per CTA = tensor-memory lanes
constexpr int kTK = 32;     // positions per tile
constexpr float kPScale = 64.0f, kPScaleLog2 = 6.0f;
constexpr float kLazy = 8.0f;  // the reference moves when a row maximum exceeds it by more than this (log2 units)
constexpr size_t kRunFloats = kPrefillRunFloats;  // a CTA's sums of the runs done, [4 coordinates][row][4]
static_assert(kRunFloats == (size_t)kRows * kHd, "a place per row and coordinate");

constexpr uint32_t kQSlab = kRows * 128, kQTile = 4 * kQSlab;  // 16 KiB per 64-coordinate slab, 64 KiB per tile
constexpr uint32_t kKVSlab = kTK * 128, kKVTile = 4 * kKVSlab;  // 4 KiB, 16 KiB
// Operand slots.  Four: K(t) then takes the place of K(t - 2), whose S products were issued when the softmax had read tile
// t - 4, so the norms of four tiles can be kept.
constexpr int kSlots = 4, kNormTiles = 4;
constexpr uint32_t kSlotBytes = 2 * kKVTile;  // hi and lo tile
// offsets from the 1024-byte aligned base
constexpr uint32_t oQlo = 0, oQhi2 = kQTile, oSlots = oQhi2 + kQTile / 2, oSmall = oSlots + kSlots * kSlotBytes;
struct SmallU {
    float givens[kHd];
    float kn[kNormTiles][kTK], lv[kNormTiles][kTK];  // ||k|| and log2 ||v|| of a tile's positions
    unsigned long long full[kSlots], empty[kSlots];  // operand slots
    unsigned long long norms[kNormTiles];            // kn, lv of a tile written
    unsigned long long s_full[2], p_full[2], o_done[2], drain;
    float mul[kRows];  // what a row's sums are multiplied by at the end
    uint32_t tmem_slot;
    int gave_up;
    int run_slot;
};
constexpr uint32_t kUmmaSmem = oSmall + 3072;
static_assert(sizeof(SmallU) <= 3072 && kUmmaSmem <= 227 * 1024, "shared memory of a CTA");
constexpr uint32_t kTmemCols = 512, kColO = 0, kColQ = 256, kColS = 320, kColP = 448;

__device__ __forceinline__ uint32_t sw_off(int rows, int row, int chunk) {  // as tile_off in bk_prefill.cu
    return (uint32_t)((chunk >> 3) * rows * 128 + row * 128 + (((chunk & 7) ^ (row & 7)) << 4));
}
__device__ __forceinline__ uint32_t expand24u(uint32_t y) {
    y &= 0x00ffffffu;
    y += (y & 0x00fff000u) * 15u;
    y += (y & 0x0fc00fc0u) * 3u;
    y += (y & 0x38383838u);
    return y;
}
__device__ __forceinline__ uint32_t expand16u(uint32_t y) {  // eight 2-bit indices -> eight nibbles
    y &= 0x0000ffffu;
    y = (y | (y << 8)) & 0x00ff00ffu;
    y = (y | (y << 4)) & 0x0f0f0f0fu;
    y = (y | (y << 2)) & 0x33333333u;
    return y;
}
// The first `rot` (0..3) of four words go to the end: the piece order of a lane, see dequant_store_shfl.
__device__ __forceinline__ void rotate4(uint32_t (&w)[4], int rot) {
    if (rot & 1) {
        const uint32_t t = w[0];
        w[0] = w[1], w[1] = w[2], w[2] = w[3], w[3] = t;
    }
    if (rot & 2) {
        const uint32_t t0 = w[0], t1 = w[1];
        w[0] = w[2], w[1] = w[3], w[2] = t0, w[3] = t1;
    }
}
// 32 coordinates (four words of eight nibbles, rotated by `rot`) -> 32 halfs as four 16-byte chunks of a tile row.
// The eight lanes of a row store chunks 4 c + ((j + c / 2) & 3) together, one per bank group (4 c + j would put them on two).
// The table sits in registers: lane i holds (hi | lo << 16) of centroid i & 15, one shuffle looks both parts of an index
// up, and no shared-memory bank is involved.  (A shuffle takes the low five bits of the lane number; the fifth, the next index's, does not matter.)
template <bool LO>
__device__ __forceinline__ void dequant_store_shfl(const uint32_t (&w)[4], uint32_t tab, uint8_t *tile_hi, uint8_t *tile_lo, int rows,
                                                   int row_hi, int row_lo, int chunk0, int rot) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
        uint32_t h[4], l[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const uint32_t v0 = __shfl_sync(0xffffffffu, tab, w[j] >> (8 * e));
            const uint32_t v1 = __shfl_sync(0xffffffffu, tab, w[j] >> (8 * e + 4));
            h[e] = __byte_perm(v0, v1, 0x5410);
            l[e] = __byte_perm(v0, v1, 0x7632);
        }
        const int chunk = chunk0 + ((j + rot) & 3);
        *reinterpret_cast<uint4 *>(tile_hi + sw_off(rows, row_hi, chunk)) = make_uint4(h[0], h[1], h[2], h[3]);
        if (LO) *reinterpret_cast<uint4 *>(tile_lo + sw_off(rows, row_lo, chunk)) = make_uint4(l[0], l[1], l[2], l[3]);
    }
}

struct PrefillUArgs {
    DecodeArgs d;
    int seq, pos0, n_tokens, tq, n_blocks, n_chunks;
    float lut_alpha;
    float *scratch;
    float *runs;      // a place of kRunFloats per resident CTA, and which of them are taken
    int *runs_taken;
    int n_runs;
    int *err_flag;
};

template <int BITS, int NREP, bool VF32 = false>
__global__ void __launch_bounds__(kUT, 1)
prefill_umma_kernel(PrefillUArgs pa, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v) {
    extern __shared__ __align__(1024) uint8_t sm[];
    const DecodeArgs &a = pa.d;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm), small = base + oSmall;
    SmallU &ss = *reinterpret_cast<SmallU *>(sm + oSmall);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    // BITS = 16 stands for an f16 cache: its rows ARE the operands, so the TMA engine drops them into the slots in
    // the swizzled layout and nothing is dequantized (no table, no norms, no Givens rotation).
    constexpr bool kF16 = BITS == 16;
    // BITS = 32 stands for an f32 cache: its rows are split into f16 hi + lo on their way into the operand tiles
    // (the lo tiles are the ones the 4-bit rows use for their rounding remainders); like f16 rows they are
    // neither rotated nor normalised.
    constexpr bool kF32 = BITS == 32, kRaw = kF16 || kF32;
    // VF32: the reference's K-only mode, planar K rows (BITS = 4 or 3) beside f32 V rows: the K side of the planar
    // kernel, the V side of the f32 one; q is rotated into the K rows' basis, the output is not rotated back.
    static_assert(!VF32 || BITS == 4 || BITS == 3, "VF32 goes with 4- or 3-bit K rows");
    constexpr bool kVRows32 = kF32 || VF32;   // V rows are floats
    constexpr bool kVPlanar = !kRaw && !VF32; // V rows are planar: a norm per row, the output is rotated back
    constexpr int kRowBytes = kF16 ? 512 : kF32 ? 1024 : 32 * BITS;  // (K rows; f32 V rows are 1024 bytes)
    // lo tiles: the rounding remainders of the 4-bit table (see bk_prefill.cu: it is only good to 1e-4), the lo parts
    // of f32 rows; beside raw V rows (several times larger than dequantized ones) the 3-bit table carries them too
    constexpr bool kLoTiles = BITS == 4 || kF32 || VF32;

    constexpr int kRun = kLoTiles ? 16 : 20;  // tiles that O collects, at most, before it is added up in f32 (see collect_o)

    // ---- which item (as in the mma.sync kernel) ---------------------------------------------
    const int item = blockIdx.x;
    // the blocks late in the prompt see the most rows: they go first
    const int chunk = item % pa.n_chunks, kv = (item / pa.n_chunks) % a.n_kv, blk = pa.n_blocks - 1 - item / (pa.n_chunks * a.n_kv);
    const int tok0 = blk * pa.tq, n_tok = min(pa.tq, pa.n_tokens - tok0), n_rows = n_tok * NREP;
    const int vis = pa.pos0 + tok0 + n_tok;
    const int L = ((vis + pa.n_chunks - 1) / pa.n_chunks + kTK - 1) / kTK * kTK;
    const int c0 = chunk * L, c1 = min(c0 + L, vis);
    const int n_tiles = c1 > c0 ? (c1 - c0 + kTK - 1) / kTK : 0;
    const int n_runs = (n_tiles + kRun - 1) / kRun, run_len = n_runs > 1 ? (n_tiles + n_runs - 1) / n_runs : kRun;

    // ---- the query rows start travelling: every row's round trip at once -----------------------------------
    const int half = a.n_rot >> 1;
    {
        const float *q0 = a.q + ((size_t)tok0 * a.n_head + kv * NREP) * kHd;
        auto row_src = [&](int r) { return q0 + ((size_t)(r / NREP) * a.n_head + r % NREP) * kHd; };
        if (((uintptr_t)a.q & 15) == 0) {
            for (int i = tid; i < n_rows * (kHd / 4); i += kUT)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(base + oSlots + 16u * i), "l"(row_src(i / (kHd / 4)) + 4 * (i % (kHd / 4)))
                             : "memory");
        } else {
            for (int i = tid; i < n_rows * kHd; i += kUT)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(base + oSlots + 4u * i), "l"(row_src(i / kHd) + i % kHd) : "memory");
        }
    }

    // ---- tables, barriers, tensor memory ----------------------------------------------------
    for (int i = tid; i < kHd; i += kUT) ss.givens[i] = a.givens[i];
    auto bar_at = [&](size_t off, int i) { return small + (uint32_t)off + 8u * (uint32_t)i; };
    const uint32_t bar_full = bar_at(offsetof(SmallU, full), 0), bar_empty = bar_at(offsetof(SmallU, empty), 0),
                   bar_norms = bar_at(offsetof(SmallU, norms), 0), bar_s = bar_at(offsetof(SmallU, s_full), 0),
                   bar_p = bar_at(offsetof(SmallU, p_full), 0), bar_o = bar_at(offsetof(SmallU, o_done), 0),
                   bar_drain = bar_at(offsetof(SmallU, drain), 0);
    if (tid == 0) {
        for (int i = 0; i < kSlots; i++) {
            mbar_init(bar_full + 8 * i, kF16 ? 1 : kProdWarps);
            mbar_init(bar_empty + 8 * i, 1);
        }
        for (int i = 0; i < kNormTiles; i++) mbar_init(bar_norms + 8 * i, 2);
        for (int i = 0; i < 2; i++) {
            mbar_init(bar_s + 8 * i, 1);
            mbar_init(bar_p + 8 * i, kSoftWarps);
            mbar_init(bar_o + 8 * i, 1);
        }
        mbar_init(bar_drain, 1);
        ss.gave_up = 0;
        ss.run_slot = 0;
        if (n_runs > 1) {
            // a place for the sums: there are as many as SMs, a CTA fills an SM and gives its place back at its end, so one is free
            uint32_t i;
            asm("mov.u32 %0, %%smid;\n" : "=r"(i));
            int tries = 0;
            for (i %= (uint32_t)pa.n_runs; atomicExch(pa.runs_taken + i, 1) != 0; i = i + 1 == (uint32_t)pa.n_runs ? 0 : i + 1)
                if (++tries > kWaitPolls) {  // (never expected)
                    ss.gave_up = 1;
                    raise_error(pa.err_flag, 4);
                    break;
                }
            __threadfence();
            ss.run_slot = (int)i;
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 0) tmem_alloc(small + (uint32_t)offsetof(SmallU, tmem_slot), kTmemCols);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, ss.tmem_slot, 0);
    auto run_sums = [&]() { return reinterpret_cast<float4 *>(pa.runs + (size_t)ss.run_slot * kRunFloats); };
    float *run_mul = reinterpret_cast<float *>(sm + oQlo);  // [row], where q_lo was: the runs' factor at the end
    const uint32_t my_tmem = tmem + ((uint32_t)((warp & 3) * 32) << 16);  // this warp's 32 lanes

    // bounded wait; after one has run out (never expected) the others of the CTA do not start to wait
    auto wait = [&](uint32_t bar, uint32_t parity) -> bool {
        volatile int *gave_up = &ss.gave_up;
        int polls = 0;
        while (!mbar_try_wait(bar, parity)) {
            if (*gave_up) return false;
            if (++polls > kWaitPolls) {
                *gave_up = 1;
                raise_error(pa.err_flag, 4);
                return false;
            }
        }
        return true;
    };

    // ---- a producer thread's share of a packed tile: position pt / 8, coordinates 32 (pt % 8) .. + 31 ------
    const int pt = (tid - 32 * kSoftWarps) & 255, my_row = pt >> 3, my_c = pt & 7, rot = my_c >> 1;
    const bool producer = warp >= kSoftWarps && warp < kMmaWarp;
    const size_t seq_rows = (size_t)pa.seq * a.seq_stride_rows;
    auto row_of = [&](int tile, int r) {  // rows past the cache's end are never used: any row of it will do
        return seq_rows + (size_t)min(c0 + tile * kTK + r, a.n_ctx - 1) * a.n_kv + kv;
    };
    uint32_t pk[4], pv[4];  // packed K of one tile and packed V of the tile before, on their way
    float pn = 0.f;
    // f32 rows: the thread's 128 bytes, its four 16-byte operand pieces in the lane's order
    [[maybe_unused]] float4 fk[kF32 ? 8 : 1], fv[kVRows32 ? 8 : 1];
    auto fetch_f32 = [&](float4 *dst, const uint8_t *rows, int tile) {
        const float4 *src = reinterpret_cast<const float4 *>(rows + row_of(tile, my_row) * 1024) + 8 * my_c;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            dst[2 * j] = __ldg(src + 2 * ((j + rot) & 3));
            dst[2 * j + 1] = __ldg(src + 2 * ((j + rot) & 3) + 1);
        }
    };
    auto fetch_packed = [&](uint32_t (&w)[4], const uint8_t *rows, int tile) {
        const uint8_t *p = rows + row_of(tile, my_row) * kRowBytes;
        if constexpr (BITS == 4) {
            const uint4 x = __ldg(reinterpret_cast<const uint4 *>(p) + my_c);
            w[0] = x.x, w[1] = x.y, w[2] = x.z, w[3] = x.w;
        } else if constexpr (BITS == 3) {
            const uint32_t *p3 = reinterpret_cast<const uint32_t *>(p) + 3 * my_c;
            w[0] = __ldg(p3), w[1] = __ldg(p3 + 1), w[2] = __ldg(p3 + 2), w[3] = 0;
        } else {  // 2 bit: 32 coordinates are 8 bytes
            const uint2 x = __ldg(reinterpret_cast<const uint2 *>(p) + my_c);
            w[0] = x.x, w[1] = x.y, w[2] = w[3] = 0;
        }
    };
    auto fetch_k = [&](int tile) {
        if constexpr (kF32) {
            fetch_f32(fk, a.k_rows, tile);
        } else if constexpr (!kF16) {
            fetch_packed(pk, a.k_rows, tile);
            if (pt < (VF32 ? kTK : 2 * kTK)) pn = __ldg((pt < kTK ? a.k_norms : a.v_norms) + row_of(tile, pt & (kTK - 1)));
        }
    };
    auto fetch_v = [&](int tile) {
        if constexpr (kVRows32) fetch_f32(fv, a.v_rows, tile);
        else if constexpr (!kF16) fetch_packed(pv, a.v_rows, tile);
    };

    // ---- q rows -> q_hi and q_lo: rope, Givens, scale, f16 hi/lo; a warp takes a row, the 32 bytes of a lane are coordinates
    // 8 lane .. + 7; the half of q_hi for tensor memory goes where the row was ---------------------------------------
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    {
        const float qscale = rsqrtf((float)kHd) * 1.4426950408889634f / pa.lut_alpha;
        // the rope entries of the warp's next two rows travel (up to 32 per row; wider rotations read the rest where they need it)
        auto rope_row = [&](int r) { return a.rope + (size_t)(pa.pos0 + tok0 + r / NREP) * half; };
        auto rope_of = [&](int r) { return r < n_rows && lane < half ? __ldg(rope_row(r) + lane) : make_float2(1.f, 0.f); };
        float2 c0r = rope_of(warp), c1r = rope_of(warp + kUWarps);
        for (int r = warp; r < kRows; r += kUWarps) {
            float *row = reinterpret_cast<float *>(sm + oSlots) + r * kHd;
            uint32_t hw[4] = {}, lw[4] = {};
            const float2 c2r = rope_of(r + 2 * kUWarps);
            if (r < n_rows) {
                for (int j = lane; j < half; j += 32) {
                    float x0 = row[j], x1 = row[j + half];
                    rope_pair(x0, x1, j < 32 ? c0r : __ldg(rope_row(r) + j));
                    row[j] = x0;
                    row[j + half] = x1;
                }
                __syncwarp();
                const float4 x0 = reinterpret_cast<const float4 *>(row)[2 * lane], x1 = reinterpret_cast<const float4 *>(row)[2 * lane + 1];
                const float x[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll
                for (int p = 0; p < 4; p++) {
                    float o0 = x[2 * p], o1 = x[2 * p + 1];
                    if constexpr (!kRaw) {
                        const int d = 8 * lane + 2 * p;
                        givens_fwd(x[2 * p], x[2 * p + 1], ss.givens[d], ss.givens[d + 1], o0, o1);
                    }
                    o0 *= qscale;
                    o1 *= qscale;
                    const __half h0 = __float2half_rn(o0), h1 = __float2half_rn(o1);
                    const __half l0 = __float2half_rn(o0 - __half2float(h0)), l1 = __float2half_rn(o1 - __half2float(h1));
                    hw[p] = (uint32_t)__half_as_ushort(h0) | ((uint32_t)__half_as_ushort(h1) << 16);
                    lw[p] = (uint32_t)__half_as_ushort(l0) | ((uint32_t)__half_as_ushort(l1) << 16);
                }
                __syncwarp();
            }
            c0r = c1r;
            c1r = c2r;
            uint4 *hi = lane < 16 ? reinterpret_cast<uint4 *>(row) + (lane ^ (r & 7)) : reinterpret_cast<uint4 *>(sm + oQhi2 + sw_off(kRows, r, lane - 16));
            *hi = make_uint4(hw[0], hw[1], hw[2], hw[3]);
            *reinterpret_cast<uint4 *>(sm + oQlo + sw_off(kRows, r, lane)) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
        }
    }
    fence_smem_to_async_proxy();
    __syncthreads();
    const int my_q = (warp & 3) * 32 + lane;  // query row of a softmax thread
    if (warp < kSoftWarps) {
#pragma unroll
        for (int b = 0; b < 2; b++) {
            uint32_t r[32];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const uint4 x = reinterpret_cast<const uint4 *>(sm + oSlots + my_q * (kHd * 4))[(8 * b + j) ^ (my_q & 7)];
                r[4 * j] = x.x, r[4 * j + 1] = x.y, r[4 * j + 2] = x.z, r[4 * j + 3] = x.w;
            }
            tmem_st32(my_tmem + kColQ + 32 * b, r);
        }
        tmem_wait_st();
        fence_smem_to_async_proxy();  // (f16: the TMA engine writes where q_hi was read)
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();

    float R = -CUDART_INF_F, lsum = 0.f;  // a query row's running reference and sum
    if (warp == kMmaWarp) {
        // ---- the products -----------------------------------------------------------------------------------
        constexpr int kKRows = kLoTiles ? 64 : 32;  // a K slab holds k_hi in rows 0-31 and k_lo in rows 32-63
        constexpr uint32_t kKSlab = kKRows * 128;
        const uint32_t idesc_s = umma_idesc_f16(kRows, kTK, 0, 0), idesc_s2 = umma_idesc_f16(kRows, kKRows, 0, 0), idesc_o = umma_idesc_f16(kRows, kHd, 0, 1);
        uint32_t slot = 0, use = 0;
        auto next_slot = [&]() {
            if (++slot == kSlots) slot = 0, use ^= 1u;
        };
        auto issue_s = [&](int tile) -> bool {
            if (!__all_sync(0xffffffffu, wait(bar_full + 8 * slot, use))) return false;
            tc_fence_after_sync();
            // columns 0-31: q_hi k_hi; 32-63: the small terms
            const uint32_t d = tmem + kColS + (uint32_t)(tile & 1) * 64u, kb = base + oSlots + slot * kSlotBytes;
            const uint64_t kd = umma_smem_desc(kb, 16, 1024, kUmmaSwizzle128), ql = umma_smem_desc(base + oQlo, 16, 1024, kUmmaSwizzle128);
            const uint64_t qh2 = umma_smem_desc(base + oQhi2, 16, 1024, kUmmaSwizzle128);
            if (elect_one()) {  // (the address field of a descriptor counts 16-byte units)
#pragma unroll
                for (int ks = 0; ks < 8; ks++)
                    umma_f16_ts(d, tmem + kColQ + 8 * ks, kd + (((ks >> 2) * kKSlab + (ks & 3) * 32) >> 4), idesc_s2, ks > 0);
#pragma unroll
                for (int ks = 8; ks < 16; ks++)
                    umma_f16_ss(d, qh2 + ((((ks >> 2) - 2) * kQSlab + (ks & 3) * 32) >> 4), kd + (((ks >> 2) * kKSlab + (ks & 3) * 32) >> 4), idesc_s2, true);
#pragma unroll
                for (int ks = 0; ks < 16; ks++)
                    umma_f16_ss(d + 32, ql + (((ks >> 2) * kQSlab + (ks & 3) * 32) >> 4), kd + (((ks >> 2) * kKSlab + (ks & 3) * 32) >> 4), idesc_s,
                                kLoTiles || ks > 0);
                umma_commit(bar_s + 8 * (tile & 1));
                umma_commit(bar_empty + 8 * slot);
            }
            __syncwarp();
            next_slot();
            return true;
        };
        bool ok = n_tiles == 0 || issue_s(0);
        int run_start = 0;
        for (int tile = 0; ok && tile < n_tiles; tile++) {
            // (S(tile + 1) goes where S(tile - 1) was, which the softmax had read when P(tile - 1) was awaited)
            if (tile + 1 < n_tiles && !issue_s(tile + 1)) break;
            ok = wait(bar_full + 8 * slot, use);
            ok = ok && wait(bar_p + 8 * (tile & 1), (uint32_t)(tile >> 1) & 1u);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after_sync();
            const uint32_t p = tmem + kColP + (uint32_t)(tile & 1) * 32u, vb = base + oSlots + slot * kSlotBytes;
            const uint64_t vd = umma_smem_desc(vb, kKVSlab, 1024, kUmmaSwizzle128);
            if (elect_one()) {
#pragma unroll
                for (int kk = 0; kk < 2; kk++) {
                    umma_f16_ts(tmem + kColO, p + 16 * kk, vd + ((kk * 2048) >> 4), idesc_o, tile != run_start || kk > 0);
                    umma_f16_ts(tmem + kColO, p + 16 * kk + 8, vd + ((kk * 2048) >> 4), idesc_o, true);
                    if constexpr (kLoTiles) umma_f16_ts(tmem + kColO, p + 16 * kk, vd + ((kKVTile + kk * 2048) >> 4), idesc_o, true);
                }
                umma_commit(bar_o + 8 * (tile & 1));
                umma_commit(bar_empty + 8 * slot);
            }
            __syncwarp();
            if (tile == run_start) run_start += run_len;
            next_slot();
        }
        // nothing in flight is left behind, whatever happened above
        if (elect_one()) umma_commit(bar_drain);
        __syncwarp();
        for (int polls = 0; !mbar_try_wait(bar_drain, 0) && polls < kWaitPolls; polls++) {}
    } else if (producer) {
        // ---- operand tiles ------------------------------------------------------------------------------------
        uint32_t slot = 0, use = 0;
        auto next_slot = [&]() {
            if (++slot == kSlots) slot = 0, use++;
        };
        auto slot_free = [&]() { return use == 0 || wait(bar_empty + 8 * slot, (use - 1) & 1u); };
        if constexpr (kF16) {
            if (warp == kSoftWarps) {
                // a tile that is whole: 8 boxes of 16 rows x 128 bytes by the TMA engine; the last one when rows of it are past
                // the chunk's end (they may hold anything, and 0 * Inf would poison the accumulators): by the warp, with zeros
                auto put = [&](int tile, const CUtensorMap *map, const uint8_t *rows) -> bool {
                    if (!__all_sync(0xffffffffu, slot_free())) return false;
                    const int valid = c1 - (c0 + tile * kTK);
                    const uint32_t bar = bar_full + 8 * slot, dst = base + oSlots + slot * kSlotBytes;
                    if (valid >= kTK) {
                        if (elect_one()) {
                            mbar_expect_tx(bar, kKVTile);
                            const int gpos = a.layer_pos0 + pa.seq * a.n_ctx + c0 + tile * kTK;
#pragma unroll
                            for (int sl = 0; sl < 4; sl++)
#pragma unroll
                                for (int hf = 0; hf < 2; hf++) tma_tile_x(dst + sl * kKVSlab + hf * 2048, map, sl * 128, kv, gpos + 16 * hf, bar);
                        }
                    } else {
                        for (int r = 0; r < kTK; r++) {
                            uint4 x = make_uint4(0, 0, 0, 0);
                            if (r < valid) x = __ldg(reinterpret_cast<const uint4 *>(rows + row_of(tile, r) * 512) + lane);
                            *reinterpret_cast<uint4 *>(sm + oSlots + slot * kSlotBytes + sw_off(kTK, r, lane)) = x;
                        }
                        fence_smem_to_async_proxy();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar);
                    }
                    __syncwarp();
                    next_slot();
                    return true;
                };
                bool ok = n_tiles == 0 || put(0, &tm_k, a.k_rows);
                for (int tile = 0; ok && tile < n_tiles; tile++) {
                    if (tile + 1 < n_tiles) ok = put(tile + 1, &tm_k, a.k_rows);
                    ok = ok && put(tile, &tm_v, a.v_rows);
                }
                if (!ok) {  // gave up: leave no copy in flight behind (every slot that was filled before this one)
                    const uint32_t filled = use * kSlots + slot;
                    for (uint32_t i = filled > kSlots ? filled - kSlots : 0; i < filled; i++) {
                        int polls = 0;
                        while (!mbar_try_wait(bar_full + 8 * (i % kSlots), (i / kSlots) & 1u) && ++polls < kWaitPolls) {}
                    }
                }
            }
        } else {
            const float cent = kRaw ? 0.f : a.book[lane & ((1 << (kRaw ? 4 : BITS)) - 1)] * pa.lut_alpha;
            const __half cent_hi = __float2half_rn(cent);
            const uint32_t tab = (uint32_t)__half_as_ushort(cent_hi) | ((uint32_t)__half_as_ushort(__float2half_rn(cent - __half2float(cent_hi))) << 16);
            // split the fetched floats into f16 hi + lo and store both as four 16-byte chunks of a tile row; rows at or past
            // the chunk's end are stored as zeros (they may hold anything, and 0 * Inf would poison the accumulators)
            auto split_store = [&](const float4 *f, uint8_t *tile_hi, uint8_t *tile_lo, int rows, int row_lo, bool live) {
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float x[8] = {f[2 * j].x, f[2 * j].y, f[2 * j].z, f[2 * j].w, f[2 * j + 1].x, f[2 * j + 1].y, f[2 * j + 1].z, f[2 * j + 1].w};
                    uint32_t h[4], l[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const float x0 = live ? x[2 * e] : 0.f, x1 = live ? x[2 * e + 1] : 0.f;
                        const __half2 hv = __floats2half2_rn(x0, x1);
                        const float2 hf = __half22float2(hv);
                        const __half2 lv = __floats2half2_rn(x0 - hf.x, x1 - hf.y);
                        h[e] = *reinterpret_cast<const uint32_t *>(&hv);
                        l[e] = *reinterpret_cast<const uint32_t *>(&lv);
                    }
                    const int ch = 4 * my_c + ((j + rot) & 3);
                    *reinterpret_cast<uint4 *>(tile_hi + sw_off(rows, my_row, ch)) = make_uint4(h[0], h[1], h[2], h[3]);
                    *reinterpret_cast<uint4 *>(tile_lo + sw_off(rows, row_lo, ch)) = make_uint4(l[0], l[1], l[2], l[3]);
                }
            };
            auto widen = [&](uint32_t (&w)[4]) {
                if constexpr (BITS == 3) {
                    const uint32_t u0 = w[0], u1 = w[1], u2 = w[2];
                    w[0] = expand24u(u0);
                    w[1] = expand24u(__funnelshift_r(u0, u1, 24));
                    w[2] = expand24u(__funnelshift_r(u1, u2, 16));
                    w[3] = expand24u(u2 >> 8);
                } else if constexpr (BITS == 2) {  // sixteen indices per word -> two words of eight nibbles
                    const uint32_t u0 = w[0], u1 = w[1];
                    w[0] = expand16u(u0);
                    w[1] = expand16u(u0 >> 16);
                    w[2] = expand16u(u1);
                    w[3] = expand16u(u1 >> 16);
                }
                rotate4(w, rot);
            };
            auto put_done = [&]() {
                fence_smem_to_async_proxy();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_full + 8 * slot);
                next_slot();
            };
            auto live = [&](int tile) { return c0 + tile * kTK + my_row < c1; };
            auto put_k = [&](int tile) -> bool {
                if (!__all_sync(0xffffffffu, slot_free())) return false;  // one answer for the warp, also when a wait runs out
                uint8_t *dst = sm + oSlots + slot * kSlotBytes;
                if constexpr (kF32) {
                    split_store(fk, dst, dst, 64, my_row + 32, live(tile));
                } else {
                    widen(pk);
                    dequant_store_shfl<kLoTiles>(pk, tab, dst, dst, kLoTiles ? 64 : 32, my_row, my_row + 32, 4 * my_c, rot);
                    if (pt < 2 * kTK) {
                        if (pt < kTK) ss.kn[tile % kNormTiles][pt] = pn;
                        else ss.lv[tile % kNormTiles][pt - kTK] = VF32 ? 0.f : fast_log2(fmaxf(pn, 1e-30f));
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar_norms + 8 * (tile % kNormTiles));
                    }
                }
                put_done();
                if (tile + 1 < n_tiles) fetch_k(tile + 1);
                return true;
            };
            auto put_v = [&](int tile) -> bool {
                if (!__all_sync(0xffffffffu, slot_free())) return false;  // one answer for the warp, also when a wait runs out
                uint8_t *dst = sm + oSlots + slot * kSlotBytes;
                if constexpr (kVRows32) {
                    split_store(fv, dst, dst + kKVTile, kTK, my_row, live(tile));
                } else {
                    widen(pv);
                    dequant_store_shfl<kLoTiles>(pv, tab, dst, dst + kKVTile, kTK, my_row, my_row, 4 * my_c, rot);
                }
                put_done();
                if (tile + 1 < n_tiles) fetch_v(tile + 1);
                return true;
            };
            if (n_tiles > 0) fetch_k(0), fetch_v(0);
            bool ok = n_tiles == 0 || put_k(0);
            for (int tile = 0; ok && tile < n_tiles; tile++) {
                if (tile + 1 < n_tiles) ok = put_k(tile + 1);
                ok = ok && put_v(tile);
            }
        }
    } else {
        // ---- softmax: thread = query row ------------------------------------------------------------------------
        const int lim = my_q < n_rows ? pa.pos0 + tok0 + my_q / NREP + 1 : 0;
        float run_R = -CUDART_INF_F;  // the reference of the sums of the runs done
        int run_start = 0;
        // O collects a run of tiles, joins the sums of the runs before, rounded to nearest, and starts again: its adds truncate at the
        // size of what it holds, so its error grows with the tiles it collects.  Against float64, channels with x20 outliers: 777
        // tokens into an f32 cache 1.36e-6 of the result (1.69e-6 without runs, 1.49e-6 with runs of up to 20 tiles), 4608 in blocks
        // of 512 2.0e-6 (3.5e-6, 2.2e-6); V of one sign, 4608 tokens, 2.8e-6 (7.9e-6).  Without lo tiles a run may be longer: fewer
        // products.  The sums stay in L2; a launch pays 5 us for the first and the last pass over them and 4 for each between: the
        // 4608 tokens 6.2 -> 6.7 ms (four layers), 777 tokens 287 -> 309 us.  The same by shorter chunks: 7.1 ms and 341 us.
        auto collect_o = [&](bool first) {
            const float f = run_R > -CUDART_INF_F ? fast_exp2(run_R - R) : 0.f;
            for (int b = 0; b < 8; b++) {
                float4 *at = run_sums() + (8 * b) * kRows + my_q;
                float4 old[8];
#pragma unroll
                for (int j = 0; j < 8; j++) old[j] = first ? make_float4(0.f, 0.f, 0.f, 0.f) : __ldcg(at + j * kRows);
                uint32_t o[32];
                tmem_ld32(my_tmem + kColO + 32 * b, o);
#pragma unroll
                for (int j = 0; j < 8; j++)
                    __stcg(at + j * kRows, make_float4(fmaf(old[j].x, f, __uint_as_float(o[4 * j])), fmaf(old[j].y, f, __uint_as_float(o[4 * j + 1])),
                                                       fmaf(old[j].z, f, __uint_as_float(o[4 * j + 2])), fmaf(old[j].w, f, __uint_as_float(o[4 * j + 3]))));
            }
            run_R = R;
        };
        for (int tile = 0; tile < n_tiles; tile++) {
            const uint32_t buf = (uint32_t)tile & 1u, par = (uint32_t)(tile >> 1) & 1u;
            if (tile == run_start && tile > 0) {  // (the next product, which starts O again, waits for this tile's weights)
                if (!__all_sync(0xffffffffu, wait(bar_o + 8 * (buf ^ 1u), (uint32_t)((tile - 1) >> 1) & 1u))) break;
                tc_fence_after_sync();
                collect_o(tile == run_len);
            }
            bool ok = wait(bar_s + 8 * buf, par);
            if constexpr (!kRaw) ok = ok && wait(bar_norms + 8 * (tile % kNormTiles), (uint32_t)(tile / kNormTiles) & 1u);
            if (tile >= 2) ok = ok && wait(bar_o + 8 * buf, par ^ 1u);  // P of two tiles ago has been used
            if (!__all_sync(0xffffffffu, ok)) break;
            tc_fence_after_sync();
            uint32_t sr[32], t[32];
            tmem_ld32(my_tmem + kColS + 64 * buf, sr);
            tmem_ld32(my_tmem + kColS + 64 * buf + 32, t);
            const float *kn = ss.kn[tile % kNormTiles], *lv = ss.lv[tile % kNormTiles];
            float mx = -CUDART_INF_F;
#pragma unroll
            for (int j = 0; j < 32; j++) {
                float s = __uint_as_float(sr[j]) + __uint_as_float(t[j]);
                if constexpr (!kRaw) s *= kn[j];
                sr[j] = __float_as_uint(s);
                t[j] = __float_as_uint(kVPlanar ? s + lv[j] : s);
            }
            const int n_ok = min(c1, lim) - (c0 + tile * kTK);  // positions of the tile that this row sees
            if (!__all_sync(0xffffffffu, n_ok >= kTK)) {
#pragma unroll
                for (int j = 0; j < 32; j++)
                    if (j >= n_ok) sr[j] = t[j] = __float_as_uint(-CUDART_INF_F);
            }
#pragma unroll
            for (int j = 0; j < 32; j++) mx = fmaxf(mx, __uint_as_float(t[j]));
            // lazy reference: move it only when this row's maximum ran ahead by more than kLazy
            const bool move = mx > -CUDART_INF_F && (R == -CUDART_INF_F || mx > R + kLazy);
            if (__any_sync(0xffffffffu, move)) {  // tensor-memory traffic is warp-collective
                const float newR = move ? mx : R;
                const float f = (move && R > -CUDART_INF_F) ? fast_exp2(R - newR) : (move ? 0.f : 1.f);
                lsum *= f;
                if (tile != run_start) {  // (the first product of a run does not add to O)
                    if (!__all_sync(0xffffffffu, wait(bar_o + 8 * (buf ^ 1u), (uint32_t)((tile - 1) >> 1) & 1u))) break;
                    tc_fence_after_sync();
                    for (int b = 0; b < 16; b++) {
                        uint32_t o[16];
                        tmem_ld16(my_tmem + kColO + 16 * b, o);
#pragma unroll
                        for (int j = 0; j < 16; j++) o[j] = __float_as_uint(__uint_as_float(o[j]) * f);
                        tmem_st16(my_tmem + kColO + 16 * b, o);
                    }
                }
                R = newR;
            }
            const float ref = (R > -CUDART_INF_F ? R : 0.f) - kPScaleLog2;
            // weights, two positions a column: for each K-step of 16 positions eight columns of hi parts and eight of lo parts;
            // lsum carries their scale
#pragma unroll
            for (int kk = 0; kk < 2; kk++) {
                uint32_t pw[16];
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    const int j = 16 * kk + 2 * e;
                    const float w0 = fast_exp2(__uint_as_float(t[j]) - ref), w1 = fast_exp2(__uint_as_float(t[j + 1]) - ref);
                    if constexpr (kVPlanar) {
                        lsum += fast_exp2(__uint_as_float(sr[j]) - ref);
                        lsum += fast_exp2(__uint_as_float(sr[j + 1]) - ref);
                    } else {
                        lsum += w0;
                        lsum += w1;
                    }
                    const __half2 h = __floats2half2_rn(w0, w1);
                    const float2 hf = __half22float2(h);
                    const __half2 l = __floats2half2_rn(w0 - hf.x, w1 - hf.y);
                    pw[e] = *reinterpret_cast<const uint32_t *>(&h);
                    pw[8 + e] = *reinterpret_cast<const uint32_t *>(&l);
                }
                tmem_st16(my_tmem + kColP + 32 * buf + 16 * kk, pw);
            }
            if (tile == run_start) run_start += run_len;
            tmem_wait_st();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_p + 8 * buf);
        }
        const float unscale = 1.0f / (kPScale * (kVPlanar ? pa.lut_alpha : 1.0f));  // (raw V rows carry no table scale)
        lsum *= 1.0f / kPScale;
        if (n_runs > 1) run_mul[my_q] = run_R > -CUDART_INF_F ? fast_exp2(run_R - R) : 0.f;
        ss.mul[my_q] = pa.n_chunks == 1 ? (lsum > 0.f ? unscale / lsum : 0.f) : unscale;
        if (pa.n_chunks > 1 && my_q < n_rows) {
            float *dst = pa.scratch + (((size_t)(tok0 + my_q / NREP) * a.n_head + kv * NREP + my_q % NREP) * pa.n_chunks + chunk) * (kHd + 2);
            dst[kHd] = R;
            dst[kHd + 1] = lsum;
        }
    }
    tc_fence_before_sync();
    __syncthreads();  // (the issuing warp has seen all its products complete)
    tc_fence_after_sync();

    // ---- epilogue: warps 0-11, 32 query rows x 32 columns at a time through a padded shared-memory block, so that the
    // global stores of a warp cover one row's 128 bytes instead of 32 rows' 8 bytes
    if (warp < kMmaWarp) {
        const bool whole = pa.n_chunks == 1;
        const float mul = ss.mul[my_q], rmul = n_runs > 1 ? run_mul[my_q] : 0.f;
        float *stg = reinterpret_cast<float *>(sm + oSlots) + warp * (32 * 33);
        const int wrow0 = (warp & 3) * 32;
        for (int b = warp >> 2; b < 8; b += 3) {
            uint32_t o[32];
            tmem_ld32(my_tmem + kColO + 32 * b, o);
            if (n_runs > 1) {
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const float4 x = __ldcg(run_sums() + (8 * b + j) * kRows + my_q);
                    o[4 * j] = __float_as_uint(fmaf(x.x, rmul, __uint_as_float(o[4 * j])));
                    o[4 * j + 1] = __float_as_uint(fmaf(x.y, rmul, __uint_as_float(o[4 * j + 1])));
                    o[4 * j + 2] = __float_as_uint(fmaf(x.z, rmul, __uint_as_float(o[4 * j + 2])));
                    o[4 * j + 3] = __float_as_uint(fmaf(x.w, rmul, __uint_as_float(o[4 * j + 3])));
                }
            }
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
                const int d = 32 * b + j;
                float o0 = n_tiles > 0 ? __uint_as_float(o[j]) * mul : 0.f, o1 = n_tiles > 0 ? __uint_as_float(o[j + 1]) * mul : 0.f;
                if (whole && kVPlanar) {
                    float r0, r1;
                    givens_inv(o0, o1, ss.givens[d], ss.givens[d + 1], r0, r1);
                    o0 = r0;
                    o1 = r1;
                }
                stg[lane * 33 + j] = o0;
                stg[lane * 33 + j + 1] = o1;
            }
            __syncwarp();
            for (int rr = 0; rr < 32; rr++) {
                const int q = wrow0 + rr;
                if (q >= n_rows) break;
                const size_t orow = (size_t)(tok0 + q / NREP) * a.n_head + kv * NREP + q % NREP;
                float *drow = whole ? a.out + orow * kHd : pa.scratch + (orow * pa.n_chunks + chunk) * (kHd + 2);
                drow[32 * b + lane] = stg[rr * 33 + lane];
            }
            __syncwarp();
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (tid == 0 && n_runs > 1) {
        __threadfence();
        atomicExch(pa.runs_taken + ss.run_slot, 0);
    }
    if (warp == 0) tmem_dealloc(tmem, kTmemCols);
}

// Merge the chunks' triples, rotate back, write: a warp per output row, so that the references and sums of up to 64 chunks
// are one or two loads and the rows' loads do not wait for them.  A chunk that the row does not see counts as zeros whatever it holds.
constexpr int kMergeWarps = 8;
__global__ void __launch_bounds__(kMergeWarps * 32) prefill_umma_merge_kernel(const float *scratch, const float *givens, int n_chunks, int n_out, float *out) {
    const int row = blockIdx.x * kMergeWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= n_out) return;
    const float *basep = scratch + (size_t)row * n_chunks * (kHd + 2);
    float m[2], f[2], l[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int c = lane + 32 * h;
        m[h] = c < n_chunks ? basep[(size_t)c * (kHd + 2) + kHd] : -CUDART_INF_F;
        l[h] = c < n_chunks ? basep[(size_t)c * (kHd + 2) + kHd + 1] : 0.f;
    }
    float M = fmaxf(m[0], m[1]);
    for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
    float Ls = 0.f;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        f[h] = m[h] > -CUDART_INF_F ? exp2f(m[h] - M) : 0.f;
        if (f[h] > 0.f) Ls = fmaf(l[h], f[h], Ls);
    }
    for (int o = 16; o > 0; o >>= 1) Ls += __shfl_xor_sync(0xffffffffu, Ls, o);
    float2 acc[4] = {};  // coordinates 2 lane, 2 lane + 1 of each quarter
#pragma unroll 4
    for (int c = 0; c < n_chunks; c++) {
        const float2 *p = reinterpret_cast<const float2 *>(basep + (size_t)c * (kHd + 2)) + lane;
        const float fc = __shfl_sync(0xffffffffu, c < 32 ? f[0] : f[1], c & 31);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float2 v = p[32 * i];
            acc[i].x = fmaf(fc > 0.f ? v.x : 0.f, fc, acc[i].x);
            acc[i].y = fmaf(fc > 0.f ? v.y : 0.f, fc, acc[i].y);
        }
    }
    const float inv = Ls > 0.f ? 1.0f / Ls : 0.f;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int d = 64 * i + 2 * lane;
        float o0 = acc[i].x * inv, o1 = acc[i].y * inv;
        if (givens) {  // planar V only
            float r0, r1;
            givens_inv(o0, o1, givens[d], givens[d + 1], r0, r1);
            o0 = r0;
            o1 = r1;
        }
        float *dst = out + (size_t)row * kHd + d;  // (the caller's alignment is only that of a float)
        dst[0] = o0;
        dst[1] = o1;
    }
}

template <int BITS, int NREP, bool VF32 = false>
bk_status launch_umma_one(bk_ctx *ctx, const PrefillUArgs &pa) {
    static std::atomic<bool> configured[64] = {};  // per device; racing first calls set the same attribute
    const int dev = ctx->device;
    if (dev < 0 || dev >= 64) return fail(ctx, BK_ERR_UNSUPPORTED, "prefill: device index above 63");
    if (!configured[dev].load()) {
        BK_CUDA(ctx, cudaFuncSetAttribute(prefill_umma_kernel<BITS, NREP, VF32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kUmmaSmem));
        configured[dev].store(true);
    }
    const int grid = pa.n_blocks * pa.d.n_kv * pa.n_chunks;
    if (!pa.d.h_tmap_k || !pa.d.h_tmap_v) return fail(ctx, BK_ERR_INVALID, "prefill: the cache has no tensor maps");
    prefill_umma_kernel<BITS, NREP, VF32><<<grid, kUT, kUmmaSmem, ctx->stream>>>(pa, *static_cast<const CUtensorMap *>(pa.d.h_tmap_k),
                                                                          *static_cast<const CUtensorMap *>(pa.d.h_tmap_v));
    ctx->launches++;
    BK_CUDA(ctx, cudaGetLastError());
    if (pa.n_chunks > 1) {
        const int n_out = pa.n_tokens * pa.d.n_head;
        prefill_umma_merge_kernel<<<(n_out + kMergeWarps - 1) / kMergeWarps, kMergeWarps * 32, 0, ctx->stream>>>(
            pa.scratch, (BITS == 16 || BITS == 32 || VF32) ? nullptr : pa.d.givens, pa.n_chunks, n_out, pa.d.out);
        ctx->launches++;
        BK_CUDA(ctx, cudaGetLastError());
    }
    return BK_OK;
}

}  // namespace

bool prefill_umma_supported(const DecodeArgs &a) {
    const int n_rep = a.n_kv > 0 ? a.n_head / a.n_kv : 0;
    const bool planar = a.k_kind == ROW_PLANAR && a.v_kind == ROW_PLANAR && (a.bits == 4 || a.bits == 3 || a.bits == 2);
    const bool f16 = a.k_kind == ROW_F16 && a.v_kind == ROW_F16 && a.k_row_bytes == 512 && a.v_row_bytes == 512;
    const bool f32 = a.k_kind == ROW_F32 && a.v_kind == ROW_F32 && a.k_row_bytes == 1024 && a.v_row_bytes == 1024;
    const bool k_only = a.k_kind == ROW_PLANAR && a.v_kind == ROW_F32 && (a.bits == 4 || a.bits == 3) && a.v_row_bytes == 1024;
    return (planar || f16 || f32 || k_only) && a.h_tmap_k && a.h_tmap_v && (n_rep == 1 || n_rep == 2 || n_rep == 4 || n_rep == 6);
}

// Into how many chunks the context is cut: the count with the least estimated time.  A CTA has an SM to itself and costs
// kFixed tiles' worth of set-up, q preparation and epilogue beside its tiles; what a launch then takes is bounded both by full rounds of its
// longest item and by its work spread evenly plus one longest item (items are handed out longest first).  Merging costs a
// launch and one read of every chunk's rows.
static int plan_chunks(int n_sms, int pos0, int n_tokens, int tq, int n_kv, int n_head) {
    constexpr double kFixed = 6.0, kMergeLaunch = 3.0, kMergeRow = 1.0 / 2048;
    const int n_blocks = (n_tokens + tq - 1) / tq, vis = pos0 + n_tokens;
    // no more than about four items per SM, which also bounds the scratch
    const int most = std::max(1, std::min({64, vis / 256, (4 * n_sms + n_blocks * n_kv - 1) / (n_blocks * n_kv)}));
    const double mean_vis = pos0 + 0.5 * (n_tokens + tq);
    double best = 0.0;
    int chunks = 1;
    for (int c = 1; c <= most; c++) {
        const double longest = kFixed + (double)((vis + c * kTK - 1) / (c * kTK)), items = (double)n_blocks * n_kv * c;
        const double mean = kFixed + std::max(1.0, mean_vis / (c * kTK));
        const double t = std::min(std::ceil(items / n_sms) * longest, items * mean / n_sms + longest) +
                         (c > 1 ? kMergeLaunch + kMergeRow * c * n_tokens * n_head / 24 : 0.0);
        if (c == 1 || t < best) {
            best = t;
            chunks = c;
        }
    }
    return chunks;
}

bk_status launch_prefill_umma(bk_ctx *ctx, const DecodeArgs &a, int seq, int pos0, int n_tokens, float alpha) {
    if (n_tokens <= 0) return BK_OK;
    const int n_rep = a.n_head / a.n_kv;
    PrefillUArgs pa{};
    pa.d = a;
    pa.seq = seq;
    pa.pos0 = pos0;
    pa.n_tokens = n_tokens;
    pa.tq = kRows / n_rep;
    pa.n_blocks = (n_tokens + pa.tq - 1) / pa.tq;
    pa.lut_alpha = alpha;
    pa.err_flag = ctx->d_err;
    const int chunks = plan_chunks(ctx->n_sms, pos0, n_tokens, pa.tq, a.n_kv, a.n_head);
    pa.n_chunks = chunks;
    pa.runs = ctx->d_prefill_runs;
    pa.runs_taken = reinterpret_cast<int *>(ctx->d_prefill_runs + ctx->n_sms * kRunFloats);
    pa.n_runs = ctx->n_sms;
    if (chunks > 1) {
        const size_t need = (size_t)n_tokens * a.n_head * chunks * (kHd + 2);
        if (ctx->d_prefill_floats < need) {
            BK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
            if (ctx->d_prefill) cudaFree(ctx->d_prefill);
            ctx->d_prefill = nullptr;
            ctx->d_prefill_floats = 0;
            BK_CUDA(ctx, cudaMalloc((void **)&ctx->d_prefill, need * sizeof(float)));
            ctx->d_prefill_floats = need;
        }
        pa.scratch = ctx->d_prefill;
    }
#define BK_PU_CASE(R)                                                                            \
    case R:                                                                                      \
        if (a.k_kind == ROW_F16) return launch_umma_one<16, R>(ctx, pa);                         \
        if (a.k_kind == ROW_F32) return launch_umma_one<32, R>(ctx, pa);                         \
        if (a.v_kind == ROW_F32) return a.bits == 3 ? launch_umma_one<3, R, true>(ctx, pa) : launch_umma_one<4, R, true>(ctx, pa); \
        if (a.bits == 2) return launch_umma_one<2, R>(ctx, pa);                                  \
        return a.bits == 3 ? launch_umma_one<3, R>(ctx, pa) : launch_umma_one<4, R>(ctx, pa);
    switch (n_rep) {
        BK_PU_CASE(1)
        BK_PU_CASE(2)
        BK_PU_CASE(4)
        BK_PU_CASE(6)
        default: return fail(ctx, BK_ERR_UNSUPPORTED, "prefill: n_head/n_kv must be 1, 2, 4 or 6");
    }
#undef BK_PU_CASE
}

}  // namespace bk
