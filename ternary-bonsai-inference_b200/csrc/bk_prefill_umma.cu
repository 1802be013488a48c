// Batched (prefill) attention over a 4-, 3- or 2-bit planar cache, or an f16 or f32 cache, on the
// 5th-generation tensor cores: the same work split and operands as bk_prefill.cu (which documents them and
// stays as the mma.sync form), with both contractions issued as tcgen05.mma and the accumulators in tensor memory.
//
// One CTA = 128 query rows (M = 128) of one kv head over a piece of the context they see, tile by tile of 32 positions.  What
// bounds it: for 4-bit and f32 rows six 128 x 32 x 256 products per tile (hi.hi, hi.lo, lo.hi twice), 1800 clocks of the tensor cores as
// issued, of a tile's 3260 clocks (f32 rows 4200, f16 and 3 bit 2650: from blocks of 512 tokens after 4096 and 16384 rows; 1.66 us at full clocks, long
// loops run into the power limit).  The tensor pipe is active for 47 % of them, tensor memory 52, shared memory about half, 44 % of the issue slots are
// taken: no unit is full, the roles wait for one another, so nothing may wait for anything else.  About 20 us of a launch lie beside the tiles.  Thirteen warps in three roles, coupled by mbarriers only:
//   * warps 4-11 (producers) turn packed rows into f16 operand tiles (for 4 bit with the rounding remainders, for
//     f32 rows hi + lo parts) in a ring of five slots, in the order of use: K0, K1, V0, K2, V1, ...  A thread's four
//     16-byte pieces of a packed row go out in an order that depends on its lane, or the eight lanes of a row would meet on
//     two of eight bank groups; of f32 rows a warp takes one at a time.  f16 rows are operands as stored and are dropped in by the TMA engine.
//   * warp 12 issues the products: S(t + 1) = Q . K^T goes ahead of O += P(t) . V, so the tensor cores work on S(t + 1)
//     under the softmax of tile t.  The small terms of S have columns of their own: the accumulator truncates, and does
//     so at the size of what it holds.
//   * warps 0-3 (thread = query row = tensor-memory lane) read S, scale by ||k||, apply the causal limit, move the
//     running reference of s + log2 ||v|| LAZILY (only when the row maximum has run ahead; their row of O is then rescaled in place) and
//     write the weights 2^(s - ref) ||v|| as f16 hi + lo.
// Tensor memory (all 512 columns): O 256 | q_hi 128 | S 2 x (32 + 32), where the weights (hi, lo) take the place of the scores.  A product
// with N = 32 costs as much as one with N = 64 (32 clocks), so q_hi meets k_hi and k_lo side by side; P and q_hi
// are A operands from tensor memory, which spares shared memory 4 KiB a product.
// Measured (4 layers, append included): a 4608-token planar4 prompt in blocks of 512 11.3 ms with one role after the other per tile, 5.95 with the
// roles and (query block, kv head, chunk) items of one length each, 4.95 in pieces (plan_pieces), 4.70 with less around the tiles of a piece
// (q's preparation 5.6 -> 3.3 us, the first tile and the epilogue 2 us each), 4.50 when a producer's first use of a row no longer stood
// right behind its load, 4.46 with all of q_hi in tensor memory, 4.2 with the append's small CTAs; a 777-token f32 prompt in one block 741, 320, 302, 288, 255
// and 233 us.  (128 registers a thread: 8 to 16 bytes spill.)
// Every mbarrier wait is bounded: one that runs out raises the context's error flag, the others of the CTA stop
// waiting, and the kernel runs on to its end, where the tensor memory is always released.
#include <cuda_fp16.h>
#include <math_constants.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <functional>

#include "bk_device.cuh"
#include "bk_internal.h"
#include "bk_mma_common.cuh"
#include "bk_umma.cuh"

namespace bk {

namespace {

constexpr int kSoftWarps = 4, kProdWarps = 8, kMmaWarp = kSoftWarps + kProdWarps, kUWarps = kMmaWarp + 1, kUT = kUWarps * 32;
constexpr int kRows = 128;  // query rows per CTA = tensor-memory lanes
constexpr int kTK = 32;     // positions per tile
// Weights are 2^(s - ref) ||v||, with the reference kBelow under a row's maximum of s + log2 ||v|| when it moves, which it does when the maximum
// has run kLazy further ahead: they stay below 2^14.
constexpr float kBelow = 6.0f, kLazy = 8.0f;
// A score is the sum of two terms that both meet ||k||, which is infinite for a K row of 1.8e19 and more: infinities of different signs would make
// a NaN of minus infinity.  Such a norm counts as kMaxFloat, which leaves the score's sign as it is and its size above kInfinite, and what is above that
// is infinite: scores of finite norms and of q's f16 parts end below 1e27.
constexpr float kMaxFloat = 3.4028235e38f, kInfinite = 1e30f;
constexpr size_t kRunFloats = kPrefillRunFloats;  // a CTA's sums of the runs done, [4 coordinates][row][4]
static_assert(kRunFloats == (size_t)kRows * kHd, "a place per row and coordinate");

constexpr uint32_t kQSlab = kRows * 128, kQTile = 4 * kQSlab;  // 16 KiB per 64-coordinate slab, 64 KiB per tile
constexpr uint32_t kKVSlab = kTK * 128, kKVTile = 4 * kKVSlab;  // 4 KiB, 16 KiB
// Operand slots.  Five: K(t) then takes the place of V(t - 4), whose products came after the softmax of tile t - 4, so the norms of
// four tiles are kept.
constexpr int kSlots = 5, kNormTiles = 4;
constexpr uint32_t kSlotBytes = 2 * kKVTile;  // hi and lo tile
// offsets from the 1024-byte aligned base
constexpr uint32_t oQlo = 0, oSlots = kQTile, oSmall = oSlots + kSlots * kSlotBytes;
struct SmallU {
    float givens[kHd];
    alignas(16) float kn[kNormTiles][kTK], vn[kNormTiles][kTK], lv[kNormTiles][kTK];  // ||k||, ||v|| and log2 ||v|| of a tile's positions
    unsigned long long full[kSlots], empty[kSlots];  // operand slots
    unsigned long long norms[kNormTiles];            // kn, lv of a tile written
    unsigned long long s_full[2], p_full[2], o_done[2], drain;
    uint32_t tmem_slot;
    int gave_up;
    int run_slot;
};
constexpr uint32_t kUmmaSmem = oSmall + 3072;
static_assert(sizeof(SmallU) <= 3072 && kUmmaSmem <= 227 * 1024, "shared memory of a CTA");
constexpr uint32_t kTmemCols = 512, kColO = 0, kColQ = 256, kColS = 384;

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
// The first `rot` (0..3) of four words go to the end: the piece order of a lane, see dequant_store.
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
// Eight nibbles of up to 7 -> eight f16 centroids, two a word, by byte permutes: a permute picks four bytes out of eight by four nibbles,
// so the table is kept as its low bytes and its high bytes.  No shared memory is involved, whose bandwidth the kernel has to spare.
struct Planes {
    uint32_t lo[2], hi[2];
    __device__ __forceinline__ void build(uint32_t tab) {  // lane i holds entry i
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const uint32_t a = __byte_perm(__shfl_sync(0xffffffffu, tab, 4 * k), __shfl_sync(0xffffffffu, tab, 4 * k + 1), 0x5410);
            const uint32_t b = __byte_perm(__shfl_sync(0xffffffffu, tab, 4 * k + 2), __shfl_sync(0xffffffffu, tab, 4 * k + 3), 0x5410);
            lo[k] = __byte_perm(a, b, 0x6420);
            hi[k] = __byte_perm(a, b, 0x7531);
        }
    }
    __device__ __forceinline__ void look_up(uint32_t x, uint32_t (&h)[4]) const {
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const uint32_t sel = x >> (16 * q), bl = __byte_perm(lo[0], lo[1], sel), bh = __byte_perm(hi[0], hi[1], sel);
            h[2 * q] = __byte_perm(bl, bh, 0x5140);
            h[2 * q + 1] = __byte_perm(bl, bh, 0x7362);
        }
    }
};

// 32 coordinates (four words of eight nibbles, rotated by `rot`) -> 32 halfs as four 16-byte chunks of a tile row.
// The eight lanes of a row store chunks 4 c + ((j + c / 2) & 3) together, one per bank group (4 c + j would put them on two).
__device__ __forceinline__ void dequant_store(const uint32_t (&w)[4], const Planes &tab, uint8_t *tile_hi, uint8_t *, int rows, int row_hi, int,
                                              int chunk0, int rot) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
        uint32_t h[4];
        tab.look_up(w[j], h);
        const int chunk = chunk0 + ((j + rot) & 3);
        *reinterpret_cast<uint4 *>(tile_hi + sw_off(rows, row_hi, chunk)) = make_uint4(h[0], h[1], h[2], h[3]);
    }
}

// The same for tables with remainders, which take 37 instructions a word by permutes: the table sits in registers, lane i holds
// (hi | lo << 16) of centroid i & 15, one shuffle looks both parts of an index up.  (A shuffle takes the low five bits of the lane number;
// the fifth, the next index's, does not matter.)
__device__ __forceinline__ void dequant_store(const uint32_t (&w)[4], uint32_t tab, uint8_t *tile_hi, uint8_t *tile_lo, int rows,
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
        *reinterpret_cast<uint4 *>(tile_lo + sw_off(rows, row_lo, chunk)) = make_uint4(l[0], l[1], l[2], l[3]);
    }
}

// An item is a (query block, kv head), the last block first.  A launch has a CTA per piece: some tiles of an item, a whole item (part < 0) or a
// part of one, which then leaves (O, m, l) of its query rows in a place of the scratch.
struct Piece {
    int item;
    uint16_t at, end;  // tiles
    int16_t part;
};
struct PieceList {
    int n;  // 0: every item whole
    Piece p[kPrefillPieces];
};
struct ItemParts {  // of every item: its first place in the scratch (they lie side by side) and how many
    int16_t first[kPrefillPieces], n[kPrefillPieces];
};
static_assert((size_t)kRows * (kHd + 2) == kPrefillPartFloats, "scratch of a piece: [row][coordinate], then [row](m, l)");

// Two f32 operations in one instruction (the softmax warps are bound by what they issue); scores come and go as words.
__device__ __forceinline__ uint64_t pair(uint32_t a, uint32_t b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t first(uint64_t x) { return (uint32_t)x; }
__device__ __forceinline__ uint32_t second(uint64_t x) { return (uint32_t)(x >> 32); }
struct PrefillUArgs {
    DecodeArgs d;
    int seq, pos0, n_tokens, tq, n_blocks;
    float lut_alpha;
    float *scratch;
    float *runs;      // a place of kRunFloats per resident CTA, and which of them are taken
    int *runs_taken;
    int n_runs;
    int *err_flag;
};

template <int BITS, int NREP, bool VF32 = false>
__global__ void __launch_bounds__(kUT, 1)
prefill_umma_kernel(const __grid_constant__ PrefillUArgs pa, const __grid_constant__ PieceList list, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v) {
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

    // ---- which piece ------------------------------------------------------------------------
    const int item = list.n ? list.p[blockIdx.x].item : blockIdx.x;
    const int kv = item % a.n_kv, blk = pa.n_blocks - 1 - item / a.n_kv;
    const int tok0 = blk * pa.tq, n_tok = min(pa.tq, pa.n_tokens - tok0), n_rows = n_tok * NREP;
    const int vis = pa.pos0 + tok0 + n_tok, at = list.n ? list.p[blockIdx.x].at : 0, t_end = list.n ? list.p[blockIdx.x].end : (vis + kTK - 1) / kTK;
    const int part = list.n ? list.p[blockIdx.x].part : -1;
    const int c0 = at * kTK, c1 = min(t_end * kTK, vis), n_tiles = t_end - at;
    const int n_runs = (n_tiles + kRun - 1) / kRun, run_len = n_runs > 1 ? (n_tiles + n_runs - 1) / n_runs : kRun;

    const int half = a.n_rot >> 1;
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
    // Nothing above was another kernel's.  The query rows start travelling: every row's round trip at once.
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
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
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, ss.tmem_slot, 0);
    auto run_sums = [&]() { return reinterpret_cast<float4 *>(pa.runs + (size_t)ss.run_slot * kRunFloats); };
    float *run_mul = reinterpret_cast<float *>(sm + oQlo), *row_mul = run_mul + kRows;  // where q_lo was: the runs' and the rows' factors at the end
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
    // f32 rows: a warp takes four rows of the tile, a lane 32 bytes of each, which become a 16-byte operand piece.  (Eight lanes a row with 128 bytes
    // each, as for packed rows, made every load touch 32 lines: 4096 clocks a tile of the load path, as much as a tile takes now.)
    [[maybe_unused]] float4 fk[kF32 ? 8 : 1], fv[kVRows32 ? 8 : 1];
    auto fetch_f32 = [&](float4 *dst, const uint8_t *rows, int tile) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float4 *src = reinterpret_cast<const float4 *>(rows + row_of(tile, (pt >> 5) * 4 + j) * 1024) + 2 * lane;
            dst[2 * j] = src[0];
            dst[2 * j + 1] = src[1];
        }
    };
    auto fetch_packed = [&](uint32_t (&w)[4], const uint8_t *rows, int tile) {
        const uint8_t *p = rows + row_of(tile, my_row) * kRowBytes;
        if constexpr (BITS == 4) {
            const uint4 x = reinterpret_cast<const uint4 *>(p)[my_c];
            w[0] = x.x, w[1] = x.y, w[2] = x.z, w[3] = x.w;
        } else if constexpr (BITS == 3) {
            const uint32_t *p3 = reinterpret_cast<const uint32_t *>(p) + 3 * my_c;
            w[0] = p3[0], w[1] = p3[1], w[2] = p3[2], w[3] = 0;
        } else {  // 2 bit: 32 coordinates are 8 bytes
            const uint2 x = reinterpret_cast<const uint2 *>(p)[my_c];
            w[0] = x.x, w[1] = x.y, w[2] = w[3] = 0;
        }
    };
    auto fetch_k = [&](int tile) {
        if constexpr (kF32) {
            fetch_f32(fk, a.k_rows, tile);
        } else if constexpr (!kF16) {
            fetch_packed(pk, a.k_rows, tile);
            if (pt < (VF32 ? kTK : 2 * kTK)) pn = (pt < kTK ? a.k_norms : a.v_norms)[row_of(tile, pt & (kTK - 1))];
        }
    };
    auto fetch_v = [&](int tile) {
        if constexpr (kVRows32) fetch_f32(fv, a.v_rows, tile);
        else if constexpr (!kF16) fetch_packed(pv, a.v_rows, tile);
    };

    if (producer) {  // the first K tile travels too (and of packed rows the first V tile)
        if constexpr (!kF32) fetch_k(0);
        if constexpr (!kVRows32) fetch_v(0);
    }

    // ---- q rows -> q_hi and q_lo: rope, Givens, scale, f16 hi/lo; a warp takes every kUWarps-th row.  Its rows' rope entries, a pair of
    // coordinates per lane, travel with the rows (up to 32 pairs; wider rotations read the others where they need them).  Then the 32 bytes
    // of a lane are coordinates 8 lane .. + 7; the half of q_hi for tensor memory goes where the row was.  (Pairs of lanes that exchange
    // their coordinates of the rotated quarter cost twice the instructions, which is what this takes: 5.5 us.)
    constexpr int kMyRows = (kRows + kUWarps - 1) / kUWarps;
    auto rope_row = [&](int r) { return a.rope + (size_t)(pa.pos0 + tok0 + r / NREP) * half; };
    float2 cs[kMyRows];
#pragma unroll
    for (int i = 0; i < kMyRows; i++) {
        const int r = warp + i * kUWarps;
        if (r < n_rows && lane < half) cs[i] = __ldg(rope_row(r) + lane);
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    {
        const float qscale = rsqrtf((float)kHd) * 1.4426950408889634f / pa.lut_alpha;
#pragma unroll
        for (int i = 0; i < kMyRows; i++) {
            const int r = warp + i * kUWarps;
            float *row = reinterpret_cast<float *>(sm + oSlots) + r * kHd;
            if (r < n_rows && lane < half) {
                float x0 = row[lane], x1 = row[lane + half];
                rope_pair(x0, x1, cs[i]);
                row[lane] = x0;
                row[lane + half] = x1;
                for (int j = lane + 32; j < half; j += 32) {
                    x0 = row[j], x1 = row[j + half];
                    rope_pair(x0, x1, __ldg(rope_row(r) + j));
                    row[j] = x0;
                    row[j + half] = x1;
                }
            }
        }
        float gv[8];
        if constexpr (!kRaw) {
            const float4 g0 = reinterpret_cast<const float4 *>(ss.givens)[2 * lane], g1 = reinterpret_cast<const float4 *>(ss.givens)[2 * lane + 1];
            gv[0] = g0.x, gv[1] = g0.y, gv[2] = g0.z, gv[3] = g0.w, gv[4] = g1.x, gv[5] = g1.y, gv[6] = g1.z, gv[7] = g1.w;
        }
        __syncwarp();
#pragma unroll 2
        for (int r = warp; r < kRows; r += kUWarps) {
            uint4 *row = reinterpret_cast<uint4 *>(sm + oSlots + r * (kHd * 4));
            uint32_t hw[4] = {}, lw[4] = {};
            if (r < n_rows) {
                const float4 x0 = reinterpret_cast<const float4 *>(row)[2 * lane], x1 = reinterpret_cast<const float4 *>(row)[2 * lane + 1];
                const float x[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll
                for (int p = 0; p < 4; p++) {
                    float o0 = x[2 * p], o1 = x[2 * p + 1];
                    if constexpr (!kRaw) givens_fwd(x[2 * p], x[2 * p + 1], gv[2 * p], gv[2 * p + 1], o0, o1);
                    o0 *= qscale;
                    o1 *= qscale;
                    const __half2 h = __floats2half2_rn(o0, o1);
                    const float2 hf = __half22float2(h);
                    const __half2 l = __floats2half2_rn(o0 - hf.x, o1 - hf.y);
                    hw[p] = *reinterpret_cast<const uint32_t *>(&h);
                    lw[p] = *reinterpret_cast<const uint32_t *>(&l);
                }
                __syncwarp();
            }
            row[lane ^ (r & 7)] = make_uint4(hw[0], hw[1], hw[2], hw[3]);
            *reinterpret_cast<uint4 *>(sm + oQlo + sw_off(kRows, r, lane)) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
        }
    }
    fence_smem_to_async_proxy();
    __syncthreads();
    const int my_q = (warp & 3) * 32 + lane;  // query row of a softmax thread
    if (warp < kSoftWarps) {
#pragma unroll
        for (int b = 0; b < 4; b++) {
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

    float ref = -CUDART_INF_F, lsum = 0.f;  // a query row's running reference and sum
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
            bool go = wait(bar_full + 8 * slot, use);
            if (tile >= 2) go = go && wait(bar_o + 8 * (tile & 1), (uint32_t)((tile - 2) >> 1) & 1u);  // P(tile - 2), in the same columns, has been used
            if (!__all_sync(0xffffffffu, go)) return false;
            tc_fence_after_sync();
            // columns 0-31: q_hi k_hi; 32-63: the small terms
            const uint32_t d = tmem + kColS + (uint32_t)(tile & 1) * 64u, kb = base + oSlots + slot * kSlotBytes;
            const uint64_t kd = umma_smem_desc(kb, 16, 1024, kUmmaSwizzle128), ql = umma_smem_desc(base + oQlo, 16, 1024, kUmmaSwizzle128);
            if (elect_one()) {  // (the address field of a descriptor counts 16-byte units)
#pragma unroll
                for (int ks = 0; ks < 16; ks++)
                    umma_f16_ts(d, tmem + kColQ + 8 * ks, kd + (((ks >> 2) * kKSlab + (ks & 3) * 32) >> 4), idesc_s2, ks > 0);
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
            if (tile + 1 < n_tiles && !issue_s(tile + 1)) break;
            ok = wait(bar_full + 8 * slot, use);
            ok = ok && wait(bar_p + 8 * (tile & 1), (uint32_t)(tile >> 1) & 1u);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after_sync();
            const uint32_t p = tmem + kColS + (uint32_t)(tile & 1) * 64u, vb = base + oSlots + slot * kSlotBytes;
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
                            if (r < valid) x = reinterpret_cast<const uint4 *>(rows + row_of(tile, r) * 512)[lane];
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
            // tables without remainders (8 entries at most) by permutes, others by shuffles
            auto make_table = [&]() {
                if constexpr (kRaw || kLoTiles) {
                    return tab;
                } else {
                    Planes p;
                    p.build(tab);
                    return p;
                }
            };
            const auto table = make_table();
            // split the fetched floats into f16 hi + lo and store both as a 16-byte chunk of a tile row each; rows at or past
            // the piece's end are stored as zeros (they may hold anything, and 0 * Inf would poison the accumulators)
            auto split_store = [&](const float4 *f, int tile, uint8_t *tile_hi, uint8_t *tile_lo, int rows, int lo_rows) {
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int r = (pt >> 5) * 4 + j;
                    const float x[8] = {f[2 * j].x, f[2 * j].y, f[2 * j].z, f[2 * j].w, f[2 * j + 1].x, f[2 * j + 1].y, f[2 * j + 1].z, f[2 * j + 1].w};
                    uint32_t h[4] = {}, l[4] = {};
                    if (c0 + tile * kTK + r < c1) {
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            const __half2 hv = __floats2half2_rn(x[2 * e], x[2 * e + 1]);
                            const float2 hf = __half22float2(hv);
                            const __half2 lv = __floats2half2_rn(x[2 * e] - hf.x, x[2 * e + 1] - hf.y);
                            h[e] = *reinterpret_cast<const uint32_t *>(&hv);
                            l[e] = *reinterpret_cast<const uint32_t *>(&lv);
                        }
                    }
                    *reinterpret_cast<uint4 *>(tile_hi + sw_off(rows, r, lane)) = make_uint4(h[0], h[1], h[2], h[3]);
                    *reinterpret_cast<uint4 *>(tile_lo + sw_off(rows, r + lo_rows, lane)) = make_uint4(l[0], l[1], l[2], l[3]);
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
            // (What is done with a fetched row begins here: left to itself the compiler puts the first of it right behind the loads.)
            auto arrived = [&](uint32_t (&w)[4]) { asm volatile("" : "+r"(w[0]), "+r"(w[1]), "+r"(w[2]), "+r"(w[3])); };
            auto arrived_f32 = [&](float4 *f) {
#pragma unroll
                for (int j = 0; j < 8; j++) asm volatile("" : "+f"(f[j].x), "+f"(f[j].y), "+f"(f[j].z), "+f"(f[j].w));
            };
            auto put_k = [&](int tile) -> bool {
                if (!__all_sync(0xffffffffu, slot_free())) return false;  // one answer for the warp, also when a wait runs out
                if constexpr (kF32) {
                    arrived_f32(fk);
                } else {
                    arrived(pk);
                    asm volatile("" : "+f"(pn));
                }
                uint8_t *dst = sm + oSlots + slot * kSlotBytes;
                if constexpr (kF32) {
                    split_store(fk, tile, dst, dst, 64, 32);
                } else {
                    widen(pk);
                    dequant_store(pk, table, dst, dst, kLoTiles ? 64 : 32, my_row, my_row + 32, 4 * my_c, rot);
                    if (pt < 2 * kTK) {
                        if (pt < kTK) ss.kn[tile % kNormTiles][pt] = pn > kMaxFloat ? kMaxFloat : pn;  // (NaN stays)
                        else if constexpr (!VF32) {
                            pn = fmaxf(pn, 1e-30f);
                            ss.vn[tile % kNormTiles][pt - kTK] = fminf(pn, kMaxFloat);  // (finite: it meets weights of 0)
                            ss.lv[tile % kNormTiles][pt - kTK] = fast_log2(pn);
                        }
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
                if constexpr (kVRows32) arrived_f32(fv);
                else arrived(pv);
                uint8_t *dst = sm + oSlots + slot * kSlotBytes;
                if constexpr (kVRows32) {
                    split_store(fv, tile, dst, dst + kKVTile, kTK, 0);
                } else {
                    widen(pv);
                    dequant_store(pv, table, dst, dst + kKVTile, kTK, my_row, my_row, 4 * my_c, rot);
                }
                put_done();
                if (tile + 1 < n_tiles) fetch_v(tile + 1);
                return true;
            };
            if constexpr (kF32) fetch_k(0);
            if constexpr (kVRows32) fetch_v(0);
            bool ok = put_k(0);
            for (int tile = 0; ok && tile < n_tiles; tile++) {
                if (tile + 1 < n_tiles) ok = put_k(tile + 1);
                ok = ok && put_v(tile);
            }
        }
    } else {
        // ---- softmax: thread = query row ------------------------------------------------------------------------
        const int lim = my_q < n_rows ? pa.pos0 + tok0 + my_q / NREP + 1 : 0;
        float run_ref = -CUDART_INF_F;  // the reference of the sums of the runs done
        int run_start = 0;
        // O collects a run of tiles, joins the sums of the runs before, rounded to nearest, and starts again: its adds truncate at the
        // size of what it holds, so its error grows with the tiles it collects.  Against float64, channels with x20 outliers: 777
        // tokens into an f32 cache 1.36e-6 of the result (1.69e-6 without runs, 1.49e-6 with runs of up to 20 tiles), 4608 in blocks
        // of 512 2.0e-6 (3.5e-6, 2.2e-6); V of one sign, 4608 tokens, 2.8e-6 (7.9e-6).  Without lo tiles a run may be longer: fewer
        // products.  The sums stay in L2.  Without runs the 4608 planar4 tokens take 4.03 ms instead of 4.19 (four layers), f16 3.26 instead of
        // 3.55, the 777 tokens 215 us instead of 233; shorter chunks cost 15 to 20 % for the same when they were tried.
        // The sums so far come in a block of 32 coordinates ahead of their use, the first before the run's last product is awaited (one block
        // after the other, each with its trip to L2, made 4 us of it).
        auto collect_o = [&](bool first_run, auto &&run_done) -> bool {
            float4 old[2][8];
            auto fetch = [&](int b, float4 (&dst)[8]) {
#pragma unroll
                for (int j = 0; j < 8; j++) dst[j] = first_run ? make_float4(0.f, 0.f, 0.f, 0.f) : __ldcg(run_sums() + (8 * b + j) * kRows + my_q);
            };
            fetch(0, old[0]);
            if (!run_done()) return false;
            const float f = run_ref > -CUDART_INF_F ? fast_exp2(run_ref - ref) : 0.f;
#pragma unroll 2
            for (int b = 0; b < 8; b++) {
                if (b < 7) fetch(b + 1, old[(b + 1) & 1]);
                uint32_t o[32];
                tmem_ld32(my_tmem + kColO + 32 * b, o);
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const float4 x = old[b & 1][j];
                    __stcg(run_sums() + (8 * b + j) * kRows + my_q,
                           make_float4(fmaf(x.x, f, __uint_as_float(o[4 * j])), fmaf(x.y, f, __uint_as_float(o[4 * j + 1])),
                                       fmaf(x.z, f, __uint_as_float(o[4 * j + 2])), fmaf(x.w, f, __uint_as_float(o[4 * j + 3]))));
                }
            }
            run_ref = ref;
            return true;
        };
        for (int tile = 0; tile < n_tiles; tile++) {
            const uint32_t buf = (uint32_t)tile & 1u, par = (uint32_t)(tile >> 1) & 1u;
            if (tile == run_start && tile > 0) {  // (the next product, which starts O again, waits for this tile's weights)
                const bool ok = collect_o(tile == run_len, [&]() {
                    if (!__all_sync(0xffffffffu, wait(bar_o + 8 * (buf ^ 1u), (uint32_t)((tile - 1) >> 1) & 1u))) return false;
                    tc_fence_after_sync();
                    return true;
                });
                if (!ok) break;
            }
            bool ok = wait(bar_s + 8 * buf, par);
            if constexpr (!kRaw) ok = ok && wait(bar_norms + 8 * (tile % kNormTiles), (uint32_t)(tile / kNormTiles) & 1u);
            if (!__all_sync(0xffffffffu, ok)) break;
            tc_fence_after_sync();
            uint32_t sr[32], t[32];
            tmem_ld32(my_tmem + kColS + 64 * buf, sr);
            tmem_ld32(my_tmem + kColS + 64 * buf + 32, t);
            // Two positions at a time: scores less the reference to sv, the same + log2 ||v|| to tv (one array for raw V rows).  The
            // reference goes in with the first product: a score of about 64 as an f32 number would be off by 2^-18.
            uint64_t sv[16], tv_[kVPlanar ? 16 : 1];
            auto tv = [&](int i) -> uint64_t & { return kVPlanar ? tv_[kVPlanar ? i : 0] : sv[i]; };
            const ulonglong2 *kn2 = reinterpret_cast<const ulonglong2 *>(ss.kn[tile % kNormTiles]), *lv2 = reinterpret_cast<const ulonglong2 *>(ss.lv[tile % kNormTiles]);
            const float base_ref = ref > -CUDART_INF_F ? ref : 0.f;
            const uint64_t nref = pair(__float_as_uint(-base_ref), __float_as_uint(-base_ref));
            float mx = -CUDART_INF_F;
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
                const uint64_t main[2] = {pair(sr[2 * i], sr[2 * i + 1]), pair(sr[2 * i + 2], sr[2 * i + 3])};
                const uint64_t small[2] = {pair(t[2 * i], t[2 * i + 1]), pair(t[2 * i + 2], t[2 * i + 3])};
                if constexpr (kRaw) {
                    sv[i] = add2(add2(main[0], nref), small[0]);
                    sv[i + 1] = add2(add2(main[1], nref), small[1]);
                } else {
                    const ulonglong2 k2 = kn2[i / 2];
                    sv[i] = fma2(small[0], k2.x, fma2(main[0], k2.x, nref));
                    sv[i + 1] = fma2(small[1], k2.y, fma2(main[1], k2.y, nref));
                }
                if constexpr (kVPlanar) {
                    const ulonglong2 l2 = lv2[i / 2];
                    tv_[i] = add2(sv[i], l2.x);
                    tv_[i + 1] = add2(sv[i + 1], l2.y);
                }
            }
            const int n_ok = min(c1, lim) - (c0 + tile * kTK);  // positions of the tile that this row sees
            if (!__all_sync(0xffffffffu, n_ok >= kTK)) {
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const uint32_t none = __float_as_uint(-CUDART_INF_F);
                    sv[i] = pair(2 * i < n_ok ? first(sv[i]) : none, 2 * i + 1 < n_ok ? second(sv[i]) : none);
                    if constexpr (kVPlanar) tv_[i] = pair(2 * i < n_ok ? first(tv_[i]) : none, 2 * i + 1 < n_ok ? second(tv_[i]) : none);
                }
            }
#pragma unroll
            for (int i = 0; i < 16; i++) mx = fmaxf(mx, fmaxf(__uint_as_float(first(tv(i))), __uint_as_float(second(tv(i)))));
            // lazy reference: move it only when this row's maximum ran ahead by more than kLazy
            const bool move = mx > -CUDART_INF_F && (ref == -CUDART_INF_F || mx > kBelow + kLazy);
            if (__any_sync(0xffffffffu, move)) {  // tensor-memory traffic is warp-collective
                const float new_ref = move ? base_ref + (mx - kBelow) : ref, by = move ? (mx < kInfinite ? new_ref - base_ref : CUDART_NAN_F) : 0.f;
                const float f = move ? (ref > -CUDART_INF_F ? fast_exp2(-by) : 0.f) : 1.f;
                const uint64_t nby = pair(__float_as_uint(-by), __float_as_uint(-by));
#pragma unroll
                for (int i = 0; i < 16; i++) sv[i] = add2(sv[i], nby);
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
                ref = new_ref;
            }
            // weights p ||v||, two positions a column: for each K-step of 16 positions eight columns of hi parts and eight of lo parts.
            // (p = 2^(s - ref) stays below 2^114: the norms are taken as 1e-30 at least.  The sum of p falls by the ratio of the norms when a row outweighs
            // those before it, so the norms that a query sees may span a factor of 1e32.)
            const ulonglong2 *vn2 = reinterpret_cast<const ulonglong2 *>(ss.vn[tile % kNormTiles]);
            uint64_t l2 = 0;
#pragma unroll
            for (int kk = 0; kk < 2; kk++) {
                uint32_t pw[16];
#pragma unroll
                for (int e = 0; e < 8; e += 2) {
                    ulonglong2 v2;
                    if constexpr (kVPlanar) v2 = vn2[4 * kk + e / 2];
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        const uint64_t x = sv[8 * kk + e + u];
                        const float p0 = fast_exp2(__uint_as_float(first(x))), p1 = fast_exp2(__uint_as_float(second(x)));
                        const uint64_t p = pair(__float_as_uint(p0), __float_as_uint(p1));
                        l2 = add2(l2, p);
                        uint64_t w = p;
                        if constexpr (kVPlanar) w = mul2(p, u ? v2.y : v2.x);
                        const float w0 = __uint_as_float(first(w)), w1 = __uint_as_float(second(w));
                        const __half2 h = __floats2half2_rn(w0, w1);
                        const float2 hf = __half22float2(h);
                        const __half2 l = __floats2half2_rn(w0 - hf.x, w1 - hf.y);
                        pw[e + u] = *reinterpret_cast<const uint32_t *>(&h);
                        pw[8 + e + u] = *reinterpret_cast<const uint32_t *>(&l);
                    }
                }
                tmem_st16(my_tmem + kColS + 64 * buf + 16 * kk, pw);  // (where this row's S was, which is in registers)
            }
            lsum += __uint_as_float(first(l2)) + __uint_as_float(second(l2));
            if (tile == run_start) run_start += run_len;
            tmem_wait_st();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_p + 8 * buf);
        }
        const float unscale = 1.0f / (kVPlanar ? pa.lut_alpha : 1.0f);  // (raw V rows carry no table scale)
        if (n_runs > 1) run_mul[my_q] = run_ref > -CUDART_INF_F ? fast_exp2(run_ref - ref) : 0.f;
        row_mul[my_q] = part < 0 ? (lsum > 0.f ? unscale / lsum : 0.f) : unscale;
        if (part >= 0 && my_q < n_rows) {
            float *dst = pa.scratch + (size_t)part * kPrefillPartFloats + kRows * kHd + 2 * my_q;
            dst[0] = ref;
            dst[1] = lsum;
        }
    }
    tc_fence_before_sync();
    __syncthreads();  // (the issuing warp has seen all its products complete)
    tc_fence_after_sync();

    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    // ---- epilogue: warps 0-11, 32 query rows x 32 columns at a time through a padded shared-memory block, so that the
    // global stores of a warp cover four rows' 128 bytes instead of 32 rows' 16 bytes
    if (warp < kMmaWarp) {
        const bool whole = part < 0, vec = !whole || ((uintptr_t)a.out & 15) == 0;
        const float mul = row_mul[my_q], rmul = n_runs > 1 ? run_mul[my_q] : 0.f;
        constexpr int kPad = 36;
        float *stg = reinterpret_cast<float *>(sm + oSlots) + warp * (32 * kPad);
        const int row0 = (warp & 3) * 32 + (lane >> 3), ch = lane & 7;
        for (int b = warp >> 2; b < 8; b += 3) {
            float4 old[8];
            if (n_runs > 1) {
#pragma unroll
                for (int j = 0; j < 8; j++) old[j] = __ldcg(run_sums() + (8 * b + j) * kRows + my_q);
            }
            uint32_t o[32];
            tmem_ld32(my_tmem + kColO + 32 * b, o);
#pragma unroll
            for (int j = 0; j < 8; j++) {
                float4 x = make_float4(__uint_as_float(o[4 * j]), __uint_as_float(o[4 * j + 1]), __uint_as_float(o[4 * j + 2]), __uint_as_float(o[4 * j + 3]));
                if (n_runs > 1)
                    x = make_float4(fmaf(old[j].x, rmul, x.x), fmaf(old[j].y, rmul, x.y), fmaf(old[j].z, rmul, x.z), fmaf(old[j].w, rmul, x.w));
                x = make_float4(x.x * mul, x.y * mul, x.z * mul, x.w * mul);
                if (whole && kVPlanar) {
                    const float4 g = *reinterpret_cast<const float4 *>(ss.givens + 32 * b + 4 * j);
                    float4 y;
                    givens_inv(x.x, x.y, g.x, g.y, y.x, y.y);
                    givens_inv(x.z, x.w, g.z, g.w, y.z, y.w);
                    x = y;
                }
                *reinterpret_cast<float4 *>(stg + lane * kPad + 4 * j) = x;
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int q = row0 + 4 * i;
                if (q >= n_rows) continue;
                const float4 x = *reinterpret_cast<const float4 *>(stg + ((lane >> 3) + 4 * i) * kPad + 4 * ch);
                float *dst = (whole ? a.out + ((size_t)(tok0 + q / NREP) * a.n_head + kv * NREP + q % NREP) * kHd
                                    : pa.scratch + (size_t)part * kPrefillPartFloats + (size_t)q * kHd) + 32 * b + 4 * ch;
                if (vec) {
                    *reinterpret_cast<float4 *>(dst) = x;
                } else {
                    dst[0] = x.x, dst[1] = x.y, dst[2] = x.z, dst[3] = x.w;
                }
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

// Merge the pieces of the items that are cut, rotate back, write: a warp per output row, so that the references and sums of all pieces
// are a few loads side by side and the rows' loads do not wait for them.  A piece that the row does not see counts as zeros whatever it holds.
constexpr int kMergeWarps = 8, kPerLane = (kPrefillParts + 31) / 32;
__global__ void __launch_bounds__(kMergeWarps * 32) prefill_umma_merge_kernel(const __grid_constant__ PrefillUArgs pa, const __grid_constant__ ItemParts parts,
                                                                              const float *givens) {
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    const int n_head = pa.d.n_head, n_rep = n_head / pa.d.n_kv, row = blockIdx.x * kMergeWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int tok = row / n_head, head = row - tok * n_head, blk = tok / pa.tq, my_q = (tok - blk * pa.tq) * n_rep + head % n_rep;
    if (tok >= pa.n_tokens) return;
    const int item = (pa.n_blocks - 1 - blk) * pa.d.n_kv + head / n_rep, n = parts.n[item];
    if (n == 0) return;  // whole: written where it was computed
    const float *base = pa.scratch + (size_t)parts.first[item] * kPrefillPartFloats;
    float f[kPerLane], l[kPerLane], M = -CUDART_INF_F, Ls = 0.f;
#pragma unroll
    for (int h = 0; h < kPerLane; h++) {
        const int i = lane + 32 * h;
        const float2 ml = i < n ? *reinterpret_cast<const float2 *>(base + i * kPrefillPartFloats + kRows * kHd + 2 * my_q) : make_float2(-CUDART_INF_F, 0.f);
        f[h] = ml.x;
        l[h] = ml.y;
        M = fmaxf(M, f[h]);
    }
    for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
#pragma unroll
    for (int h = 0; h < kPerLane; h++) {
        f[h] = f[h] > -CUDART_INF_F ? exp2f(f[h] - M) : 0.f;
        if (l[h] != l[h]) f[h] = CUDART_NAN_F;  // NaN among the row's scores, whatever became of its reference: the row is NaN
        if (f[h] != 0.f) Ls = fmaf(l[h], f[h], Ls);
    }
    for (int o = 16; o > 0; o >>= 1) Ls += __shfl_xor_sync(0xffffffffu, Ls, o);
    float4 acc[2] = {};  // coordinates 4 lane .. + 3 of each half
#pragma unroll
    for (int h = 0; h < kPerLane; h++)
#pragma unroll 4
        for (int i = 32 * h; i < min(n, 32 * h + 32); i++) {
            const float4 *p = reinterpret_cast<const float4 *>(base + i * kPrefillPartFloats + my_q * kHd) + lane;
            const float fc = __shfl_sync(0xffffffffu, f[h], i & 31);
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const float4 v = p[32 * j];
                acc[j].x = fmaf(fc > 0.f ? v.x : 0.f, fc, acc[j].x);
                acc[j].y = fmaf(fc > 0.f ? v.y : 0.f, fc, acc[j].y);
                acc[j].z = fmaf(fc > 0.f ? v.z : 0.f, fc, acc[j].z);
                acc[j].w = fmaf(fc > 0.f ? v.w : 0.f, fc, acc[j].w);
            }
        }
    const float inv = Ls > 0.f ? 1.0f / Ls : 0.f;
    const bool vec = ((uintptr_t)pa.d.out & 15) == 0;
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const int d = 128 * j + 4 * lane;
        float4 o = make_float4(acc[j].x * inv, acc[j].y * inv, acc[j].z * inv, acc[j].w * inv);
        if (givens) {  // planar V only
            const float4 g = *reinterpret_cast<const float4 *>(givens + d);
            float4 r;
            givens_inv(o.x, o.y, g.x, g.y, r.x, r.y);
            givens_inv(o.z, o.w, g.z, g.w, r.z, r.w);
            o = r;
        }
        float *dst = pa.d.out + (size_t)row * kHd + d;
        if (vec) {
            *reinterpret_cast<float4 *>(dst) = o;
        } else {  // (the caller's alignment is only that of a float)
            dst[0] = o.x, dst[1] = o.y, dst[2] = o.z, dst[3] = o.w;
        }
    }
}

template <int BITS, int NREP, bool VF32 = false>
bk_status launch_umma_one(bk_ctx *ctx, const PrefillUArgs &pa, const PieceList &list, const ItemParts &parts) {
    static std::atomic<bool> configured[64] = {};  // per device; racing first calls set the same attribute
    const int dev = ctx->device;
    if (dev < 0 || dev >= 64) return fail(ctx, BK_ERR_UNSUPPORTED, "prefill: device index above 63");
    if (!configured[dev].load()) {
        BK_CUDA(ctx, cudaFuncSetAttribute(prefill_umma_kernel<BITS, NREP, VF32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kUmmaSmem));
        configured[dev].store(true);
    }
    if (!pa.d.h_tmap_k || !pa.d.h_tmap_v) return fail(ctx, BK_ERR_INVALID, "prefill: the cache has no tensor maps");
    const int n_items = pa.n_blocks * pa.d.n_kv;
    if (list.n > n_items && !pa.scratch) return fail(ctx, BK_ERR_INVALID, "prefill: no scratch for pieces");  // (made with the cache)
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(list.n ? list.n : n_items));
    cfg.blockDim = dim3(kUT);
    cfg.dynamicSmemBytes = kUmmaSmem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // see griddepcontrol.* in the kernels
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    BK_CUDA(ctx, cudaLaunchKernelEx(&cfg, prefill_umma_kernel<BITS, NREP, VF32>, pa, list, *static_cast<const CUtensorMap *>(pa.d.h_tmap_k),
                                    *static_cast<const CUtensorMap *>(pa.d.h_tmap_v)));
    ctx->launches++;
    BK_CUDA(ctx, cudaGetLastError());
    if (list.n > n_items) {
        const int n_out = pa.n_tokens * pa.d.n_head;
        cfg.gridDim = dim3((unsigned)((n_out + kMergeWarps - 1) / kMergeWarps));
        cfg.blockDim = dim3(kMergeWarps * 32);
        cfg.dynamicSmemBytes = 0;
        BK_CUDA(ctx, cudaLaunchKernelEx(&cfg, prefill_umma_merge_kernel, pa, parts, (BITS == 16 || BITS == 32 || VF32) ? (const float *)nullptr : pa.d.givens));
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

// How the items are cut into pieces.  All tiles of all items side by side are one line, which is cut into a stretch per SM so that the longest
// stretch is as short as possible; every piece costs kFixed tiles' worth of set-up, q preparation, filling and draining of the pipeline, and
// results beside its tiles, and cutting at all costs a launch that merges.  The first CTAs get the longest piece of each stretch,
// the others follow in order of length: as the SMs come free, the SM with the shortest piece first, each finds about what its stretch had left.
// Whole items, longest first, are often spread as well, so cutting has to gain what it costs: the merge's launch, 1/45 tile for every piece that
// goes through the scratch, and a twentieth of the stretches, which the SMs do not keep to.  (us for a planar4 launch, cut / whole, 24 heads on 4:
// 512 tokens after 0, 1000 and 4000 rows 33 / 35, 76 / 87 and 178 / 234; 1000, 1500 and 2500 tokens from the start 70 / 61, 130 / 103 and 282 / 257; 48 heads
// on 8, 600 tokens 67 / 48.  Over 894 shapes of three modes the rule loses 0.1 % against the better of the two, cutting always 2.3 %.)
// With more than kPrefillItems items (four and more an SM) whole ones, longest first, are spread evenly enough.
constexpr int kPrefillItems = kPrefillPieces - kPrefillStretches;
static void plan_pieces(int n_sms, int pos0, int n_tokens, int tq, int n_kv, PieceList &list, ItemParts &parts) {
    // A piece has kLeast tiles or the rest of its item.  kFixed is less than the 12 tiles' time that a launch spends beside its tiles; 5 to 20 give the same times within 0.6 % (six modes, 76 shapes each).
    constexpr int kFixed = 7, kMerge = 3, kLeast = 4;
    const int most = std::min(n_sms, kPrefillStretches), n_blocks = (n_tokens + tq - 1) / tq, n_items = n_blocks * n_kv;
    list.n = 0;
    if (n_items > kPrefillItems || (int64_t)pos0 + n_tokens > UINT16_MAX * kTK) return;
    auto tiles_of = [&](int item) { return (std::min((n_blocks - item / n_kv) * tq, n_tokens) + pos0 + kTK - 1) / kTK; };
    int n = 0, n_stretches = 0, start[kPrefillStretches + 1];  // pieces in the order of the line, and where the stretches start
    Piece piece[kPrefillPieces];
    // into stretches of at most `budget`; false if there are not enough
    auto cut = [&](int budget) {
        n = n_stretches = 0;
        int left = 0;  // of the current stretch
        for (int item = 0, all = 0; item < n_items; item++) {
            if (item % n_kv == 0) all = tiles_of(item);
            for (int at = 0; at < all;) {
                if (left < kFixed + std::min(all - at, kLeast)) {
                    if (n_stretches == most) return false;
                    start[n_stretches++] = n;
                    left = budget;
                }
                int take = std::min(all - at, left - kFixed);
                if (all - at - take > 0 && all - at - take < kLeast) take = std::max(kLeast, all - at - kLeast);  // no short rest
                left -= kFixed + take;
                piece[n++] = Piece{item, (uint16_t)at, (uint16_t)(at + take), -1};
                at += take;
            }
        }
        start[n_stretches] = n;
        return true;
    };
    int total = 0;
    for (int b = 0; b < n_blocks; b++) total += n_kv * (kFixed + tiles_of(b * n_kv));
    // what the whole items take: each goes to the SM that is free first
    int whole = kFixed + tiles_of(0);
    if (n_items > most) {
        int load[kPrefillStretches] = {};
        for (int item = 0, all = 0; item < n_items; item++) {
            if (item % n_kv == 0) all = kFixed + tiles_of(item);
            std::pop_heap(load, load + most, std::greater<int>());
            whole = std::max(whole, load[most - 1] += all);
            std::push_heap(load, load + most, std::greater<int>());
        }
    }
    auto worth = [&](int budget, int n_parts) { return budget * 1.05 + kMerge + n_parts / 45.0 < whole; };
    int lo = std::max(kFixed + kLeast, (total + most - 1) / most), hi = lo + kFixed;
    if (!worth(lo, 0)) return;
    while (!cut(hi)) lo = hi + 1, hi += std::max(1, hi / 8);
    while (lo < hi) {
        const int mid = (lo + hi) / 2;
        if (cut(mid)) hi = mid;
        else lo = mid + 1;
    }
    cut(hi);
    // places in the scratch
    int places = 0;
    for (int i = 0; i < n_items; i++) parts.n[i] = 0;
    for (int i = 0; i < n; i++) {
        Piece &p = piece[i];
        if (p.at == 0 && p.end == tiles_of(p.item)) continue;
        if (parts.n[p.item]++ == 0) parts.first[p.item] = (int16_t)places;
        p.part = (int16_t)places++;
    }
    if (!worth(hi, places)) return;
    // order of the CTAs
    auto length = [](const Piece &p) { return p.end - p.at; };
    for (int c = 0; c < n_stretches; c++) {
        int best = start[c];
        for (int i = start[c] + 1; i < start[c + 1]; i++)
            if (length(piece[i]) > length(piece[best])) best = i;
        list.p[c] = piece[best];
        piece[best].item = -1;
    }
    list.n = n_stretches;
    for (int i = 0; i < n; i++)
        if (piece[i].item >= 0) list.p[list.n++] = piece[i];
    std::stable_sort(list.p + n_stretches, list.p + n, [&](const Piece &x, const Piece &y) { return length(x) > length(y); });
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
    pa.runs = ctx->d_prefill_runs;
    pa.runs_taken = reinterpret_cast<int *>(ctx->d_prefill_runs + ctx->n_sms * kRunFloats);
    pa.n_runs = ctx->n_sms;
    pa.scratch = ctx->d_prefill;
    PieceList list;
    ItemParts parts;
    plan_pieces(ctx->n_sms, pos0, n_tokens, pa.tq, a.n_kv, list, parts);
#define BK_PU_CASE(R)                                                                            \
    case R:                                                                                      \
        if (a.k_kind == ROW_F16) return launch_umma_one<16, R>(ctx, pa, list, parts);                         \
        if (a.k_kind == ROW_F32) return launch_umma_one<32, R>(ctx, pa, list, parts);                         \
        if (a.v_kind == ROW_F32) return a.bits == 3 ? launch_umma_one<3, R, true>(ctx, pa, list, parts) : launch_umma_one<4, R, true>(ctx, pa, list, parts); \
        if (a.bits == 2) return launch_umma_one<2, R>(ctx, pa, list, parts);                                  \
        return a.bits == 3 ? launch_umma_one<3, R>(ctx, pa, list, parts) : launch_umma_one<4, R>(ctx, pa, list, parts);
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

int32_t bk_hook_prefill_plan(int32_t n_sms, int32_t pos0, int32_t n_tokens, int32_t n_head, int32_t n_kv, int32_t capacity, int32_t *pieces) {
    bk::PieceList list;
    bk::ItemParts parts;
    bk::plan_pieces(n_sms, pos0, n_tokens, bk::kRows / (n_head / n_kv), n_kv, list, parts);
    for (int i = 0; i < std::min(list.n, capacity); i++) {
        const bk::Piece &p = list.p[i];
        const int32_t words[4] = {p.item, p.at, p.end, p.part};
        std::copy(words, words + 4, pieces + 4 * i);
    }
    return list.n;
}
