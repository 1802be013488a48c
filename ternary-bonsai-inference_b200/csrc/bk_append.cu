// Fused KV append: IMROPE on K, then store K and V rows as f32, f16 or rotated Lloyd-Max
// ("planar") rows, one launch for any number of tokens.  Replaces rope_imrope.comp (k side),
// kv_store.comp, kv_store_f16.comp and kv_store_q.comp and follows the reference CPU path
// bit for bit (src/forward.rs:259-285, src/kvquant.rs:397-412, src/rope.rs:61-69).
//
// A CTA stages 8 or 16 vectors of 256 floats ((K|V, kv head) of consecutive tokens):
//   1. coalesced 16-byte copies (cp.async) into shared memory; K vectors rotate pairs (j, j + n_rot/2) with
//      the (cos, sin) row of the token's position from the host-built rope table;
//   2. planar rows: one warp adds the 256 squares of all vectors, a vector per lane, each lane
//      in order (the reference's f32 sum is sequential, so each chain is; they run side by side);
//   3. the warps scale, Givens-rotate, find the nearest centroid (two shuffles from a host-built cell table of
//      the decision thresholds, or a binary search and a neighbour check: the same index as the reference's
//      linear scan) and write `bits` bytes per lane;
//      f32/f16 rows leave as 128-bit stores.
// Traffic per token is the algorithmic minimum: 2*n_kv*1 KiB in, rows + norms out.
#include <math_constants.h>

#include <atomic>

#include "bk_device.cuh"
#include "bk_internal.h"

namespace bk {

namespace {

constexpr int kVecPad = kHd + 4;  // floats per staged vector; +4 keeps float4 alignment and makes the
                                  // per-lane 128-bit reads of the norm pass conflict-free
constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;

// Two f32 products in one instruction, each rounded as __fmul_rn does.
__device__ __forceinline__ float2 mul_pair(float x, float y, float a, float b) { return unpack2(mul2(pack2(x, y), pack2(a, b))); }

// Eight consecutive coordinates of a staged vector for every lane without bank conflicts: two 128-bit reads
// in the staging layout (coordinates 4 l .. 4 l + 3 and 128 + 4 l .. + 3), then lanes 2m and 2m + 1 swap
// one of them: the even lane ends with group m (coordinates 8 m .. 8 m + 7), the odd one with group 16 + m.
// (Reading 8 consecutive floats per lane directly puts eight lanes on every bank.)  Returns the group.
__device__ __forceinline__ int load_group_of_8(const float *sx, int lane, float (&x)[8]) {
    const float4 a = reinterpret_cast<const float4 *>(sx)[lane], b = reinterpret_cast<const float4 *>(sx)[lane + 32];
    const bool odd = lane & 1;
    const float4 send = odd ? a : b;
    float4 recv;
    recv.x = __shfl_xor_sync(0xffffffffu, send.x, 1);
    recv.y = __shfl_xor_sync(0xffffffffu, send.y, 1);
    recv.z = __shfl_xor_sync(0xffffffffu, send.z, 1);
    recv.w = __shfl_xor_sync(0xffffffffu, send.w, 1);
    const float4 lo = odd ? recv : a, hi = odd ? b : recv;
    x[0] = lo.x; x[1] = lo.y; x[2] = lo.z; x[3] = lo.w;
    x[4] = hi.x; x[5] = hi.y; x[6] = hi.z; x[7] = hi.w;
    return odd ? 16 + (lane >> 1) : (lane >> 1);
}

// Rotate, quantize and pack the 8 coordinates of one lane; `inv` is 1 / the vector's norm (0 for a norm of up to 1e-12).
template <int BITS>
__device__ __forceinline__ void store_planar_row(const float *sx, int lane, float inv, const float *givens,
                                                 const float *sbook, uint8_t *row) {
    float x[8];
    const int group = load_group_of_8(sx, lane, x);
    const float4 g0 = reinterpret_cast<const float4 *>(givens)[2 * group], g1 = reinterpret_cast<const float4 *>(givens)[2 * group + 1];
    const float gv[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
    uint64_t packed = 0;
#pragma unroll
    for (int pr = 0; pr < 4; pr++) {
        const float a = __fmul_rn(x[2 * pr], inv), b = __fmul_rn(x[2 * pr + 1], inv);
        float r0, r1;
        givens_fwd(a, b, gv[2 * pr], gv[2 * pr + 1], r0, r1);
        packed |= (uint64_t)nearest_centroid_fast<BITS>(r0, sbook) << (BITS * (2 * pr));
        packed |= (uint64_t)nearest_centroid_fast<BITS>(r1, sbook) << (BITS * (2 * pr + 1));
    }
    store_group8<BITS>(row, group, packed);
}

// The same for codebooks of up to 16 centroids (nearest_centroid_lanes in bk_device.cuh).  The bulk kernel is bound by its
// instructions, so nothing is decided per coordinate: a finite norm bounds every rotated value by 1.5 (a norm is no
// smaller than any of its coordinates, or it is at most 1e-12 and inv is 0).  Vectors with an infinite or NaN norm take the
// scan.  A lane takes eight consecutive coordinates (two 128-bit reads, each with two lanes on a bank) and keeps their
// rotations in registers.
template <int BITS>
__device__ __forceinline__ void store_planar_row_lanes(const float *sx, int lane, float n, float inv, const float (&gv)[8], float scale,
                                                       LaneCell my, const float *book, uint8_t *row) {
    const float4 xa = reinterpret_cast<const float4 *>(sx)[2 * lane], xb = reinterpret_cast<const float4 *>(sx)[2 * lane + 1];
    const float x[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
    float v[8];
#pragma unroll
    for (int pr = 0; pr < 4; pr++) {
        // givens_fwd of the scaled pair, its six products as three
        const float2 ab = mul_pair(x[2 * pr], x[2 * pr + 1], inv, inv);
        const float c = gv[2 * pr], sn = gv[2 * pr + 1];
        const float2 by_c = mul_pair(ab.x, ab.y, c, c), by_s = mul_pair(ab.x, ab.y, sn, sn);
        v[2 * pr] = __fsub_rn(by_c.x, by_s.y);
        v[2 * pr + 1] = __fadd_rn(by_s.x, by_c.y);
    }
    uint32_t packed = 0;  // 8 indices of at most 4 bits
    if (n < CUDART_INF_F) {
#pragma unroll
        for (int i = 7; i >= 0; i--) packed = (packed << BITS) + nearest_centroid_lanes(v[i], scale, my.below, my.thr);
    } else {
#pragma unroll
        for (int i = 7; i >= 0; i--) packed = (packed << BITS) + nearest_centroid(v[i], book, 1 << BITS);
    }
    store_group8<BITS>(row, lane, (uint64_t)packed);
}

__device__ __forceinline__ void store_f32_row(const float *sx, int lane, uint8_t *row) {
    float4 *dst = reinterpret_cast<float4 *>(row);
    const float4 *src = reinterpret_cast<const float4 *>(sx);
    dst[lane] = src[lane];
    dst[lane + 32] = src[lane + 32];
}

__device__ __forceinline__ void store_f16_row(const float *sx, int lane, uint8_t *row) {
    float x[8];
    const int group = load_group_of_8(sx, lane, x);
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; i++) w[i] = pack_half2_ref(x[2 * i], x[2 * i + 1]);
    reinterpret_cast<uint4 *>(row)[group] = make_uint4(w[0], w[1], w[2], w[3]);
}

// A warp takes one K or V head of kVecs / 8 consecutive tokens, the next warp the next head (j < n_kv: K head j, else V head
// j - n_kv), so what depends on the head is worked out once a warp.  Pass 1: the warp stages its vectors and
// ropes the K ones.  Pass 2: warp 0 adds the squares of the CTA's vectors, one vector per lane, each lane in
// order (the reference's f32 sum is sequential, so the chain is; they run side by side).
// Pass 3: each warp scales, rotates, finds the nearest centroids of and stores its vectors.
// kVecs = 16 for bulk calls of planar rows (half of the lanes of the norm pass work, and five CTAs an SM are at different passes), 8 for
// smaller calls (latency: one vector per warp) and for f32 and f16 rows, which have no norm: many small CTAs load while others store.
// Us a layer of back-to-back calls of 2048 / 4096 / 8192 tokens: planar4 12.6 / 20.4 / 33.9 with 32 vectors a CTA, the head worked out per
// vector, products one at a time and five CTAs an SM, 10.3 / 17.8 / 32.2 without that and four CTAs, 9.9 / 16.8 / 29.6 with the rows staged by
// cp.async instead of through registers, 11.0 / 17.2 / 31.0 with 16 vectors (five CTAs an SM leave 48 registers, of which 4 bits spill 28 bytes and 5 to 7 bits 4 to 8; six were slower); f32 10.3 / 17.7 / 29.7 in CTAs of 32
// vectors, 7.8 / 13.5 / 25.0 of 8, 7.4 / 12.1 / 21.9 by cp.async; f16 11.1 / 17.3 / 29.5, 7.9 / 14.1 / 25.9 and 7.4 / 11.8 / 21.6.
// Sixteen vectors a CTA are taken for what follows an append, a decode of the same layer: both together 21.0 / 27.8 / 43.4 against 21.2 / 28.5 /
// 45.5 with 32 (planar4), 20.9 / 29.5 / 47.2 against 20.3 / 30.4 / 50.7 (K only).
template <int BITS, int kVecs>
__global__ void __launch_bounds__(kThreads, BITS == 0 ? 8 : kVecs == 16 ? 5 : 4) append_kernel(AppendArgs a) {
    extern __shared__ __align__(16) float smem[];
    float *snorm = smem + kVecs * kVecPad;          // the norms, and what a vector is scaled by
    [[maybe_unused]] float *sbook = snorm + 64;     // centroids (widths above 4)
    [[maybe_unused]] float *sgiv = sbook + 256;     // Givens table
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_kv = a.n_kv, per_tok = 2 * n_kv;
    constexpr int kPerWarp = kVecs / kWarps;
    const int unit = blockIdx.x * kWarps + warp, t0 = unit / per_tok * kPerWarp, j = unit % per_tok;
    const int n_here = min(kPerWarp, a.n_tokens - t0);  // (0 or less past the last token)
    const bool is_v = j >= n_kv;
    const int kv = is_v ? j - n_kv : j;
    const bool planar = a.k_kind == ROW_PLANAR || a.v_kind == ROW_PLANAR;

    if (BITS > 4) {
        for (int i = threadIdx.x; i < (1 << BITS); i += kThreads) sbook[i] = a.book[i];
        for (int i = threadIdx.x; i < kHd; i += kThreads) sgiv[i] = a.givens[i];
    }
    // k and v may come from the previous kernel in the stream: with programmatic dependent launch
    // only the table copies above run ahead of it.  Nothing after this kernel depends on more
    // than its completion, so dependents may be scheduled right away.
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");

    // ---- pass 1: stage (and rope).  All of a warp's copies and loads (rows and rope entries) are issued before any is waited for, so the
    // pass costs one round trip.
    float2 rcs[kPerWarp];
    const int half = a.n_rot >> 1;
    float *const mine = smem + warp * (kPerWarp * kVecPad);  // the warp's vectors
    const uint32_t mine_at = (uint32_t)__cvta_generic_to_shared(mine) + lane * 16;
    const float4 *src4 = reinterpret_cast<const float4 *>(is_v ? a.v : a.k) + ((size_t)t0 * n_kv + kv) * (kHd / 4) + lane;
#pragma unroll
    for (int u = 0; u < kPerWarp; u++) {
        rcs[u] = make_float2(1.f, 0.f);
        if (u < n_here) {
#pragma unroll
            for (int h = 0; h < 2; h++)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(mine_at + u * (kVecPad * 4) + h * 512),
                             "l"(src4 + (size_t)u * n_kv * (kHd / 4) + h * 32)
                             : "memory");
            if (!is_v && lane < half) {  // n_rot <= 64: one rope entry per lane
                const int pos = a.desc ? a.desc[t0 + u].z : a.pos0 + t0 + u;
                rcs[u] = __ldg(a.rope + (size_t)pos * half + lane);
            }
        }
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    if (!is_v) {
        __syncwarp();
#pragma unroll
        for (int u = 0; u < kPerWarp; u++) {
            if (u >= n_here) break;
            float *sx = mine + u * kVecPad;
            if (half <= 32) {
                if (lane < half) {
                    float x0 = sx[lane], x1 = sx[lane + half];
                    rope_pair(x0, x1, rcs[u]);
                    sx[lane] = x0;
                    sx[lane + half] = x1;
                }
            } else {  // wider rotations: entries beyond the prefetched 32 come straight from the table
                const int pos = a.desc ? a.desc[t0 + u].z : a.pos0 + t0 + u;
                const float2 *cs = a.rope + (size_t)pos * half;
                for (int p = lane; p < half; p += 32) {
                    float x0 = sx[p], x1 = sx[p + half];
                    rope_pair(x0, x1, cs[p]);
                    sx[p] = x0;
                    sx[p + half] = x1;
                }
            }
        }
    }
    __syncthreads();
    // widths up to 4: this lane's threshold cell (built once per context on the host) and rotations; not before pass 1, whose
    // loads want the registers
    [[maybe_unused]] LaneCell my = {0u, 0.f};
    [[maybe_unused]] float scale = 0.f, gv[8] = {};
    if constexpr (BITS >= 1 && BITS <= 4) {
        my = a.cells->cell[lane];
        scale = a.cells->scale;
        const float4 g0 = __ldg(reinterpret_cast<const float4 *>(a.givens) + 2 * lane), g1 = __ldg(reinterpret_cast<const float4 *>(a.givens) + 2 * lane + 1);
        gv[0] = g0.x; gv[1] = g0.y; gv[2] = g0.z; gv[3] = g0.w;
        gv[4] = g1.x; gv[5] = g1.y; gv[6] = g1.z; gv[7] = g1.w;
    }
    // ---- pass 2: sequential sums side by side ----------------------------------------------------
    if (planar && warp == 0 && lane < kVecs) {  // (a place without a vector gives a number nobody reads)
        const float4 *x4 = reinterpret_cast<const float4 *>(smem + lane * kVecPad);
        float acc = 0.0f;
#pragma unroll 8
        for (int i = 0; i < kHd / 4; i++) {
            const float4 x = x4[i];
            const float2 lo = mul_pair(x.x, x.y, x.x, x.y), hi = mul_pair(x.z, x.w, x.z, x.w);
            acc = __fadd_rn(acc, lo.x);
            acc = __fadd_rn(acc, lo.y);
            acc = __fadd_rn(acc, hi.x);
            acc = __fadd_rn(acc, hi.y);
        }
        const float n = __fsqrt_rn(acc);
        snorm[lane] = n;
        snorm[32 + lane] = (n > 1e-12f) ? __fdiv_rn(1.0f, n) : 0.0f;
    }
    __syncthreads();
    // ---- pass 3: store --------------------------------------------------------------------------------
    const int kind = is_v ? a.v_kind : a.k_kind;
    uint8_t *const rows = is_v ? a.v_rows : a.k_rows;
    [[maybe_unused]] float *const norms = is_v ? a.v_norms : a.k_norms;
    const size_t row_bytes = is_v ? a.v_row_bytes : a.k_row_bytes;
#pragma unroll
    for (int u = 0; u < kPerWarp; u++) {
        if (u >= n_here) break;
        size_t r;  // row of the cache's slab
        if (a.desc) {
            const int4 d = a.desc[t0 + u];
            r = (size_t)d.x * a.seq_stride_rows + (size_t)d.y * n_kv + kv;
        } else {
            r = (size_t)(a.row0 + t0 + u) * n_kv + kv;
        }
        const float *sx = mine + u * kVecPad;
        uint8_t *row = rows + r * row_bytes;
        if (kind == ROW_F32) {
            store_f32_row(sx, lane, row);
        } else if (BITS == 0 && kind == ROW_F16) {  // (f16 rows never lie beside planar ones)
            store_f16_row(sx, lane, row);
        } else {
            if constexpr (BITS > 0) {
                const float n = snorm[warp * kPerWarp + u], inv = snorm[32 + warp * kPerWarp + u];
                if (lane == 0) norms[r] = n;
                if constexpr (BITS <= 4) store_planar_row_lanes<BITS>(sx, lane, n, inv, gv, scale, my, a.book, row);
                else store_planar_row<BITS>(sx, lane, inv, sgiv, sbook, row);
            }
        }
    }
}


}  // namespace

bk_status launch_append(bk_ctx *ctx, const AppendArgs &a) {
    if (a.n_tokens <= 0) return BK_OK;
    const int threads = kThreads;
    const size_t n_vec = (size_t)a.n_tokens * 2 * a.n_kv;
    const bool planar = a.k_kind == ROW_PLANAR || a.v_kind == ROW_PLANAR;
    // More small CTAs than this per SM: go for throughput.  Up to 4 bits eight, the places of small CTAs on an SM twice: us a layer, 8 / 16
    // vectors a CTA, append alone, and with a decode: planar4, 1050 tokens 6.7 / 6.3, 15.8 / 17.2; 1200 tokens 8.5 / 6.6, 17.6 / 17.7; 1400 tokens
    // 9.7 / 7.3, 18.9 / 18.2 (with 32 vectors 7.1 and 18.5, 8.4 and 20.8, 9.5 and 21.5); K only, 1050 tokens 7.3 / 6.9, 16.8 / 16.5; 1200
    // tokens 8.7 / 7.2, 17.3 / 16.6.  Wider rows ten: planar8, 1200 tokens 17.8 / 17.4, 32.9 / 34.2; 1600 tokens (24.2, 42.8 with 16).
    const bool bulk = n_vec > (size_t)8 * (a.bits >= 1 && a.bits <= 4 ? 8 : 10) * ctx->n_sms;
    const int vecs = bulk && planar ? 16 : 8;
    const size_t smem = (size_t)(vecs * kVecPad + 64 + (a.bits > 4 ? 256 + kHd : 0)) * sizeof(float);
    const int per_warp = vecs / kWarps;
    const unsigned grid = (unsigned)(((size_t)(a.n_tokens + per_warp - 1) / per_warp * 2 * a.n_kv + kWarps - 1) / kWarps);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // see griddepcontrol.* in the kernel
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t err = cudaSuccess;
    // A bulk call wants five CTAs of 17 KiB or eight of 9 KiB per SM: ask for the largest shared-memory carve-out (once per
    // kernel and process; a hint, so its result is not checked).
    auto launch_bulk = [&](auto *kernel) {
        static std::atomic<bool> hinted{false};
        if (!hinted.exchange(true)) cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        return cudaLaunchKernelEx(&cfg, kernel, a);
    };
    if (!planar) {
        err = bulk ? launch_bulk(append_kernel<0, 8>) : cudaLaunchKernelEx(&cfg, append_kernel<0, 8>, a);
    } else {
        const bool ok = dispatch_bits(a.bits, [&]<int B>() {
            err = bulk ? launch_bulk(append_kernel<B, 16>) : cudaLaunchKernelEx(&cfg, append_kernel<B, 8>, a);
        });
        if (!ok) return fail(ctx, BK_ERR_INVALID, "append: bits must be 1..8");
    }
    ctx->launches++;
    BK_CUDA(ctx, err);
    BK_CUDA(ctx, cudaGetLastError());
    return BK_OK;
}

}  // namespace bk
