// Tail shared by the decode kernels: merge the split-K chunks of one (sequence, kv head) and
// write the result.  A CTA that has reduced its chunk to (acc[NREP][256], M[NREP], L[NREP]) in
// shared memory (acc relative to M, exp2 domain) calls finish_item():
//   * more than one chunk: the CTA stores its triple in the partials buffer, takes a ticket
//     from the (sequence, kv head) counter and returns unless it is the last to arrive; the
//     last one re-reads every chunk's triple and combines them.  Nobody waits for anybody.
//   * planar V: the combined accumulator is still in Givens-rotated space and is rotated back
//     once here (src/forward.rs:349, shaders/attn_out_q.comp:85-91);
//   * output: acc / L (times sigmoid(gate) when the layer form of the step passes a gate), or
//     the unnormalised (acc, m, l) triple when the caller merges chunks held by other caches /
//     GPUs itself.
#pragma once

#include <cuda/atomic>
#include <math_constants.h>

#include "bk_device.cuh"
#include "bk_internal.h"
#include "bk_mma_common.cuh"

namespace bk {

// Per-CTA time stamps for tuning builds (-DBK_PHASE): stamp i of CTA b lands in g_phase[b][i].
#ifdef BK_PHASE
static __device__ unsigned long long g_phase[1024][16];
__device__ __forceinline__ unsigned long long phase_timer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
#define BK_STAMP(i)                                                                       \
    do {                                                                                  \
        if (threadIdx.x == 0 && blockIdx.x < 1024) g_phase[blockIdx.x][i] = phase_timer(); \
    } while (0)
#else
#define BK_STAMP(i)
#endif

// A free region of shared memory through which the last arriver streams the other chunks'
// triples (the tensor-core kernels pass their drained stage ring): the TMA engine copies them in
// rounds into the region's two halves, completion on the two mbarriers at `bar` (initialised by
// the caller with count 1 and not used for anything else).  addr = 0: no region, the combine reads
// the triples with ordinary loads.
struct FinishSmem {
    uint32_t addr = 0;    // shared-window address, 16-byte aligned
    uint32_t bytes = 0;
    uint32_t bar = 0;     // shared-window address of two consecutive mbarriers
    uint8_t *ptr = nullptr;  // the same region as a generic pointer
    int *err_flag = nullptr;
};

// Context split over the GPUs of one node: dims [d0, d0 + dn) of the (acc, m, l) rows of the n_rep q heads of
// kv head `kv`: send this rank's values to slot [rank] of every rank's mailbox, wait (bounded) for the same
// values of every rank in this rank's own mailbox, and write the log-sum-exp merge to a.out.
// A mailbox is [2 parities][world][n_head][hd + 2] eight-byte words (value bits, sequence number).  A word is
// stored with one 8-byte store, which arrives whole, so it validates itself: the receiver reads it until its
// second half is the call's sequence number.  Nothing else is needed - no arrival flags, no fence between data
// and flag, one trip over the link instead of three.  The CTA that holds coordinate 0 also sends the heads' m
// and l.  The word grid does not depend on how a rank has cut its work, so ranks whose launches have different
// shapes (or that send from the stand-alone exchange kernel) understand each other.  Slots alternate with the
// parity of the sequence number: a rank can be at most one call ahead of another (it needs the other's rows to
// finish a call), so a word is never overwritten before it was read.  vals: [n_rep][dn] in shared memory,
// relative to s_M (exp2 domain), not normalised.  Every thread of the CTA must call; on a time-out the
// affected outputs are zeros and the context's error word is raised.
// One mailbox word: value and sequence number in a single 8-byte store (never two 4-byte ones).
__device__ __forceinline__ void store_word(uint2 *p, float value, unsigned seqno) {
    asm volatile("st.volatile.global.v2.u32 [%0], {%1, %2};\n" ::"l"(p), "r"(__float_as_uint(value)), "r"(seqno) : "memory");
}

__device__ __forceinline__ void exchange_slice(const DecodeArgs &a, int n_rep, int slot, int kv, int d0, int dn,
                                               const float *vals, const float *s_M, const float *s_L) {
    constexpr int kStride = kHd + 2;
    const int tid = threadIdx.x, nt = blockDim.x;
    const int world = a.xch_world, rank = a.xch_rank, n_rows = a.n_head, row0 = kv * n_rep;
    const unsigned seqno = a.xch_seqno, par = seqno & 1u;
    const size_t slot_w = (size_t)n_rows * kStride;
    BK_STAMP(10);
    for (int r = 0; r < world; r++) {
        uint2 *dst = reinterpret_cast<uint2 *>(a.xch_peer[r]) + ((size_t)par * world + rank) * slot_w + (size_t)row0 * kStride;
        for (int i = tid; i < n_rep * dn; i += nt) {
            const int rr = i / dn, d = i - rr * dn;
            store_word(dst + rr * kStride + d0 + d, vals[i], seqno);
        }
        if (d0 == 0 && tid < n_rep) {
            store_word(dst + tid * kStride + kHd, s_M[tid] * 0.6931471805599453f, seqno);  // log2 -> ln
            store_word(dst + tid * kStride + kHd + 1, s_L[tid], seqno);
        }
    }
    const uint2 *mbox = reinterpret_cast<const uint2 *>(a.xch_peer[rank]) + (size_t)par * world * slot_w + (size_t)row0 * kStride;
    bool first = true;
    for (int i = tid; i < n_rep * dn; i += nt) {
        const int rr = i / dn, d = d0 + (i - rr * dn);
        // every rank's (m, l, value): all loads of a round are issued together; words that have not arrived yet
        // are read again
        uint2 wm[kMaxWorld], wl[kMaxWorld], wx[kMaxWorld];
        unsigned pending = (world >= 32) ? 0xffffffffu : ((1u << world) - 1u);
        int polls = 0;
        bool ok = true;
        while (pending) {
#pragma unroll
            for (int r = 0; r < kMaxWorld; r++)
                if (pending >> r & 1u) {
                    const uint2 *p = mbox + (size_t)r * slot_w + (size_t)rr * kStride;
                    wm[r] = __ldcv(p + kHd);
                    wl[r] = __ldcv(p + kHd + 1);
                    wx[r] = __ldcv(p + d);
                }
#pragma unroll
            for (int r = 0; r < kMaxWorld; r++)
                if ((pending >> r & 1u) && wm[r].y == seqno && wl[r].y == seqno && wx[r].y == seqno) pending &= ~(1u << r);
            if (pending) {
                if (++polls > a.xch_spin) {  // a peer never sent: leave a mark and go on rather than hang
                    ok = false;
                    raise_error(a.xch_err, 3);
                    break;
                }
                if (polls > 2048) __nanosleep(64);  // the first microseconds without a pause: the ranks run in lock step
            }
        }
        if (first) {
            BK_STAMP(11);
            first = false;
        }
        float Mx = -CUDART_INF_F;
#pragma unroll
        for (int r = 0; r < kMaxWorld; r++)
            if (r < world && ok && __uint_as_float(wl[r].x) > 0.f) Mx = fmaxf(Mx, __uint_as_float(wm[r].x));
        float Ls = 0.f, sum = 0.f;
#pragma unroll
        for (int r = 0; r < kMaxWorld; r++)
            if (r < world && ok && __uint_as_float(wl[r].x) > 0.f) {
                const float f = expf(__uint_as_float(wm[r].x) - Mx);
                Ls = fmaf(__uint_as_float(wl[r].x), f, Ls);
                sum = fmaf(__uint_as_float(wx[r].x), f, sum);
            }
        a.out[((size_t)slot * a.n_head + row0 + rr) * kHd + d] = (ok && Ls > 0.f) ? sum / Ls : 0.f;
    }
    BK_STAMP(12);
}

// ---- Set-up shared by the tensor-core kernels ----------------------------------------------------------------
// One warp prepares one q head: lane l holds coordinates 8 l .. 8 l + 7.  load() issues every load (the rope partners
// among them, whatever n_rot), so that tile copies can be issued behind them; finish() applies RMSNorm
// (src/forward.rs:242-243; q is not stored, so a tree sum will do) and rope.  A warp per head needs no barrier between
// the steps: q was ready 2.5 us after the dependency wait with the CTA's threads spread over all heads, 1.8 us now.
struct QHead {
    float x[8], y[8];  // the lane's coordinates and their rope partners
    __device__ __forceinline__ void load(const float *row, int lane, int half) {
        const int d = 8 * lane;
        if ((reinterpret_cast<uintptr_t>(row) & 15) == 0) {
            const float4 u = reinterpret_cast<const float4 *>(row + d)[0], v = reinterpret_cast<const float4 *>(row + d)[1];
            x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w;
            x[4] = v.x; x[5] = v.y; x[6] = v.z; x[7] = v.w;
        } else {
#pragma unroll
            for (int e = 0; e < 8; e++) x[e] = row[d + e];
        }
#pragma unroll
        for (int e = 0; e < 8; e++) {
            y[e] = 0.f;
            if (d + e < 2 * half) y[e] = row[d + e < half ? d + e + half : d + e - half];
        }
    }
    __device__ __forceinline__ void finish(int lane, int half, const float *norm_w /* shared memory, or null */, float eps, const float2 *rope_row) {
        const int d = 8 * lane;
        if (norm_w) {
            float ss = 0.f;
#pragma unroll
            for (int e = 0; e < 8; e++) ss = fmaf(x[e], x[e], ss);
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
            const float sc = 1.0f / sqrtf(ss / (float)kHd + eps);
#pragma unroll
            for (int e = 0; e < 8; e++) {
                x[e] = x[e] * sc * norm_w[d + e];
                if (d + e < 2 * half) y[e] = y[e] * sc * norm_w[d + e < half ? d + e + half : d + e - half];
            }
        }
#pragma unroll
        for (int e = 0; e < 8; e++)
            if (d + e < 2 * half) {
                const bool first = d + e < half;
                float x0 = first ? x[e] : y[e], x1 = first ? y[e] : x[e];
                rope_pair(x0, x1, rope_row[first ? d + e : d + e - half]);
                x[e] = first ? x0 : x1;
            }
    }
};

// The newest token's K row (role 0) or V row (role 1) of a kv head on its way to the cache: one warp loads it, norms
// (layer form, src/forward.rs:244-245) and ropes K, and leaves it in sx (shared memory, 16-byte aligned), with the
// append kernel's arithmetic.
__device__ __forceinline__ void prepare_new_row(const DecodeArgs &a, int role, int lane, float4 lo, float4 hi, float *sx, const float2 *rope_row) {
    reinterpret_cast<float4 *>(sx)[lane] = lo;
    reinterpret_cast<float4 *>(sx)[lane + 32] = hi;
    __syncwarp();
    if (role == 0 && a.k_norm_w) {
        float w[kHd / 32];
#pragma unroll
        for (int j = 0; j < kHd / 32; j++) w[j] = __ldg(a.k_norm_w + lane + 32 * j);
        float sc = 0.f;
        if (lane == 0) sc = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(serial_sumsq256(sx), (float)kHd), a.eps)));
        sc = __shfl_sync(0xffffffffu, sc, 0);
#pragma unroll
        for (int j = 0; j < kHd / 32; j++) sx[lane + 32 * j] = __fmul_rn(__fmul_rn(sx[lane + 32 * j], sc), w[j]);
        __syncwarp();
    }
    if (role == 0 && !a.no_rope) {
        const int half = a.n_rot >> 1;
        for (int j = lane; j < half; j += 32) {
            float x0 = sx[j], x1 = sx[j + half];
            rope_pair(x0, x1, rope_row[j]);
            sx[j] = x0;
            sx[j + half] = x1;
        }
        __syncwarp();
    }
}
// The row in sx as `BITS`-wide indices (src/kvquant.rs:397-412): eight indices per lane; returns the norm (every lane).
template <int BITS>
__device__ __forceinline__ float quantize_new_row(const float *sx, int lane, const float *givens, const float *book, uint64_t &packed) {
    float n = 0.f;
    if (lane == 0) n = __fsqrt_rn(serial_sumsq256(sx));
    n = __shfl_sync(0xffffffffu, n, 0);
    const float inv = (n > 1e-12f) ? __fdiv_rn(1.0f, n) : 0.0f;
    packed = 0;
#pragma unroll
    for (int pr = 0; pr < 4; pr++) {
        const int i = lane * 4 + pr;  // pair index: coordinates 2i, 2i+1
        float r0, r1;
        givens_fwd(__fmul_rn(sx[2 * i], inv), __fmul_rn(sx[2 * i + 1], inv), givens[2 * i], givens[2 * i + 1], r0, r1);
        packed |= (uint64_t)nearest_centroid_fast<BITS>(r0, book) << (BITS * (2 * pr));
        packed |= (uint64_t)nearest_centroid_fast<BITS>(r1, book) << (BITS * (2 * pr + 1));
    }
    return n;
}

// Bounded wait for an mbarrier by a whole warp.
__device__ __forceinline__ void wait_bar(uint32_t bar, uint32_t parity, int lane, int *err_flag) {
    int polls = 0;
    while (!mbar_try_wait(bar, parity)) {
        if (++polls > kWaitPolls) {  // never expected; leave a mark and go on rather than hang
            if (lane == 0) raise_error(err_flag, 1);
            break;
        }
    }
}

// ---- The slice form of the split-K combine ----------------------------------------------------------------
// When every CTA of a (sequence, kv head) is resident at the same time (the launcher sets DecodeArgs::dist only
// then), each CTA sends its chunk's result to the CTAs that combine it and then combines ONE slice of the output
// itself: all heads of the group, D consecutive coordinates (whole Givens pairs, so the inverse rotation, the
// division by l and the gate happen here too).
//
// The boxes (DecodeArgs::boxes) are empty between launches: every 32-bit word holds kEmptyWord, a NaN pattern that
// no sender ever stores.  A word therefore validates itself: the owner of a slice reads it until it is not empty,
// uses it and empties it again.  No counter, no fence between data and flag, no set-up from launch to launch: one
// trip through L2 instead of three (stores, ticket, loads of the triples).  What bounds this stage is that trip and
// the barriers around it; from the last chunk's sums to the end of the launch 4.0 to 4.7 us with a ticket
// counter, 3.3 us now (planar4 9000 rows, f16 8192 rows).
//
// A wait that runs out leaves words behind that the next launch would take for its own, so it also marks the boxes as foul
// (DecodeArgs::box_state).  While they are, launches that are already queued write nothing and raise the
// error again; the host empties the boxes and takes the mark off when it reports the error.
//
// Boxes of a (sequence, kv head) start at first_item * NREP * kBoxFloats:
//     values  [slice][chunk][NREP][D]     relative to the chunk's maximum, not normalised
//     (m, l)  [slice][chunk][NREP][2]     a copy per slice, so that every word has one reader
constexpr unsigned kEmptyWord = 0xffffffffu;
// 16-byte columns per head in a slice, as a power of two (the index arithmetic below is shifts), and how many slices that
// makes.  The context split wants slices on its mailbox's octet grid.
__host__ __device__ constexpr int slice_lg(int n_chunks, bool exchange) {
    int lg = exchange ? 1 : 0;
    while ((kHd / 4 >> lg) > n_chunks) lg++;
    return lg;
}
constexpr bool boxes_fit() {
    for (int n = 2; n <= kFactorCap; n++)
        for (int x = 0; x < 2; x++) {
            const int n_slices = kHd / 4 >> slice_lg(n, x != 0);
            if (kHd + 2 * n_slices > kBoxFloats || n_slices > n) return false;
        }
    return true;
}
static_assert(boxes_fit(), "a box does not hold a chunk's values and (m, l) pairs, or a slice has no owner");

// Are the boxes fit for use?  Read by one thread of a CTA beside its first boxes.
__device__ __forceinline__ bool boxes_clean(const DecodeArgs &a) {
    unsigned w;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];\n" : "=r"(w) : "l"(a.box_state) : "memory");
    return w == kEmptyWord;
}
__device__ __forceinline__ float box_word(float x) {  // kEmptyWord becomes the ordinary NaN
    return __float_as_uint(x) == kEmptyWord ? __uint_as_float(0x7fffffffu) : x;
}
__device__ __forceinline__ void box_store(float *p, float x) {
    asm volatile("st.relaxed.gpu.global.f32 [%0], %1;\n" ::"l"(p), "f"(box_word(x)) : "memory");
}
__device__ __forceinline__ float4 box_load4(const float *p) {
    float4 v;
    asm volatile("ld.relaxed.gpu.global.v4.f32 {%0,%1,%2,%3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ float2 box_load2(const float *p) {
    float2 v;
    asm volatile("ld.relaxed.gpu.global.v2.f32 {%0,%1}, [%2];\n" : "=f"(v.x), "=f"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ bool box_full(float x) { return __float_as_uint(x) != kEmptyWord; }
__device__ __forceinline__ bool box_full4(float4 v) { return box_full(v.x) && box_full(v.y) && box_full(v.z) && box_full(v.w); }

// sums[r]: this chunk's value of coordinate tid (threads 0..255) of head r; s_M, s_L: its maxima and sums.  `red` is
// free shared memory (16-byte aligned, kCombineBytes); *s_ok is 1 on entry.  Every thread of the CTA calls.
// A thread merges a few chunks of one 16-byte column on its own (its own reference, no exchange of maxima), the threads
// that write the output merge the thread groups: one barrier between the loads and the output.
constexpr uint32_t kCombineBytes = 12288;
template <int NREP>
__device__ __forceinline__ void combine_slice(const DecodeArgs &a, int slot, int kv, int my_chunk, int n_chunks, int first_item,
                                              const float (&sums)[NREP], const float *s_M, const float *s_L, float *red, int *s_ok,
                                              bool v_planar, const float *givens, int *err_flag) {
    const int tid = threadIdx.x, nthr = (int)blockDim.x;
    const int lg = slice_lg(n_chunks, a.xch_peer != nullptr), D4 = 1 << lg, D = 4 * D4, n_slices = kHd / 4 >> lg;
    float *const boxes = a.boxes + (size_t)first_item * NREP * kBoxFloats;
    float *const ml = boxes + (size_t)n_slices * n_chunks * NREP * D;
    bool clean = true;
    if (tid == nthr - 1) clean = boxes_clean(a);
    // ---- send
    if (tid < kHd) {
        const int sl = tid >> (lg + 2);
        float *dst = boxes + (size_t)(sl * n_chunks + my_chunk) * NREP * D + (tid & (D - 1));
#pragma unroll
        for (int r = 0; r < NREP; r++) box_store(dst + r * D, sums[r]);
    }
    for (int i = tid; i < n_slices * NREP; i += nthr) {
        const int sl = i / NREP, r = i - sl * NREP;
        float *dst = ml + 2 * ((size_t)(sl * n_chunks + my_chunk) * NREP + r);
        asm volatile("st.relaxed.gpu.global.v2.f32 [%0], {%1, %2};\n" ::"l"(dst), "f"(box_word(s_M[r])), "f"(box_word(s_L[r])) : "memory");
    }
    BK_STAMP(6);
    if (my_chunk >= n_slices) return;
    // ---- receive
    const int d0 = my_chunk * D, n_col = NREP << lg;  // n_col: 16-byte columns of this slice (192 for two chunks)
    const int j_col = tid & (D4 - 1), rest = tid >> lg, grp = rest / NREP, r_col = rest - grp * NREP;
    const int n_grp = (256 >> lg) / NREP;             // thread groups; group g takes chunks g, g + n_grp, ...
    const int n_out = NREP * D;                       // (up to 768 outputs for a slice of half a row)
    constexpr int kPre = 4;                           // enough for every chunk of up to 168 (a.xch_peer: 84); else several rounds
    float *src = boxes + ((size_t)my_chunk * n_chunks * NREP + r_col) * D + 4 * j_col;
    float *my_ml = ml + 2 * (size_t)my_chunk * n_chunks * NREP;
    // the gate of this thread's first output travels with the first loads
    const float *gate = (a.gate && !a.partial) ? a.gate + ((size_t)slot * a.n_head + (size_t)kv * NREP) * a.gate_stride + d0 : nullptr;
    float gate0 = 0.f;
    if (gate && tid < n_out) gate0 = gate[(size_t)(tid >> (lg + 2)) * a.gate_stride + (tid & (D - 1))];
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
    float M = -CUDART_INF_F, L = 0.f;
    if (grp < n_grp) {
        int left = a.box_polls;
        for (int c0 = grp; c0 < n_chunks; c0 += kPre * n_grp) {
            float4 v[kPre];
            float2 x[kPre];
#pragma unroll
            for (int u = 0; u < kPre; u++) {
                const int c = c0 + u * n_grp;
                v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                x[u] = make_float2(-CUDART_INF_F, 0.f);
                if (c < n_chunks) {
                    v[u] = box_load4(src + (size_t)c * NREP * D);
                    x[u] = box_load2(my_ml + 2 * (c * NREP + r_col));
                }
            }
            bool full;
            do {  // words that were empty are read again, all of a thread's together
                full = true;
#pragma unroll
                for (int u = 0; u < kPre; u++) {
                    const int c = c0 + u * n_grp;
                    if (!(box_full4(v[u]) && box_full(x[u].x) && box_full(x[u].y))) {
                        v[u] = box_load4(src + (size_t)c * NREP * D);
                        x[u] = box_load2(my_ml + 2 * (c * NREP + r_col));
                        full = false;
                    }
                }
            } while (!full && --left > 0);
            float Mn = M;
#pragma unroll
            for (int u = 0; u < kPre; u++) Mn = fmaxf(Mn, x[u].x);
            if (c0 > grp) {
                const float f = M > -CUDART_INF_F ? fast_exp2(M - Mn) : 0.f;
                sum.x *= f; sum.y *= f; sum.z *= f; sum.w *= f;
                L *= f;
            }
            M = Mn;
#pragma unroll
            for (int u = 0; u < kPre; u++)
                if (x[u].x > -CUDART_INF_F) {  // an empty chunk's accumulator is never looked at
                    const float f = fast_exp2(x[u].x - M);
                    L = fmaf(x[u].y, f, L);
                    sum.x = fmaf(v[u].x, f, sum.x);
                    sum.y = fmaf(v[u].y, f, sum.y);
                    sum.z = fmaf(v[u].z, f, sum.z);
                    sum.w = fmaf(v[u].w, f, sum.w);
                }
        }
        if (left <= 0) {  // never expected: leave marks, write nothing
            *s_ok = 0;
            asm volatile("st.relaxed.gpu.global.u32 [%0], %1;\n" ::"l"(a.box_state), "r"(0u) : "memory");
        }
    }
    if (!clean) *s_ok = 0;
    float2 *s_ml = reinterpret_cast<float2 *>(red);  // [n_grp][NREP]
    float *s_sum = red + 2 * 256;                     // [n_grp][NREP][D]
    if (grp < n_grp) {
        reinterpret_cast<float4 *>(s_sum)[(grp * NREP + r_col) * D4 + j_col] = sum;
        if (j_col == 0) s_ml[grp * NREP + r_col] = make_float2(M, L);
    }
    float *s_Mg = s_sum + 1024, *s_Lg = s_Mg + 8, *snd = s_Lg + 8;  // context split: what this slice sends
    __syncthreads();
    BK_STAMP(7);
    if (!*s_ok) {
        if (tid == 0) raise_error(err_flag, 6);
        return;
    }
    // ---- merge the groups in a fixed order and write.  Whole warps, because a Givens pair is two neighbouring lanes.
    for (int i0 = tid & ~31; i0 < n_out; i0 += nthr) {
        const int i = i0 + (tid & 31), r_o = i < n_out ? i >> (lg + 2) : 0, d_o = i & (D - 1);
        float Mx = -CUDART_INF_F, Ls = 0.f, o = 0.f;
        for (int g0 = 0; g0 < n_grp; g0 += 8) {
            float2 x[8];
            float v[8], Mn = Mx;
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const bool in = i < n_out && g0 + u < n_grp;
                x[u] = in ? s_ml[(g0 + u) * NREP + r_o] : make_float2(-CUDART_INF_F, 0.f);
                v[u] = in ? s_sum[(g0 + u) * n_out + i] : 0.f;
                Mn = fmaxf(Mn, x[u].x);
            }
            const float keep = Mx > -CUDART_INF_F ? fast_exp2(Mx - Mn) : 0.f;
            Ls *= keep;
            o *= keep;
            Mx = Mn;
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const float f = x[u].x > -CUDART_INF_F ? fast_exp2(x[u].x - Mx) : 0.f;
                Ls = fmaf(x[u].y, f, Ls);
                o = fmaf(v[u], f, o);
            }
        }
        if (v_planar) {  // undo the Givens rotation (src/forward.rs:349)
            const float p = __shfl_xor_sync(0xffffffffu, o, 1);
            const int pr = (d0 + d_o) >> 1;
            float o0, o1;
            givens_inv((i & 1) ? p : o, (i & 1) ? o : p, givens[2 * pr], givens[2 * pr + 1], o0, o1);
            o = (i & 1) ? o1 : o0;
        }
        if (i < n_out) {
            if (a.xch_peer) {
                snd[i] = o;
                if (d_o == 0) {
                    s_Mg[r_o] = Mx;
                    s_Lg[r_o] = Ls;
                }
            } else if (a.partial) {
                float *po = a.out + ((size_t)slot * a.n_head + (size_t)kv * NREP + r_o) * kPartStride;
                po[d0 + d_o] = o;
                if (d0 + d_o == 0) {
                    po[kHd] = Mx * 0.6931471805599453f;  // log2 -> ln
                    po[kHd + 1] = Ls;
                }
            } else {
                o = Ls == 0.f ? 0.f : o / Ls;  // (a sum that is NaN makes a result that is)
                // src/forward.rs:379-382 with src/kernels.rs:162: out *= 1 / (1 + exp(-gate))
                if (gate) o *= 1.0f / (1.0f + expf(-(i == tid ? gate0 : gate[(size_t)r_o * a.gate_stride + d_o])));
                a.out[((size_t)slot * a.n_head + (size_t)kv * NREP + r_o) * kHd + d0 + d_o] = o;
            }
        }
    }
    BK_STAMP(8);
    // ---- empty the boxes again (behind the output: only the end of the launch waits for it).  Everything this CTA
    // owns has been read.
    {
        float4 *p = reinterpret_cast<float4 *>(boxes + (size_t)my_chunk * n_chunks * NREP * D);
        const float e = __uint_as_float(kEmptyWord);
        for (int i = tid; i < n_chunks * n_col; i += nthr) p[i] = make_float4(e, e, e, e);
        for (int i = tid; i < n_chunks * NREP; i += nthr) reinterpret_cast<float2 *>(my_ml)[i] = make_float2(e, e);
    }
    if (a.xch_peer) {  // context split: this slice goes to every rank and is merged with theirs
        __syncthreads();
        exchange_slice(a, NREP, slot, kv, d0, D, snd, s_Mg, s_Lg);
    }
}

template <int NREP, bool STREAM = false>
__device__ __forceinline__ void finish_item(const DecodeArgs &a, int slot, int s, int kv, int item, int n_chunks,
                                            int first_item, float *s_acc /* [NREP][kHd] */, float *s_M, float *s_L,
                                            int *s_last, bool v_planar,
                                            const float *givens = nullptr /* shared-memory copy, if the caller has one */,
                                            FinishSmem fs = FinishSmem()) {
    // the chunks' factors: at the front of the caller's region in the streamed form, which would otherwise lose a
    // ring stage to them
    constexpr uint32_t kFactorBytes = (kFactorCap * NREP + 8) * sizeof(float);
    float *s_f;
    if constexpr (STREAM) {
        s_f = reinterpret_cast<float *>(fs.ptr);
        fs.ptr += kFactorBytes;
        fs.addr += kFactorBytes;
        fs.bytes -= kFactorBytes;
    } else {
        __shared__ float s_static[kFactorCap * NREP + 8];
        s_f = s_static;
    }
    float *s_scale = s_f + kFactorCap * NREP;
    // the first 256 threads work; a larger CTA's remaining threads only take part in the barriers
    const int tid = threadIdx.x, nt = 256;
    const bool act = threadIdx.x < 256;
    const int tid0 = act ? tid : (1 << 30);  // loop start that keeps idle threads out of strided loops
    const int warp = tid >> 5, lane = tid & 31;
    // gate values of this thread's outputs (coordinate tid of every head); the CTA that writes the
    // output fetches them as early as it knows it is the one, so they travel with the partials
    const float *gate = (a.gate && !a.partial && act)
                            ? a.gate + ((size_t)slot * a.n_head + (size_t)kv * NREP) * a.gate_stride + tid : nullptr;
    float gv[NREP];
    auto load_gate = [&]() {
#pragma unroll
        for (int r = 0; r < NREP; r++) gv[r] = gate ? gate[(size_t)r * a.gate_stride] : 0.f;
    };
    if (n_chunks <= 1) load_gate();
    if (n_chunks > 1) {
        float *part = a.partials + ((size_t)item * NREP) * kScratchStride;
        for (int i = tid0; i < NREP * kHd; i += nt) {
            const int r = i / kHd, d = i - r * kHd;
            part[(size_t)r * kScratchStride + d] = s_acc[i];
        }
        if (tid < NREP) {
            part[(size_t)tid * kScratchStride + kHd] = s_M[tid];
            part[(size_t)tid * kScratchStride + kHd + 1] = s_L[tid];
        }
        // Publish: the barrier orders every thread's stores before thread 0's release, which
        // makes them visible to whoever later acquires the counter (cumulativity), so no thread
        // needs a full __threadfence().
        __syncthreads();
        if (tid == 0) {
            cuda::atomic_ref<unsigned, cuda::thread_scope_device> cnt(a.counters[s * a.n_kv + kv]);
            const unsigned ticket = cnt.fetch_add(1u, cuda::memory_order_acq_rel);
            *s_last = (ticket == (unsigned)(n_chunks - 1));
        }
        if (STREAM) asm volatile("fence.proxy.async;\n" ::: "memory");  // this thread's shared-memory traffic before the copies below
        __syncthreads();
        if (!*s_last) return;
        const float *base = a.partials + (size_t)first_item * NREP * kScratchStride;
        constexpr uint32_t kChunkBytes = NREP * kScratchStride * sizeof(float);
        const int cap = STREAM ? min((int)((fs.bytes / 2) / kChunkBytes), 32) : 0;  // chunks per half
        if (STREAM && cap >= 1 && fs.bytes >= (blockDim.x >> 6) * NREP * kHd * sizeof(float)) {
            // ---- streamed combine: chunks arrive through the TMA engine, two rounds in flight ------
            const int n_rounds = (n_chunks + cap - 1) / cap;
            const uint32_t half_bytes = (uint32_t)cap * kChunkBytes;
            auto issue_round = [&](int rd) {
                const int c0 = rd * cap, nc = min(cap, n_chunks - c0);
                const uint32_t bar = fs.bar + (uint32_t)(rd & 1) * 8u, dst = fs.addr + (uint32_t)(rd & 1) * half_bytes;
                mbar_expect_tx(bar, (uint32_t)nc * kChunkBytes);
                for (int c = 0; c < nc; c++)
                    tma_bulk(dst + (uint32_t)c * kChunkBytes, base + (size_t)(c0 + c) * NREP * kScratchStride, kChunkBytes, bar);
            };
            if (tid == 0) {
                // the other CTAs' stores (generic proxy, acquired through the ticket) before the async-proxy reads
                asm volatile("fence.proxy.async;\n" ::: "memory");
                issue_round(0);
                if (n_rounds > 1) issue_round(1);
            }
            load_gate();
            const int n_g = (int)blockDim.x >> 6, rg = tid >> 6, x = tid & 63;  // 64 threads span a row with float4
            float4 sum[NREP];
#pragma unroll
            for (int r = 0; r < NREP; r++) sum[r] = make_float4(0.f, 0.f, 0.f, 0.f);
            float M_run = -CUDART_INF_F, L_run = 0.f;  // warp r < NREP: running max and sum of head r
            for (int rd = 0; rd < n_rounds; rd++) {
                const int nc = min(cap, n_chunks - rd * cap);
                const uint32_t bar = fs.bar + (uint32_t)(rd & 1) * 8u, parity = (uint32_t)(rd >> 1) & 1u;
                int polls = 0;
                while (!mbar_try_wait(bar, parity)) {
                    if (++polls > kWaitPolls) {  // never expected; leave a mark and go on rather than hang
                        if (tid == 0) raise_error(fs.err_flag, 3);
                        break;
                    }
                }
                const float *H = reinterpret_cast<const float *>(fs.ptr + (size_t)(rd & 1) * half_bytes);
                if (warp < NREP) {  // one warp per head: this round's factors, online in the running max
                    const int r = warp;
                    const bool valid = lane < nc;
                    const float2 ml = valid ? *reinterpret_cast<const float2 *>(H + ((size_t)lane * NREP + r) * kScratchStride + kHd)
                                            : make_float2(-CUDART_INF_F, 0.f);
                    float mx = ml.x;
#pragma unroll
                    for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
                    const float Mn = fmaxf(M_run, mx);
                    const float fc = ml.x > -CUDART_INF_F ? exp2f(ml.x - Mn) : 0.f;
                    const float keep = M_run > -CUDART_INF_F ? exp2f(M_run - Mn) : 0.f;
                    float ls = ml.y * fc;
#pragma unroll
                    for (int off = 16; off > 0; off >>= 1) ls += __shfl_xor_sync(0xffffffffu, ls, off);
                    L_run = fmaf(L_run, keep, ls);
                    M_run = Mn;
                    if (valid) s_f[lane * NREP + r] = fc;
                    if (lane == 0) s_scale[r] = keep;
                }
                __syncthreads();
#pragma unroll
                for (int r = 0; r < NREP; r++) {
                    const float k = s_scale[r];
                    sum[r].x *= k; sum[r].y *= k; sum[r].z *= k; sum[r].w *= k;
                }
                for (int c = rg; c < nc; c += n_g) {
#pragma unroll
                    for (int r = 0; r < NREP; r++) {
                        const float4 v = reinterpret_cast<const float4 *>(H + ((size_t)c * NREP + r) * kScratchStride)[x];
                        const float f = s_f[c * NREP + r];
                        sum[r].x = fmaf(v.x, f, sum[r].x);
                        sum[r].y = fmaf(v.y, f, sum[r].y);
                        sum[r].z = fmaf(v.z, f, sum[r].z);
                        sum[r].w = fmaf(v.w, f, sum[r].w);
                    }
                }
                __syncthreads();  // this half and the factors are free again
                if (tid == 0 && rd + 2 < n_rounds) issue_round(rd + 2);
            }
            if (warp < NREP && lane == 0) {
                s_M[warp] = M_run;
                s_L[warp] = L_run;
            }
            // the groups' sums meet in the first half (every copy into it has been consumed), fixed order
            float4 *scratch = reinterpret_cast<float4 *>(fs.ptr);  // [n_g][NREP][64]
#pragma unroll
            for (int r = 0; r < NREP; r++) scratch[((size_t)rg * NREP + r) * 64 + x] = sum[r];
            __syncthreads();
            if (act) {
                const float *sf = reinterpret_cast<const float *>(fs.ptr);
#pragma unroll
                for (int r = 0; r < NREP; r++) {
                    float t = 0.f;
                    for (int g2 = 0; g2 < n_g; g2++) t += sf[((size_t)g2 * NREP + r) * kHd + tid];
                    s_acc[r * kHd + tid] = t;
                }
            }
            if (tid == 0) a.counters[s * a.n_kv + kv] = 0;  // ready for the next launch
            __syncthreads();
        } else {
        // 64 threads span one 256-float row with float4 loads; the four 64-thread groups take
        // every fourth chunk.  The (head, chunk) pairs of a thread form one flat list walked 24
        // independent 16-byte loads at a time.  The first batch is issued before the m/l sweep
        // below so that both travel in the same L2 round trip.
        const int rg = tid >> 6, x = tid & 63;
        const int per_rg = (n_chunks - rg + 3) / 4;  // chunks rg, rg+4, ...
        const int n_pairs = act ? per_rg * NREP : 0;
        constexpr int kBatch = (NREP == 6) ? 30 : 32;  // a multiple of NREP: slot u is always head u % NREP
        float4 v[kBatch];
        auto load_batch = [&](int i0) {
#pragma unroll
            for (int u = 0; u < kBatch; u++) {
                const int i = i0 + u, r = u % NREP;
                const int c = rg + 4 * (i / NREP);
                if (i < n_pairs)
                    v[u] = __ldcg(reinterpret_cast<const float4 *>(base + ((size_t)c * NREP + r) * kScratchStride) + x);
                else
                    v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        };
        load_batch(0);
        load_gate();
        // one warp per head: global max, the chunks' rescale factors and the merged l, from one
        // sweep over the (m, l) pairs
        if (warp < NREP) {
            const int r = warp;
            constexpr int kPer = kFactorCap / 32;  // (m, l) pairs a lane keeps in registers
            float2 ml[kPer];
            float M = -CUDART_INF_F;
#pragma unroll
            for (int u = 0; u < kPer; u++) {
                const int c = lane + 32 * u;
                ml[u] = make_float2(-CUDART_INF_F, 0.f);
                if (c < n_chunks)
                    ml[u] = __ldcg(reinterpret_cast<const float2 *>(base + ((size_t)c * NREP + r) * kScratchStride + kHd));
                M = fmaxf(M, ml[u].x);
            }
            for (int c = kFactorCap + lane; c < n_chunks; c += 32)  // beyond the cached range (rare)
                M = fmaxf(M, __ldcg(base + ((size_t)c * NREP + r) * kScratchStride + kHd));
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
            float Lsum = 0.f;
#pragma unroll
            for (int u = 0; u < kPer; u++) {
                const int c = lane + 32 * u;
                const float f = ml[u].x > -CUDART_INF_F ? exp2f(ml[u].x - M) : 0.f;
                Lsum = fmaf(ml[u].y, f, Lsum);
                if (c < n_chunks) s_f[c * NREP + r] = f;
            }
            for (int c = kFactorCap + lane; c < n_chunks; c += 32) {
                const float2 x2 = __ldcg(reinterpret_cast<const float2 *>(base + ((size_t)c * NREP + r) * kScratchStride + kHd));
                Lsum = fmaf(x2.y, x2.x > -CUDART_INF_F ? exp2f(x2.x - M) : 0.f, Lsum);
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) Lsum += __shfl_xor_sync(0xffffffffu, Lsum, off);
            if (lane == 0) {
                s_M[r] = M;
                s_L[r] = Lsum;
            }
        }
        __syncthreads();
        float4 sum[NREP];
#pragma unroll
        for (int r = 0; r < NREP; r++) sum[r] = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int i0 = 0; i0 < n_pairs; i0 += kBatch) {
            if (i0 > 0) load_batch(i0);
#pragma unroll
            for (int u = 0; u < kBatch; u++) {
                const int i = i0 + u, r = u % NREP;
                const int c = rg + 4 * (i / NREP);
                float f = 0.f;
                if (i < n_pairs) {
                    if (c < kFactorCap) f = s_f[c * NREP + r];
                    else {
                        const float mc = __ldcg(base + ((size_t)c * NREP + r) * kScratchStride + kHd);
                        f = mc > -CUDART_INF_F ? exp2f(mc - s_M[r]) : 0.f;
                    }
                }
                sum[r].x = fmaf(v[u].x, f, sum[r].x);
                sum[r].y = fmaf(v[u].y, f, sum[r].y);
                sum[r].z = fmaf(v[u].z, f, sum[r].z);
                sum[r].w = fmaf(v[u].w, f, sum[r].w);
            }
        }
        // fixed order over the four groups keeps the result deterministic
        for (int gsel = 0; gsel < 4; gsel++) {
            if (rg == gsel) {
#pragma unroll
                for (int r = 0; r < NREP; r++) {
                    float4 *dst = reinterpret_cast<float4 *>(s_acc + r * kHd) + x;
                    if (gsel == 0) *dst = sum[r];
                    else {
                        float4 o = *dst;
                        o.x += sum[r].x; o.y += sum[r].y; o.z += sum[r].z; o.w += sum[r].w;
                        *dst = o;
                    }
                }
            }
            __syncthreads();
        }
        if (tid == 0) a.counters[s * a.n_kv + kv] = 0;  // ready for the next launch
        __syncthreads();
        }
    }

    if (v_planar) {
        for (int i = tid0; i < NREP * (kHd / 2); i += nt) {
            const int r = i / (kHd / 2), pr = i - r * (kHd / 2);
            float o0, o1;
            const float *gv = givens ? givens : a.givens;
            givens_inv(s_acc[r * kHd + 2 * pr], s_acc[r * kHd + 2 * pr + 1], gv[2 * pr], gv[2 * pr + 1],
                       o0, o1);
            s_acc[r * kHd + 2 * pr] = o0;
            s_acc[r * kHd + 2 * pr + 1] = o1;
        }
        __syncthreads();
    }
    if (a.xch_peer) {
        // ---- context split: send this kv head's rows to every rank, wait for everybody's, merge ----
        exchange_slice(a, NREP, slot, kv, 0, kHd, s_acc, s_M, s_L);
    } else if (a.partial) {
        float *out = a.out + ((size_t)slot * a.n_head + (size_t)kv * NREP) * kPartStride;
        for (int i = tid0; i < NREP * kHd; i += nt) {
            const int r = i / kHd, d = i - r * kHd;
            out[(size_t)r * kPartStride + d] = s_acc[i];
        }
        if (tid < NREP) {
            out[(size_t)tid * kPartStride + kHd] = s_M[tid] * 0.6931471805599453f;  // log2 -> ln
            out[(size_t)tid * kPartStride + kHd + 1] = s_L[tid];
        }
    } else {
        float *out = a.out + ((size_t)slot * a.n_head + (size_t)kv * NREP) * kHd;
        if (act) {
#pragma unroll
            for (int r = 0; r < NREP; r++) {
                const float Ls = s_L[r];
                float o = Ls == 0.f ? 0.f : s_acc[r * kHd + tid] / Ls;  // (a sum that is NaN makes a result that is)
                // src/forward.rs:379-382 with src/kernels.rs:162: out *= 1 / (1 + exp(-gate))
                if (gate) o *= 1.0f / (1.0f + expf(-gv[r]));
                out[r * kHd + tid] = o;
            }
        }
    }
}

}  // namespace bk
