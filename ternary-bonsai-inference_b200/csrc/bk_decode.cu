// GQA decode attention over the KV cache: split-K flash decoding, all cache modes.
// Replaces attn_scores*.comp + softmax_inplace.comp + attn_out*.comp (7 dispatches per layer
// in src/gdev.rs:584-829) and the CPU loop src/forward.rs:287-375 with one launch.
//
// Work item = (sequence, kv head, chunk of positions); one CTA of 8 warps per item.  A warp
// takes every 8th position of the chunk; its 32 lanes split the 256 coordinates of a row, so a
// row is read once with full-width coalesced loads and serves all q heads of the GQA group
// (the reference reads every row once per q head).  Scores are completed with xor-shuffle
// reductions, the softmax is the online (running max / running sum) form in the exp2 domain,
// and V is accumulated in registers.  Warps merge through shared memory, CTAs through a
// partials buffer in global memory; the CTA that arrives last for a (sequence, kv head)
// combines the chunks, undoes the Givens rotation for planar V and writes the output, so there
// is no second launch.  No CTA ever waits on another.
//
// Algorithmic traffic per (position, kv head): K row + V row (+ 2 norms); q and out once.
#include <math_constants.h>

#include <algorithm>

#include "bk_decode_common.cuh"

namespace bk {

namespace {

constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;

// Coordinate held in slot e (0..7) of lane l.  Planar and f16 rows: 8 consecutive coordinates
// (one packed group / one 16-byte load).  f32 rows: two float4 halves 128 coordinates apart so
// that both loads are fully coalesced.
template <int KIND>
__device__ __forceinline__ int dim_of(int lane, int e) {
    if constexpr (KIND == ROW_F32) return (e < 4) ? lane * 4 + e : 128 + lane * 4 + (e - 4);
    else return lane * 8 + e;
}

template <int KIND>
struct RawRow {};
template <>
struct RawRow<ROW_F32> { float4 a, b; };
template <>
struct RawRow<ROW_F16> { uint4 a; };

template <int KIND>
__device__ __forceinline__ RawRow<KIND> load_row(const uint8_t *row, int lane) {
    RawRow<KIND> x;
    if constexpr (KIND == ROW_F32) {
        x.a = reinterpret_cast<const float4 *>(row)[lane];
        x.b = reinterpret_cast<const float4 *>(row)[32 + lane];
    } else {
        x.a = reinterpret_cast<const uint4 *>(row)[lane];
    }
    return x;
}

// Expand a raw row piece to 8 floats.
template <int KIND>
__device__ __forceinline__ void expand_row(const RawRow<KIND> &x, float (&v)[8]) {
    if constexpr (KIND == ROW_F32) {
        v[0] = x.a.x; v[1] = x.a.y; v[2] = x.a.z; v[3] = x.a.w;
        v[4] = x.b.x; v[5] = x.b.y; v[6] = x.b.z; v[7] = x.b.w;
    } else {
        const uint32_t w[4] = {x.a.x, x.a.y, x.a.z, x.a.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            v[2 * i] = half_bits_to_f32((uint16_t)(w[i] & 0xffffu));
            v[2 * i + 1] = half_bits_to_f32((uint16_t)(w[i] >> 16));
        }
    }
}

template <int KIND, int NREP>
__global__ void __launch_bounds__(kThreads) decode_kernel(DecodeArgs a, DecodeMeta meta) {
    __shared__ __align__(16) float s_q[NREP][kHd];       // roped q; later the merged acc
    __shared__ float s_m[kWarps][NREP], s_l[kWarps][NREP];
    __shared__ float s_M[NREP], s_L[NREP];
    __shared__ int s_last;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    // ---- which item --------------------------------------------------------
    const int item = blockIdx.x;
    int s = 0;
    while (s + 1 < meta.n_seqs && meta.item_start[s + 1] <= item) s++;
    const int n_pos = meta.n_pos[s];
    const int L = meta.chunk_len;
    const int n_chunks = (n_pos + L - 1) / L;
    const int local = item - meta.item_start[s];
    const int kv = local / n_chunks, chunk = local - kv * n_chunks;
    const int p0 = chunk * L, p1 = min(p0 + L, n_pos);
    const int seq = meta.seq_id[s];

    // ---- q: rope, fold scale*log2(e) ------------------------------------------
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    {
        const float *q = a.q + ((size_t)meta.slot[s] * a.n_head + (size_t)kv * NREP) * kHd;
        for (int i = tid; i < NREP * kHd; i += kThreads) (&s_q[0][0])[i] = q[i];
        __syncthreads();
        if (!a.no_rope) {
            const int half = a.n_rot >> 1;
            const float2 *cs = a.rope + (size_t)meta.q_pos[s] * half;
            for (int i = tid; i < NREP * half; i += kThreads) {
                const int r = i / half, j = i - r * half;
                float x0 = s_q[r][j], x1 = s_q[r][j + half];
                rope_pair(x0, x1, cs[j]);
                s_q[r][j] = x0;
                s_q[r][j + half] = x1;
            }
            __syncthreads();
        }
    }
    const float qscale = rsqrtf((float)kHd) * 1.4426950408889634f;  // 1/sqrt(hd) * log2(e)
    float qr[NREP][8];
#pragma unroll
    for (int r = 0; r < NREP; r++)
#pragma unroll
        for (int e = 0; e < 8; e++) qr[r][e] = s_q[r][dim_of<KIND>(lane, e)] * qscale;

    // ---- scan --------------------------------------------------------------
    float m[NREP], l[NREP], acc[NREP][8];
#pragma unroll
    for (int r = 0; r < NREP; r++) {
        m[r] = -CUDART_INF_F;
        l[r] = 0.f;
#pragma unroll
        for (int e = 0; e < 8; e++) acc[r][e] = 0.f;
    }
    const size_t seq_rows = (size_t)seq * a.seq_stride_rows;
    int p = p0 + warp;
    RawRow<KIND> kraw{}, vraw{};
    if (p < p1) {
        const size_t r = seq_rows + (size_t)p * a.n_kv + kv;
        kraw = load_row<KIND>(a.k_rows + r * a.k_row_bytes, lane);
        vraw = load_row<KIND>(a.v_rows + r * a.v_row_bytes, lane);
    }
    while (p < p1) {
        const RawRow<KIND> kc = kraw, vc = vraw;
        const int pn = p + kWarps;
        if (pn < p1) {  // prefetch the warp's next position
            const size_t r = seq_rows + (size_t)pn * a.n_kv + kv;
            kraw = load_row<KIND>(a.k_rows + r * a.k_row_bytes, lane);
            vraw = load_row<KIND>(a.v_rows + r * a.v_row_bytes, lane);
        }
        float kvv[8];
        expand_row<KIND>(kc, kvv);
        float sc[NREP];
#pragma unroll
        for (int r = 0; r < NREP; r++) {
            float d = 0.f;
#pragma unroll
            for (int e = 0; e < 8; e++) d = fmaf(qr[r][e], kvv[e], d);
            sc[r] = d;
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
#pragma unroll
            for (int r = 0; r < NREP; r++) sc[r] += __shfl_xor_sync(0xffffffffu, sc[r], off);
        float vv[8];
        expand_row<KIND>(vc, vv);
#pragma unroll
        for (int r = 0; r < NREP; r++) {
            const float sr = sc[r];
            if (sr > m[r]) {
                const float corr = exp2f(m[r] - sr);  // 0 on the first position (m = -inf)
                l[r] *= corr;
#pragma unroll
                for (int e = 0; e < 8; e++) acc[r][e] *= corr;
                m[r] = sr;
            }
            const float pr = exp2f(sr - m[r]);
            l[r] += pr;
#pragma unroll
            for (int e = 0; e < 8; e++) acc[r][e] = fmaf(pr, vv[e], acc[r][e]);
        }
        p = pn;
    }

    // ---- merge the 8 warps --------------------------------------------------
    if (lane == 0)
#pragma unroll
        for (int r = 0; r < NREP; r++) {
            s_m[warp][r] = m[r];
            s_l[warp][r] = l[r];
        }
    __syncthreads();  // also: every warp is done reading s_q
    if (tid < NREP) {
        float M = -CUDART_INF_F;
        for (int w = 0; w < kWarps; w++) M = fmaxf(M, s_m[w][tid]);
        float Lsum = 0.f;
        for (int w = 0; w < kWarps; w++)  // (without a maximum: no row, or none but NaN, which the sum tells)
            Lsum += s_l[w][tid] * (s_m[w][tid] > -CUDART_INF_F ? exp2f(s_m[w][tid] - M) : 0.f);
        s_M[tid] = M;
        s_L[tid] = Lsum;
    }
    for (int i = tid; i < NREP * kHd; i += kThreads) (&s_q[0][0])[i] = 0.f;
    __syncthreads();
    for (int w = 0; w < kWarps; w++) {  // fixed order keeps the sum deterministic
        if (warp == w) {
#pragma unroll
            for (int r = 0; r < NREP; r++) {
                const float f = (m[r] > -CUDART_INF_F) ? exp2f(m[r] - s_M[r]) : 0.f;
#pragma unroll
                for (int e = 0; e < 8; e++) s_q[r][dim_of<KIND>(lane, e)] += acc[r][e] * f;
            }
        }
        __syncthreads();
    }

    // ---- merge the chunks of this (sequence, kv head), write ------
    const int first_item = meta.item_start[s] + kv * n_chunks;
    finish_item<NREP>(a, meta.slot[s], s, kv, item, n_chunks, first_item, &s_q[0][0], s_M, s_L, &s_last, false);
}

// ---- planar rows ------------------------------------------------------------------------------------------
// The same split of the work and the same f32 arithmetic for planar K rows (V planar or f32), arranged by what bounds it, the
// instructions per row.  A warp takes four consecutive positions at a time:
//   * a centroid is one conflict-free shared-memory read from a table with a column per lane (a plain table has three or four lanes
//     on a bank); for 8 bits the entries are 256 bytes apart and the table 64 KiB aligned, so that one byte permute makes the address;
//   * products run as pairs of f32;
//   * 4 x NREP sums over 32 lanes take 27 shuffles for six heads (120 as butterflies): a lane keeps half of its sums at every
//     step.  It never has to choose which: it loads the positions, and holds q's heads, in an order that makes the sums it
//     keeps the first ones.  At the end a lane has the scores of one position and half of the heads, and does that part of the softmax;
//   * the weights come back through shared memory as pairs, two positions a read; the running maxima move under one vote.
// rows come through a ring of three groups a warp (cp.async): loaded into registers a group ahead, they are
//     waited for (8 bit, 131000 rows: 182 to 235 us a layer).
// Measured (24 q heads on 4, us a layer of a 16-layer step, append included, a row a step before / now): 8 bit, 40 rows 23 / 15, 100 rows 27 / 17, 1000 rows
// 28 / 20, 9000 rows 90 / 32, 32768 rows 155 / 55, 131000 rows 370 / 145; 5 bit, 9000 rows 103 / 31; 8 bit K beside f32 V, 9000 rows 87 / 33.
// 177 instructions a row now (215 with rows loaded into registers); the f32 pipe is the busiest.  With twelve warps (168 registers) 56 to 84 bytes
// spill for four and six heads, none for one and two.
constexpr int kGroup = 4;  // positions a warp works on at a time

// More than twelve warps do not fit with q and the sums of six heads in registers (168 each); eight heads, or rows of f32, want 255.
template <int VK, int NREP>
constexpr int kPlanarWarps = (VK == ROW_PLANAR && NREP <= 6) ? 12 : 8;
// Bytes from one centroid's 32 copies to the next one's (beside f32 rows there is no room for the wide form).
template <int VK, int BITS>
constexpr uint32_t kTabStride = BITS == 8 && VK == ROW_PLANAR ? 256 : 128;
template <int VK, int BITS>
constexpr uint32_t kTabBytes = kTabStride<VK, BITS> << BITS;
// A stage: a group's K rows, V rows and 2 x 4 norms.  A warp has three.
constexpr int kStages = 3;
template <int BITS>
constexpr uint32_t kGroupK = kGroup * 32 * BITS;
template <int VK, int BITS>
constexpr uint32_t kGroupV = VK == ROW_PLANAR ? kGroupK<BITS> : kGroup * kHd * 4;
template <int VK, int BITS>
constexpr uint32_t kStageBytes = (kGroupK<BITS> + kGroupV<VK, BITS> + 32 + 127) / 128 * 128;
template <int VK, int BITS, int NREP>
constexpr uint32_t kRingBytes = kPlanarWarps<VK, NREP> * kStages * kStageBytes<VK, BITS>;
// The ring, then the table, aligned to its size; the warps' sums take the place of both.
template <int VK, int BITS, int NREP>
constexpr uint32_t kPlanarSmem = std::max(kRingBytes<VK, BITS, NREP> + 2 * kTabBytes<VK, BITS>, (uint32_t)(kPlanarWarps<VK, NREP> * NREP * kHd * 4));

// Eight indices -> eight centroids as four pairs.  tab: the aligned table's shared-memory address plus 4 * lane.
template <int BITS, uint32_t STRIDE>
__device__ __forceinline__ void expand_group(uint64_t packed, uint32_t tab, uint64_t (&v)[4]) {
    float f[8];
#pragma unroll
    for (int e = 0; e < 8; e++) {
        uint32_t at;
        if constexpr (STRIDE == 256) at = __byte_perm((uint32_t)(packed >> (e & 4 ? 32 : 0)), tab, 0x7604u | (uint32_t)((e & 3) << 4));
        else at = (((uint32_t)(packed >> (BITS * e)) & ((1u << BITS) - 1u)) << 7) | tab;
        asm("ld.shared.f32 %0, [%1];\n" : "=f"(f[e]) : "r"(at));
    }
#pragma unroll
    for (int i = 0; i < 4; i++) v[i] = pack2(f[2 * i], f[2 * i + 1]);
}

template <int VK, int BITS, int NREP>
__global__ void __launch_bounds__(kPlanarWarps<VK, NREP> * 32, 1) decode_planar_kernel(const __grid_constant__ DecodeArgs a,
                                                                                      const __grid_constant__ DecodeMeta meta) {
    constexpr int kW = kPlanarWarps<VK, NREP>, kNT = kW * 32;
    constexpr int kHalf = NREP % 2 == 0 ? NREP / 2 : NREP;  // heads whose scores a lane ends up with
    constexpr uint32_t kTab = kTabBytes<VK, BITS>, kStride = kTabStride<VK, BITS>, kStage = kStageBytes<VK, BITS>;
    extern __shared__ __align__(128) uint8_t dyn[];         // see kPlanarSmem
    __shared__ __align__(16) float s_q[NREP][kHd];          // roped and rotated q; later the merged sums
    __shared__ __align__(16) float2 s_w[kW][2][NREP][kGroup];  // a warp's weights, twice each
    __shared__ float s_m[kW][NREP], s_l[kW][NREP];
    __shared__ float s_M[NREP], s_L[NREP];
    __shared__ int s_last;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    // ---- which item --------------------------------------------------------
    const int item = blockIdx.x;
    int s = 0;
    while (s + 1 < meta.n_seqs && meta.item_start[s + 1] <= item) s++;
    const int n_pos = meta.n_pos[s], L = meta.chunk_len, n_chunks = (n_pos + L - 1) / L;
    const int local = item - meta.item_start[s], kv = local / n_chunks, chunk = local - kv * n_chunks;
    const int p0 = chunk * L, p1 = min(p0 + L, n_pos);

    // ---- the table: it is constant, so it is filled under the end of the kernel before ----
    const uint32_t raw = (uint32_t)__cvta_generic_to_shared(dyn), base = (raw + kRingBytes<VK, BITS, NREP> + kTab - 1) & ~(kTab - 1);
    uint8_t *const table = dyn + (base - raw);
    for (int i = tid; i < 8 << BITS; i += kNT) {
        const float c = __ldg(a.book + (i >> 3));
        *reinterpret_cast<float4 *>(table + (uint32_t)(i >> 3) * kStride + (i & 7) * 16) = make_float4(c, c, c, c);
    }
    asm volatile("griddepcontrol.wait;\n" ::: "memory");

    // ---- the first groups' rows ----
    const uint8_t *const ring = dyn + (uint32_t)warp * (kStages * kStage);
    const uint32_t ring_at = raw + (uint32_t)warp * (kStages * kStage);
    const size_t row_base = (size_t)meta.seq_id[s] * a.seq_stride_rows + kv;
    const uint32_t k_pitch = (uint32_t)a.n_kv * (uint32_t)a.k_row_bytes, v_pitch = (uint32_t)a.n_kv * (uint32_t)a.v_row_bytes;
    auto copy = [&](uint32_t dst, const void *src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory"); };
    auto issue = [&](int g, int stage) {  // rows past the chunk: its last row stands in, without weight
        if (g < p1) {
            const int last = p1 - 1 - g;
            const size_t r = row_base + (size_t)g * a.n_kv;
            const uint32_t at = ring_at + (uint32_t)stage * kStage;
            const uint8_t *kr = a.k_rows + r * a.k_row_bytes, *vr = a.v_rows + r * a.v_row_bytes;
            constexpr int kChunksK = 2 * BITS, kChunksV = kGroupV<VK, BITS> / (kGroup * 16);  // 16-byte pieces of a row
#pragma unroll
            for (int c0 = 0; c0 < kGroup * kChunksK; c0 += 32) {
                const int c = c0 + lane, row = c / kChunksK;
                if (c0 + 32 <= kGroup * kChunksK || c < kGroup * kChunksK)
                    copy(at + c * 16, kr + (uint32_t)min(row, last) * k_pitch + (c - row * kChunksK) * 16);
            }
#pragma unroll
            for (int c0 = 0; c0 < kGroup * kChunksV; c0 += 32) {
                const int c = c0 + lane, row = c / kChunksV;
                if (c0 + 32 <= kGroup * kChunksV || c < kGroup * kChunksV)
                    copy(at + kGroupK<BITS> + c * 16, vr + (uint32_t)min(row, last) * v_pitch + (c - row * kChunksV) * 16);
            }
            if (lane < (VK == ROW_PLANAR ? 2 * kGroup : kGroup)) {
                const float *norms = lane < kGroup ? a.k_norms : a.v_norms;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(at + kGroupK<BITS> + kGroupV<VK, BITS> + lane * 4),
                             "l"(norms + r + (uint32_t)min(lane & (kGroup - 1), last) * (uint32_t)a.n_kv)
                             : "memory");
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    int g = p0 + warp * kGroup;
    for (int i = 0; i < kStages - 1; i++) issue(g + i * (kW * kGroup), i);

    // ---- q: rope, Givens rotation (the rows are rotated unit vectors, src/forward.rs:304) -------------------------------------
    {
        const float *q = a.q + ((size_t)meta.slot[s] * a.n_head + (size_t)kv * NREP) * kHd;
        for (int i = tid; i < NREP * kHd; i += kNT) (&s_q[0][0])[i] = q[i];
        __syncthreads();
        if (!a.no_rope) {
            const int half = a.n_rot >> 1;
            const float2 *cs = a.rope + (size_t)meta.q_pos[s] * half;
            for (int i = tid; i < NREP * half; i += kNT) {
                const int r = i / half, j = i - r * half;
                float x0 = s_q[r][j], x1 = s_q[r][j + half];
                rope_pair(x0, x1, cs[j]);
                s_q[r][j] = x0;
                s_q[r][j + half] = x1;
            }
            __syncthreads();
        }
        for (int i = tid; i < NREP * (kHd / 2); i += kNT) {
            const int r = i / (kHd / 2), pr = i - r * (kHd / 2);
            float o0, o1;
            givens_fwd(s_q[r][2 * pr], s_q[r][2 * pr + 1], a.givens[2 * pr], a.givens[2 * pr + 1], o0, o1);
            s_q[r][2 * pr] = o0;
            s_q[r][2 * pr + 1] = o1;
        }
        __syncthreads();
    }
    // The lane's place: it ends up with position `mine` of a group and the heads head0 .. head0 + kHalf - 1.  Sum slot (j, h) of a lane is
    // for position j ^ mine and head (h + head0) % NREP.
    const int mine = lane >> 3, head0 = kHalf < NREP && (lane & 4) ? kHalf : 0;
    const float qscale = rsqrtf((float)kHd) * 1.4426950408889634f;  // 1/sqrt(hd) * log2(e)
    uint64_t qr[NREP][4], acc[NREP][4];
#pragma unroll
    for (int h = 0; h < NREP; h++) {
        const int head = h + head0 < NREP ? h + head0 : h + head0 - NREP;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            qr[h][i] = pack2(s_q[head][lane * 8 + 2 * i] * qscale, s_q[head][lane * 8 + 2 * i + 1] * qscale);
            acc[h][i] = 0;
        }
    }
    float m[kHalf], l[kHalf];
#pragma unroll
    for (int i = 0; i < kHalf; i++) m[i] = -CUDART_INF_F, l[i] = 0.f;

    // ---- scan --------------------------------------------------------------
    const uint32_t tab = base + lane * 4;
    int st = 0;
    for (int turn = 0; g < p1; turn ^= 1) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kStages - 2) : "memory");
        __syncwarp();  // the group is there, and the one before it has been read
        issue(g + (kStages - 1) * (kW * kGroup), st == 0 ? kStages - 1 : st - 1);
        const uint8_t *const k_rows = ring + (uint32_t)st * kStage, *const v_rows = k_rows + kGroupK<BITS>;
        const float *const norms = reinterpret_cast<const float *>(v_rows + kGroupV<VK, BITS>);
        const float kn = norms[mine], vn = VK == ROW_PLANAR ? norms[kGroup + mine] : 1.f;
        float sc[kGroup][NREP];
#pragma unroll
        for (int j = 0; j < kGroup; j++) {
            uint64_t k2[4];
            expand_group<BITS, kStride>(load_group8<BITS>(k_rows + (j ^ mine) * (32 * BITS), lane), tab, k2);
#pragma unroll
            for (int h = 0; h < NREP; h++) {
                uint64_t d = mul2(qr[h][0], k2[0]);
#pragma unroll
                for (int i = 1; i < 4; i++) d = fma2(qr[h][i], k2[i], d);
                const float2 xy = unpack2(d);
                sc[j][h] = xy.x + xy.y;
            }
        }
#pragma unroll
        for (int h = 0; h < NREP; h++) {
            sc[0][h] += __shfl_xor_sync(0xffffffffu, sc[2][h], 16);
            sc[1][h] += __shfl_xor_sync(0xffffffffu, sc[3][h], 16);
        }
#pragma unroll
        for (int h = 0; h < NREP; h++) sc[0][h] += __shfl_xor_sync(0xffffffffu, sc[1][h], 8);
#pragma unroll
        for (int i = 0; i < kHalf; i++) {
            sc[0][i] += __shfl_xor_sync(0xffffffffu, sc[0][kHalf < NREP ? i + kHalf : i], 4);
            sc[0][i] += __shfl_xor_sync(0xffffffffu, sc[0][i], 2);
            sc[0][i] += __shfl_xor_sync(0xffffffffu, sc[0][i], 1);
        }
        const bool real = g + mine < p1;
        bool ahead = false;
#pragma unroll
        for (int i = 0; i < kHalf; i++) {
            sc[0][i] *= kn;
            ahead |= sc[0][i] > m[i] && real;
        }
        if (__any_sync(0xffffffffu, ahead)) {  // the maxima move
            float corr[kHalf];
#pragma unroll
            for (int i = 0; i < kHalf; i++) {
                float top = real ? sc[0][i] : -CUDART_INF_F;
                top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 8));
                top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 16));
                corr[i] = 1.f;
                if (top > m[i]) {
                    corr[i] = exp2f(m[i] - top);  // 0 at first (m = -inf)
                    l[i] *= corr[i];
                    m[i] = top;
                }
            }
#pragma unroll
            for (int h = 0; h < NREP; h++) {
                const float f = __shfl_sync(0xffffffffu, corr[h % kHalf], h >= kHalf ? 4 : 0);
#pragma unroll
                for (int i = 0; i < 4; i++) acc[h][i] = mul2(pack2(f, f), acc[h][i]);
            }
        }
#pragma unroll
        for (int i = 0; i < kHalf; i++) {
            const float pr = real ? exp2f(sc[0][i] - m[i]) : 0.f, w = real ? pr * vn : 0.f;
            l[i] += pr;
            if ((lane & 3) == 0) s_w[warp][turn][head0 + i][mine] = make_float2(w, w);
        }
        __syncwarp();  // (the other buffer's last readers are behind this too)
        uint64_t v2[kGroup][4];
#pragma unroll
        for (int j = 0; j < kGroup; j++) {
            if constexpr (VK == ROW_PLANAR) {
                expand_group<BITS, kStride>(load_group8<BITS>(v_rows + j * (32 * BITS), lane), tab, v2[j]);
            } else {
                const float4 *row = reinterpret_cast<const float4 *>(v_rows + j * (kHd * 4));
                float4 x = row[lane], y = row[32 + lane];
                if (g + j >= p1) x = y = make_float4(0.f, 0.f, 0.f, 0.f);  // (a row that stands in may hold infinities)
                v2[j][0] = pack2(x.x, x.y), v2[j][1] = pack2(x.z, x.w), v2[j][2] = pack2(y.x, y.y), v2[j][3] = pack2(y.z, y.w);
            }
        }
        // A group's terms are added up before they join the sums: a quarter of the roundings at the size of the sums.
#pragma unroll
        for (int h = 0; h < NREP; h++) {
            uint64_t w[kGroup];
#pragma unroll
            for (int j = 0; j < kGroup; j += 2) {
                const ulonglong2 two = *reinterpret_cast<const ulonglong2 *>(&s_w[warp][turn][h][j]);
                w[j] = two.x, w[j + 1] = two.y;
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                uint64_t t = mul2(w[0], v2[0][i]);
#pragma unroll
                for (int j = 1; j < kGroup; j++) t = fma2(w[j], v2[j][i], t);
                acc[h][i] = add2(acc[h][i], t);
            }
        }
        g += kW * kGroup;
        if (++st == kStages) st = 0;
    }

    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");

    // ---- merge the warps -----------------------------------------------------
    // a lane's l is its position's part of the sum
#pragma unroll
    for (int i = 0; i < kHalf; i++) {
        l[i] += __shfl_xor_sync(0xffffffffu, l[i], 8);
        l[i] += __shfl_xor_sync(0xffffffffu, l[i], 16);
        if ((lane & 27) == 0) s_m[warp][head0 + i] = m[i], s_l[warp][head0 + i] = l[i];
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();  // also: every warp is done with the ring and the table
    float *const part = reinterpret_cast<float *>(dyn);  // [warp][head][kHd]
#pragma unroll
    for (int h = 0; h < NREP; h++) {
        float2 x[4];
#pragma unroll
        for (int i = 0; i < 4; i++) x[i] = unpack2(acc[h][i]);
        float *dst = part + (size_t)(warp * NREP + h) * kHd;
        *reinterpret_cast<float4 *>(dst + dim_of<VK>(lane, 0)) = make_float4(x[0].x, x[0].y, x[1].x, x[1].y);
        *reinterpret_cast<float4 *>(dst + dim_of<VK>(lane, 4)) = make_float4(x[2].x, x[2].y, x[3].x, x[3].y);
    }
    if (tid < NREP) {
        float M = -CUDART_INF_F, sum = 0.f;
        for (int w = 0; w < kW; w++) M = fmaxf(M, s_m[w][tid]);
        for (int w = 0; w < kW; w++) {
            const float f = s_m[w][tid] > -CUDART_INF_F ? exp2f(s_m[w][tid] - M) : 0.f;
            sum += s_l[w][tid] * f;
            s_m[w][tid] = f;
        }
        s_M[tid] = M;
        s_L[tid] = sum;
    }
    __syncthreads();
    for (int i = tid; i < NREP * kHd; i += kNT) {
        const int r = i / kHd;
        float sum = 0.f;
#pragma unroll
        for (int w = 0; w < kW; w++) sum += part[w * (NREP * kHd) + i] * s_m[w][r];
        (&s_q[0][0])[i] = sum;
    }
    __syncthreads();

    const int first_item = meta.item_start[s] + kv * n_chunks;
    finish_item<NREP>(a, meta.slot[s], s, kv, item, n_chunks, first_item, &s_q[0][0], s_M, s_L, &s_last, VK == ROW_PLANAR);
}

// out[row][d] = sum_g acc_g[d] e^{m_g - M} / sum_g l_g e^{m_g - M}
__global__ void lse_merge_kernel(int n_parts, int n_rows, int hd, const float *parts, float *out) {
    const int row = blockIdx.x;
    const int stride = hd + 2;
    float M = -CUDART_INF_F;
    for (int g = 0; g < n_parts; g++) {
        const float *p = parts + ((size_t)g * n_rows + row) * stride;
        if (p[hd + 1] > 0.f) M = fmaxf(M, p[hd]);
    }
    float Ls = 0.f;
    for (int g = 0; g < n_parts; g++) {
        const float *p = parts + ((size_t)g * n_rows + row) * stride;
        if (p[hd + 1] > 0.f) Ls += p[hd + 1] * expf(p[hd] - M);
    }
    for (int d = threadIdx.x; d < hd; d += blockDim.x) {
        float sum = 0.f;
        for (int g = 0; g < n_parts; g++) {
            const float *p = parts + ((size_t)g * n_rows + row) * stride;
            if (p[hd + 1] > 0.f) sum = fmaf(p[d], expf(p[hd] - M), sum);
        }
        out[(size_t)row * hd + d] = Ls > 0.f ? sum / Ls : 0.f;
    }
}

// Both kernels wait for the kernel before them themselves, so they may be launched under its end.
template <typename Kernel>
bk_status launch_pdl(bk_ctx *ctx, Kernel *kernel, int threads, size_t smem, const DecodeArgs &a, const DecodeMeta &m) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)m.n_items);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    BK_CUDA(ctx, cudaLaunchKernelEx(&cfg, kernel, a, m));
    ctx->launches++;
    BK_CUDA(ctx, cudaGetLastError());
    return BK_OK;
}

template <int VK, int BITS, int NREP>
bk_status launch_planar(bk_ctx *ctx, const DecodeArgs &a, const DecodeMeta &m) {
    constexpr size_t smem = kPlanarSmem<VK, BITS, NREP>;
    static PerDevice opted_in;
    BK_CUDA(ctx, opted_in.once(ctx->device, [] {
        return cudaFuncSetAttribute(decode_planar_kernel<VK, BITS, NREP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPlanarSmem<VK, BITS, NREP>);
    }));
    return launch_pdl(ctx, decode_planar_kernel<VK, BITS, NREP>, kPlanarWarps<VK, NREP> * 32, smem, a, m);
}

template <typename F>
bk_status with_rep(bk_ctx *ctx, const DecodeArgs &a, F &&f) {
    switch (a.n_head / a.n_kv) {
        case 1: return f.template operator()<1>();
        case 2: return f.template operator()<2>();
        case 4: return f.template operator()<4>();
        case 6: return f.template operator()<6>();
        case 8: return f.template operator()<8>();
        default: return fail(ctx, BK_ERR_UNSUPPORTED, "decode: n_head/n_kv must be 1, 2, 4, 6 or 8");
    }
}

}  // namespace

bk_status launch_decode(bk_ctx *ctx, const DecodeArgs &a, const DecodeMeta &m) {
    if (m.n_items <= 0) return BK_OK;
    if (a.k_kind == ROW_F32 && a.v_kind == ROW_F32)
        return with_rep(ctx, a, [&]<int R>() { return launch_pdl(ctx, decode_kernel<ROW_F32, R>, kThreads, 0, a, m); });
    if (a.k_kind == ROW_F16 && a.v_kind == ROW_F16)
        return with_rep(ctx, a, [&]<int R>() { return launch_pdl(ctx, decode_kernel<ROW_F16, R>, kThreads, 0, a, m); });
    if (a.k_kind == ROW_PLANAR) {
        bk_status st = BK_ERR_INVALID;
        const bool vq = a.v_kind == ROW_PLANAR;
        const bool ok = dispatch_bits(a.bits, [&]<int B>() {
            st = with_rep(ctx, a, [&]<int R>() { return vq ? launch_planar<ROW_PLANAR, B, R>(ctx, a, m) : launch_planar<ROW_F32, B, R>(ctx, a, m); });
        });
        if (!ok) return fail(ctx, BK_ERR_INVALID, "decode: bits must be 1..8");
        return st;
    }
    return fail(ctx, BK_ERR_UNSUPPORTED, "decode: unsupported K/V row combination");
}

bk_status launch_lse_merge(bk_ctx *ctx, int n_parts, int n_rows, int hd, const float *parts, float *out) {
    if (n_rows <= 0) return BK_OK;
    lse_merge_kernel<<<n_rows, 256, 0, ctx->stream>>>(n_parts, n_rows, hd, parts, out);
    ctx->launches++;
    BK_CUDA(ctx, cudaGetLastError());
    return BK_OK;
}

}  // namespace bk
