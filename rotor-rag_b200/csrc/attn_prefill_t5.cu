// Softmax attention for prompt prefill on the fifth-generation tensor cores (head_dim 128).
//
// Reference: MultiHeadAttention.forward (src/rotor/transformer.py:249-283): scores
// Q K^T / sqrt(head_dim) over the cache, optional causal mask, softmax, times V, K/V shared by the
// query heads of a group.  Same contract and row mapping as the mma.sync kernel
// (attn_prefill_tc.cu), which stays for head_dim 64 and as the comparison path.
//
// CTA: 128 query rows of one KV head (128 / G positions x G heads of the group), keys walked 64
// at a time.  Both products run as tcgen05.mma.kind::f16 with bf16 operands and float32
// accumulators in tensor memory, every operand split into hi + lo bf16 terms (16 operand mantissa bits), which holds
// the 1e-3-of-RMS bound of the float32 reference.  O takes lo*hi + hi*lo + hi*hi; S takes lo*lo too, and both add the small
// products first: an accumulator that stays in tensor memory over a row's keys rounds more than tiles that are added in registers,
// and the scores give it back (error of the attention layer against float64, three activation terms, 2 x 700 positions of the 2B
// shape: 7.68e-6 with each tile added in registers, 7.94e-6 with three products in S, 6.53e-6 so; one prompt of 2048 8.07e-6, 8.46e-6,
// 6.96e-6; 6 layers of 8 x 2048 11.08 / 11.30 ms with three / four).
//   S = Q K^T : A = Q hi / lo from TENSOR MEMORY (scaled, split and written once per CTA), B = K hi / lo tiles
//               [64 keys][128] by TMA; accumulator 128 lanes x 64 columns.
//   O += P V  : A = P hi / lo from tensor memory (written by the softmax warps over the S buffer they have just
//               read), B = V^T hi / lo tiles [128][64 keys] by TMA (the split kernel stores V transposed per key
//               tile so that this operand is K-major too); accumulator 128 lanes x 128 columns.
// Two groups of four warps, a thread per query row: group 0 takes the even key tiles, group 1 the odd ones, each with
// an S buffer, a reference maximum, a sum and an accumulator of its own, so that one group's softmax runs while the tensor
// pipe works for the other and no barrier joins them before the end, where a row's two results are weighed against each
// other.  The accumulator stays in tensor memory: it is rescaled only when a tile's maximum passes the reference by more
// than 2^8 (weights up to 2^8 lose nothing in float32), and then the tile's S being complete means that the products
// before it are too.  With the shared-memory Q of before a 64-column S product read more shared memory (6 KB per
// instruction of 32 clocks) than its port gives; all columns of tensor memory are used now (S 2 x 64, O 2 x 128, Q 2 x 64).
// Persistent: one CTA per SM walks the query tiles, longest first, back and forth over the CTAs so that their sums agree.  The
// next tile's Q arrives while the present one is worked on; when its products are done the Q goes to tensor memory first, so that
// the next scores run beside the present tile's outputs (a CTA per tile spent 16 us before and behind its first key tile).
// 2B shape, 8 x 2048 causal, a layer: 692 us with one stream of eight warps that met at two barriers a tile and added each
// product to registers, 599 as above with a CTA per tile, 443 persistent, 480 with the scores' fourth product.
// Warps 8 and 9: TMA producers of the K and the V^T tiles -- separate two-deep rings, because a K
// tile is free again as soon as its S product has run, while a V^T tile stays until P V.  Warp 10: MMA issue.  Warp 11: Q rows.
// Every wait is bounded; a wait that runs out records a code in the library status word, the CTA
// stops issuing work, frees its tensor memory and returns.  No multicast, this GPU's memory only.
#include <cuda.h>
#include <cuda_bf16.h>

#include <cstdlib>
#include <type_traits>

#include "model.cuh"
#include "tc5.cuh"

namespace rb {

constexpr int A5_BM = 128, A5_BN = 64, A5_D = 128;
constexpr int A5_THREADS = 384;  // 8 softmax / output warps, two TMA warps, MMA warp, Q warp
constexpr int A5_SOFT = 256;     // threads of the softmax warps
constexpr int A5_Q_ROW = 132;             // floats per staged query row (padding: rows start in different banks)
constexpr int A5_Q_BYTES = A5_BM * A5_Q_ROW * 4;
constexpr int A5_K_BYTES = 32768;         // one K tile: hi panel 0, 1; lo panel 0, 1 (64 rows x 128 bytes each)
constexpr int A5_V_BYTES = 32768;         // one V^T tile: hi, lo (128 rows x 128 bytes each)
constexpr int A5_STAGES = 2;              // depth of the K ring and of the V^T ring
constexpr int A5_OUT_ROW = 80;            // bytes per staged output row of 16 columns
constexpr int A5_OUT_BYTES = 8 * 32 * A5_OUT_ROW;
constexpr int A5_SMEM = A5_Q_BYTES + A5_OUT_BYTES + A5_STAGES * (A5_K_BYTES + A5_V_BYTES) + 1024;
constexpr int A5_TMEM_COLS = 512;         // S0 [0,64)  S1 [64,128)  O0 [128,256)  O1 [256,384)  Q hi [384,448)  Q lo [448,512)
constexpr uint32_t A5_O = 128, A5_QT = 384;
constexpr float A5_SLACK = 8.f;           // log2 of the largest weight before the reference maximum moves

struct A5Params {
    const float* q;        // [rows][n_heads * 128]
    float* out;            // [rows][n_heads * 128]
    const int* past_len;
    unsigned* status;
    int n_heads, n_kv_heads, seq, max_seq, causal;
    int split_seq;         // rows per (sequence, KV head) in the K planes (max_seq rounded up to 64)
    int batch, nqt;        // sequences, query tiles of each (sequence, KV head)
};

// ACC == 0: the accumulator is overwritten (first MMA of a tile), 1: accumulated into.
template <int ACC>
__device__ __forceinline__ void a5_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t db, uint32_t idesc) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t"
        "}\n" ::"r"(d_tmem),
        "r"(a_tmem), "l"(db), "r"(idesc), "n"(ACC), "r"(0u)
        : "memory");
}
__device__ __forceinline__ void a5_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}

// hi + lo split of two floats, packed as bf16x2 (first value in the low half): one packed conversion
// per term, the hi values widened again by shifting
__device__ __forceinline__ void a5_split2(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    const float xh = __uint_as_float(hi << 16), yh = __uint_as_float(hi & 0xffff0000u);
    const __nv_bfloat162 l = __floats2bfloat162_rn(x - xh, y - yh);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}
__device__ __forceinline__ float a5_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Splits the float32 K/V cache rows of key tile blockIdx.x (64 keys) of one (sequence, KV head)
// into hi / lo bf16 planes laid out for the tensor-core kernel:
//   K hi, K lo : [sequence][KV head][split_seq][128]          (row = key)
//   V hi, V lo : [sequence][KV head][tile][128][64]           (transposed inside the key tile)
// Keys past the sequence's length inside a started tile are written as zeros (their probabilities
// are zero, and zero times stale memory could be NaN); tiles past the length are not touched.
__global__ void __launch_bounds__(256) kv_split_t5_kernel(const float* __restrict__ k_cache, const float* __restrict__ v_cache,
                                                          const int* __restrict__ past_len, int seq, int max_seq,
                                                          int n_kv_heads, int split_seq, __nv_bfloat16* __restrict__ planes,
                                                          size_t plane) {
    __shared__ float vs[A5_BN][A5_D + 1];
    const int tile = blockIdx.x, hk = blockIdx.y, b = blockIdx.z;
    int t_all = past_len[b] + seq;
    if (t_all > max_seq) t_all = max_seq;
    const int t0 = tile * A5_BN;
    if (t0 >= t_all) return;
    const size_t head = (size_t)b * n_kv_heads + hk;
    const float* kc = k_cache + head * max_seq * A5_D;
    const float* vc = v_cache + head * max_seq * A5_D;
    __nv_bfloat16* kh = planes + (head * split_seq + t0) * A5_D;
    __nv_bfloat16* kl = kh + plane;
    for (int idx = threadIdx.x; idx < A5_BN * (A5_D / 4); idx += 256) {
        const int r = idx / (A5_D / 4), c4 = idx - r * (A5_D / 4);
        float4 k = make_float4(0.f, 0.f, 0.f, 0.f), v = k;
        if (t0 + r < t_all) {
            k = *reinterpret_cast<const float4*>(kc + (size_t)(t0 + r) * A5_D + 4 * c4);
            v = *reinterpret_cast<const float4*>(vc + (size_t)(t0 + r) * A5_D + 4 * c4);
        }
        uint2 h2, l2;
        a5_split2(k.x, k.y, h2.x, l2.x);
        a5_split2(k.z, k.w, h2.y, l2.y);
        *reinterpret_cast<uint2*>(kh + (size_t)r * A5_D + 4 * c4) = h2;
        *reinterpret_cast<uint2*>(kl + (size_t)r * A5_D + 4 * c4) = l2;
        vs[r][4 * c4] = v.x;
        vs[r][4 * c4 + 1] = v.y;
        vs[r][4 * c4 + 2] = v.z;
        vs[r][4 * c4 + 3] = v.w;
    }
    __syncthreads();
    __nv_bfloat16* vh = planes + 2 * plane + (head * (split_seq / A5_BN) + tile) * (size_t)(A5_D * A5_BN);
    __nv_bfloat16* vl = vh + plane;
    for (int idx = threadIdx.x; idx < A5_D * (A5_BN / 2); idx += 256) {
        const int d = idx / (A5_BN / 2), kp = idx - d * (A5_BN / 2);  // keys 2 kp, 2 kp + 1
        uint32_t h, l;
        a5_split2(vs[2 * kp][d], vs[2 * kp + 1][d], h, l);
        *reinterpret_cast<uint32_t*>(vh + (size_t)d * A5_BN + 2 * kp) = h;
        *reinterpret_cast<uint32_t*>(vl + (size_t)d * A5_BN + 2 * kp) = l;
    }
}

__global__ void __launch_bounds__(A5_THREADS, 1)
attn_prefill_t5_kernel(const __grid_constant__ CUtensorMap tm_kh, const __grid_constant__ CUtensorMap tm_kl,
                       const __grid_constant__ CUtensorMap tm_vh, const __grid_constant__ CUtensorMap tm_vl,
                       const __grid_constant__ A5Params p) {
    extern __shared__ unsigned char a5_raw[];
    __shared__ __align__(8) unsigned long long s_kfull[A5_STAGES], s_kempty[A5_STAGES], s_vfull[A5_STAGES],
        s_vempty[A5_STAGES], s_sfull[2], s_pfull[2], s_ofull, s_qready, s_qfull, s_qempty, s_oread;
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;
    __shared__ float s_m[2][2][A5_BM], s_l[2][2][A5_BM];  // by tile parity: each group's reference maximum and sum of a row
    const uint32_t kring = (smem_u32(a5_raw) + 1023u) & ~1023u, vring = kring + A5_STAGES * A5_K_BYTES;
    const uint32_t qstage = vring + A5_STAGES * A5_V_BYTES, ostage = qstage + A5_Q_BYTES;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int G = p.n_heads / p.n_kv_heads, lg = 31 - __clz(G), QT = A5_BM >> lg;  // (G divides 128)
    const int items = p.nqt * p.n_kv_heads * p.batch;
    volatile int* abort_flag = &s_abort;

    // The k-th query tile of this CTA; n: its key tiles (0: there is none).
    struct Item {
        int s0, hk, b, past, last, t_all, n;
    };
    auto item = [&](int k) {
        Item o = {};
        const int i = k * (int)gridDim.x + ((k & 1) ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x);
        if (i >= items) return o;
        const int per = p.n_kv_heads * p.batch, qt = p.nqt - 1 - i / per, e = i % per;
        o.hk = e % p.n_kv_heads;
        o.b = e / p.n_kv_heads;
        o.s0 = qt * QT;
        o.past = __ldg(p.past_len + o.b);
        o.last = min(o.s0 + QT, p.seq) - 1;
        o.t_all = min(o.past + (p.causal ? o.last + 1 : p.seq), p.max_seq);
        o.n = (o.t_all + A5_BN - 1) / A5_BN;
        return o;
    };
    const int rounds = (items + (int)gridDim.x - 1) / (int)gridDim.x;  // (the last may hold no tile for this CTA)

    if (threadIdx.x == 0) {
        s_abort = 0;
        auto init = [](unsigned long long* bar, int count) { t5_bar_init(smem_u32(bar), count); };
        for (int s = 0; s < A5_STAGES; ++s) {
            init(&s_kfull[s], 1);
            init(&s_kempty[s], 1);
            init(&s_vfull[s], 1);
            init(&s_vempty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            init(&s_sfull[s], 1);
            init(&s_pfull[s], 4);   // one arrival per warp of the group
        }
        init(&s_ofull, 1);
        init(&s_qready, 8);
        init(&s_qfull, 1);
        init(&s_qempty, 8);
        init(&s_oread, 8);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 8) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                     "r"(A5_TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;

    if (warp < 8) {
        const int half = warp >> 2, wq = warp & 3;
        const int r = wq * 32 + lane;  // this thread's query row
        const uint32_t lane_base = tmem + ((uint32_t)(wq * 32) << 16);
        const uint32_t sbuf = lane_base + 64u * half, obuf = lane_base + A5_O + 128u * half;
        const uint32_t blk = ostage + (uint32_t)warp * (32u * A5_OUT_ROW);
        bool ok = true;
        int tiles = 0;          // of this group, over all query tiles: phases of its barriers
        Item prev = {};         // the tile whose products are done and whose outputs are still in tensor memory
        float w0 = 0.f, w1 = 0.f;
        // (after a failed wait every further one returns at once; the warps still meet at each barrier)
        for (int k = 0; k <= rounds; ++k) {
            const Item it = k < rounds ? item(k) : Item{};
            if (it.n) {
                // ---------------- Q: rows out of shared memory, scaled and split into tensor memory
                const float scale = 1.4426950408889634f / sqrtf((float)A5_D);  // scores come out in units of log2: p = 2^(s - m)
                ok = ok && t5_wait(smem_u32(&s_qfull), (uint32_t)k & 1u, abort_flag, p.status, 0x7b00000bu);
                uint32_t qh[32], ql[32];  // columns [64 half, +64) of the row
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    float4 v;
                    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                                 : "r"(qstage + (uint32_t)(r * A5_Q_ROW + 64 * half + 4 * i) * 4u));
                    a5_split2(v.x * scale, v.y * scale, qh[2 * i], ql[2 * i]);
                    a5_split2(v.z * scale, v.w * scale, qh[2 * i + 1], ql[2 * i + 1]);
                }
                __syncwarp();
                if (lane == 0) t5_bar_arrive(smem_u32(&s_qempty));
                t5_st32(lane_base + A5_QT + 32u * half, qh);
                t5_st32(lane_base + A5_QT + 64u + 32u * half, ql);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) t5_bar_arrive(smem_u32(&s_qready));
            }
            if (prev.n && __all_sync(0xffffffffu, ok)) {
                // ---------------- outputs of the tile before, columns [64 half, +64) of both accumulators.  A lane holds
                // consecutive outputs of ONE row, so a 16-byte store instruction of the warp would touch 32 different lines:
                // the rows cross a per-warp block and leave as 64-byte pieces, eight rows per instruction.
#pragma unroll 1
                for (uint32_t c = 0; c < 64u; c += 16u) {
                    uint32_t o0[32], o1[32];
                    t5_ld16(lane_base + A5_O + 64u * half + c, o0);
                    if (prev.n > 1) t5_ld16(lane_base + A5_O + 128u + 64u * half + c, o1);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    float o[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        o[i] = __uint_as_float(o0[i]) * w0;
                        if (prev.n > 1) o[i] += __uint_as_float(o1[i]) * w1;
                    }
#pragma unroll
                    for (int i = 0; i < 16; i += 4)
                        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(blk + (uint32_t)lane * A5_OUT_ROW + 4u * i),
                                     "f"(o[i]), "f"(o[i + 1]), "f"(o[i + 2]), "f"(o[i + 3])
                                     : "memory");
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int rr = 8 * i + (lane >> 2), chunk = lane & 3;
                        float4 w;
                        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                                     : "=f"(w.x), "=f"(w.y), "=f"(w.z), "=f"(w.w)
                                     : "r"(blk + (uint32_t)rr * A5_OUT_ROW + 16u * chunk));
                        const int r2 = wq * 32 + rr, srow = prev.s0 + (r2 >> lg), gi = r2 & (G - 1);
                        if (srow < p.seq)
                            *reinterpret_cast<float4*>(p.out + ((size_t)prev.b * p.seq + srow) * p.n_heads * A5_D +
                                                       (size_t)(prev.hk * G + gi) * A5_D + half * 64 + c + 4 * chunk) = w;
                    }
                    __syncwarp();
                }
                // read by every warp before the next tile's first product: the groups read both accumulators
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) t5_bar_arrive(smem_u32(&s_oread));
            }
            prev = it;
            if (!it.n) continue;
            // ---------------- softmax of this group's key tiles
            const int srow = it.s0 + (r >> lg);
            int lim = p.causal ? it.past + (srow < p.seq ? srow : it.last) + 1 : it.past + p.seq;
            if (lim > it.t_all) lim = it.t_all;
            float m_ref = -INFINITY, l_run = 0.f;
            for (int j = half; j < it.n; j += 2, ++tiles) {
                ok = ok && t5_wait(smem_u32(&s_sfull[half]), (uint32_t)tiles & 1u, abort_flag, p.status, 0x7b000001u);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                uint32_t sa[2][32];
                t5_ld32(sbuf, sa[0]);
                t5_ld32(sbuf + 32u, sa[1]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                const int kb = j * A5_BN;
                if (kb + A5_BN > lim) {  // only the last tiles of a row need the mask
#pragma unroll
                    for (int c = 0; c < 64; ++c)
                        if (kb + c >= lim) sa[c >> 5][c & 31] = 0xff800000u;  // -inf
                }
                float t0 = -INFINITY, t1 = t0;
#pragma unroll
                for (int c = 0; c < 32; c += 2) {
                    t0 = fmaxf(t0, fmaxf(__uint_as_float(sa[0][c]), __uint_as_float(sa[0][c + 1])));
                    t1 = fmaxf(t1, fmaxf(__uint_as_float(sa[1][c]), __uint_as_float(sa[1][c + 1])));
                }
                const float tmax = fmaxf(t0, t1);
                // (each row for itself: what another row of the warp does, one past the sequence above all, changes nothing here)
                const bool far = tmax > m_ref + A5_SLACK;
                if (__any_sync(0xffffffffu, far)) {  // the first tile, then rarely
                    const float alpha = !far ? 1.f : m_ref == -INFINITY ? 0.f : a5_exp2(m_ref - tmax);
                    if (far) m_ref = tmax;
                    l_run *= alpha;
                    if (j >= 2) {
#pragma unroll 1
                        for (uint32_t c = 0; c < 128u; c += 32u) {
                            uint32_t ov[32];
                            t5_ld32(obuf + c, ov);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                            for (int i = 0; i < 32; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * alpha);
                            t5_st32(obuf + c, ov);
                        }
                    }
                }
                const float m_use = m_ref == -INFINITY ? 0.f : m_ref;  // (no visible key yet: every weight is 2^-inf)
                float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t ph[16], pl[16];
#pragma unroll
                    for (int c = 0; c < 16; ++c) {
                        const float e0 = a5_exp2(__uint_as_float(sa[h][2 * c]) - m_use), e1 = a5_exp2(__uint_as_float(sa[h][2 * c + 1]) - m_use);
                        sum0 += e0;
                        sum1 += e1;
                        a5_split2(e0, e1, ph[c], pl[c]);  // keys 32 h + 2 c, + 1 -> column 16 h + c
                    }
                    a5_st16(sbuf + 16u * h, ph);        // P hi: 64 bf16 in columns [0, 32) of the S buffer
                    a5_st16(sbuf + 32u + 16u * h, pl);  // P lo: columns [32, 64)
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) t5_bar_arrive(smem_u32(&s_pfull[half]));
                l_run += sum0 + sum1;
            }
            // ---------------- the groups' results of a row, weighed against each other
            float(*sm)[A5_BM] = s_m[k & 1], (*sl)[A5_BM] = s_l[k & 1];
            sm[half][r] = m_ref;
            sl[half][r] = l_run;
            asm volatile("bar.sync 1, %0;" ::"n"(A5_SOFT) : "memory");
            const float m0 = sm[0][r], m1 = sm[1][r], M = fmaxf(m0, m1);
            w0 = m0 == -INFINITY ? 0.f : a5_exp2(m0 - M);
            w1 = m1 == -INFINITY ? 0.f : a5_exp2(m1 - M);
            const float inv = 1.0f / (sl[0][r] * w0 + sl[1][r] * w1);
            w0 *= inv;
            w1 *= inv;
            ok = ok && t5_wait(smem_u32(&s_ofull), (uint32_t)k & 1u, abort_flag, p.status, 0x7b000002u);
            ok = __all_sync(0xffffffffu, ok);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
    } else if (warp == 8) {
        // ---------------- K tiles by TMA
        if (elect_lane()) {
            int t = 0;
            bool ok = true;
            for (int k = 0; k < rounds && ok; ++k) {
                const Item it = item(k);
                const int krow0 = (it.b * p.n_kv_heads + it.hk) * p.split_seq;
                for (int j = 0; j < it.n; ++j, ++t) {
                    const int s = t & 1;
                    ok = t5_wait(smem_u32(&s_kempty[s]), ((uint32_t)(t >> 1) & 1u) ^ 1u, abort_flag, p.status, 0x7b000003u);
                    if (!ok) break;
                    const uint32_t bar = smem_u32(&s_kfull[s]), st = kring + (uint32_t)s * A5_K_BYTES;
                    t5_bar_expect(bar, A5_K_BYTES);
#pragma unroll
                    for (int pn = 0; pn < 2; ++pn) {
                        t5_tma_2d(st + (uint32_t)pn * 8192u, &tm_kh, pn * 64, krow0 + j * A5_BN, bar);
                        t5_tma_2d(st + 16384u + (uint32_t)pn * 8192u, &tm_kl, pn * 64, krow0 + j * A5_BN, bar);
                    }
                }
            }
        }
    } else if (warp == 9) {
        // ---------------- V^T tiles by TMA
        if (elect_lane()) {
            int t = 0;
            bool ok = true;
            for (int k = 0; k < rounds && ok; ++k) {
                const Item it = item(k);
                const int vrow0 = (it.b * p.n_kv_heads + it.hk) * (p.split_seq / A5_BN) * A5_D;
                for (int j = 0; j < it.n; ++j, ++t) {
                    const int s = t & 1;
                    ok = t5_wait(smem_u32(&s_vempty[s]), ((uint32_t)(t >> 1) & 1u) ^ 1u, abort_flag, p.status, 0x7b000009u);
                    if (!ok) break;
                    const uint32_t bar = smem_u32(&s_vfull[s]), st = vring + (uint32_t)s * A5_V_BYTES;
                    t5_bar_expect(bar, A5_V_BYTES);
                    t5_tma_2d(st, &tm_vh, 0, vrow0 + j * A5_D, bar);
                    t5_tma_2d(st + 16384u, &tm_vl, 0, vrow0 + j * A5_D, bar);
                }
            }
        }
    } else if (warp == 11) {
        // ---------------- Q rows of the next tile (rows past the sequence keep what lies there: nobody stores their outputs)
        bool ok = true;
        for (int k = 0; k < rounds && ok; ++k) {
            const Item it = item(k);
            if (!it.n) break;
            ok = t5_wait(smem_u32(&s_qempty), ((uint32_t)k & 1u) ^ 1u, abort_flag, p.status, 0x7b00000cu);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            const uint32_t bar = smem_u32(&s_qfull);
            const int live = (it.last - it.s0 + 1) << lg;
            if (lane == 0) t5_bar_expect(bar, (uint32_t)live * (A5_D * 4));
            __syncwarp();
            for (int rr = lane; rr < live; rr += 32) {
                const float* src = p.q + ((size_t)it.b * p.seq + it.s0 + (rr >> lg)) * p.n_heads * A5_D + (size_t)(it.hk * G + (rr & (G - 1))) * A5_D;
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                 qstage + (uint32_t)(rr * A5_Q_ROW) * 4u),
                             "l"(src), "r"(A5_D * 4), "r"(bar)
                             : "memory");
            }
        }
    } else {
        // ---------------- MMA issue
        if (elect_lane()) {
            // kind::f16: float32 accumulate (bit 4), A and B bf16 (bits 7, 10), both K-major, N >> 3 at 17, M >> 4 at 24
            const uint32_t idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(A5_BN >> 3) << 17) | ((128u >> 4) << 24);
            const uint32_t idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(A5_D >> 3) << 17) | ((128u >> 4) << 24);
            // One thread issues every MMA of the CTA, so its instruction count per MMA bounds the tensor pipe:
            // the descriptors of a tile are its base descriptor plus compile-time constants (the address field
            // counts 16-byte units and no operand crosses the field's range), nothing is recomputed per MMA.
            // j: key tile of the query tile (its group's buffers); t: over all query tiles (ring slots)
            auto issue_s = [&](int j, int t) {
                const uint64_t dk_hi = t5_desc(kring + (uint32_t)(t & 1) * A5_K_BYTES), dk_lo = dk_hi + (16384u >> 4);
                const uint32_t d = tmem + (uint32_t)(j & 1) * 64u;
#pragma unroll
                for (int term = 3; term >= 0; --term)  // lo lo, lo hi, hi lo, hi hi
#pragma unroll
                    for (int k16 = 0; k16 < A5_D / 16; ++k16) {
                        const uint64_t ko = (uint64_t)(((k16 >> 2) * 8192 + (k16 & 3) * 32) >> 4);
                        const uint32_t qa = tmem + A5_QT + (term >= 2 ? 64u : 0u) + (uint32_t)k16 * 8u;
                        const uint64_t db = ((term & 1) ? dk_lo : dk_hi) + ko;
                        if (term == 3 && k16 == 0)
                            a5_mma_ts<0>(d, qa, db, idesc_s);
                        else
                            a5_mma_ts<1>(d, qa, db, idesc_s);
                    }
                t5_commit(smem_u32(&s_sfull[j & 1]));
                t5_commit(smem_u32(&s_kempty[t & 1]));
            };
            auto issue_pv = [&](int j, int t, auto first) {
                const uint64_t dv_hi = t5_desc(vring + (uint32_t)(t & 1) * A5_V_BYTES), dv_lo = dv_hi + (16384u >> 4);
                const uint32_t pbase = tmem + (uint32_t)(j & 1) * 64u, d = tmem + A5_O + (uint32_t)(j & 1) * 128u;
#pragma unroll
                for (int term = 2; term >= 0; --term)  // lo hi, hi lo, hi hi
#pragma unroll
                    for (int k16 = 0; k16 < A5_BN / 16; ++k16) {
                        const uint32_t pa = pbase + (term == 2 ? 32u : 0u) + (uint32_t)k16 * 8u;
                        const uint64_t db = (term == 1 ? dv_lo : dv_hi) + (uint64_t)((k16 * 32) >> 4);
                        if (decltype(first)::value && term == 2 && k16 == 0)
                            a5_mma_ts<0>(d, pa, db, idesc_o);
                        else
                            a5_mma_ts<1>(d, pa, db, idesc_o);
                    }
                t5_commit(smem_u32(&s_vempty[t & 1]));
            };
            bool ok = true;
            int base = 0;                // key tiles of the query tiles before
            uint32_t phases = 0;         // of the groups' weights, a bit each
            for (int k = 0; k < rounds && ok; ++k) {
                const Item it = item(k);
                if (!it.n) break;
                ok = t5_wait(smem_u32(&s_qready), (uint32_t)k & 1u, abort_flag, p.status, 0x7b000004u);
                auto scores = [&](int j) {
                    const int t = base + j;
                    ok = ok && t5_wait(smem_u32(&s_kfull[t & 1]), (uint32_t)(t >> 1) & 1u, abort_flag, p.status, 0x7b000005u);
                    if (!ok) return;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    issue_s(j, t);
                };
                for (int j = 0; j < 2 && j < it.n; ++j) scores(j);
                for (int j = 0; j < it.n && ok; ++j) {
                    const int t = base + j;
                    ok = t5_wait(smem_u32(&s_pfull[j & 1]), (phases >> (j & 1)) & 1u, abort_flag, p.status, 0x7b000007u);
                    phases ^= 1u << (j & 1);
                    if (ok && j == 0 && k > 0) ok = t5_wait(smem_u32(&s_oread), (uint32_t)(k - 1) & 1u, abort_flag, p.status, 0x7b00000du);
                    if (ok) ok = t5_wait(smem_u32(&s_vfull[t & 1]), (uint32_t)(t >> 1) & 1u, abort_flag, p.status, 0x7b00000au);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (j < 2)
                        issue_pv(j, t, std::true_type());
                    else
                        issue_pv(j, t, std::false_type());
                    if (j + 2 < it.n) scores(j + 2);  // (over the P that this product has read)
                }
                if (ok) t5_commit(smem_u32(&s_ofull));
                base += it.n;
            }
        }
    }

    // ---------------- common exit: nothing of this CTA may still be in flight when it returns
    if (*abort_flag && threadIdx.x == 0) {
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000LL) {
        }  // about a millisecond for copies already issued to land
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 8) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(A5_TMEM_COLS));
    }
}

static PerDevice<bool> g_a5_ready;

int configure_attn_prefill_t5() {
    if (g_a5_ready.here()) return ROTOR_B200_OK;
    RB_CUDA(cudaFuncSetAttribute(attn_prefill_t5_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, A5_SMEM));
    g_a5_ready.here() = true;
    return ROTOR_B200_OK;
}

// Shapes the tensor-memory kernel takes: head_dim 128, split planes present (prompts of 16 positions
// and more), a group size that divides the 128-row tile.
bool attn_prefill_t5_supported(const AttnParams& p, int rows) {
    static const bool off = getenv("ROTOR_B200_NO_TCGEN05") != nullptr;  // comparison aid: the mma.sync kernel
    if (off || p.head_dim != A5_D || !p.kv_split || p.seq < 16) return false;
    const int G = p.n_heads / p.n_kv_heads;
    return G >= 1 && G <= A5_BM && A5_BM % G == 0 && rows % p.seq == 0 && ((uintptr_t)p.kv_split & 127) == 0 &&
           ((uintptr_t)p.q & 15) == 0;
}

int launch_attn_prefill_t5(const AttnParams& p, int rows, cudaStream_t st) {
    int rc = configure_attn_prefill_t5();
    if (rc) return rc;
    const int G = p.n_heads / p.n_kv_heads, QT = A5_BM / G;
    const int batch = rows / p.seq;
    const int split_seq = (p.max_seq + A5_BN - 1) / A5_BN * A5_BN;
    if ((size_t)batch * p.n_kv_heads * split_seq * A5_D > p.split_plane) return ROTOR_B200_ERR_WORKSPACE;
    // ---- hi / lo planes of this call's cache rows
    dim3 sgrid(split_seq / A5_BN, p.n_kv_heads, batch);
    kv_split_t5_kernel<<<sgrid, 256, 0, st>>>(p.k_cache, p.v_cache, p.past_len, p.seq, p.max_seq, p.n_kv_heads, split_seq,
                                              p.kv_split, p.split_plane);
    rc = launch_status();
    if (rc) return rc;
    // ---- tensor maps: K planes [rows][128] in boxes of 64 columns x 64 rows, V^T planes [rows][64] in boxes of 64 x 128
    CUtensorMap tm[4];
    const size_t krows = (size_t)batch * p.n_kv_heads * split_seq, vrows = krows / A5_BN * A5_D;
    for (int i = 0; i < 4; ++i) {
        const __nv_bfloat16* plane = p.kv_split + (size_t)i * p.split_plane;
        if (!(i < 2 ? t5_map_bf16(&tm[i], plane, krows, A5_D, A5_D, A5_BN) : t5_map_bf16(&tm[i], plane, vrows, A5_BN, A5_BN, A5_D)))
            return ROTOR_B200_ERR_CUDA;
    }
    A5Params a;
    a.q = p.q;
    a.out = p.out;
    a.past_len = p.past_len;
    a.status = library_status_word();
    a.n_heads = p.n_heads;
    a.n_kv_heads = p.n_kv_heads;
    a.seq = p.seq;
    a.max_seq = p.max_seq;
    a.causal = p.causal;
    a.split_seq = split_seq;
    if (!a.status) return ROTOR_B200_ERR_CUDA;
    a.batch = batch;
    a.nqt = (p.seq + QT - 1) / QT;
    const int items = a.nqt * p.n_kv_heads * batch, sms = fused_sm_count();
    attn_prefill_t5_kernel<<<items < sms ? items : sms, A5_THREADS, A5_SMEM, st>>>(tm[0], tm[1], tm[2], tm[3], a);
    return launch_status();
}

}  // namespace rb
