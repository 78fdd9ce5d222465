// Ternary BitLinear integer core for prompt prefill on the fifth-generation tensor cores:
// acc[c][o] = sum_k xq[c][k] * w[o][k], exact int32, for hundreds to thousands of
// activation columns c (tokens).
//
// CTA tile: 256 tokens x 256 weight rows, K walked 128 at a time through a 3-stage ring of
// shared-memory operand tiles.  tcgen05.mma.kind::i8 (M = 128 tokens, N = 256 weight rows, K = 32 per
// instruction) accumulates into tensor memory: two 128-lane int32 accumulators of N columns (all 512
// TMEM columns of the SM).  A token half without tokens is skipped.  Per stage:
//   * the token operand (2 x 128 rows of 128 int8) arrives by TMA
//     (cp.async.bulk.tensor.2d, 128-byte swizzle, rows past the last token zero filled),
//   * eight decoder warps turn the stage's packed weight tiles (2 bits per weight; 16 tiles = 8 KB)
//     into bytes (32 KB) in the same swizzled K-major layout: a lane's 128-bit tile word holds, per
//     row, 32 consecutive K positions, i.e. two 16-byte chunks of the operand row,
//   * one thread issues the eight MMAs and commits them to the stage's "empty" barrier.
// The weight operand holds the codes w + 1 (0, 1, 2) as unsigned bytes against signed activations;
// the read-back subtracts the token's activation sum.  After the last stage the decoder warps read
// the accumulators back (tcgen05.ld 32 lanes x 32 columns: a lane holds 32 consecutive outputs of
// one token) and pass them through a per-warp shared-memory block so that they leave as whole
// 128-byte rows.  Products of more than 128 tokens mostly take gemm_pair_kernel below (takes_pairs), with further read-backs:
// PAIR_GATED (gate/up product: activation and product, float32 out) and PAIR_QKV (dequantise, rotary, cache append).  When
// 256-row tiles do not cover the GPU the K range is split over blockIdx.z and the partial sums are added with
// integer atomics (64-row tiles remain for products too short to split).
// Every wait is bounded by a cycle count; a wait that runs out records a code in the library status
// word, the CTA stops issuing work, lets its copies land, frees its tensor memory and returns.
#include <cuda.h>

#include <cstdlib>

#include "model.cuh"
#include "tc5.cuh"

RB_TRACE_DEFINE(rotor_b200_trace_read_gemm5)

namespace rb {

// Tokens per CTA is a template argument too: 256 (two MMA M halves, all 512 tensor-memory columns) or 128 (one
// half) for at most 128 tokens: the product is then bound by the weight stream, and the halved token operand leaves
// room for a fourth stage; four K steps of weights are requested ahead instead of two.
// Decoder warps (they also read the accumulators back), then one TMA + TMEM warp and one MMA warp.
// Eight decoders for 256-row tiles: a lone warp per scheduler issues about one instruction every
// four cycles, and at four warps the decode of a K step (about 550 instructions per warp) took
// twice as long as its eight MMAs; two warps per scheduler hide each other's latencies.
// Weight rows per CTA (MMA N) is a template argument: 256 for large grids; 64 when 256-row tiles
// would leave most SMs without a CTA (few tokens and a narrow output, e.g. 64 tokens x 8192 rows).
template <int ROWS, int TOK = 256>
struct T5Cfg {
    static constexpr int A_BYTES = TOK * TILE_K;                   // token operand per stage
    static constexpr int B_BYTES = ROWS * TILE_K;                  // weight operand per stage
    static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
    // ring depth and decoder look-ahead: with 64-row tiles a stage is only four short MMAs, so the
    // copy and weight-load latencies need more stages in flight to stay hidden
    static constexpr int STAGES = TOK == 128 ? 4 : (ROWS >= 256 ? 3 : 5);
    // decoder warps take every GROUPS-th K step with GROUPS times the tiles: one chain of wait, decode, fence and arrival per
    // GROUPS steps (with this, an arrival per warp and dependent launches a step of 64 sequences of the 2B shape, 12 layers, went
    // from 1653 to 1546 us, of 32 from 1316 to 1162, of 64 of the XL shape, 4 layers, from 1464 to 1408)
    static constexpr int GROUPS = ROWS >= 256 ? 2 : 1;
    static constexpr int PREFETCH = ROWS < 256 ? 6 : TOK == 128 ? 4 : 2;           // of its K steps that a warp requests ahead
    static constexpr int SMEM = STAGES * STAGE_BYTES + 1024;       // + slack to align the ring to 1024 bytes
    static constexpr int TMEM_COLS = (TOK / 128) * ROWS < 32 ? 32 : (TOK / 128) * ROWS;  // one accumulator of ROWS columns per token half
    static constexpr int DECODERS = ROWS >= 256 ? 8 : 4;           // decoder warps
    static constexpr int THREADS = (DECODERS + 2) * 32;
    static constexpr int TILES_PER_WARP = ROWS / TILE_ROWS * GROUPS / DECODERS;  // row tiles a decoder warp handles a step
};
constexpr int T5_SCATTER_COLS = 48;  // columns up to which a split product's sums are added by a lane per token
constexpr int T5_DEEP_STEPS = 12;  // K steps of a CTA from which the 128-token variant is taken
struct Tc5Params {
    const uint4* tiles;
    const int32_t* xsum;  // [ncols] sum of each token's int8 activations (removes the +1 of the weight codes)
    int32_t* acc;       // [ncols][out]
    unsigned* status;
    int out, nrt, nkt, ncols;
    int kt_per_split;   // > 0: CTA z takes K steps [z kt_per_split, +kt_per_split) and ADDS its sums into zeroed acc
    int box_rows;       // token rows of a copy
    int mt, nt;         // pairs: tiles of 256 tokens, of 256 weight rows (128 channels when gated)
    // PAIR_GATED: `tiles` holds the gate matrix followed by the up matrix (ff rows
    // each); a tile takes 128 gate rows and the matching 128 up rows, and the read-back writes
    // gated[token][channel] = act(gate * sx[token] * sg) * (up * sx[token] * su) as float32 instead
    // of two int32 accumulators per channel
    float* gated;       // [ncols][ff]
    const float* sx;    // [ncols] activation scales (one term per token)
    float sg, su;
    int ff, ffn_act;
    // PAIR_QKV (head_dim 128): `tiles` is the stacked [q; k; v] matrix; the read-back
    // dequantises (sx[token] * sq / sk / sv), rotates q and k (half-split pairs i, i + 64) and writes q rows
    // and the K / V cache rows of the token's position; no int32 accumulator leaves the kernel
    int dq, dkv, seq, max_seq;
    const int* past_len;   // [batch] cached length per sequence
    const float2* rope;    // [max_seq][64] (cos, sin), or null
    float* qout;           // [ncols][dq]
    float* k_cache;        // [batch][dkv / 128][max_seq][128]
    float* v_cache;
    float sq, sk, sv;
};

template <int ROWS, int T5_TOK = 256>
__global__ void __launch_bounds__(T5Cfg<ROWS, T5_TOK>::THREADS, 1)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ Tc5Params p) {
    using Cfg = T5Cfg<ROWS, T5_TOK>;
    constexpr int T5_A_BYTES = Cfg::A_BYTES, A_HALF = 128 * TILE_K;
    constexpr int T5_ROWS = ROWS, T5_STAGE_BYTES = Cfg::STAGE_BYTES, TPW = Cfg::TILES_PER_WARP;
    constexpr int T5_STAGES = Cfg::STAGES, PF = Cfg::PREFETCH, NDW = Cfg::DECODERS, GR = Cfg::GROUPS;
#ifdef RB_TRACE
    const unsigned long long t_entry = gtime();
#endif
    extern __shared__ unsigned char t5_raw[];
    __shared__ __align__(8) unsigned long long s_full[T5_STAGES], s_empty[T5_STAGES], s_accf;
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;
    const uint32_t ring = (smem_u32(t5_raw) + 1023u) & ~1023u;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tok0 = blockIdx.x * T5_TOK, rt0 = blockIdx.y * (T5_ROWS / TILE_ROWS);
    const int nhalf = (T5_TOK > 128 && p.ncols - tok0 > 128) ? 2 : 1;  // token halves of this CTA that hold any token
    // K steps of this CTA: all of them, or its share when the K range is split over blockIdx.z.  Loops
    // below count local steps 0 .. nk-1; ktb + step is the position in the matrix.
    const int ktb = p.kt_per_split ? (int)blockIdx.z * p.kt_per_split : 0;
    const int nk = p.kt_per_split ? min(p.kt_per_split, p.nkt - ktb) : p.nkt;
    volatile int* abort_flag = &s_abort;

    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int s = 0; s < T5_STAGES; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&s_full[s])), "r"(NDW / GR + 1));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&s_empty[s])), "r"(1));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&s_accf)), "r"(1));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == NDW) {  // the whole warp allocates the accumulators' tensor-memory columns (one CTA per SM)
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                     "r"(Cfg::TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;

    if (warp < NDW) {
        // ---------------- weight decoders: warp w of a group owns row tiles TPW w .. TPW w + TPW - 1 of the CTA's
        const int g = lane >> 2, t = lane & 3, w = warp % (NDW / GR), grp0 = warp / (NDW / GR);
        // weight tiles (constants) are requested PF of the warp's steps ahead of their decode, the first before the launch wait
        uint4 wv[PF][TPW];
        auto fetch = [&](int kt, uint4 (&dst)[TPW]) {
#pragma unroll
            for (int u = 0; u < TPW; ++u) {
                const int rt = rt0 + w * TPW + u;
                dst[u] = (rt < p.nrt && kt < nk)
                             ? ld_stream_v4(p.tiles + ((size_t)rt * p.nkt + ktb + kt) * 32 + lane)
                             : make_uint4(0x55555555u, 0x55555555u, 0x55555555u, 0x55555555u);
            }
        };
#pragma unroll
        for (int par = 0; par < PF; ++par) fetch(GR * par + grp0, wv[par]);
#ifdef RB_TRACE
        TraceRec trd = {};
        const bool tracedd = blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0;
        unsigned long long tld = gtime(), t0d = tld;
#endif
        bool going = true;
        for (int kt2 = grp0; kt2 < nk && going; kt2 += GR * PF) {
#pragma unroll
          for (int par = 0; par < PF; ++par) {
            const int kt = kt2 + GR * par;
            if (kt >= nk) break;
            const int s = kt % T5_STAGES;
            going = t5_wait(smem_u32(&s_empty[s]), ((kt / T5_STAGES) & 1) ^ 1, abort_flag, p.status, 0x7c000001u);
            if (!__all_sync(0xffffffffu, going)) {
                going = false;
                break;
            }
#ifdef RB_TRACE
            if (tracedd) { const unsigned long long n_ = gtime(); trd.t[0] += n_ - tld; tld = n_; }
#endif
            const uint32_t bbase = ring + s * T5_STAGE_BYTES + T5_A_BYTES;
#pragma unroll
            for (int u = 0; u < TPW; ++u) {
                const uint32_t pw[4] = {wv[par][u].x, wv[par][u].y, wv[par][u].z, wv[par][u].w};
#pragma unroll
                for (int rh = 0; rh < 2; ++rh) {
                    // operand row R = 16 (TPW w + u) + g + 8 rh; R % 8 == g; K bytes [32 t, 32 t + 32)
                    const uint32_t row = bbase + (uint32_t)((w * TPW + u) * 2 + rh) * 1024u + (uint32_t)g * 128u;
                    const uint32_t lo = pw[rh], hi = pw[rh + 2];
#pragma unroll
                    for (int c = 0; c < 2; ++c) {  // 16-byte chunk 2 t + c holds bit pairs 2 c and 2 c + 1
                        // the operand bytes are the codes w + 1 themselves (unsigned operand); the read-back
                        // subtracts the token's activation sum
                        const uint32_t a0 = (lo >> (4 * c)) & 0x03030303u;
                        const uint32_t a1 = (hi >> (4 * c)) & 0x03030303u;
                        const uint32_t a2 = (lo >> (4 * c + 2)) & 0x03030303u;
                        const uint32_t a3 = (hi >> (4 * c + 2)) & 0x03030303u;
                        const uint32_t dst = row + (uint32_t)(((2 * t + c) ^ g) << 4);
                        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(a0), "r"(a1), "r"(a2),
                                     "r"(a3)
                                     : "memory");
                    }
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic writes -> tensor-core reads
            __syncwarp();
            if (lane == 0) t5_bar_arrive(smem_u32(&s_full[s]));  // (an arrival a thread: 256 in turn on one word)
            fetch(kt + GR * PF, wv[par]);
#ifdef RB_TRACE
            if (tracedd) { const unsigned long long n_ = gtime(); trd.t[1] += n_ - tld; tld = n_; }
#endif
          }
        }
        pdl_wait();  // sums of the activations, and what is added to, belong to earlier kernels until here
        pdl_trigger();
#ifdef RB_TRACE
        if (tracedd) {
            trd.t[2] = gtime() - t0d;
            trd.t[3] = t0d - t_entry;  // kernel entry -> first K step
            trd.t[7] = (unsigned long long)p.nkt;
            tld = gtime();
        }
#endif
        // ---------------- epilogue: lane = token, 32 columns (weight rows) per load
        // (warp-uniform decision: the tensor-memory loads below are warp-wide instructions)
        const bool acc_ok = !*abort_flag && t5_wait(smem_u32(&s_accf), 0, abort_flag, p.status, 0x7c000002u);
#ifdef RB_TRACE
        if (tracedd) { const unsigned long long n_ = gtime(); trd.t[4] = n_ - tld; tld = n_; }
#endif
        if (__all_sync(0xffffffffu, acc_ok)) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int row0 = rt0 * TILE_ROWS;
            // a warp reaches the tensor-memory lanes of its quarter (warp % 4); with eight warps the two
            // groups of four split the (token half, 32-row chunk) pairs between them
            constexpr int NCH = T5_ROWS / 32, GROUPS = NDW / 4;
            const int wq = warp & 3, grp = warp >> 2;
#pragma unroll 1
            for (int item = grp; item < nhalf * NCH; item += GROUPS) {
                const int half = item / NCH, ch = item - half * NCH;
                const int token = tok0 + half * 128 + wq * 32 + lane;
                {
                    uint32_t v[32];
                    const uint32_t taddr = tmem + ((uint32_t)(wq * 32) << 16) + (uint32_t)(half * ROWS + ch * 32);
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
                          "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
                          "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]),
                          "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]),
                          "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                        : "r"(taddr));
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    const int rbase = row0 + ch * 32;
                    if (rbase < p.out) {  // warp-uniform
                        const int tok_base = tok0 + half * 128 + wq * 32;
                        // remove the +1 of the codes: once per output, i.e. in the first K split only
                        const uint32_t xs =
                            ((p.kt_per_split && blockIdx.z) || token >= p.ncols) ? 0u : (uint32_t)__ldcg(p.xsum + token);
#pragma unroll
                        for (int q = 0; q < 32; ++q) v[q] -= xs;
                        if (p.kt_per_split) {  // one of several partial sums: exact, in any order
                            // A lane per token adds to 32 lines an instruction and takes longer with every token; whole lines at a
                            // time take the same time for any number.  us at 36 / 48 / 64 columns: 2560 x 2560 12.5 / 14.5 / 16.7
                            // against 14.5 / 14.7 / 14.5, 8192 x 8192 18.4 / 20.5 / 23.0 against 21.6 / 21.9 / 21.8, 1000 x 1000
                            // 12.1 / 13.7 / 15.7 against 14.7, 13824 x 2560 17.9 / 20.2 / 21.9 against 18.5 / 18.7 / 18.7 (903
                            // columns of 2560 x 2560: 56.8 against 25.4).
                            if (p.ncols <= T5_SCATTER_COLS) {
                                if (token < p.ncols) {
                                    int32_t* dst = p.acc + (size_t)token * p.out + rbase;
#pragma unroll
                                    for (int q = 0; q < 32; ++q)
                                        if (rbase + q < p.out) atomicAdd(dst + q, (int32_t)v[q]);
                                }
                            } else {
                                t5_put_rows<true>(ring + (uint32_t)warp * T5_XPOSE_BYTES, v, p.acc + (size_t)tok_base * p.out + rbase,
                                                  (size_t)p.out, p.out - rbase, tok_base, p.ncols, lane);
                            }
                        } else if (rbase + 32 <= p.out && (p.out & 3) == 0) {
                            t5_store_rows(ring + (uint32_t)warp * T5_XPOSE_BYTES, v, p.acc + (size_t)tok_base * p.out + rbase,
                                          (size_t)p.out * sizeof(int32_t), tok_base, p.ncols, lane);
                        } else if (token < p.ncols) {
                            int32_t* dst = p.acc + (size_t)token * p.out + rbase;
#pragma unroll
                            for (int q = 0; q < 32; ++q)
                                if (rbase + q < p.out) dst[q] = (int32_t)v[q];
                        }
                    }
                }
            }
        }
#ifdef RB_TRACE
        if (tracedd) {
            trd.t[5] = gtime() - tld;  // read-back and stores
            trd.kind = 601;
            unsigned idx_ = atomicAdd(&g_trace_n, 1u);
            if (idx_ < 4096) g_trace[idx_] = trd;
        }
#endif
    } else if (warp == NDW) {
        // ---------------- token operand by TMA
        if (elect_lane()) {
            pdl_wait();  // the tokens are the work of the kernel before
            for (int kt = 0; kt < nk; ++kt) {
                const int s = kt % T5_STAGES;
                if (!t5_wait(smem_u32(&s_empty[s]), ((kt / T5_STAGES) & 1) ^ 1, abort_flag, p.status, 0x7c000003u)) break;
                const uint32_t bar = smem_u32(&s_full[s]);
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                             "r"(nhalf * p.box_rows * TILE_K)
                             : "memory");
                for (int half = 0; half < nhalf; ++half) {
                    const uint32_t dst = ring + s * T5_STAGE_BYTES + half * A_HALF;
                    asm volatile(
                        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes "
                        "[%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
                        "l"(&tmap), "r"((ktb + kt) * TILE_K), "r"(tok0 + half * 128), "r"(bar)
                        : "memory");
                }
            }
        }
    } else {
        // ---------------- MMA issue
        if (elect_lane()) {
            // kind::i8, S32 accumulate, signed tokens (A) x unsigned weight codes (B), both K-major, N = ROWS, M = 128
            const uint32_t idesc = (2u << 4) | (1u << 7) | (0u << 10) | ((uint32_t)(T5_ROWS >> 3) << 17) | ((128u >> 4) << 24);
            bool ok = true;
#ifdef RB_TRACE
            TraceRec trm = {};
            const bool traced = blockIdx.x == 0 && blockIdx.y == 0;
            unsigned long long tl = gtime(), t0m = tl;
#endif
            for (int kt = 0; kt < nk && ok; ++kt) {
                const int s = kt % T5_STAGES;
                ok = t5_wait(smem_u32(&s_full[s]), (kt / T5_STAGES) & 1, abort_flag, p.status, 0x7c000004u);
                if (!ok) break;
#ifdef RB_TRACE
                if (traced) { const unsigned long long n_ = gtime(); trm.t[0] += n_ - tl; tl = n_; }
#endif
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t abase = ring + s * T5_STAGE_BYTES, bbase = abase + T5_A_BYTES;
                for (int half = 0; half < nhalf; ++half)
#pragma unroll
                    for (int k4 = 0; k4 < TILE_K / 32; ++k4) {
                        const uint64_t da = t5_desc(abase + half * A_HALF + k4 * 32);
                        const uint64_t db = t5_desc(bbase + k4 * 32);
                        const uint32_t accumulate = (kt > 0 || k4 > 0) ? 1u : 0u;
                        asm volatile(
                            "{\n\t"
                            ".reg .pred p;\n\t"
                            "setp.ne.b32 p, %4, 0;\n\t"
                            "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t"
                            "}\n" ::"r"(tmem + (uint32_t)(half * ROWS)),
                            "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u)
                            : "memory");
                    }
                // arrives on the stage's "empty" barrier once these MMAs have read their operands
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 smem_u32(&s_empty[s]))
                             : "memory");
#ifdef RB_TRACE
                if (traced) { const unsigned long long n_ = gtime(); trm.t[1] += n_ - tl; tl = n_; }
#endif
            }
#ifdef RB_TRACE
            if (traced) {
                trm.t[2] = gtime() - t0m;
                trm.t[7] = (unsigned long long)p.nkt;
                trm.kind = 600;
                unsigned idx_ = atomicAdd(&g_trace_n, 1u);
                if (idx_ < 4096) g_trace[idx_] = trm;
            }
#endif
            if (ok)
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 smem_u32(&s_accf))
                             : "memory");
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
    if (warp == NDW) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Cfg::TMEM_COLS));
    }
}

// ---------------------------------------------------------------------------------------
// Products of more than 128 tokens (takes_pairs; gate/up and q/k/v always): a pair of CTAs per tile, tcgen05.mma.cta_group::2
// (M = 256 tokens, N = 256 weight rows, K = 32).  Each CTA holds 128 tokens and decodes 128 weight rows; the tensor cores of
// both SMs read both halves of the weights.  A CTA's accumulator is then 128 lanes x 256 columns, so that two fit tensor memory
// and the read-back of one tile runs beside the MMAs of the next, and a K step of the pair moves through each SM's shared
// memory 16 KB of tokens and 16 KB of decoded weights for 128 x 256 outputs (a CTA by itself: 32 + 32 KB for twice the
// outputs, and the read-back outside the K loop).  Persistent: one pair per two SMs walks the tiles.
// 16384 tokens, us with a CTA per 256 x 256 tile / now: gate/up 2 x 6912 x 2560 523 / 353, o 2560 x 2560 105 / 78, down
// 2560 x 6912 220 / 171, q/k/v 3840 x 2560 233 / 140; 1500 tokens: gate/up 63 / 45, q/k/v 35 / 29.
// Per CTA: warps 0-3 decode the even and 4-7 the odd K steps, two 16-row tiles each, 8-15 read back, 16 loads tokens (TMA), 17 issues MMAs (rank 0).
// Barriers: full (of rank 0: both CTAs' copies and decoder warps), empty (one per CTA, a commit to both), accumulator full (the
// same) and empty (of rank 0: both CTAs' read-back warps).
enum { PAIR_SUMS = 0, PAIR_GATED = 1, PAIR_QKV = 2 };
constexpr int PR_DEC = 8, PR_EPI = 8, PR_THREADS = (PR_DEC + PR_EPI + 2) * 32;
constexpr int PR_STAGES = 5, PR_HALF = 128 * TILE_K, PR_STAGE = 2 * PR_HALF, PR_AHEAD = 4;  // PR_AHEAD: steps of a decoder warp
constexpr int PR_SMEM = PR_STAGES * PR_STAGE + PR_EPI * (int)T5_XPOSE_BYTES + 1024;

// An mbarrier of CTA 0 of the pair.
__device__ __forceinline__ uint32_t pr_lead(uint32_t bar) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(bar));
    return r;
}
// Release at cluster scope: what this CTA's decoders wrote to its shared memory is read by an MMA that a thread of the other CTA
// issues (which waits with an acquire of that scope).  Restricted to shared memory: the unrestricted form also waits for the
// weights that the warp has requested ahead (13824 x 2560, 16384 tokens, int32 sums: 742 us, so 400; one thread of CTA 1 that
// passes its warps' arrivals on 867).
__device__ __forceinline__ void pr_arrive(uint32_t cluster_bar) {
    asm volatile(
        "fence.release.sync_restrict::shared::cta.cluster;\n\t"
        "mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar)
        : "memory");
}
__device__ __forceinline__ void pr_commit(uint32_t bar) {  // to the same barrier of both CTAs
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3)
        : "memory");
}
__device__ __forceinline__ void pr_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
template <int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PR_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ Tc5Params p) {
    extern __shared__ unsigned char t5_raw[];
    __shared__ __align__(8) unsigned long long s_full[PR_STAGES], s_empty[PR_STAGES], s_accf[2], s_acce[2];
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;
    const uint32_t ring = (smem_u32(t5_raw) + 1023u) & ~1023u, xpose = ring + PR_STAGES * PR_STAGE;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = blockIdx.x & 1;
    const int nk = p.nkt, ntiles = p.mt * p.nt, pair0 = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    volatile int* abort_flag = &s_abort;

    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int s = 0; s < PR_STAGES; ++s) {
            t5_bar_init(smem_u32(&s_full[s]), PR_DEC + 1);  // half of each CTA's decoders, the copies
            t5_bar_init(smem_u32(&s_empty[s]), 1);
        }
        for (int s = 0; s < 2; ++s) {
            t5_bar_init(smem_u32(&s_accf[s]), 1);
            t5_bar_init(smem_u32(&s_acce[s]), 2 * PR_EPI);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == PR_DEC + PR_EPI) {  // all columns of both SMs (one CTA per SM)
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    pr_sync();  // both CTAs' barriers are initialised
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;

    // tiles in blocks of 16 token tiles, token tiles fastest: the pairs of a wave share weight tiles
    auto place = [&](int t, int& m, int& n) {
        const int block = t / (16 * p.nt), bm = min(16, p.mt - block * 16), r = t - block * 16 * p.nt;
        n = r / bm;
        m = block * 16 + (r - n * bm);
    };

    if (warp < PR_DEC) {
        // ---------------- weight decoders: a warp turns row tiles 2 w and 2 w + 1 of this CTA's half of every other K step into
        // operand bytes (one chain of wait, decode, fence and arrival per two steps and two tiles: with a tile of every step a
        // warp the 13824 x 2560 product of 16384 tokens took 439 us, so 353)
        const int g = lane >> 2, t4 = lane & 3, w = warp & 3, odd = warp >> 2;
        const uint4 none = make_uint4(0x55555555u, 0x55555555u, 0x55555555u, 0x55555555u);  // zero weights
        auto row_of = [&](int t, int u) -> const uint4* {
            int m, n;
            place(t, m, n);
            int rt = n * 16 + rank * 8 + 2 * w + u;
            if constexpr (EPI == PAIR_GATED) {  // rank 0: 128 gate rows; rank 1: the same channels of the up matrix
                const int ch = n * 8 + 2 * w + u, ff_rt = p.ff / TILE_ROWS;
                rt = ch < ff_rt ? rank * ff_rt + ch : p.nrt;
            }
            return rt < p.nrt ? p.tiles + (size_t)rt * nk * 32 + lane : nullptr;
        };
        // requested PR_AHEAD of its steps before their decode, across tiles
        int ft = pair0, fk = 0;
        const uint4 *fp0 = nullptr, *fp1 = nullptr;
        auto enter = [&] {
            if (ft < ntiles) {
                fp0 = row_of(ft, 0);
                fp1 = row_of(ft, 1);
            }
        };
        auto skip = [&](int steps) {
            fk += steps;
            if (fk < nk) return;
            do {
                fk -= nk;
                ft += pairs;
            } while (fk >= nk);
            enter();
        };
        auto fetch = [&](uint4 (&dst)[2]) {
            if (ft >= ntiles) return;
            dst[0] = fp0 ? ld_stream_v4(fp0 + (size_t)fk * 32) : none;
            dst[1] = fp1 ? ld_stream_v4(fp1 + (size_t)fk * 32) : none;
            skip(2);
        };
        enter();
        skip(odd);
        uint4 wv[PR_AHEAD][2];
#pragma unroll
        for (int u = 0; u < PR_AHEAD; ++u) fetch(wv[u]);
        const int total = pair0 < ntiles ? ((ntiles - pair0 + pairs - 1) / pairs) * nk : 0;
        int s = odd;
        uint32_t parity = 1;
        bool ok = true;
        for (int it0 = odd; it0 < total && ok; it0 += 2 * PR_AHEAD) {
#pragma unroll
            for (int u = 0; u < PR_AHEAD; ++u) {
                if (it0 + 2 * u >= total) break;
                ok = t5_wait(smem_u32(&s_empty[s]), parity, abort_flag, p.status, 0x7c000011u);
                if (!__all_sync(0xffffffffu, ok)) {
                    ok = false;
                    break;
                }
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    const uint32_t base = ring + s * PR_STAGE + PR_HALF + (uint32_t)(2 * w + v) * 2048u + (uint32_t)g * 128u;
                    const uint32_t pw[4] = {wv[u][v].x, wv[u][v].y, wv[u][v].z, wv[u][v].w};
#pragma unroll
                    for (int rh = 0; rh < 2; ++rh) {
                        const uint32_t lo = pw[rh], hi = pw[rh + 2];
#pragma unroll
                        for (int c = 0; c < 2; ++c) {  // 16-byte chunk 2 t4 + c holds bit pairs 2 c and 2 c + 1
                            const uint32_t a0 = (lo >> (4 * c)) & 0x03030303u, a1 = (hi >> (4 * c)) & 0x03030303u;
                            const uint32_t a2 = (lo >> (4 * c + 2)) & 0x03030303u, a3 = (hi >> (4 * c + 2)) & 0x03030303u;
                            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(base + rh * 1024u + (uint32_t)(((2 * t4 + c) ^ g) << 4)),
                                         "r"(a0), "r"(a1), "r"(a2), "r"(a3)
                                         : "memory");
                        }
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic writes -> tensor-core reads
                __syncwarp();
                if (lane == 0) pr_arrive(pr_lead(smem_u32(&s_full[s])));
                fetch(wv[u]);
                s += 2;
                if (s >= PR_STAGES) {
                    s -= PR_STAGES;
                    parity ^= 1u;
                }
            }
        }
    } else if (warp < PR_DEC + PR_EPI) {
        // ---------------- read-back: lane = token, 32 columns (weight rows) per load; the two warps of a lane quarter alternate
        const int wq = warp & 3, grp = (warp - PR_DEC) >> 2;
        const uint32_t stage = xpose + (uint32_t)(warp - PR_DEC) * T5_XPOSE_BYTES;
        int lt = 0;
        for (int t = pair0; t < ntiles; t += pairs, ++lt) {
            int m, n;
            place(t, m, n);
            const int buf = lt & 1, tok_base = m * 256 + rank * 128 + wq * 32, token = tok_base + lane;
            const bool good = t5_wait<true>(smem_u32(&s_accf[buf]), (lt >> 1) & 1, abort_flag, p.status, 0x7c000012u);
            if (!__all_sync(0xffffffffu, good)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t acc = tmem + ((uint32_t)(wq * 32) << 16) + (uint32_t)buf * 256u;
            const bool live = token < p.ncols;
            const int32_t xs = live ? __ldg(p.xsum + token) : 0;
            // the accumulator is free again once every warp has its last columns in registers
            auto release = [&] {
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) pr_arrive(pr_lead(smem_u32(&s_acce[buf])));
            };
            if constexpr (EPI == PAIR_QKV) {
                // per item a head of the tile (0 / 1) and 16 pairs of its rows, 16 pc + i with 64 + 16 pc + i.  They are rotated on
                // their way out, where four lanes share a token and read its angles as whole sectors (a lane per token read 32
                // lines an instruction, and the read-back took 17 us a tile)
                const int bb = live ? token / p.seq : 0;
                const int pos = live ? __ldg(p.past_len + bb) + (token - bb * p.seq) : 0;
                const float sxv = live ? __ldg(p.sx + token) : 0.f;
#pragma unroll 1
                for (int item = grp; item < 8; item += 2) {
                    const int hh = item >> 2, pc = item & 3;
                    const int R0 = n * 256 + hh * 128;  // first row of the head in the stacked matrix
                    uint32_t gv[32], uv[32];
                    t5_ld16(acc + (uint32_t)(hh * 128 + pc * 16), gv);
                    t5_ld16(acc + (uint32_t)(hh * 128 + pc * 16 + 64), uv);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (item + 2 >= 8) release();
                    if (R0 >= p.out) continue;  // warp-uniform
                    const int kind = R0 < p.dq ? 0 : (R0 < p.dq + p.dkv ? 1 : 2);  // q, k, v
                    const int head = (kind == 0 ? R0 : (kind == 1 ? R0 - p.dq : R0 - p.dq - p.dkv)) >> 7;
                    const float sc = kind == 0 ? p.sq : (kind == 1 ? p.sk : p.sv);
                    float* cache = kind == 1 ? p.k_cache : p.v_cache;
#pragma unroll
                    for (int q = 0; q < 16; q += 4) {
                        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(stage + (uint32_t)lane * 144u + 4u * q),
                                     "f"(((float)((int32_t)gv[q] - xs) * sxv) * sc), "f"(((float)((int32_t)gv[q + 1] - xs) * sxv) * sc),
                                     "f"(((float)((int32_t)gv[q + 2] - xs) * sxv) * sc), "f"(((float)((int32_t)gv[q + 3] - xs) * sxv) * sc)
                                     : "memory");
                        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(stage + (uint32_t)lane * 144u + 64u + 4u * q),
                                     "f"(((float)((int32_t)uv[q] - xs) * sxv) * sc), "f"(((float)((int32_t)uv[q + 1] - xs) * sxv) * sc),
                                     "f"(((float)((int32_t)uv[q + 2] - xs) * sxv) * sc), "f"(((float)((int32_t)uv[q + 3] - xs) * sxv) * sc)
                                     : "memory");
                    }
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int tl = 8 * i + (lane >> 2), at = 16 * pc + 4 * (lane & 3), t2 = tok_base + tl;
                        const int pos2 = __shfl_sync(0xffffffffu, pos, tl), b2 = __shfl_sync(0xffffffffu, bb, tl);
                        float4 a, c;
                        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                                     : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w)
                                     : "r"(stage + (uint32_t)tl * 144u + 16u * (lane & 3)));
                        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                                     : "=f"(c.x), "=f"(c.y), "=f"(c.z), "=f"(c.w)
                                     : "r"(stage + (uint32_t)tl * 144u + 64u + 16u * (lane & 3)));
                        if (t2 >= p.ncols) continue;
                        if (kind != 2 && p.rope != nullptr && pos2 < p.max_seq) {
                            const float4* cs4 = reinterpret_cast<const float4*>(p.rope + (size_t)pos2 * 64 + at);
                            const float4 s0 = __ldg(cs4), s1 = __ldg(cs4 + 1);  // (cos, sin) of four pairs
                            const float4 r = make_float4(a.x * s0.x - c.x * s0.y, a.y * s0.z - c.y * s0.w, a.z * s1.x - c.z * s1.y,
                                                         a.w * s1.z - c.w * s1.w);
                            c = make_float4(c.x * s0.x + a.x * s0.y, c.y * s0.z + a.y * s0.w, c.z * s1.x + a.z * s1.y, c.w * s1.z + a.w * s1.w);
                            a = r;
                        }
                        float* dst;  // the token's q row, or its position's row of the head's cache
                        if (kind == 0)
                            dst = p.qout + (size_t)t2 * p.dq + (size_t)head * 128;
                        else if (pos2 < p.max_seq)
                            dst = cache + (((size_t)b2 * (p.dkv >> 7) + head) * p.max_seq + pos2) * 128;
                        else
                            continue;
                        *reinterpret_cast<float4*>(dst + at) = a;
                        *reinterpret_cast<float4*>(dst + 64 + at) = c;
                    }
                    __syncwarp();  // the block is rewritten by the next item
                }
            } else if constexpr (EPI == PAIR_GATED) {
                // per item 32 channels: gate sums in columns [32 ch, +32), up in [128 + 32 ch, +32)
                const float sxv = live ? __ldg(p.sx + token) : 0.f;
#pragma unroll 1
                for (int ch = grp; ch < 4; ch += 2) {
                    uint32_t gv[32], uv[32];
                    t5_ld32(acc + (uint32_t)(ch * 32), gv);
                    t5_ld32(acc + (uint32_t)(ch * 32 + 128), uv);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (ch + 2 >= 4) release();
                    const int c0 = n * 128 + ch * 32;
                    if (c0 >= p.ff) continue;  // warp-uniform
                    // the gated values replace the gate sums in place (bit patterns of float32)
#pragma unroll
                    for (int q = 0; q < 32; ++q) {
                        const float g = ((float)((int32_t)gv[q] - xs) * sxv) * p.sg, u = ((float)((int32_t)uv[q] - xs) * sxv) * p.su;
                        float r;
                        if (p.ffn_act == ROTOR_B200_FFN_RELU2) {
                            const float a = fmaxf(g, 0.f);
                            r = a * a * u;
                        } else {
                            const float c = fminf(fmaxf(u, -20.f), 20.f);
                            r = g * (c / (1.f + expf(-c)));
                        }
                        gv[q] = __float_as_uint(r);
                    }
                    if (c0 + 32 <= p.ff && (p.ff & 3) == 0) {
                        t5_store_rows(stage, gv, p.gated + (size_t)tok_base * p.ff + c0, (size_t)p.ff * sizeof(float), tok_base, p.ncols, lane);
                    } else if (live) {
                        float* dst = p.gated + (size_t)token * p.ff + c0;
#pragma unroll
                        for (int q = 0; q < 32; ++q)
                            if (c0 + q < p.ff) dst[q] = __uint_as_float(gv[q]);
                    }
                }
            } else {
#pragma unroll 1
                for (int ch = grp; ch < 8; ch += 2) {
                    uint32_t v[32];
                    t5_ld32(acc + (uint32_t)(ch * 32), v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (ch + 2 >= 8) release();
                    const int rbase = n * 256 + ch * 32;
                    if (rbase >= p.out) continue;  // warp-uniform
#pragma unroll
                    for (int q = 0; q < 32; ++q) v[q] -= (uint32_t)xs;
                    if (rbase + 32 <= p.out && (p.out & 3) == 0) {
                        t5_store_rows(stage, v, p.acc + (size_t)tok_base * p.out + rbase, (size_t)p.out * sizeof(int32_t), tok_base, p.ncols, lane);
                    } else {
                        t5_put_rows<false>(stage, v, p.acc + (size_t)tok_base * p.out + rbase, (size_t)p.out, p.out - rbase, tok_base, p.ncols, lane);
                    }
                }
            }
        }
    } else if (warp == PR_DEC + PR_EPI) {
        // ---------------- token operand by TMA: this CTA's 128 tokens, counted by rank 0's barrier
        if (elect_lane()) {
            int s = 0;
            uint32_t parity = 1;
            bool ok = true;
            for (int t = pair0; t < ntiles && ok; t += pairs) {
                int m, n;
                place(t, m, n);
                for (int kt = 0; kt < nk; ++kt) {
                    ok = t5_wait(smem_u32(&s_empty[s]), parity, abort_flag, p.status, 0x7c000013u);
                    if (!ok) break;
                    const uint32_t bar = smem_u32(&s_full[s]);
                    if (rank == 0) t5_bar_expect(bar, 2 * PR_HALF);
                    asm volatile(
                        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
                        "[%0], [%1, {%2, %3}], [%4];" ::"r"(ring + s * PR_STAGE),
                        "l"(&tmap), "r"(kt * TILE_K), "r"(m * 256 + rank * 128), "r"(pr_lead(bar))
                        : "memory");
                    if (++s == PR_STAGES) {
                        s = 0;
                        parity ^= 1u;
                    }
                }
            }
            for (int i = 0; i < PR_STAGES && ok; ++i) {  // the last commits to this CTA's barriers have landed
                ok = t5_wait(smem_u32(&s_empty[s]), parity, abort_flag, p.status, 0x7c000016u);
                if (++s == PR_STAGES) {
                    s = 0;
                    parity ^= 1u;
                }
            }
        }
    } else if (rank == 0) {
        // ---------------- MMA issue for both SMs
        if (elect_lane()) {
            // kind::i8, S32 accumulate, signed tokens (A) x unsigned weight codes (B), both K-major, M = 256, N = 256
            constexpr uint32_t idesc = (2u << 4) | (1u << 7) | ((256u >> 3) << 17) | ((256u >> 4) << 24);
            int s = 0, lt = 0;
            uint32_t parity = 0;
            bool ok = true;
            for (int t = pair0; t < ntiles && ok; t += pairs, ++lt) {
                const int buf = lt & 1;
                ok = t5_wait<true>(smem_u32(&s_acce[buf]), ((lt >> 1) & 1) ^ 1, abort_flag, p.status, 0x7c000014u);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int kt = 0; kt < nk; ++kt) {
                    ok = t5_wait<true>(smem_u32(&s_full[s]), parity, abort_flag, p.status, 0x7c000015u);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t da = t5_desc(ring + s * PR_STAGE), db = t5_desc(ring + s * PR_STAGE + PR_HALF);
#pragma unroll
                    for (int k4 = 0; k4 < TILE_K / 32; ++k4)
                        asm volatile(
                            "{\n\t"
                            ".reg .pred p;\n\t"
                            "setp.ne.b32 p, %4, 0;\n\t"
                            "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t"
                            "}\n" ::"r"(tmem + (uint32_t)buf * 256u),
                            "l"(da + 2 * k4), "l"(db + 2 * k4), "r"(idesc), "r"((uint32_t)(kt > 0 || k4 > 0)), "r"(0u)
                            : "memory");
                    pr_commit(smem_u32(&s_empty[s]));
                    if (++s == PR_STAGES) {
                        s = 0;
                        parity ^= 1u;
                    }
                }
                if (ok) pr_commit(smem_u32(&s_accf[buf]));
            }
        }
    }

    // ---------------- common exit: nothing of either CTA may still be in flight when one returns
    __syncwarp();
    if (*abort_flag && threadIdx.x == 0) {
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000LL) {
        }  // about a millisecond for copies already issued to land
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    pr_sync();
    if (warp == PR_DEC + PR_EPI) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
    }
}

static PerDevice<bool> g_tc5_ready;

// Shapes this kernel takes: enough tokens to be worth its tile, 16-byte aligned operands.
bool gemm_tcgen05_supported(size_t out, size_t in, int ncols, const void* xq) {
    static const bool off = getenv("ROTOR_B200_NO_TCGEN05") != nullptr;  // measurement aid: legacy mma.sync path
    // with fewer than 256 tokens the tile is partly empty, but the product is then bound by the weight stream
    return !off && ncols > ACC_FEW_COLS && out >= 16 && in >= 4 && ((uintptr_t)xq & 15) == 0;
}

int configure_gemm_tcgen05() {
    if (g_tc5_ready.here()) return ROTOR_B200_OK;
    if (!t5_encoder()) return ROTOR_B200_ERR_CUDA;
    RB_CUDA(cudaFuncSetAttribute(gemm_tcgen05_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, T5Cfg<256>::SMEM));
    RB_CUDA(cudaFuncSetAttribute(gemm_tcgen05_kernel<256, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize, T5Cfg<256, 128>::SMEM));
    RB_CUDA(cudaFuncSetAttribute(gemm_tcgen05_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, T5Cfg<64>::SMEM));
    RB_CUDA(cudaFuncSetAttribute(gemm_pair_kernel<PAIR_SUMS>, cudaFuncAttributeMaxDynamicSharedMemorySize, PR_SMEM));
    RB_CUDA(cudaFuncSetAttribute(gemm_pair_kernel<PAIR_GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, PR_SMEM));
    RB_CUDA(cudaFuncSetAttribute(gemm_pair_kernel<PAIR_QKV>, cudaFuncAttributeMaxDynamicSharedMemorySize, PR_SMEM));
    g_tc5_ready.here() = true;
    return ROTOR_B200_OK;
}

// The token operand: int8 rows of kpad bytes, boxes of 128 tokens x 128 bytes; rows past the last token read zeros.
// (rows: of a box, fewer where there are fewer tokens: what lies behind lands in accumulator lanes that nobody reads)
static bool encode_tokens(CUtensorMap* tmap, const void* xq, size_t kpad, int ncols, int rows = 128) {
    const cuuint64_t gdim[2] = {(cuuint64_t)kpad, (cuuint64_t)ncols};
    const cuuint64_t gstride[1] = {(cuuint64_t)kpad};  // bytes between token rows
    const cuuint32_t box[2] = {(cuuint32_t)TILE_K, (cuuint32_t)rows};
    const cuuint32_t estride[2] = {1u, 1u};
    const T5EncodeFn encode = t5_encoder();
    return encode && encode(tmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(xq), gdim, gstride, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Whether a product goes to pairs of CTAs: tiles for every pair, or, above 128 columns, K ranges so short that splitting them
// only adds read-backs, or a pair for every fourth tile whose K range is not too long for the pairs that are left idle.  us of a layer
// call, split / paired: 3840 x 2560 129 columns 24.9 / 22.8, 1500 65.8 / 55.6; 1000 x 1000 256 29.1 / 18.8; 4096 x 4096 (16 tiles) 129
// 25.0 / 26.9, (32) 257 37.3 / 29.1; 8192 x 8192 (32) 129 35.2 / 39.4, 144 39.1 / 41.3, 168 43.4 / 41.5, (64) 257 55.7 / 45.4; 2560 x
// 6912 (10) 256 33.2 / 35.1, (20) 300 37.3 / 36.9, (40) 903 53.7 / 47.4; 4096 x 11008 (16) 256 43.7 / 49.8, (32) 257 49.6 / 51.0, (64) 903
// 92.5 / 81.7; 8192 x 28672 (32) 129 66.0 / 95.4, 256 83.3 / 104.0, (64) 257 112.8 / 102.7.  A whole tile a CTA / paired, 57344 x
// 8192: 129 145.7 / 151.9, 257 242.0 / 253.5, 512 328 / 306, 1500 824 / 761.  Rows of sums off a 16-byte boundary leave
// a value at a time and take longer: 3001 x 1923 129 23.2 / 26.9, 168 31.2 / 28.5; 8001 x 8190 (32) 256 47.5 / 51.8, (64) 257 55.9 /
// 52.8; 2562 x 6912 (33) 700 47.5 / 49.5, (44) 903 53.7 / 53.1; 999 x 8000 (24) 1500 53.4 / 59.7; too short a K range to be split
// (5003 x 777) 192 25.0 / 29.0, 300 33.0 / 29.0.
static bool takes_pairs(size_t out, int ncols, int nkt, int tiles256) {
    const bool ragged = out & 3;
    if (ncols <= 128 || 2 * tiles256 >= fused_sm_count()) return ncols > 128;
    if (nkt <= 24) return !ragged || ncols > (nkt < 8 ? 256 : 144);
    return tiles256 >= (ragged ? 40 : 20) && nkt <= 4 * tiles256 && ncols > 144;
}

// fewer 256-row tiles than SMs: split the K range so that the grid covers the GPU (a K step of a
// 256-row tile costs a decoder less per weight than four steps of 64-row tiles); at least four K
// steps per CTA, partial sums added into the zeroed accumulators
int gemm_tcgen05_splits(size_t out, size_t in, int ncols) {
    const int nkt = (int)(kpad_of(in) / TILE_K), rows = (int)opad_of(out);
    const int tiles256 = (ncols + 255) / 256 * ((rows + 255) / 256), sms = fused_sm_count();
    int splits = tiles256 < sms && !takes_pairs(out, ncols, nkt, tiles256) ? sms / tiles256 : 1;
    if (splits > nkt / 4) splits = nkt / 4;
    if (splits < 2) return 1;
    const int per = (nkt + splits - 1) / splits;
    return (nkt + per - 1) / per;
}

// dependent: the launch may start while the kernel before it ends (the weights are older than that kernel).
template <int ROWS, int TOK>
static int launch_t5(const CUtensorMap& tmap, const Tc5Params& p, dim3 grid, bool dependent, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(T5Cfg<ROWS, TOK>::THREADS);
    cfg.dynamicSmemBytes = T5Cfg<ROWS, TOK>::SMEM;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_use_pdl && dependent ? 1 : 0;
    if (cudaLaunchKernelEx(&cfg, gemm_tcgen05_kernel<ROWS, TOK>, tmap, p) != cudaSuccess) {
        ++g_launch_count;
        return ROTOR_B200_ERR_CUDA;
    }
    return launch_status();
}

// n: weight rows (or pairs of gate and up rows, two each) that the tiles of 256 cover.
template <int EPI>
static int launch_pair(const CUtensorMap& tmap, Tc5Params& p, int n, cudaStream_t st) {
    p.mt = (p.ncols + 255) / 256;
    p.nt = (n + 255) / 256;
    const int tiles = p.mt * p.nt, pairs = fused_sm_count() / 2;
    gemm_pair_kernel<EPI><<<2 * (tiles < pairs ? tiles : pairs), PR_THREADS, PR_SMEM, st>>>(tmap, p);
    return launch_status();
}

int launch_gemm_tcgen05(const void* tiles, size_t out, size_t in, const int8_t* xq, const int32_t* xsum, int ncols,
                        int32_t* acc, cudaStream_t st, bool zeroed, bool dependent) {
    int rc = configure_gemm_tcgen05();
    if (rc) return rc;
    Tc5Params p = {};
    p.tiles = (const uint4*)tiles;
    p.xsum = xsum;
    p.acc = acc;
    p.status = library_status_word();
    p.out = (int)out;
    p.nrt = (int)(opad_of(out) / TILE_ROWS);
    p.nkt = (int)(kpad_of(in) / TILE_K);
    p.ncols = ncols;
    if (!p.status) return ROTOR_B200_ERR_CUDA;
    CUtensorMap tmap;
    p.box_rows = ncols < 128 ? (ncols + 7) / 8 * 8 : 128;
    if (!encode_tokens(&tmap, xq, kpad_of(in), ncols, p.box_rows)) return ROTOR_B200_ERR_CUDA;
    const int tok_tiles = (ncols + 255) / 256, rows = p.nrt * TILE_ROWS;
    const int sms = fused_sm_count(), tiles256 = tok_tiles * ((rows + 255) / 256);
    int splits = gemm_tcgen05_splits(out, in, ncols);
    if (takes_pairs(out, ncols, p.nkt, tiles256)) return launch_pair<PAIR_SUMS>(tmap, p, rows, st);
    auto launch256 = [&](dim3 grid) {
        // (64 tokens, 57344 x 8192: 78.3 -> 66.9 us, 8192 x 28672: 44.7 -> 38.7; runs of fewer steps end before the
        // deeper look-ahead is filled and take the variant with less code)
        if (ncols <= 128 && (p.kt_per_split ? p.kt_per_split : p.nkt) >= T5_DEEP_STEPS) return launch_t5<256, 128>(tmap, p, grid, dependent, st);
        return launch_t5<256, 256>(tmap, p, grid, dependent, st);
    };
    if (splits >= 2) {
        p.kt_per_split = (p.nkt + splits - 1) / splits;
        if (!zeroed) RB_CUDA(cudaMemsetAsync(acc, 0, (size_t)ncols * out * sizeof(int32_t), st));
        return launch256(dim3(tok_tiles, (rows + 255) / 256, splits));
    } else if (tiles256 < sms) {  // 256-row tiles would leave SMs idle
        return launch_t5<64, 256>(tmap, p, dim3(tok_tiles, (rows + 63) / 64), dependent, st);
    }
    return launch256(dim3(tok_tiles, (rows + 255) / 256));
}

// Gate/up product with the gating in the epilogue: `tiles` holds the gate matrix followed by the up
// matrix (ff rows each, ff a multiple of 16), one activation term per token.  Writes
// gated[token][channel] as float32; no int32 accumulator leaves the kernel.
bool gemm_tcgen05_gated_supported(size_t ff, size_t in, int ncols, const void* xq) {
    return ff % TILE_ROWS == 0 && ncols > 128 && gemm_tcgen05_supported(2 * ff, in, ncols, xq);
}

int launch_gemm_tcgen05_gated(const void* tiles, size_t ff, size_t in, const int8_t* xq, const float* sx,
                              const int32_t* xsum, int ncols, float sg, float su, int ffn_act, float* gated,
                              cudaStream_t st) {
    int rc = configure_gemm_tcgen05();
    if (rc) return rc;
    if (!gemm_tcgen05_gated_supported(ff, in, ncols, xq)) return ROTOR_B200_ERR_SHAPE;
    Tc5Params p = {};
    p.tiles = (const uint4*)tiles;
    p.status = library_status_word();
    p.out = (int)(2 * ff);
    p.nrt = (int)(2 * ff / TILE_ROWS);
    p.nkt = (int)(kpad_of(in) / TILE_K);
    p.ncols = ncols;
    p.gated = gated;
    p.sx = sx;
    p.xsum = xsum;
    p.sg = sg;
    p.su = su;
    p.ff = (int)ff;
    p.ffn_act = ffn_act;
    if (!p.status) return ROTOR_B200_ERR_CUDA;
    CUtensorMap tmap;
    if (!encode_tokens(&tmap, xq, kpad_of(in), ncols)) return ROTOR_B200_ERR_CUDA;
    return launch_pair<PAIR_GATED>(tmap, p, (int)(2 * ((ff + 127) / 128 * 128)), st);
}

// q/k/v product with dequantisation, rotary and the cache append in its read-back: head_dim 128, one
// activation term per token, more than 128 tokens.
bool gemm_tcgen05_qkv_supported(size_t dq, size_t dkv, size_t in, int head_dim, int ncols, const void* xq) {
    return head_dim == 128 && dq % 128 == 0 && dkv % 128 == 0 && ncols > 128 &&
           gemm_tcgen05_supported(dq + 2 * dkv, in, ncols, xq);
}

int launch_gemm_tcgen05_qkv(const void* tiles, size_t in, const int8_t* xq, const float* sx, const int32_t* xsum,
                            int ncols, const QkvFinishParams& f, cudaStream_t st) {
    int rc = configure_gemm_tcgen05();
    if (rc) return rc;
    const size_t dq = (size_t)f.n_heads * f.head_dim, dkv = (size_t)f.n_kv_heads * f.head_dim;
    if (!gemm_tcgen05_qkv_supported(dq, dkv, in, f.head_dim, ncols, xq) || f.terms != 1) return ROTOR_B200_ERR_SHAPE;
    Tc5Params p = {};
    p.tiles = (const uint4*)tiles;
    p.status = library_status_word();
    p.out = (int)(dq + 2 * dkv);
    p.nrt = (int)(opad_of(dq + 2 * dkv) / TILE_ROWS);
    p.nkt = (int)(kpad_of(in) / TILE_K);
    p.ncols = ncols;
    p.sx = sx;
    p.xsum = xsum;
    p.dq = (int)dq;
    p.dkv = (int)dkv;
    p.seq = f.seq;
    p.max_seq = f.max_seq;
    p.past_len = f.past_len;
    p.rope = f.rope;
    p.qout = f.q;
    p.k_cache = f.k_cache;
    p.v_cache = f.v_cache;
    p.sq = f.sq;
    p.sk = f.sk;
    p.sv = f.sv;
    if (!p.status) return ROTOR_B200_ERR_CUDA;
    CUtensorMap tmap;
    if (!encode_tokens(&tmap, xq, kpad_of(in), ncols)) return ROTOR_B200_ERR_CUDA;
    return launch_pair<PAIR_QKV>(tmap, p, p.nrt * TILE_ROWS, st);
}

}  // namespace rb
