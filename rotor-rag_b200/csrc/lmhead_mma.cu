// Tied LM head for many rows at once (batched generation steps, logits of every prompt
// position): logits[r][v] = sum_d x[r][d] * E[v][d] with the bf16 table E read ONCE for up to 128
// rows, instead of once per four rows (lmhead.cu).
//
// Reference: BitNetModel.forward, src/rotor/bitnet_model.py:235-242 (np.dot(hidden, embed.T));
// greedy pick: GreedySampling.sample, src/rotor/generation.py:31-42 (lowest index on ties).
//
// Bound by the table's stream from HBM up to about 64 rows, so the layout serves the stream: one CTA per SM owns a
// run of vocabulary rows (units of 16 rows, so that all CTAs end within 16 rows of one another), walks them 256 rows
// at a time and d 64 columns a stage, and keeps 3 to 6 stages (up to 200 KB) of TMA loads in flight.  The vocabulary
// rows are the MMA's M (two halves of 128, tcgen05.mma.kind::f16, one issuing thread), the token rows its N: the
// table is bf16 already, the float32 rows x are split once into hi + lo bf16 terms (x_split_kernel) and every tile
// costs E*hi + E*lo into one float32 accumulator, which keeps 16 mantissa bits of x.  256 vocabulary rows share one
// load of the token tiles: at 64 rows these are half the bytes of the table's and come from L2.  Two accumulators in
// tensor memory, so that four read-back warps empty one tile while the next is computed; a lane holds one vocabulary
// row, so a token's 32 logits leave as one 128-byte line, and its pick is one warp reduction over order-preserving
// keys.  Table loads of the first stages are issued before the launch wait (they depend on nothing).
// Measured (table 128256 wide, x split included; before: an mma.sync kernel of 128 x 64 tiles with two cp.async
// stages): 8 rows of d 2560 305 -> 131 us = 5.0 TB/s, 64 rows of d 8192 920 -> 404 us = 5.2 TB/s.  Loads of 128 rows
// instead of 16 gave 10 %, evicting the table's lines first up to 10 % more; two 64-column panels a stage nothing.
// Outputs: logits (optional) and one (max, argmax) partial per CTA and token row, merged by argmax_final_kernel.
// (The file, its entry points and ROTOR_B200_NO_LMHEAD_MMA keep the name of the mma.sync kernel that stood here before.)
#include <cuda_bf16.h>

#include <cstdlib>

#include "model.cuh"
#include "tc5.cuh"

namespace rb {

constexpr int LM5_V = 256;        // vocabulary rows per tile: two M halves
constexpr int LM5_K = 64;         // d per stage
constexpr int LM5_UNIT = 16;      // granularity of a CTA's share, and rows per table load where a half tile is not whole
constexpr int LM5_THREADS = 192;  // TMA warp, MMA warp, four read-back warps

template <int NT>
struct Lm5 {
    static constexpr int E_BYTES = LM5_V * LM5_K * 2, X_BYTES = NT * LM5_K * 2;
    static constexpr int STAGE = E_BYTES + 2 * X_BYTES;
    static constexpr int STAGES = NT >= 128 ? 3 : NT == 64 ? 4 : NT == 32 ? 5 : 6;
    static constexpr int SMEM = STAGES * STAGE + 1024;
    static constexpr int TMEM_COLS = 4 * NT;  // two accumulators of two halves
};

// x float32 [rows][d] -> hi / lo bf16 planes [rows][d] (lo plane at hi + rows * d)
__global__ void __launch_bounds__(256) x_split_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ out,
                                                      size_t n4, size_t plane) {
    pdl_trigger();  // launched without the attribute: everything before it is complete, the table may be requested
    const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= n4) return;
    const float4 v = reinterpret_cast<const float4*>(x)[i];
    const float f[4] = {v.x, v.y, v.z, v.w};
    __nv_bfloat16 h[4], l[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        h[e] = __float2bfloat16_rn(f[e]);
        l[e] = __float2bfloat16_rn(f[e] - __bfloat162float(h[e]));
    }
    *reinterpret_cast<uint2*>(out + 4 * i) = *reinterpret_cast<const uint2*>(h);
    *reinterpret_cast<uint2*>(out + plane + 4 * i) = *reinterpret_cast<const uint2*>(l);
}

struct Lm5Params {
    unsigned* status;
    int vocab, d, rows;
    float* logits;               // optional [rows][vocab]
    float* part_val;             // optional [rows][gridDim.x]: best logit of this CTA's vocabulary rows
    int* part_idx;
};

// Float to an unsigned key of the same order (both zeros alike); below every number: 0 for NaN, which is never picked.
__device__ __forceinline__ unsigned lm5_key(float v) {
    const unsigned u = __float_as_uint(v + 0.f);
    return v == v ? (u & 0x80000000u ? ~u : u | 0x80000000u) : 0u;
}
__device__ __forceinline__ float lm5_unkey(unsigned k) {
    return k ? __uint_as_float(k & 0x80000000u ? k & 0x7fffffffu : ~k) : -INFINITY;
}

template <int NT>
__global__ void __launch_bounds__(LM5_THREADS, 1)
lmhead_t5_kernel(const __grid_constant__ CUtensorMap tm_e, const __grid_constant__ CUtensorMap tm_unit,
                 const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ Lm5Params p) {
    using C = Lm5<NT>;
    constexpr int ST = C::STAGES;
    extern __shared__ unsigned char lm5_raw[];
    __shared__ __align__(8) unsigned long long s_full[ST], s_empty[ST], s_accf[2], s_acce[2];
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;
    __shared__ unsigned s_key[4][NT];
    __shared__ int s_idx[4][NT];
    const uint32_t ring = (smem_u32(lm5_raw) + 1023u) & ~1023u;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r0 = blockIdx.y * NT, nk = p.d / LM5_K;
    // this CTA's vocabulary rows [v0, v1)
    const long long units = (p.vocab + LM5_UNIT - 1) / LM5_UNIT;
    const int v0 = (int)(units * blockIdx.x / gridDim.x) * LM5_UNIT, v1 = (int)(units * (blockIdx.x + 1) / gridDim.x) * LM5_UNIT;
    volatile int* abort_flag = &s_abort;

    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int s = 0; s < ST; ++s) {
            t5_bar_init(smem_u32(&s_full[s]), 1);
            t5_bar_init(smem_u32(&s_empty[s]), 1);
        }
        for (int s = 0; s < 2; ++s) {
            t5_bar_init(smem_u32(&s_accf[s]), 1);
            t5_bar_init(smem_u32(&s_acce[s]), 4);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(C::TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;

    if (warp == 0) {
        if (elect_lane()) {
            // a stage's table rows (only those of the CTA's share: the tile's other rows keep what was there, in
            // accumulator lanes nobody reads) and the hi and lo token tiles
            auto table = [&](int it, int vt, int kt) {
                const uint32_t bar = smem_u32(&s_full[it % ST]), st = ring + (it % ST) * C::STAGE;
                const int n = min(LM5_V, v1 - vt);
                t5_bar_expect(bar, n * LM5_K * 2 + 2 * C::X_BYTES);
                int r = 0;
                for (; r + 128 <= n; r += 128) t5_tma_2d_once(st + r * LM5_K * 2, &tm_e, kt * LM5_K, vt + r, bar);
                for (; r < n; r += LM5_UNIT) t5_tma_2d_once(st + r * LM5_K * 2, &tm_unit, kt * LM5_K, vt + r, bar);
            };
            auto tokens = [&](int it, int kt) {
                const uint32_t bar = smem_u32(&s_full[it % ST]), st = ring + (it % ST) * C::STAGE + C::E_BYTES;
                t5_tma_2d(st, &tm_x, kt * LM5_K, r0, bar);
                t5_tma_2d(st + C::X_BYTES, &tm_x, kt * LM5_K, p.rows + r0, bar);
            };
            const int total = (v1 - v0 + LM5_V - 1) / LM5_V * nk, ahead = min(ST, total);
            for (int it = 0; it < ahead; ++it) table(it, v0 + it / nk * LM5_V, it % nk);
            pdl_wait();
            for (int it = 0; it < ahead; ++it) tokens(it, it % nk);
            int vt = v0 + ahead / nk * LM5_V, kt = ahead % nk;
            for (int it = ahead; it < total; ++it) {
                if (!t5_wait(smem_u32(&s_empty[it % ST]), ((it / ST) & 1) ^ 1, abort_flag, p.status, 0x78000001u)) break;
                table(it, vt, kt);
                tokens(it, kt);
                if (++kt == nk) {
                    kt = 0;
                    vt += LM5_V;
                }
            }
        }
    } else if (warp == 1) {
        if (elect_lane()) {
            constexpr uint32_t idesc = t5_idesc_bf16(128, NT);
            int it = 0, lt = 0;
            bool ok = true;
            for (int vt = v0; vt < v1 && ok; vt += LM5_V, ++lt) {
                const int buf = lt & 1, halves = v1 - vt > 128 ? 2 : 1;
                ok = t5_wait(smem_u32(&s_acce[buf]), ((lt >> 1) & 1) ^ 1, abort_flag, p.status, 0x78000002u);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int kt = 0; kt < nk; ++kt, ++it) {
                    const int s = it % ST;
                    ok = t5_wait(smem_u32(&s_full[s]), (it / ST) & 1, abort_flag, p.status, 0x78000003u);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t st = ring + s * C::STAGE;
                    const uint64_t dh = t5_desc(st + C::E_BYTES), dl = t5_desc(st + C::E_BYTES + C::X_BYTES);
                    for (int h = 0; h < halves; ++h) {
                        const uint64_t da = t5_desc(st + h * 128 * LM5_K * 2);
                        const uint32_t d = tmem + (uint32_t)(2 * buf + h) * NT;
#pragma unroll
                        for (int k16 = 0; k16 < 4; ++k16) {
                            t5_mma_ss(d, da + 2 * k16, dh + 2 * k16, idesc, (kt > 0 || k16 > 0) ? 1u : 0u);
                            t5_mma_ss(d, da + 2 * k16, dl + 2 * k16, idesc, 1u);
                        }
                    }
                    t5_commit(smem_u32(&s_empty[s]));
                }
                if (ok) t5_commit(smem_u32(&s_accf[buf]));
            }
        }
    } else {
        const int wq = warp & 3;  // the quarter of the tensor-memory lanes this warp reaches
        const int ntok = min(NT, p.rows - r0);
        // the warp's running pick of every token, in shared memory; vocabulary rows come in ascending order, so only a
        // larger key replaces it
        for (int i = lane; i < NT; i += 32) {
            s_key[wq][i] = 0u;
            s_idx[wq][i] = 0x7fffffff;
        }
        __syncwarp();
        int lt = 0;
        for (int vt = v0; vt < v1; vt += LM5_V, ++lt) {
            const int buf = lt & 1;
            const bool good = t5_wait(smem_u32(&s_accf[buf]), (lt >> 1) & 1, abort_flag, p.status, 0x78000004u);
            if (!__all_sync(0xffffffffu, good)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                const int vw = vt + h * 128 + wq * 32, v = vw + lane;
                const bool live = v < min(v1, p.vocab);
                if (vw >= v1) break;  // warp-uniform
                const uint32_t ta = tmem + ((uint32_t)(wq * 32) << 16) + (uint32_t)(2 * buf + h) * NT;
                constexpr int CH = NT < 32 ? NT : 32;
#pragma unroll 1
                for (int c = 0; c < ntok; c += CH) {
                    uint32_t w[32];
                    if constexpr (CH == 32) {
                        t5_ld32(ta + c, w);
                    } else {
                        t5_ld16(ta, w);
                    }
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int q = 0; q < CH; ++q) {
                        if (c + q >= ntok) continue;  // warp-uniform
                        const float val = __uint_as_float(w[q]);
                        if (p.logits && live) p.logits[(size_t)(r0 + c + q) * p.vocab + v] = val;
                        if (p.part_val) {
                            const unsigned key = live ? lm5_key(val) : 0u, top = __reduce_max_sync(0xffffffffu, key);
                            const int first = __ffs(__ballot_sync(0xffffffffu, key == top)) - 1;
                            if (lane == q && top > s_key[wq][c + q]) {
                                s_key[wq][c + q] = top;
                                s_idx[wq][c + q] = vw + first;
                            }
                        }
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) t5_bar_arrive(smem_u32(&s_acce[buf]));
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
    if (p.part_val && threadIdx.x < NT && r0 + (int)threadIdx.x < p.rows) {
        unsigned bk = s_key[0][threadIdx.x];
        int bi = s_idx[0][threadIdx.x];
        for (int w = 1; w < 4; ++w) {
            const unsigned ok = s_key[w][threadIdx.x];
            const int oi = s_idx[w][threadIdx.x];
            if (ok > bk || (ok == bk && oi < bi)) {
                bk = ok;
                bi = oi;
            }
        }
        p.part_val[(size_t)(r0 + threadIdx.x) * gridDim.x + blockIdx.x] = lm5_unkey(bk);
        p.part_idx[(size_t)(r0 + threadIdx.x) * gridDim.x + blockIdx.x] = bi;
    }
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::TMEM_COLS));
    }
}

// Partials per token row: one per CTA.  CTAs: one per SM, fewer where a share would be below a half tile of rows.
int lmhead_mma_parts(int vocab) {
    const int most = (vocab + 127) / 128, sms = fused_sm_count();
    return most < sms ? most : sms;
}

// Whether the many-row kernel takes this call (d in whole stages, 16-byte aligned rows).
bool lmhead_mma_supported(int rows, int d) {
    static const bool off = getenv("ROTOR_B200_NO_LMHEAD_MMA") != nullptr;  // comparison aid
    return !off && rows > 4 && d % LM5_K == 0;
}

int configure_lmhead_mma() {
    RB_CUDA(cudaFuncSetAttribute(lmhead_t5_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, Lm5<16>::SMEM));
    RB_CUDA(cudaFuncSetAttribute(lmhead_t5_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, Lm5<32>::SMEM));
    RB_CUDA(cudaFuncSetAttribute(lmhead_t5_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, Lm5<64>::SMEM));
    RB_CUDA(cudaFuncSetAttribute(lmhead_t5_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, Lm5<128>::SMEM));
    return t5_encoder() && library_status_word() ? ROTOR_B200_OK : ROTOR_B200_ERR_CUDA;
}

template <int NT>
static int lm5_launch(const __nv_bfloat16* embed, const __nv_bfloat16* xsplit, const Lm5Params& p, cudaStream_t st) {
    CUtensorMap te, tu, tx;
    if (!t5_map_bf16(&te, embed, p.vocab, p.d, p.d, 128) || !t5_map_bf16(&tu, embed, p.vocab, p.d, p.d, LM5_UNIT) ||
        !t5_map_bf16(&tx, xsplit, 2 * (size_t)p.rows, p.d, p.d, NT))
        return ROTOR_B200_ERR_CUDA;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(lmhead_mma_parts(p.vocab), (p.rows + NT - 1) / NT);
    cfg.blockDim = dim3(LM5_THREADS);
    cfg.dynamicSmemBytes = Lm5<NT>::SMEM;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_use_pdl ? 1 : 0;
    if (cudaLaunchKernelEx(&cfg, lmhead_t5_kernel<NT>, te, tu, tx, p) != cudaSuccess) {
        ++g_launch_count;
        return ROTOR_B200_ERR_CUDA;
    }
    return launch_status();
}

// x: float32 [rows][d]; xsplit: scratch of 2 * rows * d bf16; part_*: [rows][lmhead_mma_parts(vocab)] or null.
int launch_lmhead_mma(const __nv_bfloat16* embed, const float* x, __nv_bfloat16* xsplit, int rows, int vocab, int d,
                      float* logits, float* part_val, int* part_idx, cudaStream_t st) {
    Lm5Params p;
    p.status = library_status_word();
    if (!p.status) return ROTOR_B200_ERR_CUDA;
    const size_t plane = (size_t)rows * d, n4 = plane / 4;
    x_split_kernel<<<(unsigned)((n4 + 255) / 256), 256, 0, st>>>(x, xsplit, n4, plane);
    int rc = launch_status();
    if (rc) return rc;
    p.vocab = vocab;
    p.d = d;
    p.rows = rows;
    p.logits = logits;
    p.part_val = part_val;
    p.part_idx = part_idx;
    // The token tile: all rows up to 128 in one pass over the table; a vocabulary of fewer shares than SMs takes narrower
    // tiles while the grid still fits one CTA to an SM (its table is small and comes from L2: 200 rows of 512 x 512 19.1 -> 9.1 us).
    int nt = rows <= 16 ? 16 : rows <= 32 ? 32 : rows <= 64 ? 64 : 128;
    while (nt > 16 && lmhead_mma_parts(vocab) * ((rows + nt / 2 - 1) / (nt / 2)) <= fused_sm_count()) nt /= 2;
    switch (nt) {
        case 16: return lm5_launch<16>(embed, xsplit, p, st);
        case 32: return lm5_launch<32>(embed, xsplit, p, st);
        case 64: return lm5_launch<64>(embed, xsplit, p, st);
    }
    return lm5_launch<128>(embed, xsplit, p, st);
}

}  // namespace rb
