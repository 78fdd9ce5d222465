// Ternary BitLinear integer core: acc[c][o] = sum_k xq[c][k] * w[o][k].
//
// HBM-bound: the kernel streams each 512-byte weight tile exactly once with one
// 128-bit load per lane, stages the int8 activation columns in shared memory with a
// bulk (TMA) copy, and decodes in registers with one AND per operand word:
// (word & (0x03030303 << 2j)) is the int8x4 vector 4^j * (w+1).  Partial sums are
// kept per bit-pair j and rescaled exactly (arithmetic shift) at the end; the "+1"
// of the code is removed by subtracting sum_k xq[c][k] (xsum).
//
// Two instruction mixes share the layout:
//   DP4A : dp4a.u32.s32 lanes, up to 4 columns a launch (decode work is per weight,
//          multiply work per weight per column);
//   MMA  : mma.sync m16n8k32 u8 x s8 -> s32; the tile IS the A fragment, 8 columns
//          at the cost of one, which also carries the residual terms of the
//          multi-term activation quantiser; up to 40 columns a launch.
#include "gemv_core.cuh"
#include "leanstage.cuh"
#include "model.cuh"

namespace rb {

// Activation columns are staged into shared memory with bulk async (TMA) copies that
// signal an mbarrier.  stage_init() may run before the producer of xq has finished;
// stage_issue() must run after it; stage_wait() spins with a bound and returns false
// when it gave up (the caller records it; results are then undefined but every access
// stays in bounds).
__device__ __forceinline__ void stage_init(uint64_t* bar) {
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)));
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
}

__device__ __forceinline__ void stage_issue(uint64_t* bar, int8_t* xs, int xs_stride, const int8_t* src,
                                            size_t src_stride, int ncols, uint32_t bytes) {
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                     "r"(bytes * (uint32_t)ncols)
                     : "memory");
        for (int c = 0; c < ncols; ++c)
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                    smem_u32(xs + (size_t)c * xs_stride)),
                "l"(src + (size_t)c * src_stride), "r"(bytes), "r"(smem_u32(bar))
                : "memory");
    }
}

// Call after a __syncthreads() that follows stage_issue.
__device__ __forceinline__ bool stage_wait(uint64_t* bar) {
    uint32_t ok = 0;
    const long long start = clock64();
    // bounded: gives up after ~2e8 SM cycles (about 0.1 s) instead of waiting for ever
    while (!ok) {
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0; selp.u32 %0, 1, 0, p; }"
            : "=r"(ok)
            : "r"(smem_u32(bar))
            : "memory");
        if (!ok && clock64() - start > 200000000LL) break;
    }
    return ok != 0;
}

// Sums that the product adds to are cleared by the quantiser, a share per row, so that no memset stands between the two, up to
// this many bytes a row: 8192 -> 28672, 8 rows (115 KB) 27.1 / 27.5 us, 5 rows of two terms (229 KB) 43.4 / 41.9, of three
// (344 KB) 56.8 / 53.1.  The product starts early where it is one launch (4096 -> 11008, 8 rows: 10.6 against 12.6 us).
constexpr size_t LINEAR_CLEAR_MAX = 128 * 1024;
constexpr int ACC_MMA_COLS = 40;   // columns of one launch of the MMA variant
// Columns up to which the MMA variant is faster than the tiled tensor-core kernel, which takes the same time for any number up to
// 128 but sixteen rows at a time reads its columns over and over in a large matrix.  us, MMA variant / tiled: 2560 x 2560 40 columns 6.5 /
// 12.5, 48 9.1 / 14.1; 13824 x 2560 40 14.1 / 17.7, 48 21.9 / 20.1; 2560 x 6912 40 12.4 / 15.7, 48 19.0 / 16.9; 8192 x 8192 24 15.9 /
// 17, 32 25.9 / 17.4; 10240 x 8192 24 18.5 / 20, 32 29.0 / 20.7; 8192 x 28672 16 30.4 / 34, 24 43.4 / 34; 57344 x 8192 16 56.1 / 62,
// 24 77.5 / 62.
static int acc_most_cols(size_t out, size_t in) {
    const size_t weights = out * in;
    return weights <= ((size_t)48 << 20) ? ACC_MMA_COLS : weights <= ((size_t)128 << 20) ? 24 : ACC_FEW_COLS;
}
// Whether a product takes the tiled kernels.
static bool takes_tiles(size_t out, size_t in, size_t ncols, int variant) {
    return variant == ROTOR_B200_VARIANT_AUTO && ncols > (size_t)acc_most_cols(out, in);
}
constexpr size_t LINEAR_FUSED_ROWS = 4, LINEAR_FUSED_COLS = 6;  // a stand-alone layer call in one launch: see its rule

struct AccParams {
    const uint4* tiles;
    const int8_t* xq;      // [ncols][kpad]
    const int32_t* xsum;   // [ncols]
    int32_t* acc;          // [ncols][out]
    unsigned* status;      // device word, set to ROTOR_B200_ERR_TIMEOUT on a staging timeout
    int out;
    int nkt;               // k-tiles per row of tiles
    int nrt;               // row tiles
    int row_tiles;         // row tiles of a CTA, one after the other against the same staged columns
    int kt_per_split;
    int ncols;
    int atomic;            // gridDim.y > 1: accumulate with integer atomics into zeroed acc
    size_t plane_stride;   // != 0: K split s stores its partial sums to acc + s*plane_stride instead
    // whole K ranges (one split): finished float rows [y_rows][out] instead of sums, y_terms columns each
    float* y;
    const float *y_sx, *y_scales;
    float y_scale;
    int y_rows, y_terms;
};

// NT: groups of eight columns of the MMA variant.  A weight word is loaded and masked once for all of them, so that more columns
// cost shared-memory reads and MMAs but no further pass over the matrix.  A step of the 2B shape (12 layers), a launch for every eight
// columns / one for all: 12 sequences 843 / 734 us, 16 876 / 750, 24 1090 / 921; three terms 5 sequences 952 / 829, 8 1132 / 940.
// FORM: what a launch needs is compiled for it alone (2B step of two sequences, 12 layers, 579 us; with the loop of ACC_MANY compiled
// into it 623, with the finished rows 585; two groups: 96 registers let five CTAs share an SM, at 99 only four, and a step of 16
// sequences took 759 instead of 744).
enum { ACC_ONE = 0, ACC_MANY = 1, ACC_FINISH = 2 };  // one row tile a CTA; several (acc_row_tiles); one, finished rows
template <int WARPS, int UMAX, bool USE_MMA, int NCOL, int NT, int FORM>
__global__ void __launch_bounds__(WARPS * 32, NT == 2 && FORM == ACC_ONE ? 5 : 0) bitlinear_acc_kernel(const __grid_constant__ AccParams p) {
    constexpr bool MANY = FORM == ACC_MANY;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int rt0 = MANY ? blockIdx.x * p.row_tiles : blockIdx.x, rt1 = MANY ? min(p.nrt, rt0 + p.row_tiles) : rt0 + 1;
    const int kt0 = blockIdx.y * p.kt_per_split;
    const int kt1 = min(p.nkt, kt0 + p.kt_per_split);
    const int ks = (kt1 - kt0) * TILE_K;
    const int xs_stride = p.kt_per_split * TILE_K + XS_PAD;
    const int kbase = kt0 * TILE_K;

    uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw);
    int* red = reinterpret_cast<int*>(smem_raw + 16);            // [WARPS][NT][128]; MANY: two of them, in turn
    int8_t* xs = reinterpret_cast<int8_t*>(smem_raw + 16 + (MANY ? 2 : 1) * WARPS * NT * 128 * 4);

    stage_init(bar);

    const uint4* trow = p.tiles + ((size_t)rt0 * p.nkt) * 32 + lane;
    // The first batch of a row tile's weights: of the CTA's first one before the activations are waited for, of the others
    // before the sums of the one before are put together.
    uint4 wv[UMAX];
    auto first = [&]() {
        const int base = kt0 + warp;
#pragma unroll
        for (int u = 0; u < UMAX; ++u)
            if (base + u * WARPS < kt1) wv[u] = ld_stream_v4(trow + (size_t)(base + u * WARPS) * 32);
    };
    first();
    pdl_wait();     // weights above are constants; everything below depends on the producer kernel
    pdl_trigger();  // after the wait: see the rule in common.cuh
    stage_issue(bar, xs, xs_stride, p.xq + (size_t)kt0 * TILE_K, (size_t)p.nkt * TILE_K, p.ncols, (uint32_t)ks);
    __syncthreads();  // mbarrier initialised, bulk copies issued
    if (!stage_wait(bar) && threadIdx.x == 0) atomicMax(p.status, (unsigned)ROTOR_B200_ERR_TIMEOUT);

    int rt = rt0;
    do {
        int accm[NT][4][4];      // MMA: [bit pair j][fragment register]
        int accd[2][4][NCOL];    // DP4A: [row half][bit pair j][column]
#pragma unroll
        for (int j = 0; j < 4; ++j) {
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int r = 0; r < 4; ++r) accm[n][j][r] = 0;
#pragma unroll
            for (int c = 0; c < NCOL; ++c) accd[0][j][c] = accd[1][j][c] = 0;
        }
        int base = kt0 + warp;
        while (base < kt1) {
#pragma unroll
            for (int u = 0; u < UMAX; ++u) {
                const int kt = base + u * WARPS;
                if (kt < kt1) {
                    const uint32_t pw[4] = {wv[u].x, wv[u].y, wv[u].z, wv[u].w};
                    const int koff = kt * TILE_K - kbase + 32 * t;
#pragma unroll
                    for (int n = 0; n < NT; ++n)
                        tile_mac<USE_MMA, NCOL>(pw, xs + (size_t)8 * n * xs_stride, xs_stride, koff, g, p.ncols - 8 * n, accm[n], accd);
                }
            }
            base += UMAX * WARPS;
#pragma unroll
            for (int u = 0; u < UMAX; ++u)
                if (base + u * WARPS < kt1) wv[u] = ld_stream_v4(trow + (size_t)(base + u * WARPS) * 32);
        }
        if (MANY && rt + 1 < rt1) {
            trow += (size_t)p.nkt * 32;
            first();
        }

        // exact rescale of the per-bit-pair partial sums, then reduce across the CTA
        int* cta_red = red + (MANY ? ((rt - rt0) & 1) * WARPS * NT * 128 : 0);
        int* myred = cta_red + warp * NT * 128;
        if constexpr (USE_MMA) {
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const int v = accm[n][0][r] + (accm[n][1][r] >> 2) + (accm[n][2][r] >> 4) + (accm[n][3][r] >> 6);
                    const int row_l = g + 8 * (r >> 1), col = 2 * t + (r & 1);
                    myred[n * 128 + row_l * 8 + col] = v;
                }
        } else {
#pragma unroll
            for (int rh = 0; rh < 2; ++rh)
#pragma unroll
                for (int c = 0; c < NCOL; ++c) {
                    int v = accd[rh][0][c] + (accd[rh][1][c] >> 2) + (accd[rh][2][c] >> 4) + (accd[rh][3][c] >> 6);
                    v += __shfl_xor_sync(0xffffffffu, v, 1);
                    v += __shfl_xor_sync(0xffffffffu, v, 2);
                    if (t == 0) myred[(g + 8 * rh) * 8 + c] = v;
                }
        }
        __syncthreads();  // (the other half is written next: whoever still reads this one has passed the barrier before that)
        if constexpr (FORM == ACC_FINISH) {  // whole sums: finished rows, rounded as dequant_kernel rounds
            for (int e = threadIdx.x; e < 16 * p.y_rows; e += WARPS * 32) {
                const int row_l = e & 15, m = e >> 4, row = rt * TILE_ROWS + row_l;
                if (row >= p.out) continue;
                float v = 0.f;
                for (int tt = 0; tt < p.y_terms; ++tt) {
                    const int col = m * p.y_terms + tt;
                    int s = -__ldcg(p.xsum + col);
#pragma unroll
                    for (int w = 0; w < WARPS; ++w) s += cta_red[(w * NT + (col >> 3)) * 128 + row_l * 8 + (col & 7)];
                    v = __fadd_rn(v, __fmul_rn((float)s, __ldcg(p.y_sx + col)));
                }
                p.y[(size_t)m * p.out + row] = __fmul_rn(v, p.y_scales ? __ldg(p.y_scales + row) : p.y_scale);
            }
        } else
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            for (int e = threadIdx.x; e < 128; e += WARPS * 32) {
                // several groups: a warp's sums of one column lie in consecutive rows (a quarter of a line an instruction)
                const int row_l = NT > 1 ? e & 15 : e >> 3, col_l = NT > 1 ? e >> 4 : e & 7, col = 8 * n + col_l;
                const int row = rt * TILE_ROWS + row_l;
                if (col < p.ncols && row < p.out) {
                    int s = 0;
#pragma unroll
                    for (int w = 0; w < WARPS; ++w) s += cta_red[(w * NT + n) * 128 + row_l * 8 + col_l];
                    if (blockIdx.y == 0) s -= p.xsum[col];
                    int32_t* dst = p.acc + (size_t)blockIdx.y * p.plane_stride + (size_t)col * p.out + row;
                    if (p.atomic)
                        atomicAdd(dst, s);
                    else
                        *dst = s;
                }
            }
        }
    } while (MANY && ++rt < rt1);
}

// Row tiles of a CTA.  One after the other against the same staged columns: a CTA a row tile copies the columns of its K
// range for every 16 rows, which from two groups of eight on is more than the weights.  Kept small enough that the grid covers
// the GPU.  us with 1 / 2 / 4 row tiles: 8 columns 57344 x 8192 36.4 / 35.0 / 36.1; 16 columns 8192 x 8192 14.1 / 12.2 / 11.8, 57344 x 8192
// 71.7 / 60.4 / 56.1; 24 columns 2560 x 6912 8.7 / 7.1 / 9.4, 57344 x 8192 107.9 / 85.3 / 77.5; 40 columns 13824 x 2560 19.7 / 15.9 / 14.1.
static int acc_row_tiles(int nrt, int ksplit, int groups) {
    if (groups == 1) return 1;
    const int least = groups == 2 ? 1000 : 240;  // CTAs left
    int r = 1;
    while (r < 4 && nrt * ksplit >= 2 * r * least) r *= 2;
    return r;
}

__global__ void dequant_kernel(const int32_t* acc, const float* sx, int m, int terms,
                               int out, float wscale, const float* wscale_vec,
                               float* y) {
    pdl_wait();
    const size_t total = (size_t)m * out;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int r = (int)(i / out), o = (int)(i % out);
        float v = 0.f;
        for (int tt = 0; tt < terms; ++tt)
            v = __fadd_rn(v, __fmul_rn((float)__ldcg(acc + ((size_t)r * terms + tt) * out + o), __ldcg(sx + r * terms + tt)));
        y[i] = __fmul_rn(v, wscale_vec ? __ldg(wscale_vec + o) : wscale);
    }
}

template <int WARPS, int UMAX, bool USE_MMA, int NCOL, int NT, int FORM>
static int launch_acc_kind(const AccParams& p, int nrt, int ksplit, cudaStream_t st) {
    constexpr bool MANY = FORM == ACC_MANY;
    auto kern = bitlinear_acc_kernel<WARPS, UMAX, USE_MMA, NCOL, NT, FORM>;
    const size_t smem = 16 + (MANY ? 2 : 1) * WARPS * NT * 128 * 4 + (size_t)p.ncols * (p.kt_per_split * TILE_K + XS_PAD);
    if (smem > 200 * 1024) return ROTOR_B200_ERR_SHAPE;
    if (smem > 48 * 1024) {
        static PerDevice<size_t> once;  // per instantiation and device
        size_t& configured = once.here();
        if (smem > configured) {
            RB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
            configured = 200 * 1024;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(MANY ? (nrt + p.row_tiles - 1) / p.row_tiles : nrt, ksplit);
    cfg.blockDim = dim3(WARPS * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_use_pdl ? 1 : 0;
    if (cudaLaunchKernelEx(&cfg, kern, p) != cudaSuccess) {
        ++g_launch_count;
        return ROTOR_B200_ERR_CUDA;
    }
    return launch_status();
}

template <int WARPS, int UMAX, bool USE_MMA, int NCOL, int NT = 1>
static int launch_acc(const AccParams& pin, int nrt, int ksplit, cudaStream_t st) {
    AccParams p = pin;
    p.nrt = nrt;
    if constexpr (USE_MMA) {
        if (p.y) return launch_acc_kind<WARPS, UMAX, USE_MMA, NCOL, NT, ACC_FINISH>(p, nrt, ksplit, st);
    }
    p.row_tiles = acc_row_tiles(nrt, ksplit, NT);
    if constexpr (NT > 1) {
        if (p.row_tiles > 1) return launch_acc_kind<WARPS, UMAX, USE_MMA, NCOL, NT, ACC_MANY>(p, nrt, ksplit, st);
    }
    return launch_acc_kind<WARPS, UMAX, USE_MMA, NCOL, NT, ACC_ONE>(p, nrt, ksplit, st);
}

// Split the K range over gridDim.y so that the grid covers the GPU a few times and
// the staged activations stay below ~64 KB per CTA.
static int choose_ksplit(int nrt, int nkt, int ncols, int warps) {
    int ks = 1;
    while (ks < nkt) {
        const int per = (nkt + ks - 1) / ks;
        const bool enough_ctas = (long)nrt * ks >= 2 * 148;
        const bool smem_ok = (size_t)ncols * (per * TILE_K + XS_PAD) <= 64 * 1024;
        const bool too_thin = per / 2 < warps;  // keep at least one tile per warp after doubling
        if (smem_ok && (enough_ctas || too_thin)) break;
        ks *= 2;
    }
    return ks > nkt ? nkt : ks;
}

static int dispatch_acc(const AccParams& p, int nrt, int ksplit, int variant, cudaStream_t st) {
    constexpr int WARPS = 4, UMAX = 8;
    if (variant == ROTOR_B200_VARIANT_MMA) {
        switch ((p.ncols + 7) / 8) {
            case 1: return launch_acc<WARPS, UMAX, true, 1>(p, nrt, ksplit, st);
            case 2: return launch_acc<WARPS, UMAX, true, 1, 2>(p, nrt, ksplit, st);
            case 3: return launch_acc<WARPS, UMAX, true, 1, 3>(p, nrt, ksplit, st);
            case 4: return launch_acc<WARPS, UMAX, true, 1, 4>(p, nrt, ksplit, st);
            case 5: return launch_acc<WARPS, UMAX, true, 1, 5>(p, nrt, ksplit, st);
        }
        return ROTOR_B200_ERR_ARG;
    }
    switch (p.ncols) {
        case 1: return launch_acc<WARPS, UMAX, false, 1>(p, nrt, ksplit, st);
        case 2: return launch_acc<WARPS, UMAX, false, 2>(p, nrt, ksplit, st);
        case 3: return launch_acc<WARPS, UMAX, false, 3>(p, nrt, ksplit, st);
        case 4: return launch_acc<WARPS, UMAX, false, 4>(p, nrt, ksplit, st);
    }
    return ROTOR_B200_ERR_ARG;
}

template <bool USE_MMA, int NCOL, int NT = 1, int FORM = ACC_ONE>
static int configure_one() {
    RB_CUDA(cudaFuncSetAttribute(bitlinear_acc_kernel<4, 8, USE_MMA, NCOL, NT, FORM>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    if constexpr (FORM == ACC_ONE && USE_MMA) {
        if (int rc = configure_one<USE_MMA, NCOL, NT, ACC_FINISH>()) return rc;
        if constexpr (NT > 1) return configure_one<USE_MMA, NCOL, NT, ACC_MANY>();
    }
    return ROTOR_B200_OK;
}

// Done once, outside any stream capture: status word and the shared-memory opt-ins.
int configure_gemv_kernels() {
    int rc = (library_status_word() ? ROTOR_B200_OK : ROTOR_B200_ERR_CUDA);
    if (rc) return rc;
    if ((rc = configure_one<true, 1>()) || (rc = configure_one<true, 1, 2>()) || (rc = configure_one<true, 1, 3>()) ||
        (rc = configure_one<true, 1, 4>()) || (rc = configure_one<true, 1, 5>()))
        return rc;
    if ((rc = configure_one<false, 1>())) return rc;
    if ((rc = configure_one<false, 2>())) return rc;
    if ((rc = configure_one<false, 3>())) return rc;
    return configure_one<false, 4>();
}

static int pick_variant(int variant, int ncols) {
    if (variant != ROTOR_B200_VARIANT_AUTO) return variant;
    return ncols <= 2 ? ROTOR_B200_VARIANT_DP4A : ROTOR_B200_VARIANT_MMA;
}

GemvPlan plan_gemv(size_t out, size_t in, int ncols) {
    const int nkt = (int)(kpad_of(in) / TILE_K), nrt = (int)(opad_of(out) / TILE_ROWS);
    const int per_pass = ncols < ACC_MMA_COLS ? ncols : ACC_MMA_COLS;
    int ks = choose_ksplit(nrt, nkt, per_pass, 4);
    GemvPlan g;
    g.kt_per_split = (nkt + ks - 1) / ks;
    g.ksplit = (nkt + g.kt_per_split - 1) / g.kt_per_split;
    return g;
}

bool gemv_adds(size_t out, size_t in, int ncols, const void* xq, int variant) {
    if (takes_tiles(out, in, ncols, variant))
        return gemm_tcgen05_supported(out, in, ncols, xq) && gemm_tcgen05_splits(out, in, ncols) >= 2;
    return plan_gemv(out, in, ncols).ksplit > 1;
}

int launch_gemv_planes(const void* tiles, size_t out, size_t in, const int8_t* xq, const int32_t* xsum, int ncols,
                       int32_t* acc, size_t plane_stride, const GemvPlan& plan, int variant, cudaStream_t st, bool zeroed) {
    int rc = (library_status_word() ? ROTOR_B200_OK : ROTOR_B200_ERR_CUDA);
    if (rc) return rc;
    if (takes_tiles(out, in, ncols, variant)) {
        // compute-bound regime: the tiled GEMM writes complete sums into plane 0 (callers use one plane)
        if (gemm_tcgen05_supported(out, in, ncols, xq)) return launch_gemm_tcgen05(tiles, out, in, xq, xsum, ncols, acc, st, zeroed, true);
        return launch_gemm_mma(tiles, out, in, xq, xsum, ncols, acc, st);
    }
    const int nkt = (int)(kpad_of(in) / TILE_K), nrt = (int)(opad_of(out) / TILE_ROWS);
    const size_t kpad = kpad_of(in);
    variant = pick_variant(variant, ncols);
    const int chunk = variant == ROTOR_B200_VARIANT_MMA ? ACC_MMA_COLS : 4;
    for (int c0 = 0; c0 < ncols; c0 += chunk) {
        AccParams p = {};
        p.tiles = (const uint4*)tiles;
        p.xq = xq + (size_t)c0 * kpad;
        p.xsum = xsum + c0;
        p.acc = acc + (size_t)c0 * out;
        p.status = library_status_word();
        p.out = (int)out;
        p.nkt = nkt;
        p.kt_per_split = plan.kt_per_split;
        p.ncols = (ncols - c0) < chunk ? (ncols - c0) : chunk;
        // plane_stride 0 with a split K range: the splits add into one zeroed plane (exact in any order)
        p.atomic = plane_stride == 0 && plan.ksplit > 1;
        p.plane_stride = plane_stride;
        if (p.atomic && !zeroed) RB_CUDA(cudaMemsetAsync(p.acc, 0, (size_t)p.ncols * out * sizeof(int32_t), st));
        rc = dispatch_acc(p, nrt, plan.ksplit, variant, st);
        if (rc) return rc;
    }
    return ROTOR_B200_OK;
}

// Whether a product can finish its rows itself: one launch of whole K ranges, where the matrix has enough row tiles and few
// enough K tiles for that (else the K range is split and the sums are put together in memory).  The staged columns have to leave an SM
// room for three CTAs, or, where one round of two an SM takes all row tiles, for two.  us of a layer call, sums in memory / finished:
// 1000 x 1000 5-40 columns 10.5 / 8.2-9; 2560 x 2560 8 10.7 / 8.1, 32 11.4 / 10.7; 13824 x 2560 8 12.5 / 8.9, 17 14.8 / 14.7, 24 14.8 /
// 16.2; 4096 x 4096 16 10.9 / 8.7, 20 12.5 / 10.7; 6144 x 4096 16 13.5 / 10.4, 20 12.7 / 16.6; 16384 x 4096 13 20.4 / 18.6, 17 20.9 /
// 23.0, 20 20.9 / 27.0; 22016 x 4096 16 23.0 / 20.9, 20 27.1 / 32.9; 2560 x 6912 9 10.9 / 10.7, 17 12.7 / 18.8; 8192 x 8192 6 13.0 /
// 12.2, 8 14.0 / 14.5, 16 18.6 / 26.8; 4096 x 11008 6 16.8 / 14.5, 12 18.9 / 21.7.
bool acc_finish_supported(size_t out, size_t in, size_t ncols, int variant) {
    if (variant != ROTOR_B200_VARIANT_AUTO || out >= (1u << 30) || in > 49152 || ncols < 3 || ncols > (size_t)ACC_MMA_COLS || takes_tiles(out, in, ncols, variant))
        return false;
    const int nkt = (int)(kpad_of(in) / TILE_K), nrt = (int)(opad_of(out) / TILE_ROWS);
    const size_t staged = ncols * (nkt * TILE_K + XS_PAD);  // (16 columns of 6912 leave one CTA an SM: feed-forward of 16 rows 22.2 -> 23.0 us)
    const size_t most = nkt > 32 ? 64 : nrt <= 2 * fused_sm_count() ? 96 : 68;  // KB
    return choose_ksplit(nrt, nkt, (int)ncols, 4) == 1 || (nrt >= 128 && nkt <= 64 && staged <= most * 1024);
}

// y[rows][out] from quantised rows of `terms` columns each.
int launch_acc_finish(const void* tiles, size_t out, size_t in, const int8_t* xq, const float* sx, const int32_t* xsum, int rows, int terms,
                      float wscale, const float* wscale_vec, float* y, cudaStream_t st) {
    AccParams p = {};
    p.tiles = (const uint4*)tiles;
    p.xq = xq;
    p.xsum = xsum;
    p.status = library_status_word();
    if (!p.status) return ROTOR_B200_ERR_CUDA;
    p.out = (int)out;
    p.nkt = p.kt_per_split = (int)(kpad_of(in) / TILE_K);
    p.ncols = rows * terms;
    p.y = y;
    p.y_sx = sx;
    p.y_scales = wscale_vec;
    p.y_scale = wscale;
    p.y_rows = rows;
    p.y_terms = terms;
    return dispatch_acc(p, (int)(opad_of(out) / TILE_ROWS), 1, ROTOR_B200_VARIANT_MMA, st);
}

}  // namespace rb

using namespace rb;

// dependent: the kernel before is this call's own (its weights are older).
static int run_acc(const void* tiles, size_t out, size_t in, const int8_t* xq, const int32_t* xsum, size_t ncols,
                   int32_t* acc, int variant, cudaStream_t st, bool zeroed, bool dependent) {
    RB_REQUIRE(tiles && xq && xsum && acc && out > 0 && in > 0 && ncols > 0);
    RB_REQUIRE(out < (1u << 30) && in < (1u << 30));
    RB_REQUIRE(((uintptr_t)tiles & 15) == 0 && ((uintptr_t)xq & 15) == 0);
    RB_REQUIRE(variant >= ROTOR_B200_VARIANT_AUTO && variant <= ROTOR_B200_VARIANT_MMA);
    int rc = (library_status_word() ? ROTOR_B200_OK : ROTOR_B200_ERR_CUDA);
    if (rc) return rc;
    const int nkt = (int)(kpad_of(in) / TILE_K), nrt = (int)(opad_of(out) / TILE_ROWS);
    const size_t kpad = kpad_of(in);
    if (takes_tiles(out, in, ncols, variant)) {
        if (gemm_tcgen05_supported(out, in, (int)ncols, xq))
            return launch_gemm_tcgen05(tiles, out, in, xq, xsum, (int)ncols, acc, st, zeroed, dependent);
        return launch_gemm_mma(tiles, out, in, xq, xsum, (int)ncols, acc, st);
    }
    // small matrices, up to eight columns: the staged kernel (every CTA's share of the tiles sits in shared
    // memory before the activations are needed, which a chain of dependent launches can overlap)
    if (ncols <= 8 && staged_acc_supported(out, in, (int)ncols, variant))
        return launch_staged_acc(tiles, out, in, xq, xsum, (int)ncols, acc, variant, st);
    variant = pick_variant(variant, (int)(ncols < 8 ? ncols : 8));
    const size_t chunk = variant == ROTOR_B200_VARIANT_MMA ? ACC_MMA_COLS : 4;
    for (size_t c0 = 0; c0 < ncols; c0 += chunk) {
        const int nc = (int)((ncols - c0) < chunk ? (ncols - c0) : chunk);
        const int ksplit = choose_ksplit(nrt, nkt, nc, 4);
        AccParams p = {};
        p.tiles = (const uint4*)tiles;
        p.xq = xq + c0 * kpad;
        p.xsum = xsum + c0;
        p.acc = acc + c0 * out;
        p.status = library_status_word();
        p.out = (int)out;
        p.nkt = nkt;
        p.kt_per_split = (nkt + ksplit - 1) / ksplit;
        p.ncols = nc;
        const int ksplit_eff = (nkt + p.kt_per_split - 1) / p.kt_per_split;
        p.atomic = ksplit_eff > 1;
        p.plane_stride = 0;
        if (p.atomic && !zeroed) RB_CUDA(cudaMemsetAsync(p.acc, 0, (size_t)nc * out * sizeof(int32_t), st));
        rc = dispatch_acc(p, nrt, ksplit_eff, variant, st);
        if (rc) return rc;
    }
    return ROTOR_B200_OK;
}

// Whether run_acc adds to acc for any of its column chunks (it then clears acc first unless it is told `zeroed`).
static bool acc_adds(size_t out, size_t in, size_t ncols, const int8_t* xq, int variant) {
    if (takes_tiles(out, in, ncols, variant))
        return gemm_tcgen05_supported(out, in, (int)ncols, xq) && gemm_tcgen05_splits(out, in, (int)ncols) >= 2;
    if (ncols <= 8 && staged_acc_supported(out, in, (int)ncols, variant)) return false;
    const size_t chunk = pick_variant(variant, (int)(ncols < 8 ? ncols : 8)) == ROTOR_B200_VARIANT_MMA ? ACC_MMA_COLS : 4;
    const int nkt = (int)(kpad_of(in) / TILE_K), nrt = (int)(opad_of(out) / TILE_ROWS), rest = (int)(ncols % chunk);
    return (ncols >= chunk && choose_ksplit(nrt, nkt, (int)chunk, 4) > 1) || (rest && choose_ksplit(nrt, nkt, rest, 4) > 1);
}

extern "C" {

int rotor_b200_bitlinear_acc(const void* tiles, size_t out, size_t in, const int8_t* xq, const int32_t* xsum,
                             size_t ncols, int32_t* acc, int variant, void* stream) {
    return run_acc(tiles, out, in, xq, xsum, ncols, acc, variant, as_stream(stream), false, false);
}

int rotor_b200_bitlinear_dequant(const int32_t* acc, const float* sx, size_t m, int terms, size_t out,
                                 float wscale, const float* wscale_vec, float* y, void* stream) {
    RB_REQUIRE(acc && sx && y && m > 0 && out > 0 && terms >= 1 && terms <= 4);
    const size_t total = m * out;
    unsigned grid = (unsigned)((total + 255) / 256);
    if (grid > 148 * 16) grid = 148 * 16;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(256);
    cfg.stream = as_stream(stream);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_use_pdl ? 1 : 0;
    if (cudaLaunchKernelEx(&cfg, dequant_kernel, acc, sx, (int)m, terms, (int)out, wscale, wscale_vec, y) != cudaSuccess) {
        ++g_launch_count;
        return ROTOR_B200_ERR_CUDA;
    }
    return launch_status();
}

static inline size_t al256(size_t v) { return (v + 255) & ~(size_t)255; }

size_t rotor_b200_bitlinear_workspace_bytes(size_t out, size_t in, size_t m, int terms) {
    const size_t nc = m * (size_t)terms;
    return al256(nc * kpad_of(in)) + al256(nc * 4) + al256(nc * 4) + al256(nc * out * 4);
}

int rotor_b200_bitlinear_forward(const void* tiles, size_t out, size_t in, const float* x, size_t m, int terms,
                                 float wscale, const float* wscale_vec, float* y, void* workspace,
                                 size_t workspace_bytes, int variant, void* stream) {
    RB_REQUIRE(tiles && x && y && workspace && m > 0 && out > 0 && in > 0 && terms >= 1 && terms <= 4);
    RB_REQUIRE(((uintptr_t)workspace & 255) == 0);
    if (workspace_bytes < rotor_b200_bitlinear_workspace_bytes(out, in, m, terms)) return ROTOR_B200_ERR_WORKSPACE;
    const size_t nc = m * (size_t)terms;
    // A few rows: one launch, the rows are quantised in the product's prologue by every CTA (a row and term costs each about
    // a microsecond, the two launches saved cost four) and leave it as floats.  Every CTA reads x, so y must not lie on it.
    // On the GPU, one launch against three: 1 row of 2560 -> 6912 4.5 / 8.3 us, 4 rows 8.5 / 8.5, 2 rows of three terms
    // 9.9 / 12.2, 3 of two 9.9 / 9.9, 4 of two 12.6 / 11.3; 8192 -> 8192 8.0 / 12.2, 14.4 / 13.7, 16.6 / 19.3, 16.7 / 16.7,
    // 19.8 / 17.6.  Up to six columns the two are within 5 % at worst and the host saves two launches (25.8 -> 19.4 us a call).
    const uintptr_t x0 = (uintptr_t)x, x1 = x0 + m * in * sizeof(float), y0 = (uintptr_t)y, y1 = y0 + m * out * sizeof(float);
    if (variant == ROTOR_B200_VARIANT_AUTO && !wscale_vec && m <= LINEAR_FUSED_ROWS && nc <= LINEAR_FUSED_COLS && (x0 & 15) == 0 &&
        ((uintptr_t)tiles & 15) == 0 && out < (1u << 30) && in <= 49152 && (y1 <= x0 || x1 <= y0) &&
        fused_gemv_supported(out, in, (int)m, terms, 1, 0)) {
        LeanStage stage = {};
        stage.mode = LM_PLAIN;
        stage.n = (int)in;
        stage.y = x;
        stage.terms = terms;
        stage.kpad = (int)kpad_of(in);
        const float scale[3] = {wscale, wscale, wscale};
        return launch_fused_gemv(tiles, out, in, 1, (int)m, stage, y, scale, (int)out, (int)out, 0, as_stream(stream), nullptr, true);
    }
    unsigned char* w = (unsigned char*)workspace;
    int8_t* xq = (int8_t*)w;
    w += al256(nc * kpad_of(in));
    float* sx = (float*)w;
    w += al256(nc * 4);
    int32_t* xsum = (int32_t*)w;
    w += al256(nc * 4);
    int32_t* acc = (int32_t*)w;
    if (((uintptr_t)tiles & 15) == 0 && acc_finish_supported(out, in, nc, variant)) {
        // the product leaves finished rows: no sums to clear before it, no launch behind it (13 rows of 1923 -> 3001, three terms:
        // 14.3 us a call with both, 12.2 so)
        const int rc = launch_quantize_rows(x, m, in, terms, xq, sx, xsum, nullptr, 0, true, as_stream(stream));
        return rc ? rc : launch_acc_finish(tiles, out, in, xq, sx, xsum, (int)m, terms, wscale, wscale_vec, y, as_stream(stream));
    }
    const bool adds = out < (1u << 30) && in <= 49152 && nc * out * sizeof(int32_t) <= m * LINEAR_CLEAR_MAX && acc_adds(out, in, nc, xq, variant);
    int rc = launch_quantize_rows(x, m, in, terms, xq, sx, xsum, adds ? acc : nullptr, adds ? nc * out : 0, !takes_tiles(out, in, nc, variant), as_stream(stream));
    if (rc) return rc;
    rc = run_acc(tiles, out, in, xq, xsum, nc, acc, variant, as_stream(stream), adds, true);
    if (rc) return rc;
    return rotor_b200_bitlinear_dequant(acc, sx, m, terms, out, wscale, wscale_vec, y, stream);
}

/* ---------------------------------------------------------------------------------------
 * Allocation-free layer forward.
 *
 * rotor_b200_bitlinear_forward needs a caller-provided workspace, and the accumulate step
 * behind it creates a small device status word with cudaMalloc on first use.  Some hosts
 * cannot do either: a plug-in driven through the reference's backend call
 * (ternary_matmul(packed, scales, input_vec, in_dim, out_dim) has no workspace argument),
 * or a serving loop that has already handed every remaining byte of device memory to its
 * own pool, where cudaMalloc would fail -- and, when it succeeds, stalls all streams of the
 * device while it runs.  For them the scratch lives in a fixed array inside the library:
 * ROTOR_B200_STATIC_SCRATCH_BYTES per GPU, resident from library load to process exit on
 * every GPU that loads the library.
 *
 * Rules of use
 *  - Problems whose scratch need exceeds the array are refused with ROTOR_B200_ERR_TOO_LARGE;
 *    nothing is launched.  rotor_b200_bitlinear_static_fits() answers the question up front.
 *  - The first call on each device looks up the array's device address
 *    (cudaGetSymbolAddress).  Make that first call before starting any stream capture.
 *  - All calls on one GPU share the array, and it keeps the previous call's contents; the
 *    entry point clears what has to start at zero.  Two calls that overlap on the GPU
 *    (different streams, no ordering between them) race on the array: serialise them.
 *  - No cudaMalloc, cudaFree or other allocating routine is called on this path. */
static __device__ __align__(256) unsigned char g_static_scratch[ROTOR_B200_STATIC_SCRATCH_BYTES];

static PerDevice<unsigned char*> g_static_addr;  // device address of the array, once looked up on that device

static int static_scratch_address(unsigned char** out) {
    int dev = -1;
    RB_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= RB_MAX_DEVICES) return ROTOR_B200_ERR_ARG;
    unsigned char*& addr = g_static_addr.v[dev];
    if (!addr) {
        // g_static_scratch names the array in device code only; host code must ask for its address
        void* p = nullptr;
        RB_CUDA(cudaGetSymbolAddress(&p, g_static_scratch));
        addr = static_cast<unsigned char*>(p);
        g_extra_status.v[dev] = reinterpret_cast<unsigned*>(addr);  // (its status word is at the start)
    }
    *out = addr;
    return ROTOR_B200_OK;
}

static size_t static_need(size_t out, size_t in, size_t m, int terms) {
    return 256 + rotor_b200_bitlinear_workspace_bytes(out, in, m, terms);  // status word + stage buffers
}

int rotor_b200_bitlinear_static_fits(size_t out, size_t in, size_t m, int terms) {
    if (out == 0 || in == 0 || m == 0 || terms < 1 || terms > 4) return 0;
    return static_need(out, in, m, terms) <= ROTOR_B200_STATIC_SCRATCH_BYTES;
}

int rotor_b200_bitlinear_forward_static(const void* tiles, size_t out, size_t in, const float* x, size_t m,
                                        int terms, float wscale, const float* wscale_vec, float* y, int variant,
                                        void* stream) {
    RB_REQUIRE(tiles && x && y && m > 0 && out > 0 && in > 0 && terms >= 1 && terms <= 4);
    RB_REQUIRE(out < (1u << 30) && in < (1u << 30));
    RB_REQUIRE(((uintptr_t)tiles & 15) == 0);
    RB_REQUIRE(variant >= ROTOR_B200_VARIANT_AUTO && variant <= ROTOR_B200_VARIANT_MMA);
    if (static_need(out, in, m, terms) > ROTOR_B200_STATIC_SCRATCH_BYTES) return ROTOR_B200_ERR_TOO_LARGE;
    unsigned char* base = nullptr;
    int rc = static_scratch_address(&base);
    if (rc) return rc;
    cudaStream_t st = as_stream(stream);
    // carve: [status word, 256 B][xq][sx][xsum][acc]
    unsigned* status = reinterpret_cast<unsigned*>(base);
    unsigned char* w = base + 256;
    const size_t nc = m * (size_t)terms, kpad = kpad_of(in);
    int8_t* xq = (int8_t*)w;
    w += al256(nc * kpad);
    float* sx = (float*)w;
    w += al256(nc * 4);
    int32_t* xsum = (int32_t*)w;
    w += al256(nc * 4);
    int32_t* acc = (int32_t*)w;
    // the status word starts at zero (the array is zero-initialised when the library is loaded) and is
    // cleared only by rotor_b200_device_status(), which reads it: a timed-out wait is never lost
    rc = rotor_b200_quantize_rows(x, m, in, terms, xq, sx, xsum, stream);
    if (rc) return rc;
    const int nkt = (int)(kpad / TILE_K), nrt = (int)(opad_of(out) / TILE_ROWS);
    variant = pick_variant(variant, (int)(nc < 8 ? nc : 8));
    const size_t chunk = variant == ROTOR_B200_VARIANT_MMA ? ACC_MMA_COLS : 4;
    for (size_t c0 = 0; c0 < nc; c0 += chunk) {
        const int ncols = (int)((nc - c0) < chunk ? (nc - c0) : chunk);
        const int ksplit = choose_ksplit(nrt, nkt, ncols, 4);
        AccParams p = {};
        p.tiles = (const uint4*)tiles;
        p.xq = xq + c0 * kpad;
        p.xsum = xsum + c0;
        p.acc = acc + c0 * out;
        p.status = status;
        p.out = (int)out;
        p.nkt = nkt;
        p.kt_per_split = (nkt + ksplit - 1) / ksplit;
        p.ncols = ncols;
        const int ksplit_eff = (nkt + p.kt_per_split - 1) / p.kt_per_split;
        p.atomic = ksplit_eff > 1;
        p.plane_stride = 0;
        // split-K partial sums are added into the accumulators: they must start at zero
        if (p.atomic) RB_CUDA(cudaMemsetAsync(p.acc, 0, (size_t)ncols * out * sizeof(int32_t), st));
        rc = dispatch_acc(p, nrt, ksplit_eff, variant, st);
        if (rc) return rc;
    }
    return rotor_b200_bitlinear_dequant(acc, sx, m, terms, out, wscale, wscale_vec, y, stream);
}

int rotor_b200_ternary_matmul_host(const void* tiles, const float* scales_host, const float* x_host, size_t in,
                                   size_t out, int terms, float* y_host) {
    RB_REQUIRE(tiles && scales_host && x_host && y_host && in > 0 && out > 0 && terms >= 1 && terms <= 4);
    // grow-only staging area owned by the library: this seam is synchronous and single-threaded
    static unsigned char* stage = nullptr;
    static size_t stage_bytes = 0;
    const size_t ws = rotor_b200_bitlinear_workspace_bytes(out, in, 1, terms);
    const size_t need = al256(in * 4) + 2 * al256(out * 4) + ws;
    if (need > stage_bytes) {
        if (stage) RB_CUDA(cudaFree(stage));
        stage = nullptr;
        stage_bytes = 0;
        RB_CUDA(cudaMalloc(&stage, need));
        stage_bytes = need;
    }
    float* dx = (float*)stage;
    float* dsc = (float*)(stage + al256(in * 4));
    float* dy = (float*)(stage + al256(in * 4) + al256(out * 4));
    void* dws = stage + al256(in * 4) + 2 * al256(out * 4);
    RB_CUDA(cudaMemcpy(dx, x_host, in * 4, cudaMemcpyHostToDevice));
    RB_CUDA(cudaMemcpy(dsc, scales_host, out * 4, cudaMemcpyHostToDevice));
    int rc = rotor_b200_bitlinear_forward(tiles, out, in, dx, 1, terms, 1.0f, dsc, dy, dws, ws,
                                          ROTOR_B200_VARIANT_AUTO, nullptr);
    if (rc) return rc;
    RB_CUDA(cudaMemcpy(y_host, dy, out * 4, cudaMemcpyDeviceToHost));
    return ROTOR_B200_OK;
}

}  // extern "C"
