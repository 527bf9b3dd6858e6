// f32 convolutions with stride 1 and up to 64 channels as six bf16 products on tcgen05 (the arithmetic of
// gemm_tcx.cuh: three planes per operand, sums of 64 k read out and added in registers, in the same order, so the bits are
// those of the gathered engine).
//
// One pass writes the source as channels-last planes inside its zero padding, [plane][image][y][x][Cp] with Cp = 16, 32 or
// 64 channels, a pixel being one row of 32, 64 or 128 bytes, and the filters as [plane][tap][n][Cp].  The source of a
// batch is then a matrix of rows, and the A operand of tap (fi, fj) is that of tap (0, 0) moved down fi * Wp + fj rows: a
// tile of 128 rows loads ONE box of 128 + (fh - 1) * Wp + fw - 1 rows per plane by TMA, and every tap's products start that
// many rows further on in it (as in conv_tc_halo.cu; the 32- and 64-byte swizzles too are functions of the absolute
// shared-memory address).  The filters of all taps stay in shared memory.  Rows that are no outputs, the right-hand columns
// and bottom rows of every image, are computed and dropped.
//
// The gathered engine fetches and splits every element once per tap (16 channels 3 x 3: 92 KB per tile from L1 and L2, and
// most of its instructions); here a tile's box is 19 KB and no thread touches an operand.  What bounds it: products of 32 to
// 128 columns, of which each takes some 45 cycles, and the pass ahead of it.
//
// Warps: 0 loads, 1 issues, 2 - 9 read accumulators, in two sets that take turns at tiles, each with two accumulators
// (leading block and corrections) of its own.
#include <cuda.h>

#include "conv_halo_f32.cuh"
#include "gemm_tcx.cuh"

namespace ag {
namespace halo32 {

using namespace ::ag::tc;

namespace {

constexpr int kWarps = 10, kThreads = kWarps * 32, kStages = 4, kBuffers = 4, kMostTaps = 25;
constexpr int kMarkWords = 128;          // a bit per epilogue warp and tile of a CTA
constexpr int kMostTiles = kMarkWords * 8;
constexpr int kControl = 256 + kMarkWords * 4 + 1024;

struct Params {
    int R, tiles;                        // rows of the framed source
    int hp, wp, oh, ow, n;
    int fh, fw, halo_rows, stages, groups;   // groups of 64 k
    FastDiv div_wp, div_image;
    const float *bias;
    int relu;
    float *y;
    int *status;
    // the operands as they were given (redo)
    const float *src, *w;
    int channels, h, wd, pad_h, pad_w;
    int64_t s_row, s_c;
    int reversed;
};

template <int RB>
__device__ __forceinline__ uint64_t operand(uint32_t addr) {
    constexpr uint64_t layout = RB == 32 ? 6ull : RB == 64 ? 4ull : 2ull;   // swizzle of 32, 64, 128 bytes
    uint64_t d = (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((8 * RB) >> 4) << 32;
    d |= 1ull << 46;
    return d | layout << 61;
}

__device__ __forceinline__ void load_box(uint32_t dst, const CUtensorMap *map, uint32_t bar, int row, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
            dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(0), "r"(row), "r"(z)
        : "memory");
}

// Output position of row q.
struct Position {
    int b, y, x;
    bool valid;
};
__device__ __forceinline__ Position position(const Params &p, int q) {
    uint32_t b, r, y, x;
    p.div_image.divmod((uint32_t)q, b, r);
    p.div_wp.divmod(r, y, x);
    return Position{(int)b, (int)y, (int)x, q < p.R && (int)y < p.oh && (int)x < p.ow};
}
__device__ __forceinline__ float finish(const Params &p, float v, float bias) {
    if (p.bias != nullptr) v = __fadd_rn(v, bias);
    return p.relu && !(v >= 0.f) ? 0.f : v;
}

// The marked blocks (32 positions), dealt to all warps eight columns at a time: FMAs over (tap, channel) in order.
__device__ __noinline__ void redo(const Params &p, const unsigned *marks) {
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, taps = p.fh * p.fw;
    int turn = 0;
    for (int tile = blockIdx.x, i = 0; tile < p.tiles; tile += gridDim.x, ++i)
        for (int quarter = 0; quarter < 4; ++quarter) {
            if (!(marks[i / 8] >> (i % 8 * 4 + quarter) & 1u)) continue;
            const Position at = position(p, tile * 128 + quarter * 32 + lane);
            for (int n0 = 0; n0 < p.n; n0 += 8) {
                if (turn++ % kWarps != warp || !at.valid) continue;
                float acc[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[j] = 0.f;
                for (int tap = 0; tap < taps; ++tap) {
                    const int sy = at.y + tap / p.fw - p.pad_h, sx = at.x + tap % p.fw - p.pad_w;
                    const bool in = sy >= 0 && sy < p.h && sx >= 0 && sx < p.wd;
                    const float *s = p.src + (int64_t)at.b * p.channels * p.h * p.wd + (in ? sy * p.wd + sx : 0);
                    const float *w = p.w + n0 * p.s_row + (p.reversed ? taps - 1 - tap : tap);
                    for (int c = 0; c < p.channels; ++c) {
                        const float v = in ? s[(int64_t)c * p.h * p.wd] : 0.f;
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            if (n0 + j < p.n) acc[j] = fmaf(v, w[j * p.s_row + c * p.s_c], acc[j]);
                    }
                }
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (n0 + j < p.n)
                        p.y[(((int64_t)at.b * p.n + n0 + j) * p.oh + at.y) * p.ow + at.x] =
                            finish(p, acc[j], p.bias != nullptr ? p.bias[n0 + j] : 0.f);
            }
        }
}

template <int RB, int BN>
__global__ void __launch_bounds__(kThreads, 1)
    conv_halo_f32_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                         const __grid_constant__ Params p) {
    constexpr int W_PLANE = BN * RB, STEPS = RB / 32, COLS = 2 * BN;   // k steps of a tap, columns of an accumulator
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int taps = p.fh * p.fw, box = p.halo_rows * RB;
    uint8_t *smem_a = smem + (taps * 3 * W_PLANE + 1023) / 1024 * 1024;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem_a + p.stages * 3 * box);
    uint64_t *full_bar = bars, *empty_bar = bars + kStages, *acc_full = bars + 2 * kStages;
    uint64_t *acc_empty = acc_full + kBuffers, *w_full = acc_empty + kBuffers;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(w_full + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    volatile int *any_mark = reinterpret_cast<volatile int *>(tmem_slot + 2);
    unsigned *marks = reinterpret_cast<unsigned *>(reinterpret_cast<uint8_t *>(bars) + 256);
    float *s_bias = reinterpret_cast<float *>(marks + kMarkWords);
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;

    if (threadIdx.x == 0) {
        prefetch_tmap(&map_x);
        prefetch_tmap(&map_w);
        for (int s = 0; s < kStages; ++s) {
            mbar_init(smem_u32(&full_bar[s]), 1);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        for (int s = 0; s < kBuffers; ++s) {
            mbar_init(smem_u32(&acc_full[s]), 1);
            mbar_init(smem_u32(&acc_empty[s]), 4);
        }
        mbar_init(smem_u32(w_full), 1);
        *abort_flag = 0;
        *any_mark = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (threadIdx.x < kMarkWords) marks[threadIdx.x] = 0;
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), kBuffers * COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    let_dependents_launch();
    dependency_wait();
    if (threadIdx.x < BN) s_bias[threadIdx.x] = p.bias != nullptr && threadIdx.x < p.n ? p.bias[threadIdx.x] : 0.f;
    __syncthreads();

    if (warp == 0) {
        if (elect_one()) {
            mbar_arrive_expect_tx(smem_u32(w_full), (uint32_t)(taps * 3 * W_PLANE));
            for (int t = 0; t < taps; ++t)
                for (int pl = 0; pl < 3; ++pl)
                    load_box(smem_u32(smem + (t * 3 + pl) * W_PLANE), &map_w, smem_u32(w_full), 0, pl * taps + t);
            int stage = 0;
            uint32_t phase = 0;
            for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x) {
                if (!mbar_wait(smem_u32(&empty_bar[stage]), phase ^ 1, abort_flag)) {
                    atomicExch(p.status, 210);
                    break;
                }
                mbar_arrive_expect_tx(smem_u32(&full_bar[stage]), (uint32_t)(3 * box));
                load_box(smem_u32(smem_a + stage * 3 * box), &map_x, smem_u32(&full_bar[stage]), tile * 128, 0);
                if (++stage == p.stages) {
                    stage = 0;
                    phase ^= 1;
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (elect_one()) {
            constexpr uint32_t id1 = make_idesc(false, false, 128, BN), id2 = make_idesc(false, false, 128, 2 * BN);
            const uint64_t w0 = operand<RB>(smem_u32(smem));
            const uint32_t plane = (uint32_t)box >> 4, next_row = (uint32_t)((p.wp - p.fw + 1) * RB) >> 4;
            const int steps = taps * STEPS;
            int stage = 0, set = 0;
            uint32_t phase = 0, used[2] = {0, 0};   // accumulators that a set's tiles have taken
            bool ok = mbar_wait(smem_u32(w_full), 0, abort_flag);
            if (!ok) atomicExch(p.status, 211);
            for (int tile = blockIdx.x; ok && tile < p.tiles; tile += gridDim.x) {
                if (!mbar_wait(smem_u32(&full_bar[stage]), phase, abort_flag)) {
                    atomicExch(p.status, 212);
                    break;
                }
                uint64_t a = operand<RB>(smem_u32(smem_a + stage * 3 * box)), b = w0;
                int fj = 0, ks = 0;
                uint32_t index = used[set];
                for (int s0 = 0; s0 < steps; s0 += 4, ++index) {
                    const int buf = 2 * set + (int)(index & 1);
                    if (!mbar_wait(smem_u32(&acc_empty[buf]), (index / 2 + 1) & 1u, abort_flag)) {
                        atomicExch(p.status, 213);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t d = tmem + buf * COLS;
                    // corrections first, as in gemm_tcx.cuh: hi.mid and mid.hi beside the leading products, hi.lo, mid.mid and
                    // lo.hi in the second block
                    uint64_t at[4], bt[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (s0 + i >= steps) break;
                        at[i] = a + 2 * ks;
                        bt[i] = b + 2 * ks;
                        umma_bf16(d, at[i], bt[i] + (W_PLANE >> 4), id2, i > 0);
                        umma_bf16(d, at[i] + plane, bt[i], id2, 1);
                        umma_bf16(d + BN, at[i] + 2 * plane, bt[i], id1, 1);
                        if (++ks == STEPS) {
                            ks = 0;
                            b += 3 * (W_PLANE >> 4);
                            if (++fj == p.fw) {
                                fj = 0;
                                a += next_row;
                            } else {
                                a += RB >> 4;
                            }
                        }
                    }
                    umma_bf16_shift8(d, at[0], bt[0], id1);
#pragma unroll
                    for (int i = 1; i < 4; ++i)
                        if (s0 + i < steps) umma_bf16(d, at[i], bt[i], id1, 1);
                    umma_commit(smem_u32(&acc_full[buf]));
                }
                if (!ok) break;
                used[set] = index;
                set ^= 1;
                umma_commit(smem_u32(&empty_bar[stage]));
                if (++stage == p.stages) {
                    stage = 0;
                    phase ^= 1;
                }
            }
        }
        __syncwarp();
    } else {
        const int quarter = warp % 4, set = (warp - 2) / 4;
        bool ok = true;
        uint32_t index = 0;
        for (int tile = blockIdx.x + set * gridDim.x, i = set; ok && tile < p.tiles; tile += 2 * gridDim.x, i += 2) {
            float sum[BN];
#pragma unroll
            for (int j = 0; j < BN; ++j) sum[j] = 0.f;
            for (int g = 0; g < p.groups; ++g, ++index) {
                const int buf = 2 * set + (int)(index & 1);
                if (!mbar_wait(smem_u32(&acc_full[buf]), index / 2 & 1u, abort_flag)) {
                    if (lane == 0) atomicExch(p.status, 214);
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t t = tmem + buf * COLS + ((uint32_t)(quarter * 32) << 16);
#pragma unroll
                for (int c = 0; c < BN; c += 16) {
                    uint32_t r0[16], r1[16];
                    tmem_ld_32x16(t + c, r0);
                    tmem_ld_32x16(t + BN + c, r1);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) sum[c + j] += fmaf(__uint_as_float(r1[j]), 0x1p-16f, __uint_as_float(r0[j]));
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&acc_empty[buf]));
            }
            if (!ok) break;
            const Position at = position(p, tile * 128 + quarter * 32 + lane);
            float finite = 0.f;
#pragma unroll
            for (int j = 0; j < BN; ++j) finite = fmaf(sum[j], 0.f, finite);
            if (__any_sync(0xffffffffu, at.valid && !(finite == 0.f))) {
                if (lane == 0) {
                    atomicOr(marks + i / 8, 1u << (i % 8 * 4 + quarter));
                    *any_mark = 1;
                }
            } else if (at.valid) {
                float *q = p.y + ((int64_t)at.b * p.n * p.oh + at.y) * p.ow + at.x;
                const int64_t step = (int64_t)p.oh * p.ow;
#pragma unroll
                for (int j = 0; j < BN; ++j, q += step)
                    if (j < p.n) *q = finish(p, sum[j], s_bias[j]);
            }
            __syncwarp();
        }
    }

    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {   // loads and products that were issued may still be running
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, kBuffers * COLS);
    }
    if (*any_mark && !*abort_flag) redo(p, marks);
}

// ------------------------------------------------------------------ planes
struct SourceJob {
    const float *src;
    uint4 *dst;
    int64_t plane;            // 16-byte pieces per plane
    int channels, h, wd, pad_h, pad_w, groups;
    uint32_t total;           // images x groups x framed pixels
    FastDiv div_frame, div_wp, div_groups;
};
struct FilterJob {
    const float *w;
    uint4 *dst;
    int64_t plane, s_row, s_c;
    int channels, groups, taps, n, reversed;
    uint32_t total;           // n x groups x taps
    FastDiv div_taps, div_groups;
};

__device__ __forceinline__ void store_planes(const float (&x)[8], uint4 *dst, int64_t plane) {
    uint32_t h[4], m[4], l[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        uint32_t hb[2], mb[2], lb[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) tcx::split3(x[2 * e + u], hb[u], mb[u], lb[u]);
        h[e] = tcx::upper_halves(hb[0], hb[1]);
        m[e] = tcx::upper_halves(mb[0], mb[1]);
        l[e] = tcx::upper_halves(lb[0], lb[1]);
    }
    dst[0] = make_uint4(h[0], h[1], h[2], h[3]);
    dst[plane] = make_uint4(m[0], m[1], m[2], m[3]);
    dst[2 * plane] = make_uint4(l[0], l[1], l[2], l[3]);
}

// A thread makes eight channels of a pixel of the frame (or of a filter's tap); a warp reads neighbouring pixels.
__global__ void __launch_bounds__(256) planes_kernel(const SourceJob s, const FilterJob f) {
    let_dependents_launch(kAlwaysEarly);
    dependency_wait();
    float x[8];
    if (blockIdx.y == 0) {
        for (uint32_t i = blockIdx.x * 256u + threadIdx.x; i < s.total; i += gridDim.x * 256u) {
            uint32_t t, at, image, group, py, px;
            s.div_frame.divmod(i, t, at);
            s.div_groups.divmod(t, image, group);
            s.div_wp.divmod(at, py, px);
            const int y = (int)py - s.pad_h, xx = (int)px - s.pad_w, c0 = (int)group * 8;
            const bool in = y >= 0 && y < s.h && xx >= 0 && xx < s.wd;
            const int64_t hw = (int64_t)s.h * s.wd;
            const float *q = s.src + ((int64_t)image * s.channels + c0) * hw + (in ? y * s.wd + xx : 0);
#pragma unroll
            for (int e = 0; e < 8; ++e, q += hw) x[e] = load_or_zero(q, in && c0 + e < s.channels);
            store_planes(x, s.dst + ((int64_t)image * s.div_frame.d + at) * s.groups + group, s.plane);
        }
    } else {
        for (uint32_t i = blockIdx.x * 256u + threadIdx.x; i < f.total; i += gridDim.x * 256u) {
            uint32_t t, tap, row, group;
            f.div_taps.divmod(i, t, tap);
            f.div_groups.divmod(t, row, group);
            const int c0 = (int)group * 8;
            const float *q = f.w + row * f.s_row + c0 * f.s_c + (f.reversed ? f.taps - 1 - (int)tap : (int)tap);
#pragma unroll
            for (int e = 0; e < 8; ++e, q += f.s_c) x[e] = load_or_zero(q, c0 + e < f.channels);
            store_planes(x, f.dst + ((int64_t)tap * f.n + row) * f.groups + group, f.plane);
        }
    }
}

// ---------------------------------------------------------------------- host
struct Plan {
    int rb, bn, halo_rows, stages, smem;
    int64_t hp, wp, rows, tiles;
};
bool make_plan(ag_device *dev, const Problem &p, Plan *l) {
    if (p.channels < 1 || p.channels > 64 || p.n < 1 || p.n > 64 || p.fh * p.fw > kMostTaps) return false;
    if (p.pad_h < 0 || p.pad_w < 0 || encode_tiled_fn() == nullptr) return false;
    l->rb = p.channels <= 16 ? 32 : p.channels <= 32 ? 64 : 128;
    l->bn = p.n <= 16 ? 16 : p.n <= 32 ? 32 : 64;
    l->hp = p.h + 2 * p.pad_h;
    l->wp = p.wd + 2 * p.pad_w;
    l->rows = p.bs * l->hp * l->wp;
    if (l->hp >= (1 << 15) || l->wp >= (1 << 15) || p.bs >= (1 << 20) || l->rows >= (int64_t(1) << 27)) return false;
    const int64_t halo = (128 + (p.fh - 1) * l->wp + p.fw - 1 + 31) / 32 * 32;
    if (halo > 256) return false;
    l->halo_rows = (int)halo;
    const int weights = (p.fh * p.fw * 3 * l->bn * l->rb + 1023) / 1024 * 1024, box = (int)halo * l->rb * 3;
    l->stages = (226 * 1024 - 1024 - kControl - weights) / box;
    if (l->stages < 2) return false;
    if (l->stages > kStages) l->stages = kStages;
    l->smem = weights + l->stages * box + 1024 + kControl;
    l->tiles = ceil_div(l->rows, 128);
    return l->tiles <= (int64_t)kMostTiles * dev->sm_count;
}

// A map of {channels, rows, z} with boxes of all channels, `rows` rows and `deep` of z.
int make_map(CUtensorMap *map, const void *base, int rb, int64_t rows, int64_t z, int box_rows, int deep) {
    const cuuint64_t dims[3] = {(cuuint64_t)rb / 2, (cuuint64_t)rows, (cuuint64_t)z};
    const cuuint64_t strides[2] = {(cuuint64_t)rb, (cuuint64_t)rb * (cuuint64_t)rows};
    const cuuint32_t box[3] = {(cuuint32_t)rb / 2, (cuuint32_t)box_rows, (cuuint32_t)deep}, one[3] = {1, 1, 1};
    const CUresult r = encode_tiled_fn()(
        map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(base), dims, strides, box, one,
        CU_TENSOR_MAP_INTERLEAVE_NONE,
        rb == 32 ? CU_TENSOR_MAP_SWIZZLE_32B : rb == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    AG_REQUIRE(r == CUDA_SUCCESS, AG_ERR_CUDA, "cuTensorMapEncodeTiled failed (CUresult %d)", (int)r);
    return AG_OK;
}

template <int RB, int BN>
int launch(ag_device *dev, const Plan &l, const CUtensorMap &mx, const CUtensorMap &mw, const Params &a) {
    auto kernel = conv_halo_f32_kernel<RB, BN>;
    const int smem = l.smem < kOneCtaPerSm ? kOneCtaPerSm : l.smem;
    static int configured_on[64] = {};
    int &configured = configured_on[dev->ordinal & 63];
    if (smem > configured) {
        AG_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        configured = smem;
    }
    const int grid = l.tiles < dev->sm_count ? (int)l.tiles : dev->sm_count;
    return launch_dependent(dev, kernel, dim3((unsigned)grid), kThreads, smem, mx, mw, a);
}

}  // namespace

// Against the gathered engine, us here and there, images x channels x side -> columns, 3 x 3 unless said: forward 64 x 16 x
// 32 -> 32 17.9 and 24.3, 144 x 32 x 28 -> 6 27 and 39, 61 x 32 x 51 -> 16 37 and 62, 134 x 6 x 29 -> 64 27 and 34, 94 x 32 x
// 12 -> 32 11.7 and 13.0; input gradients 64 x 32 x 32 -> 16 20.7 and 30.9, 171 x 16 x 42 -> 64 65 and 96, 13 x 32 x 39 -> 6
// 12.1 and 17.6.  It is two launches and pads channels to 16 and columns too: 47 x 6 x 21 -> 32 12.0 and 9.1, 11 x 3 x 59 ->
// 32 14.0 and 9.5, 5 x 5 45 x 6 x 61 -> 32 64 and 59, input gradients 30 x 6 x 35 -> 32 13.6 and 12.6.  Many channels into
// few columns are faster as products with every tap: 134 x 64 x 29 -> 6 53 and 39, 245 x 32 x 38 -> 3 81 and 65.  Over 110
// drawn f32 convolutions the passes that come here take 0.75 of their time, one in thirty more than it.
bool takes(ag_device *dev, const Problem &p) {
    Plan l;
    if (!make_plan(dev, p, &l)) return false;
    const int64_t taps = p.fh * p.fw;
    if (p.channels <= 4 || (p.channels < 12 && taps > 9)) return false;
    if ((p.channels > 32 && p.n * taps <= 128) || (p.channels > 16 && p.n <= 4)) return false;
    if (2 * p.oh * p.ow < l.hp * l.wp) return false;   // rows of the frame that are outputs
    return p.bs * p.oh * p.ow * taps * p.channels * (p.n < 16 ? 16 : p.n) >= 80000000;
}

int run(ag_device *dev, const Problem &p, const float *bias, bool relu, float *y, bool *taken) {
    Plan l;
    *taken = false;
    AG_REQUIRE(make_plan(dev, p, &l), AG_ERR_UNSUPPORTED, "convolution not taken");
    const int groups = l.rb / 16, taps = p.fh * p.fw;
    SourceJob s;
    s.src = p.src;
    s.plane = l.rows * groups;
    s.channels = (int)p.channels;
    s.h = (int)p.h; s.wd = (int)p.wd;
    s.pad_h = p.pad_h; s.pad_w = p.pad_w;
    s.groups = groups;
    s.total = (uint32_t)s.plane;
    s.div_frame = FastDiv((uint32_t)(l.hp * l.wp));
    s.div_wp = FastDiv((uint32_t)l.wp);
    s.div_groups = FastDiv((uint32_t)groups);
    FilterJob f;
    f.w = p.w;
    f.s_row = p.s_row; f.s_c = p.s_c;
    f.channels = (int)p.channels;
    f.groups = groups;
    f.taps = taps;
    f.n = (int)p.n;
    f.reversed = p.reversed;
    f.plane = (int64_t)taps * p.n * groups;
    f.total = (uint32_t)f.plane;
    f.div_taps = FastDiv((uint32_t)taps);
    f.div_groups = s.div_groups;
    const int64_t source_bytes = (s.plane * 48 + 1023) / 1024 * 1024;
    void *ws = nullptr;
    if (staging(dev, (size_t)(source_bytes + f.plane * 48), &ws) != AG_OK) return AG_OK;
    *taken = true;
    s.dst = (uint4 *)ws;
    f.dst = (uint4 *)((char *)ws + source_bytes);
    const int64_t blocks = ceil_div(s.total > f.total ? s.total : f.total, 256), cap = (int64_t)dev->sm_count * 16;
    AG_TRY(launch_dependent(dev, planes_kernel, dim3((unsigned)(blocks < cap ? blocks : cap), 2), 256, 0, s, f));

    Params a;
    a.R = (int)l.rows;
    a.tiles = (int)l.tiles;
    a.hp = (int)l.hp; a.wp = (int)l.wp;
    a.oh = (int)p.oh; a.ow = (int)p.ow;
    a.n = (int)p.n;
    a.fh = p.fh; a.fw = p.fw;
    a.halo_rows = l.halo_rows;
    a.stages = l.stages;
    a.groups = (int)ceil_div((int64_t)taps * (l.rb / 32), 4);
    a.div_wp = s.div_wp;
    a.div_image = s.div_frame;
    a.bias = bias;
    a.relu = relu ? 1 : 0;
    a.y = y;
    a.status = dev->status_dev;
    a.src = p.src; a.w = p.w;
    a.channels = (int)p.channels;
    a.h = (int)p.h; a.wd = (int)p.wd;
    a.pad_h = p.pad_h; a.pad_w = p.pad_w;
    a.s_row = p.s_row; a.s_c = p.s_c;
    a.reversed = p.reversed;
    CUtensorMap mx, mw;
    AG_TRY(make_map(&mx, s.dst, l.rb, l.rows, 3, l.halo_rows, 3));
    AG_TRY(make_map(&mw, f.dst, l.rb, p.n, 3 * taps, l.bn, 1));
    if (l.rb == 32)
        return l.bn == 16 ? launch<32, 16>(dev, l, mx, mw, a)
             : l.bn == 32 ? launch<32, 32>(dev, l, mx, mw, a) : launch<32, 64>(dev, l, mx, mw, a);
    if (l.rb == 64)
        return l.bn == 16 ? launch<64, 16>(dev, l, mx, mw, a)
             : l.bn == 32 ? launch<64, 32>(dev, l, mx, mw, a) : launch<64, 64>(dev, l, mx, mw, a);
    return l.bn == 16 ? launch<128, 16>(dev, l, mx, mw, a)
         : l.bn == 32 ? launch<128, 32>(dev, l, mx, mw, a) : launch<128, 64>(dev, l, mx, mw, a);
}

}  // namespace halo32
}  // namespace ag
