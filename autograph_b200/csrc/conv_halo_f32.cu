// f32 convolutions with stride 1 and up to 64 channels as six bf16 products on tcgen05 (the arithmetic of
// gemm_tcx.cuh: three planes per operand, sums of 64 k read out and added in registers, in the same order, so the bits are
// those of the gathered engine).
//
// The source, channels last and inside its zero padding, [image][y][x][Cp] with Cp = 16, 32 or 64 channels, a pixel being one
// row of 32, 64 or 128 bytes, is a matrix of rows, and the A operand of tap (fi, fj) is that of tap (0, 0) moved down fi * Wp +
// fj rows: a tile of 128 rows needs ONE box of 128 + (fh - 1) * Wp + fw - 1 rows per plane, and every tap's products start that
// many rows further on in it (as in conv_tc_halo.cu; the 32- and 64-byte swizzles too are functions of the absolute
// shared-memory address).  The filters of all taps stay in shared memory.  Rows that are no outputs, the right-hand columns
// and bottom rows of every image, are computed and dropped.
//
// The gathered engine fetches and splits every element once per tap (16 channels 3 x 3: 92 KB per tile from L1 and L2, and
// most of its instructions); here it is once per box, whose rows are rounded up to 32: 224 rows for a tile of 128 of a 32 x 32
// image in its frame, so 1.75 times over all.  A pass that wrote the rows for TMA to load was half of the operator's time.
// What bounds it is latency: at 64 x 16 x 32 x 32 -> 32, four tiles an SM, the tensor pipe is active 12 % (input gradient 9 %) and
// warps wait for loads of pixels (long scoreboard, 2.5 and 4.7 per issue) and, in the epilogue, for the other ones (barrier 2.5).
//
// Warps: 1 issues, 2 - 9 split the filters and then read accumulators, in two sets that take turns at tiles, each with two
// accumulators (leading block and corrections) of its own, 0 and 10 - 15 load and split rows.
#include "conv_halo_device.cuh"

namespace ag {
namespace halo32 {

using namespace ::ag::tc;

namespace {

constexpr int kWarps = 9 + kFillers, kThreads = kWarps * 32, kStages = 4, kBuffers = 4, kMostTaps = 25;
constexpr int kMarkWords = 128;          // a bit per epilogue warp and tile of a CTA
constexpr int kMostTiles = kMarkWords * 8;
constexpr int kControl = 256 + kMarkWords * 4 + 1024;

struct Params {
    Source x;
    int tiles, oh, ow, n;
    int wp, fh, fw, halo_rows, stages, groups;   // groups of 64 k
    FastDiv div_taps;
    const float *w;
    int64_t s_row, s_c;
    int reversed;
    const float *bias;
    int relu;
    float *y;
    int *status;
};

// Output position of row q.
struct Position {
    int b, y, x;
    bool valid;
};
__device__ __forceinline__ Position position(const Params &p, int q) {
    uint32_t b, r, y, x;
    p.x.div_image.divmod((uint32_t)q, b, r);
    p.x.div_wp.divmod(r, y, x);
    return Position{(int)b, (int)y, (int)x, q < p.x.rows && (int)y < p.oh && (int)x < p.ow};
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
                    const int sy = at.y + tap / p.fw - p.x.pad_h, sx = at.x + tap % p.fw - p.x.pad_w;
                    const bool in = sy >= 0 && sy < p.x.h && sx >= 0 && sx < p.x.wd;
                    const float *s = p.x.src + (int64_t)at.b * p.x.channels * p.x.h * p.x.wd + (in ? sy * p.x.wd + sx : 0);
                    const float *w = p.w + n0 * p.s_row + (p.reversed ? taps - 1 - tap : tap);
                    for (int c = 0; c < p.x.channels; ++c) {
                        const float v = in ? s[(int64_t)c * p.x.h * p.x.wd] : 0.f;
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
    conv_halo_f32_kernel(const __grid_constant__ Params p) {
    constexpr int W_PLANE = BN * RB, STEPS = RB / 32, COLS = 2 * BN;   // k steps of a tap, columns of an accumulator
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int taps = p.fh * p.fw, box = p.halo_rows * RB, items = p.halo_rows / 32 * STEPS;
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
        for (int s = 0; s < kStages; ++s) {
            mbar_init(smem_u32(&full_bar[s]), (uint32_t)items);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        for (int s = 0; s < kBuffers; ++s) {
            mbar_init(smem_u32(&acc_full[s]), 1);
            mbar_init(smem_u32(&acc_empty[s]), 4);
        }
        mbar_init(smem_u32(w_full), 8);
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

    if (warp == 0 || warp > 9) {
        const int worker = warp == 0 ? 0 : warp - 9;
        Item item{0, (int)blockIdx.x, 0, 1u};
        item.forward(worker, items, p.stages);
        float v[16];
        const auto load = [&](const Item &i, float (&to)[16]) {
            if (i.tile < p.tiles) load_row(p.x, i.tile * 128 + i.at / STEPS * 32 + lane, i.at % STEPS * 16, to);
        };
        load(item, v);
        while (item.tile < p.tiles) {
            Item next = item;
            next.forward(kFillers, items, p.stages);
            float ahead[16];
            load(next, ahead);
            if (!mbar_wait(smem_u32(&empty_bar[item.stage]), item.phase, abort_flag)) {
                if (lane == 0) atomicExch(p.status, 210);
                break;
            }
            const uint32_t offset = (item.at / STEPS * 32 + lane) * RB + item.at % STEPS * 32;
            uint8_t *dst = smem_a + item.stage * 3 * box;
            store_pieces<RB>(v, dst, offset, box);
            store_pieces<RB>(v + 8, dst, offset + 16, box);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&full_bar[item.stage]));
            item = next;
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = ahead[e];
        }
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
        // [tap][plane][n][Cp], eight channels at a time
        constexpr int MANY = 3;
        const int pieces = taps * BN * STEPS * 2;
        for (int i0 = threadIdx.x - 64; i0 < pieces; i0 += 256 * MANY) {
            float v[MANY][8];
            uint32_t offset[MANY];
#pragma unroll
            for (int m = 0; m < MANY; ++m) {
                uint32_t t, tap;
                p.div_taps.divmod((uint32_t)(i0 + 256 * m), t, tap);
                const int n = (int)t / (STEPS * 2), c0 = (int)t % (STEPS * 2) * 8;
                const float *q = p.w + n * p.s_row + c0 * p.s_c + (p.reversed ? taps - 1 - (int)tap : (int)tap);
                offset[m] = tap * 3 * W_PLANE + n * RB + c0 * 2;
#pragma unroll
                for (int e = 0; e < 8; ++e, q += p.s_c) v[m][e] = load_or_zero(q, n < p.n && c0 + e < p.x.channels);
            }
#pragma unroll
            for (int m = 0; m < MANY; ++m)
                if (i0 + 256 * m < pieces) store_pieces<RB>(v[m], smem, offset[m], W_PLANE);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(w_full));

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
    if (*abort_flag) {   // products that were issued may still be running
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, kBuffers * COLS);
    }
    if (*any_mark && !*abort_flag) redo(p, marks);
}

// ---------------------------------------------------------------------- host
struct Plan {
    int rb, bn, halo_rows, stages, smem;
    int64_t hp, wp, rows, tiles;
};
bool make_plan(ag_device *dev, const Problem &p, Plan *l) {
    if (p.channels < 1 || p.channels > 64 || p.n < 1 || p.n > 64 || p.fh * p.fw > kMostTaps) return false;
    if (p.pad_h < 0 || p.pad_w < 0) return false;
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
    l->stages = (kMostSmem - 1024 - kControl - weights) / box;
    if (l->stages < 2) return false;
    if (l->stages > kStages) l->stages = kStages;
    l->smem = weights + l->stages * box + 1024 + kControl;
    l->tiles = ceil_div(l->rows, 128);
    return l->tiles <= (int64_t)kMostTiles * dev->sm_count;
}

template <int RB, int BN>
int launch(ag_device *dev, const Plan &l, const Params &a) {
    auto kernel = conv_halo_f32_kernel<RB, BN>;
    const int smem = l.smem < kOneCtaPerSm ? kOneCtaPerSm : l.smem;
    static SmemAllowed allowed;
    AG_TRY(allow_smem(dev, kernel, allowed));
    const int grid = l.tiles < dev->sm_count ? (int)l.tiles : dev->sm_count;
    return launch_dependent(dev, kernel, dim3((unsigned)grid), kThreads, smem, a);
}

}  // namespace

// Against the gathered engine and an earlier form with its rows written by a pass (that did not take calls below 8e7), us there and
// here, images x channels x side -> columns, 3 x 3 unless said: forward 64 x 16 x 32 -> 32 24.3, 17.8 and 13.0, 243 x 64 x 35 -> 16 167
// and 85, 134 x 6 x 29 -> 64 34, 27 and 23, 232 x 1 x 60 -> 32 126 and 76; input gradients (of that forward) 64 x 16 x 32 -> 32 30.9,
// 20.8 and 16.9, 171 x 64 x 42 -> 16 96 and 65; small ones 5 x 16 x 39 -> 16 9.5 and 5.5, 133 x 6 x 13 -> 32 12.4 and 9.2, 38 x
// 6 x 26 -> 16's input gradient 17.6 and 6.9.
// Every CTA splits all filters before its first product: many filters want more work (19 x 16 x 20 -> 64 5 x 5 15.6 and 17.5, 5 x 32 x
// 40 -> 64 13.2 and 14.4, 10 x 32 x 42 -> 64's input gradient 19.2 and 21.5).  Channels are padded to 16 and columns to 16, 32 or 64: up to
// 4 channels gain where there is much work (189 x 3 x 20 -> 64 18.5 and 21.2, 246 x 3 x 55 -> 64 146 and 111), 94 x 6 x 31
// -> 64 5 x 5 43 and 46.  Many channels into few columns are faster as products with every tap: 189 x 3 x 20 -> 64's input
// gradient 22.7 and 30.8, 232 x 1 x 60 -> 32's 101 and 138, 658 x 3 x 27 -> 20 5 x 5's 178 and 222, but 8 x 1 x 61 -> 32's 14.6 and 11.6.
bool takes(ag_device *dev, const Problem &p) {
    Plan l;
    if (!make_plan(dev, p, &l)) return false;
    const int64_t taps = p.fh * p.fw, work = p.bs * p.oh * p.ow * taps * p.channels * (p.n < 16 ? 16 : p.n);
    if (p.channels < 12 && taps > 9 && p.n > 32) return false;
    if ((p.channels > 32 && p.n * taps <= 128) || (p.channels > 16 && p.n <= 2 && work > (taps > 9 ? 100000000 : 300000000)) ||
        (p.channels > 16 && p.n <= 4 && taps > 9 && work > 300000000))
        return false;
    if (2 * p.oh * p.ow < l.hp * l.wp) return false;   // rows of the frame that are outputs
    if (p.channels <= 4) return taps <= 9 && work >= 200000000;
    const int64_t filters = taps * l.bn * (l.rb / 2);
    return work >= (filters <= 7000 ? 15000000 : filters <= 14000 ? 80000000 : 400000000);
}

int run(ag_device *dev, const Problem &p, const float *bias, bool relu, float *y) {
    Plan l;
    AG_REQUIRE(make_plan(dev, p, &l), AG_ERR_UNSUPPORTED, "convolution not taken");
    const int taps = p.fh * p.fw;
    Params a;
    a.x = source(p.src, p.channels, p.h, p.wd, p.pad_h, p.pad_w, l.hp, l.wp, l.rows);
    a.tiles = (int)l.tiles;
    a.oh = (int)p.oh; a.ow = (int)p.ow;
    a.n = (int)p.n;
    a.wp = (int)l.wp;
    a.fh = p.fh; a.fw = p.fw;
    a.halo_rows = l.halo_rows;
    a.stages = l.stages;
    a.groups = (int)ceil_div((int64_t)taps * (l.rb / 32), 4);
    a.div_taps = FastDiv((uint32_t)taps);
    a.w = p.w;
    a.s_row = p.s_row; a.s_c = p.s_c;
    a.reversed = p.reversed;
    a.bias = bias;
    a.relu = relu ? 1 : 0;
    a.y = y;
    a.status = dev->status_dev;
    if (l.rb == 32)
        return l.bn == 16 ? launch<32, 16>(dev, l, a)
             : l.bn == 32 ? launch<32, 32>(dev, l, a) : launch<32, 64>(dev, l, a);
    if (l.rb == 64)
        return l.bn == 16 ? launch<64, 16>(dev, l, a)
             : l.bn == 32 ? launch<64, 32>(dev, l, a) : launch<64, 64>(dev, l, a);
    return l.bn == 16 ? launch<128, 16>(dev, l, a)
         : l.bn == 32 ? launch<128, 32>(dev, l, a) : launch<128, 64>(dev, l, a);
}

}  // namespace halo32
}  // namespace ag
