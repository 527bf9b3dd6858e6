// Weight gradients of f32 convolutions with stride 1 from up to 64 channels into up to 32 on tcgen05 (three bf16 planes per operand
// and sums of 64 k read out and added in registers, as in gemm_tcx.cuh).
//
//   dw[n][c][fi][fj] = sum over rows r of x[r + fj][c] * dy[r - fi * Wp][n]
//
// on the matrices of rows that conv_halo_f32.cu works on: x channels last inside its zero padding, and dy on the same grid of
// Hp x Wp rows per image, zero where a row is no output, so that one index serves both.  The reduction runs over rows, and both
// operands are read across them (MN-major).  A tile is 128 rows: one box of as many rows of x and a few more, one of 128 + (fh -
// 1) * Wp rows of dy, three planes each, loaded and split once.  The taps are the operands moved by rows, which is what a
// descriptor's stride between blocks says: the M index of a product is blocks of Cp channels that start one row apart
// (eight, four or two taps of a filter row; what lies beyond fw is not looked at), its N index is fh blocks of dy's columns that
// start Wp rows apart.  So a product has all taps of 3 x 3 filters at up to 32 channels, where one per filter row with planes of
// dy side by side takes twice as many products of some 45 cycles each.  Every CTA leaves the sums of its tiles, a second
// kernel adds them in order.
//
// The gathered engine makes a [taps x channels] x [positions] matrix of it and fetches and splits an element once per tap.
#include "conv_halo_device.cuh"

namespace ag {
namespace halo32 {

using namespace ::ag::tc;

namespace {

constexpr int kWarps = 9 + kFillers, kThreads = kWarps * 32, kStages = 4;
constexpr int kControl = 256;
constexpr int kMostSums = 6;   // accumulators of 16 columns that a warp's registers hold

struct WgradParams {
    Source x, dy;
    int tiles, wp, fh, fw, products;      // products: blocks of taps of a filter row
    int x_rows, dy_rows, stages;          // of a box
    float *partial;                       // [CTA][product][filter row, last first][n][128]
    int *status;
};

// RB, RN: bytes of a row of x and dy.
template <int RB, int RN>
__global__ void __launch_bounds__(kThreads, 1)
    conv_halo_wgrad_kernel(const __grid_constant__ WgradParams p) {
    constexpr int N = RN / 2, BLOCKS = 256 / RB;   // columns; taps of a product
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int x_plane = p.x_rows * RB, dy_plane = p.dy_rows * RN, stage_bytes = 3 * (x_plane + dy_plane);
    const int accs = p.fh * p.products;
    const int buffers = accs * 2 * N <= 256 ? 2 : 1;   // of tensor memory, which has 512 columns
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + p.stages * stage_bytes);
    uint64_t *full_bar = bars, *empty_bar = bars + kStages, *acc_full = bars + 2 * kStages, *acc_empty = acc_full + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + 2);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    constexpr int X_PAIRS = RB / 32, DY_PAIRS = RN / 32;
    const int x_items = p.x_rows / 32 * X_PAIRS, items = x_items + p.dy_rows / 32 * DY_PAIRS;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(smem_u32(&full_bar[s]), (uint32_t)items);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(smem_u32(&acc_full[s]), 1);
            mbar_init(smem_u32(&acc_empty[s]), 8);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    let_dependents_launch();
    dependency_wait();

    if (warp == 0 || warp > 9) {
        const int worker = warp == 0 ? 0 : warp - 9;
        Item item{0, (int)blockIdx.x, 0, 1u};
        item.forward(worker, items, p.stages);
        float v[16];
        const auto load = [&](const Item &i, float (&to)[16]) {
            if (i.tile >= p.tiles) return;
            if (i.at < x_items) {
                load_row(p.x, i.tile * 128 + i.at / X_PAIRS * 32 + lane, i.at % X_PAIRS * 16, to);
            } else {
                const int at = i.at - x_items;
                load_row(p.dy, i.tile * 128 - (p.fh - 1) * p.wp + at / DY_PAIRS * 32 + lane, at % DY_PAIRS * 16, to);
            }
        };
        load(item, v);
        while (item.tile < p.tiles) {
            Item next = item;
            next.forward(kFillers, items, p.stages);
            float ahead[16];
            load(next, ahead);
            if (!mbar_wait(smem_u32(&empty_bar[item.stage]), item.phase, abort_flag)) {
                if (lane == 0) atomicExch(p.status, 220);
                break;
            }
            uint8_t *dst = smem + item.stage * stage_bytes;
            if (item.at < x_items) {
                const uint32_t offset = (item.at / X_PAIRS * 32 + lane) * RB + item.at % X_PAIRS * 32;
                store_pieces<RB>(v, dst, offset, x_plane);
                store_pieces<RB>(v + 8, dst, offset + 16, x_plane);
            } else {
                const int at = item.at - x_items;
                const uint32_t offset = (at / DY_PAIRS * 32 + lane) * RN + at % DY_PAIRS * 32;
                store_pieces<RN>(v, dst + 3 * x_plane, offset, dy_plane);
                store_pieces<RN>(v + 8, dst + 3 * x_plane, offset + 16, dy_plane);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&full_bar[item.stage]));
            item = next;
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = ahead[e];
        }
    } else if (warp == 1) {
        if (elect_one()) {
            const int width = p.fh * N;
            const uint32_t idesc = make_idesc(true, true, 128, width), xp = (uint32_t)x_plane >> 4, yp = (uint32_t)dy_plane >> 4;
            int stage = 0, buf = 0;
            uint32_t phase = 0, acc_phase = 0;
            bool ok = true;
            for (int tile = blockIdx.x; ok && tile < p.tiles; tile += gridDim.x) {
                if (!mbar_wait(smem_u32(&full_bar[stage]), phase, abort_flag)) {
                    atomicExch(p.status, 221);
                    break;
                }
                const uint32_t base = smem_u32(smem + stage * stage_bytes);
                const uint64_t a0 = operand<RB>(base) | (uint64_t)(RB >> 4) << 16;   // blocks one row apart
                const uint64_t b0 = operand<RN>(base + 3 * x_plane) | (uint64_t)(p.wp * (RN >> 4)) << 16;   // Wp rows
                for (int half = 0; half < 2; ++half) {   // 64 rows
                    if (!mbar_wait(smem_u32(&acc_empty[buf]), acc_phase ^ 1, abort_flag)) {
                        atomicExch(p.status, 222);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    uint32_t d = tmem + buf * 256;
                    for (int pr = 0; pr < p.products; ++pr, d += 2 * width) {
                        const uint64_t a = a0 + (uint64_t)((pr * BLOCKS + half * 64) * (RB >> 4));
                        const uint64_t b = b0 + (uint64_t)(half * 64 * (RN >> 4));
                        // corrections first, as in gemm_tcx.cuh; hi.lo, mid.mid and lo.hi in the second block
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const uint64_t ak = a + k * RB, bk = b + k * RN;   // 16 rows further on
                            umma_bf16(d, ak, bk + yp, idesc, k > 0);
                            umma_bf16(d, ak + xp, bk, idesc, 1);
                            umma_bf16(d + width, ak, bk + 2 * yp, idesc, k > 0);
                            umma_bf16(d + width, ak + xp, bk + yp, idesc, 1);
                            umma_bf16(d + width, ak + 2 * xp, bk, idesc, 1);
                        }
                        umma_bf16_shift8(d, a, b, idesc);
#pragma unroll
                        for (int k = 1; k < 4; ++k) umma_bf16(d, a + k * RB, b + k * RN, idesc, 1);
                    }
                    umma_commit(smem_u32(&acc_full[buf]));
                    if (++buf == buffers) {
                        buf = 0;
                        acc_phase ^= 1;
                    }
                }
                if (!ok) break;
                umma_commit(smem_u32(&empty_bar[stage]));
                if (++stage == p.stages) {
                    stage = 0;
                    phase ^= 1;
                }
            }
        }
        __syncwarp();
    } else {
        // 32 rows and 16 columns of every accumulator
        const int quarter = warp % 4, part = (warp - 2) / 4;
        const bool mine = part * 16 < N;
        // taps of a product's rows; those beyond the filter are neither read nor stored
        const int first = quarter * 64 / RB, tap = (quarter * 32 + lane) * 2 / RB;
        float sum[kMostSums][16];
#pragma unroll
        for (int i = 0; i < kMostSums; ++i)
#pragma unroll
            for (int j = 0; j < 16; ++j) sum[i][j] = 0.f;
        int buf = 0;
        uint32_t acc_phase = 0;
        bool ok = true;
        for (int tile = blockIdx.x; ok && tile < p.tiles; tile += gridDim.x)
            for (int half = 0; ok && half < 2; ++half) {
                if (!mbar_wait(smem_u32(&acc_full[buf]), acc_phase, abort_flag)) {
                    if (lane == 0) atomicExch(p.status, 223);
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t t = tmem + buf * 256 + ((uint32_t)(quarter * 32) << 16) + part * 16;
                if (mine)
#pragma unroll
                    for (int i = 0; i < kMostSums; ++i)
                        if (i < accs && i / p.fh * BLOCKS + first < p.fw) {
                            const uint32_t at = t + (i + i / p.fh * p.fh) * N;   // a product's two blocks of fh * N
                            uint32_t r0[16], r1[16];
                            tmem_ld_32x16(at, r0);
                            tmem_ld_32x16(at + p.fh * N, r1);
                            tmem_ld_wait();
#pragma unroll
                            for (int j = 0; j < 16; ++j) sum[i][j] += fmaf(__uint_as_float(r1[j]), 0x1p-16f, __uint_as_float(r0[j]));
                        }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&acc_empty[buf]));
                if (++buf == buffers) {
                    buf = 0;
                    acc_phase ^= 1;
                }
            }
        if (ok && mine) {
            float *q = p.partial + ((int64_t)blockIdx.x * accs * N + part * 16) * 128 + quarter * 32 + lane;
#pragma unroll
            for (int i = 0; i < kMostSums; ++i)
                if (i < accs && i / p.fh * BLOCKS + tap < p.fw)
#pragma unroll
                    for (int j = 0; j < 16; ++j) q[(i * N + j) * 128] = sum[i][j];
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
        tmem_dealloc(tmem, 512);
    }
}

struct WgradSum {
    const float *partial;
    int planes, n, channels, cp, fh, fw, products;
    float beta;
    float *dw;
    // the operands, for sums that are not finite
    const float *x, *dy;
    int bs, h, wd, oh, ow, pad_h, pad_w;
    int dy_channels;
};
// dw = beta * dw + the CTAs' sums: 32 neighbouring (tap, channel) of one n by 32 rows of CTAs, whose sums are added as a tree (in
// row order the chain of roundings left errors of up to 1.14 of the gathered engine's, now 0.35 to 0.86).
// A sum that is not finite (a split infinity is a NaN, and rows that are no outputs multiply pixels by zero) is computed
// again from the operands by the whole block.
constexpr int W_ROWS = 32;
__global__ void __launch_bounds__(32 * W_ROWS) conv_halo_wgrad_sum_kernel(const __grid_constant__ WgradSum p) {
    let_dependents_launch(kAlwaysEarly);
    dependency_wait();
    __shared__ float part[W_ROWS][33];
    __shared__ unsigned again;
    const int values = p.fh * p.fw * p.channels, n = blockIdx.y;
    const int i = blockIdx.x * 32 + threadIdx.x;
    const bool live = i < values;
    const int tap = live ? i / p.channels : 0, c = live ? i % p.channels : 0;
    const int fi = tap / p.fw, fj = tap % p.fw, blocks = 128 / p.cp;
    const float *src = p.partial + ((int64_t)(fj / blocks * p.fh + p.fh - 1 - fi) * p.n + n) * 128 + fj % blocks * p.cp + c;
    const int64_t plane = (int64_t)p.fh * p.products * p.n * 128;
    float s = 0.f;
    if (live)
        for (int z = threadIdx.y; z < p.planes; z += 5 * W_ROWS) {
            float v[5];
#pragma unroll
            for (int j = 0; j < 5; ++j) v[j] = z + W_ROWS * j < p.planes ? src[(z + W_ROWS * j) * plane] : 0.f;
#pragma unroll
            for (int j = 0; j < 5; ++j) s += v[j];
        }
    part[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    float *out = p.dw + ((int64_t)n * p.channels + c) * p.fh * p.fw + tap;
    if (threadIdx.y == 0) {
        float v[W_ROWS];
        v[0] = s;
#pragma unroll
        for (int r = 1; r < W_ROWS; ++r) v[r] = part[r][threadIdx.x];
#pragma unroll
        for (int half = W_ROWS / 2; half > 0; half /= 2)
#pragma unroll
            for (int r = 0; r < half; ++r) v[r] += v[r + half];
        s = v[0];
        const bool finite = s - s == 0.f;
        const unsigned bad = __ballot_sync(0xffffffffu, live && !finite);
        if (threadIdx.x == 0) again = bad;
        if (live && finite) *out = p.beta != 0.f ? s + p.beta * *out : s;
    }
    __syncthreads();
    for (unsigned bad = again; bad != 0; bad &= bad - 1) {
        const int j = __ffs(bad) - 1, at = blockIdx.x * 32 + j, t = at / p.channels, ch = at % p.channels;
        const int di = t / p.fw - p.pad_h, dj = t % p.fw - p.pad_w;
        const int tid = threadIdx.y * 32 + threadIdx.x;
        float sum = 0.f;
        for (int64_t e = tid; e < (int64_t)p.bs * p.oh * p.ow; e += 32 * W_ROWS) {
            const int b = (int)(e / (p.oh * p.ow)), r = (int)(e % (p.oh * p.ow)), y = r / p.ow + di, x = r % p.ow + dj;
            const float v = y >= 0 && y < p.h && x >= 0 && x < p.wd
                                ? p.x[(((int64_t)b * p.channels + ch) * p.h + y) * p.wd + x] : 0.f;
            sum = fmaf(v, p.dy[((int64_t)b * p.dy_channels + n) * p.oh * p.ow + r], sum);
        }
        __syncthreads();
        part[threadIdx.y][threadIdx.x] = sum;
        __syncthreads();
        if (tid == 0) {
            float total = 0.f;
            for (int r = 0; r < W_ROWS; ++r)
                for (int k = 0; k < 32; ++k) total += part[r][k];
            float *q = p.dw + ((int64_t)n * p.channels + ch) * p.fh * p.fw + t;
            *q = p.beta != 0.f ? total + p.beta * *q : total;
        }
    }
}

struct WgradPlan {
    int rb, rn, x_rows, dy_rows, stages, smem, products;
    int64_t hp, wp, rows, tiles;
};
bool make_wgrad_plan(const Wgrad &p, WgradPlan *l) {
    if (p.bs < 1 || p.channels < 1 || p.channels > 64 || p.n < 1 || p.n > 32 || p.fh * p.fw > 25) return false;
    l->rb = p.channels <= 16 ? 32 : p.channels <= 32 ? 64 : 128;
    l->rn = p.n <= 16 ? 32 : 64;
    const int blocks = 256 / l->rb;
    l->products = (int)ceil_div(p.fw, blocks);
    const int accs = p.fh * l->products, n = l->rn / 2;
    if (accs * 2 * n > 512 || accs > kMostSums) return false;   // tensor memory and the registers that add its sums
    l->hp = p.h + 2 * p.pad_h;
    l->wp = p.wd + 2 * p.pad_w;
    l->rows = p.bs * l->hp * l->wp;
    if (l->hp >= (1 << 15) || l->wp >= (1 << 15) || p.bs >= (1 << 20) || l->rows >= (int64_t(1) << 27)) return false;
    l->x_rows = (int)ceil_div(127 + l->products * blocks, 32) * 32;
    if (l->wp * (l->rn >> 4) >= (1 << 14)) return false;   // a descriptor's stride
    l->dy_rows = (int)ceil_div(128 + (p.fh - 1) * l->wp, 32) * 32;
    const int64_t stage = 3 * ((int64_t)l->x_rows * l->rb + (int64_t)l->dy_rows * l->rn);
    l->stages = (int)((kMostSmem - 1024 - kControl) / stage);
    if (l->stages < 2) return false;
    if (l->stages > kStages) l->stages = kStages;
    l->smem = l->stages * (int)stage + 1024 + kControl;
    l->tiles = ceil_div(l->rows, 128);
    return true;
}

template <int RB, int RN>
int launch_wgrad(ag_device *dev, const WgradPlan &l, int grid, const WgradParams &a) {
    auto kernel = conv_halo_wgrad_kernel<RB, RN>;
    const int smem = l.smem < kOneCtaPerSm ? kOneCtaPerSm : l.smem;
    static SmemAllowed allowed;
    AG_TRY(allow_smem(dev, kernel, allowed));
    return launch_dependent(dev, kernel, dim3((unsigned)grid), kThreads, smem, a);
}

}  // namespace

// Against the gathered engine, us there and here, images x channels x side -> columns, 3 x 3 unless said: 64 x 16 x 32 -> 32 34.2 and
// 21.7, 163 x 32 x 40 -> 16 117 and 42, 144 x 64 x 56 -> 6 438 and 124, 136 x 16 x 53 -> 32 149 and 78, 231 x 6 x 57 -> 6 5 x 5 248
// and 100, 53 x 3 x 48 -> 16 28 and 20, 87 x 1 x 17 -> 6 14.3 and 11.3, 4 x 64 x 39 -> 16 16.2 and 15.7.
// It pads channels and columns and has two launches: 17 x 16 x 22 -> 32 5 x 5 13.7 and 18.0, 5 x 64 x 47 -> 32 21.9 and 25.4 (61 x 64
// x 31 -> 32 57 and 45), 136 x 1 x 57 -> 32 5 x 5 70 and 123, 14 x 64 x 10 -> 6 9.9 and 12.7.  With 64 columns a tile's sums are 96
// registers a thread and its boxes leave two stages: 72 x 16 x 57 -> 64 100 and 97, 130 x 6 x 42 -> 64 48 and 78, so
// there are none.  One channel with 5 x 5 filters is a sixteenth of its rows and slower here (121 x 1 x 43 -> 16 42.9 and 45.2), and
// so are few positions of many channels (50 x 64 x 12 -> 16 13.9 and 15.3).  Over 331 drawn gradients those that come here take
// 0.69 of their time, all but one (278 x 3 x 17 x 45 -> 6 5 x 1, 35.7 and 39.6) at most 1.02.
// Errors against float64 are 0.35 to 0.86 of the gathered engine's over 106 drawn gradients.
bool takes_wgrad(const Wgrad &p) {
    WgradPlan l;
    if (!make_wgrad_plan(p, &l)) return false;
    const int64_t positions = p.bs * p.oh * p.ow;
    if (2 * p.oh * p.ow < l.hp * l.wp) return false;   // rows of the frame that are outputs
    if (p.channels == 1 && p.fh * p.fw >= 25) return false;
    if (p.n <= 16) return positions >= (p.channels > 32 ? 6000 : 4000);
    return p.channels > 4 && positions >= (p.channels > 32 || p.fh * p.fw > 9 ? 40000 : 10000);
}

int run_wgrad(ag_device *dev, const Wgrad &p, float beta, float *dw, bool *taken) {
    WgradPlan l;
    *taken = false;
    AG_REQUIRE(make_wgrad_plan(p, &l), AG_ERR_UNSUPPORTED, "weight gradient not taken");
    const int grid = l.tiles < dev->sm_count ? (int)l.tiles : dev->sm_count, accs = p.fh * l.products, n = l.rn / 2;
    void *sums = nullptr;
    if (engine_scratch(dev, (size_t)grid * accs * n * 128 * sizeof(float), &sums) != AG_OK) return AG_OK;
    *taken = true;
    WgradParams a;
    a.x = source(p.x, p.channels, p.h, p.wd, p.pad_h, p.pad_w, l.hp, l.wp, l.rows);
    a.dy = source(p.dy, p.n, p.oh, p.ow, 0, 0, l.hp, l.wp, l.rows);
    a.tiles = (int)l.tiles;
    a.wp = (int)l.wp;
    a.fh = p.fh;
    a.fw = p.fw;
    a.products = l.products;
    a.x_rows = l.x_rows;
    a.dy_rows = l.dy_rows;
    a.stages = l.stages;
    a.partial = (float *)sums;
    a.status = dev->status_dev;
    const int status = l.rb == 32   ? l.rn == 32 ? launch_wgrad<32, 32>(dev, l, grid, a) : launch_wgrad<32, 64>(dev, l, grid, a)
                       : l.rb == 64 ? l.rn == 32 ? launch_wgrad<64, 32>(dev, l, grid, a) : launch_wgrad<64, 64>(dev, l, grid, a)
                       : l.rn == 32 ? launch_wgrad<128, 32>(dev, l, grid, a) : launch_wgrad<128, 64>(dev, l, grid, a);
    AG_TRY(status);
    // every column of the accumulators that is an output
    WgradSum s{(const float *)sums, grid, n, (int)p.channels, l.rb / 2, p.fh, p.fw, l.products, beta, dw, p.x, p.dy,
               (int)p.bs, (int)p.h, (int)p.wd, (int)p.oh, (int)p.ow, p.pad_h, p.pad_w, (int)p.n};
    return launch_dependent(dev, conv_halo_wgrad_sum_kernel,
                            dim3((unsigned)ceil_div((int64_t)p.fh * p.fw * p.channels, 32), (unsigned)p.n), dim3(32, W_ROWS), 0, s);
}

}  // namespace halo32
}  // namespace ag
