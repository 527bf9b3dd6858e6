// The first stage of a network on images: a convolution with few input channels, Relu and a 2 x 2 max pool, bf16.
//
// Layer by layer such a stage is memory traffic: with 256 x 3 x 64 x 64 images and 64 3 x 3 filters the convolution's
// output is 126 MB, the image 6 MB and the pooled output 31 MB, and patches, convolution, Relu + pool, their gradient
// and the weight gradient pass over a tensor of the large size seven times.  Here none of those tensors exists.
//
// Forward.  A tile is 128 pool windows (of the whole batch, in order) by 64 output channels.  The filter's k values
// (channel, row, column; padded to KP) are a row of the A operand, and the four cells of the windows are four
// products into four accumulators of the same tile, so a window's four sums meet in the registers of one thread,
// which adds the bias, applies Relu, pools, and stores the pooled value and the code of the winning cell.
//   Producers: one thread per window reads the window's (FH + 1) x (FW + 1) pixels of every channel and writes the four
//   patches, which overlap, from those registers.  Operands lie in 16-byte rows without swizzle,
//   [8 values of k][window][8]: a warp's stores are 512 consecutive bytes.
//
// Backward.  dw[oc][k] and db[oc]: the reduction runs over windows and cells.
// The operand of a cell is the pooled gradient where the code names that cell and zero elsewhere, written by the
// producers to [window][64 channels] rows (MN-major); the patches are the same rows as in the forward pass, read
// MN-major.  Two cells share an instruction: rows 0 - 63 of A are cell 2j's channels, rows 64 - 127 cell 2j + 1's, the
// columns of B the patches of both; the two diagonal blocks of the accumulator are wanted, and the instruction
// costs what one of half its rows does.  The bias gradient is added in registers by the producers: as a product with a
// k value of 1 it was a sum of all of a CTA's windows in one accumulator, which adds with truncation (1024 images of 64 x
// 64, 831 additions: more than 4e-6 of a value short, and the more the more images; a training step of a network of this
// stage and a dense layer, 256 images, takes 209 us either way).  Every CTA leaves its sums; a second kernel adds them in
// order.
//
// Measured at 256 x 3 x 64 x 64 -> 64, each kernel alone with cold caches: forward 23 us (patches, convolution and Relu +
// pool as kernels of their own 38 + 57 + 23), backward 27 + 6 (pool gradient 30, weight gradient and its sum 47); a training
// step of the wide stack 480 -> 345 us, inference 201 -> 105.  What bounds them is instructions with few warps to hide their
// latency (schedulers issue in 44 % and 38 % of the cycles); the bytes would take 7 us each.
#include "image_stage.cuh"
#include "pool_codes.cuh"
#include "tc_ptx.cuh"

namespace ag {
namespace image_stage {

using namespace ::ag::tc;

namespace {

// One geometry: the values of k, and the pixels of a window's four patches as pairs along the row.
template <int IC_, int F_>
struct Geo {
    static constexpr int IC = IC_, F = F_;
    static constexpr int K = IC * F * F;
    static constexpr int KP = (K + 1 + 15) / 16 * 16;   // a sum's column K is the bias gradient
    static constexpr int G = KP / 8;
    static constexpr int ROWS = F + 1, WORDS = (F + 1) / 2;
    static_assert(F % 2 == 1, "pairs of pixels");
    uint32_t v[IC][ROWS][WORDS];

    // `px`: the window's first pixel.  PAIRS: pairs of pixels start at 4-byte addresses.
    template <bool PAIRS>
    __device__ __forceinline__ void load(const unsigned short *px, int64_t plane, int iw) {
#pragma unroll
        for (int c = 0; c < IC; ++c)
#pragma unroll
            for (int r = 0; r < ROWS; ++r)
#pragma unroll
                for (int w = 0; w < WORDS; ++w) {
                    const unsigned short *p = px + c * plane + r * iw + 2 * w;
                    if (PAIRS)
                        v[c][r][w] = __ldg(reinterpret_cast<const uint32_t *>(p));
                    else
                        v[c][r][w] = (uint32_t)__ldg(p) | ((uint32_t)__ldg(p + 1) << 16);
                }
    }
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int c = 0; c < IC; ++c)
#pragma unroll
            for (int r = 0; r < ROWS; ++r)
#pragma unroll
                for (int w = 0; w < WORDS; ++w) v[c][r][w] = 0;
    }
    // Values k and k + 1 of cell (dy, dx)'s patch; all arguments are known when this is compiled.
    __device__ __forceinline__ uint32_t pair(int dy, int dx, int k) const {
        auto word = [&](int k) { return v[k / (F * F)][dy + k / F % F][(dx + k % F) / 2]; };
        const int s0 = (dx + k % F) % 2 ? 0x32 : 0x10, s1 = (dx + (k + 1) % F) % 2 ? 0x7600 : 0x5400;
        if (k + 1 < K) return __byte_perm(word(k), word(k + 1), s0 | s1);
        return k < K ? __byte_perm(word(k), 0u, s0 | 0x5400) : 0u;
    }
    // The four patches: cell c's group g of this window at dst + (c * G + g) * pitch.
    __device__ __forceinline__ void store(uint8_t *dst, int pitch) const {
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int g = 0; g < G; ++g)
                *reinterpret_cast<uint4 *>(dst + (c * G + g) * pitch) =
                    make_uint4(pair(c / 2, c % 2, 8 * g), pair(c / 2, c % 2, 8 * g + 2), pair(c / 2, c % 2, 8 * g + 4),
                               pair(c / 2, c % 2, 8 * g + 6));
    }
};

struct Params {
    const unsigned short *x;
    int64_t plane, image;   // elements of a channel and of an image
    int iw, oc, pairs;
    int windows, tiles;
    FastDiv per_image, per_row;
    int *status;
};

// First pixel of window `win`.
__device__ __forceinline__ const unsigned short *window_pixel(const Params &p, int win) {
    uint32_t b, r, py, px;
    p.per_image.divmod((uint32_t)win, b, r);
    p.per_row.divmod(r, py, px);
    return p.x + b * p.image + (int64_t)(2 * py) * p.iw + 2 * px;
}

template <class P>
__device__ __forceinline__ void load_window(P &patch, const Params &p, int win) {
    if (win >= p.windows)
        patch.clear();
    else if (p.pairs)
        patch.template load<true>(window_pixel(p, win), p.plane, p.iw);
    else
        patch.template load<false>(window_pixel(p, win), p.plane, p.iw);
}

// Descriptor of an operand without swizzle: 8 x 16-byte core matrices.
__device__ __forceinline__ uint64_t plain_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return make_smem_desc(addr, lbo, sbo) & ~(7ull << 61);
}

// This thread's shared-memory writes are for the tensor cores; one arrival per warp.
__device__ __forceinline__ void publish(uint32_t bar) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (threadIdx.x % 32 == 0) mbar_arrive(bar);
}

// ------------------------------------------------------------------- forward
constexpr int F_TILE = 128, F_STAGES = 2;
constexpr int F_EPI = 8, F_PROD = 8;   // warps; the producers are two teams that take turns
constexpr int F_THREADS = (F_EPI + F_PROD + 1) * 32;
constexpr int kMostChannels = 256;

template <class P>
constexpr int f_stage_bytes() { return 4 * P::KP * F_TILE * 2; }

template <class P>
__global__ void __launch_bounds__(F_THREADS, 1)
    image_stage_kernel(const Params p, const __nv_bfloat16 *__restrict__ w, const __nv_bfloat16 *__restrict__ bias,
                       __nv_bfloat16 *__restrict__ y, uint32_t *__restrict__ codes) {
    constexpr int STAGE = f_stage_bytes<P>();
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t *filters = smem + F_STAGES * STAGE;                    // [k group][oc][8]
    __shared__ uint64_t full_bar[F_STAGES], empty_bar[F_STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_word;
    __shared__ uint32_t s_bias[kMostChannels / 2];
    volatile int *abort_flag = &abort_word;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;

    if (threadIdx.x == 0) {
        for (int s = 0; s < F_STAGES; ++s) {
            mbar_init(smem_u32(&full_bar[s]), F_PROD / 2);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(smem_u32(&acc_full[s]), 1);
            mbar_init(smem_u32(&acc_empty[s]), F_EPI);
        }
        abort_word = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == F_EPI + F_PROD) {
        tmem_alloc(smem_u32(&tmem_slot), 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    let_dependents_launch();
    dependency_wait();
    for (int i = threadIdx.x; i < P::G * p.oc; i += F_THREADS) {
        const int g = i / p.oc, n = i - g * p.oc;
        uint32_t q[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int k = g * 8 + 2 * e;
            const uint32_t lo = k < P::K ? __bfloat16_as_ushort(w[n * P::K + k]) : 0u;
            const uint32_t hi = k + 1 < P::K ? __bfloat16_as_ushort(w[n * P::K + k + 1]) : 0u;
            q[e] = lo | (hi << 16);
        }
        reinterpret_cast<uint4 *>(filters)[i] = make_uint4(q[0], q[1], q[2], q[3]);
    }
    if (bias != nullptr)
        for (int i = threadIdx.x; i < p.oc / 2; i += F_THREADS)
            s_bias[i] = __bfloat16_as_ushort(bias[2 * i]) | ((uint32_t)__bfloat16_as_ushort(bias[2 * i + 1]) << 16);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();

    if (warp >= F_EPI && warp < F_EPI + F_PROD) {
        const int team = (warp - F_EPI) / 4, row = (warp - F_EPI) % 4 * 32 + lane;
        static_assert(F_STAGES == 2, "a team owns a stage");
        uint32_t phase = 0;
        for (int tile = blockIdx.x + team * gridDim.x; tile < p.tiles; tile += 2 * gridDim.x, phase ^= 1) {
            P patch;
            load_window(patch, p, tile * F_TILE + row);
            if (!mbar_wait(smem_u32(&empty_bar[team]), phase ^ 1, abort_flag)) {
                if (lane == 0) atomicExch(p.status, 200);
                break;
            }
            patch.store(smem + team * STAGE + row * 16, F_TILE * 16);
            publish(smem_u32(&full_bar[team]));
        }
    } else if (warp == F_EPI + F_PROD) {
        if (elect_one()) {
            constexpr uint32_t idesc = make_idesc(false, false, F_TILE, 64);
            const uint32_t f_lbo = (uint32_t)p.oc * 16;
            uint32_t phase = 0, acc_phase = 0;
            int stage = 0, acc = 0;
            bool ok = true;
            for (int tile = blockIdx.x; ok && tile < p.tiles; tile += gridDim.x) {
                if (!mbar_wait(smem_u32(&full_bar[stage]), phase, abort_flag)) {
                    atomicExch(p.status, 201);
                    break;
                }
                for (int n0 = 0; n0 < p.oc; n0 += 64) {
                    if (!mbar_wait(smem_u32(&acc_empty[acc]), acc_phase ^ 1, abort_flag)) {
                        atomicExch(p.status, 202);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
#pragma unroll
                    for (int c = 0; c < 4; ++c)
#pragma unroll
                        for (int k = 0; k < P::KP / 16; ++k)
                            umma_bf16(tmem + acc * 256 + c * 64,
                                      plain_desc(smem_u32(smem + stage * STAGE) + (c * P::G + 2 * k) * F_TILE * 16,
                                                 F_TILE * 16, 128),
                                      plain_desc(smem_u32(filters) + 2 * k * f_lbo + n0 * 16, f_lbo, 128), idesc, k > 0);
                    umma_commit(smem_u32(&acc_full[acc]));
                    if (++acc == 2) {
                        acc = 0;
                        acc_phase ^= 1;
                    }
                }
                umma_commit(smem_u32(&empty_bar[stage]));
                if (++stage == F_STAGES) {
                    stage = 0;
                    phase ^= 1;
                }
            }
        }
        __syncwarp();
    } else {
        const int quarter = warp % 4, half = warp / 4;   // 32 windows, 32 of 64 channels
        const bool has_bias = bias != nullptr;
        uint32_t acc_phase = 0;
        int acc = 0;
        bool ok = true;
        for (int tile = blockIdx.x; ok && tile < p.tiles; tile += gridDim.x) {
            const int win = tile * F_TILE + quarter * 32 + lane;
            for (int n0 = 0; n0 < p.oc; n0 += 64) {
                if (!mbar_wait(smem_u32(&acc_full[acc]), acc_phase, abort_flag)) {
                    if (lane == 0) atomicExch(p.status, 203);
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t t = tmem + ((uint32_t)(quarter * 32) << 16) + acc * 256 + half * 32;
                const int ch0 = n0 + half * 32;
                uint32_t code[4];
#pragma unroll
                for (int part = 0; part < 2; ++part) {   // 16 channels
                    uint32_t r[4][16];
#pragma unroll
                    for (int c = 0; c < 4; ++c) tmem_ld_32x16(t + c * 64 + part * 16, r[c]);
                    tmem_ld_wait();
                    if (part == 1) {   // the accumulators are in registers
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(smem_u32(&acc_empty[acc]));
                    }
                    uint32_t o[8];
                    code[2 * part] = code[2 * part + 1] = 0;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const uint32_t b = has_bias ? s_bias[(ch0 + part * 16) / 2 + j] : 0u;
                        uint32_t cells[4];
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            // the sum rounded, the bias added, rounded again (two bf16 values' sum in one rounding
                            // is what a sum in f32 and a rounding give)
                            __nv_bfloat162 h =
                                __floats2bfloat162_rn(__uint_as_float(r[c][2 * j]), __uint_as_float(r[c][2 * j + 1]));
                            if (has_bias) h = __hadd2(h, *reinterpret_cast<const __nv_bfloat162 *>(&b));
                            cells[c] = *reinterpret_cast<const uint32_t *>(&h);
                        }
                        uint32_t c8;
                        o[j] = nhwc::relu_pool_pair(cells, c8);
                        code[2 * part + j / 4] |= c8 << (8 * (j % 4));
                    }
                    if (win < p.windows) {
                        uint4 *q = reinterpret_cast<uint4 *>(y + (int64_t)win * p.oc + ch0 + part * 16);
                        q[0] = make_uint4(o[0], o[1], o[2], o[3]);
                        q[1] = make_uint4(o[4], o[5], o[6], o[7]);
                    }
                }
                if (codes != nullptr && win < p.windows)
                    *reinterpret_cast<uint4 *>(codes + ((int64_t)win * p.oc + ch0) / 8) =
                        make_uint4(code[0], code[1], code[2], code[3]);
                if (++acc == 2) {
                    acc = 0;
                    acc_phase ^= 1;
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {   // products that were issued may still be running
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    if (warp == F_EPI + F_PROD) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

// ------------------------------------------------------------------ backward
constexpr int B_TILE = 64;
constexpr int B_GRAD = 8, B_PATCH = 4;   // producer warps of the gradients and of the patches (two teams)
constexpr int B_THREADS = (B_GRAD + B_PATCH + 1) * 32;
constexpr int B_ATOM = B_TILE * 64 * 2;   // one cell's [64 windows][64 channels]
template <class P>
struct BCfg {
    static constexpr int STAGE = 4 * B_ATOM + 4 * P::KP * B_TILE * 2;
    static constexpr int STAGES = P::KP == 32 ? 4 : 3;
    static constexpr int COLS = 2 * P::KP <= 64 ? 64 : 128;   // of tensor memory
};

// Mask of a pair of channels from bits 8j + 7 of `lo` and `hi`.
__device__ __forceinline__ uint32_t pair_mask(uint32_t lo, uint32_t hi, int j) {
    uint32_t m;   // a selector's top bit repeats the sign of its byte
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(m) : "r"(lo), "r"(hi), "r"(0xcc88u + 0x1111u * (uint32_t)j));
    return m;
}

// BIAS: with the bias gradient.
template <class P, bool BIAS>
__global__ void __launch_bounds__(B_THREADS, 1)
    image_stage_backward_kernel(const Params p, const __nv_bfloat16 *__restrict__ dy, const uint32_t *__restrict__ codes,
                                int blocks, float *__restrict__ partial) {
    using C = BCfg<P>;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ uint64_t full_bar[C::STAGES], empty_bar[C::STAGES], done_bar;
    __shared__ float s_db[B_GRAD][64];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_word;
    volatile int *abort_flag = &abort_word;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int n0 = (int)(blockIdx.x % blocks) * 64, split = (int)(blockIdx.x / blocks), splits = (int)(gridDim.x / blocks);

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::STAGES; ++s) {
            mbar_init(smem_u32(&full_bar[s]), B_GRAD + B_PATCH / 2);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        mbar_init(smem_u32(&done_bar), 1);
        abort_word = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == B_GRAD + B_PATCH) {
        tmem_alloc(smem_u32(&tmem_slot), C::COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    let_dependents_launch();
    dependency_wait();

    if (warp < B_GRAD) {
        // Two 16-byte pieces of the gradient per thread and tile, loaded two tiles ahead.
        const int row = warp * 4 + lane / 8, group = lane % 8;   // and row + 32
        uint4 g[2][2];
        uint32_t c[2][2];
        float db[8] = {};   // of the group's channels
        auto fetch = [&](int buf, int tile) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int win = tile * B_TILE + row + i * 32;
                g[buf][i] = make_uint4(0, 0, 0, 0);
                c[buf][i] = 0;
                if (tile < p.tiles && win < p.windows) {
                    const int64_t at = (int64_t)win * p.oc + n0 + group * 8;
                    g[buf][i] = __ldg(reinterpret_cast<const uint4 *>(dy + at));
                    c[buf][i] = __ldg(codes + at / 8);
                }
            }
        };
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        fetch(0, split);
        fetch(1, split + splits);
        for (int tile = split; ok && tile < p.tiles;) {
#pragma unroll
            for (int buf = 0; buf < 2; ++buf) {
                if (tile >= p.tiles) break;
                if (!mbar_wait(smem_u32(&empty_bar[stage]), phase ^ 1, abort_flag)) {
                    if (lane == 0) atomicExch(p.status, 204);
                    ok = false;
                    break;
                }
                uint8_t *base = smem + stage * C::STAGE;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int r = row + i * 32;
                    uint8_t *dst = base + r * 128 + ((group ^ (r & 7)) << 4);   // 128-byte swizzle
                    const uint4 v = g[buf][i];
#pragma unroll
                    for (int cell = 0; cell < 4; ++cell) {
                        // nibbles that are 4 | cell, as ones in their lowest bit
                        const uint32_t t = c[buf][i] ^ (0x44444444u + 0x11111111u * (uint32_t)cell);
                        const uint32_t hit = ~(t | (t >> 1) | (t >> 2)) & 0x11111111u;
                        const uint32_t lo = hit << 7, hi = hit << 3;
                        *reinterpret_cast<uint4 *>(dst + cell * B_ATOM) =
                            make_uint4(v.x & pair_mask(lo, hi, 0), v.y & pair_mask(lo, hi, 1), v.z & pair_mask(lo, hi, 2),
                                       v.w & pair_mask(lo, hi, 3));
                    }
                    if (!BIAS) continue;
                    const uint32_t passed = (c[buf][i] >> 2) & 0x11111111u, lo = passed << 7, hi = passed << 3;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint32_t pair = (&v.x)[j] & pair_mask(lo, hi, j);
                        db[2 * j] += __uint_as_float(pair << 16);
                        db[2 * j + 1] += __uint_as_float(pair & 0xffff0000u);
                    }
                }
                publish(smem_u32(&full_bar[stage]));
                fetch(buf, tile + 2 * splits);
                if (++stage == C::STAGES) {
                    stage = 0;
                    phase ^= 1;
                }
                tile += splits;
            }
        }
        if (BIAS) {
#pragma unroll
            for (int e = 0; e < 8; ++e) {   // lanes 8 apart have the same channels
                db[e] += __shfl_xor_sync(0xffffffffu, db[e], 8);
                db[e] += __shfl_xor_sync(0xffffffffu, db[e], 16);
                if (lane < 8) s_db[warp][group * 8 + e] = db[e];
            }
            asm volatile("bar.sync 1, %0;" ::"n"(B_GRAD * 32) : "memory");   // the producers of gradients
        }
        // the sums: rows 0 - 63 and columns below KP are the even cells', the others the odd ones'
        if (ok && warp < 4) {
            if (mbar_wait(smem_u32(&done_bar), 0, abort_flag)) {
                tc_fence_after();
                const int cell = warp / 2, oc = n0 + warp % 2 * 32 + lane;
                float bias_sum = 0.f;   // in the even cells' sums
                if (BIAS && cell == 0)
#pragma unroll
                    for (int i = 0; i < B_GRAD; ++i) bias_sum += s_db[i][warp % 2 * 32 + lane];
                float *dst = partial + ((int64_t)(2 * split + cell) * p.oc + oc) * P::KP;
#pragma unroll
                for (int k = 0; k < P::KP; k += 16) {
                    uint32_t r[16];
                    tmem_ld_32x16(tmem + ((uint32_t)(warp * 32) << 16) + cell * P::KP + k, r);
                    tmem_ld_wait();
                    if (k <= P::K && P::K < k + 16) r[P::K % 16] = __float_as_uint(bias_sum);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        reinterpret_cast<uint4 *>(dst + k)[j] = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
                }
            } else if (lane == 0) {
                atomicExch(p.status, 205);
            }
        }
    } else if (warp < B_GRAD + B_PATCH) {
        const int team = (warp - B_GRAD) / 2, row = warp % 2 * 32 + lane;
        int i = team;   // the CTA's i-th tile
        P patch;
        load_window(patch, p, min(split + team * splits, p.tiles) * B_TILE + row);
        for (int tile = split + team * splits; tile < p.tiles; tile += 2 * splits, i += 2) {
            const int stage = i % C::STAGES;
            if (!mbar_wait(smem_u32(&empty_bar[stage]), (uint32_t)(i / C::STAGES + 1) & 1u, abort_flag)) {
                if (lane == 0) atomicExch(p.status, 206);
                break;
            }
            patch.store(smem + stage * C::STAGE + 4 * B_ATOM + row * 16, B_TILE * 16);
            publish(smem_u32(&full_bar[stage]));
            load_window(patch, p, min(tile + 2 * splits, p.tiles) * B_TILE + row);
        }
    } else {
        if (elect_one()) {
            constexpr uint32_t idesc = make_idesc(true, true, 128, 2 * P::KP);
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int tile = split; tile < p.tiles; tile += splits) {
                if (!mbar_wait(smem_u32(&full_bar[stage]), phase, abort_flag)) {
                    atomicExch(p.status, 207);
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t a = smem_u32(smem + stage * C::STAGE), b = a + 4 * B_ATOM;
#pragma unroll
                for (int c = 0; c < 4; c += 2)
#pragma unroll
                    for (int k = 0; k < B_TILE / 16; ++k)
                        umma_bf16(tmem, make_smem_desc(a + c * B_ATOM + k * 16 * 128, B_ATOM, 1024),
                                  plain_desc(b + c * P::G * B_TILE * 16 + k * 16 * 16, 128, B_TILE * 16), idesc,
                                  tile > split || c > 0 || k > 0);
                umma_commit(smem_u32(&empty_bar[stage]));
                if (++stage == C::STAGES) {
                    stage = 0;
                    phase ^= 1;
                }
            }
            if (ok) umma_commit(smem_u32(&done_bar));
        }
        __syncwarp();
    }

    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {   // products that were issued may still be running
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    if (warp == B_GRAD + B_PATCH) {
        tc_fence_after();
        tmem_dealloc(tmem, C::COLS);
    }
}

// out[oc][t] = sum over planes, in a fixed order, of partial[plane][oc][first + t].  32 outputs by 32 rows of planes
// (with 8 rows 19 us of 296 planes that are not in L2); the rows' sums are added in row order.
constexpr int R_ROWS = 32;
__global__ void __launch_bounds__(32 * R_ROWS)
    image_stage_reduce_kernel(const float *__restrict__ partial, int planes, int oc, int kp, int first, int count,
                              __nv_bfloat16 *__restrict__ out) {
    let_dependents_launch(kAlwaysEarly);
    dependency_wait();
    __shared__ float part[R_ROWS][33];
    const int i = blockIdx.x * 32 + threadIdx.x;
    const bool live = i < oc * count;
    const int64_t plane = (int64_t)oc * kp;
    const float *src = partial + (live ? i / count * kp + first + i % count : 0);
    float s = 0.f;
    if (live)
        for (int z = threadIdx.y; z < planes; z += 10 * R_ROWS) {   // all of a thread's loads in flight
            float v[10];
#pragma unroll
            for (int j = 0; j < 10; ++j) v[j] = z + R_ROWS * j < planes ? src[(z + R_ROWS * j) * plane] : 0.f;
#pragma unroll
            for (int j = 0; j < 10; ++j) s += v[j];
        }
    part[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.y != 0 || !live) return;
#pragma unroll
    for (int r = 1; r < R_ROWS; ++r) s += part[r][threadIdx.x];
    out[i] = __float2bfloat16_rn(s);
}

// ---------------------------------------------------------------------- host
Params make_params(ag_device *dev, const Shape &s, const __nv_bfloat16 *x, int tile) {
    Params p;
    const int64_t ph = (s.ih - s.fh + 1) / 2, pw = (s.iw - s.fw + 1) / 2;
    p.x = reinterpret_cast<const unsigned short *>(x);
    p.plane = s.ih * s.iw;
    p.image = s.ic * p.plane;
    p.iw = (int)s.iw;
    p.oc = (int)s.oc;
    p.pairs = s.iw % 2 == 0 && (reinterpret_cast<uintptr_t>(x) & 3) == 0;
    p.windows = (int)(s.bs * ph * pw);
    p.tiles = (int)ceil_div(p.windows, tile);
    p.per_image = FastDiv((uint32_t)(ph * pw));
    p.per_row = FastDiv((uint32_t)pw);
    p.status = dev->status_dev;
    return p;
}

template <class P>
int run_forward(ag_device *dev, const Shape &s, const __nv_bfloat16 *x, const __nv_bfloat16 *w, const __nv_bfloat16 *bias,
                __nv_bfloat16 *y, uint32_t *codes) {
    const Params p = make_params(dev, s, x, F_TILE);
    constexpr int most = F_STAGES * f_stage_bytes<P>() + kMostChannels * P::KP * 2;
    constexpr int smem = most < kOneCtaPerSm ? kOneCtaPerSm : most;
    static SmemAllowed allowed;
    AG_TRY(allow_smem<smem>(dev, image_stage_kernel<P>, allowed));
    const int grid = p.tiles < dev->sm_count ? p.tiles : dev->sm_count;
    return launch_dependent(dev, image_stage_kernel<P>, dim3((unsigned)grid), F_THREADS, smem, p, w, bias, y, codes);
}

int splits_of(ag_device *dev, const Shape &s) {
    const int64_t windows = s.bs * ((s.ih - s.fh + 1) / 2) * ((s.iw - s.fw + 1) / 2);
    const int64_t tiles = ceil_div(windows, B_TILE), room = dev->sm_count / (s.oc / 64);
    return (int)(tiles < room ? tiles : room);
}

template <class P, bool BIAS>
int run_backward(ag_device *dev, const Shape &s, const __nv_bfloat16 *x, const __nv_bfloat16 *dy, const uint32_t *codes,
                 float *partial) {
    using C = BCfg<P>;
    const Params p = make_params(dev, s, x, B_TILE);
    constexpr int smem = C::STAGES * C::STAGE + 1024;
    static_assert(smem >= kOneCtaPerSm && smem <= 226 * 1024, "one CTA per SM");
    static SmemAllowed allowed;
    AG_TRY(allow_smem<smem>(dev, image_stage_backward_kernel<P, BIAS>, allowed));
    const int blocks = (int)(s.oc / 64), grid = splits_of(dev, s) * blocks;
    return launch_dependent(dev, image_stage_backward_kernel<P, BIAS>, dim3((unsigned)grid), B_THREADS, smem, p, dy, codes,
                            blocks, partial);
}

// `call` with the geometry's type, or -1.
template <class F>
int with_geometry(const Shape &s, F call) {
    if (s.fh == 3 && s.fw == 3) {
        if (s.ic == 2) return call(Geo<2, 3>{});
        if (s.ic == 3) return call(Geo<3, 3>{});
        if (s.ic == 4) return call(Geo<4, 3>{});
    } else if (s.fh == 5 && s.fw == 5) {
        if (s.ic == 1) return call(Geo<1, 5>{});
        if (s.ic == 2) return call(Geo<2, 5>{});
    }
    return -1;
}

int padded_k(const Shape &s) { return (int)((s.ic * s.fh * s.fw + 1 + 15) / 16 * 16); }

int reduce(ag_device *dev, const Shape &s, const float *partial, int first, int count, __nv_bfloat16 *out) {
    return launch_dependent(dev, image_stage_reduce_kernel, dim3((unsigned)ceil_div(s.oc * count, 32)), dim3(32, R_ROWS), 0, partial,
                            2 * splits_of(dev, s), (int)s.oc, padded_k(s), first, count, out);
}

}  // namespace

bool takes(const Shape &s) {
    const int64_t oh = s.ih - s.fh + 1, ow = s.iw - s.fw + 1;
    return with_geometry(s, [](auto) { return 1; }) == 1 && s.oc > 0 && s.oc % 64 == 0 && s.oc <= kMostChannels && oh >= 2 &&
           ow >= 2 && s.bs > 0 && s.iw < (int64_t(1) << 31) && s.bs * (oh / 2) * (ow / 2) < (int64_t(1) << 31) - F_TILE;
}

int forward(ag_device *dev, const Shape &s, const __nv_bfloat16 *x, const __nv_bfloat16 *w, const __nv_bfloat16 *bias,
            __nv_bfloat16 *y, uint32_t *codes) {
    AG_REQUIRE(takes(s), AG_ERR_UNSUPPORTED, "image stage: shape not taken");
    return with_geometry(s, [&](auto g) { return run_forward<decltype(g)>(dev, s, x, w, bias, y, codes); });
}

int64_t partial_floats(ag_device *dev, const Shape &s) { return 2ll * splits_of(dev, s) * s.oc * padded_k(s); }

int backward(ag_device *dev, const Shape &s, const __nv_bfloat16 *x, const __nv_bfloat16 *dy, const uint32_t *codes, bool bias,
             float *partial) {
    AG_REQUIRE(takes(s) && (s.ih - s.fh + 1) % 2 == 0 && (s.iw - s.fw + 1) % 2 == 0, AG_ERR_UNSUPPORTED,
               "image stage: shape not taken");
    return with_geometry(s, [&](auto g) {
        return bias ? run_backward<decltype(g), true>(dev, s, x, dy, codes, partial)
                    : run_backward<decltype(g), false>(dev, s, x, dy, codes, partial);
    });
}

int weight_gradient(ag_device *dev, const Shape &s, const float *partial, __nv_bfloat16 *dw) {
    return reduce(dev, s, partial, 0, (int)(s.ic * s.fh * s.fw), dw);
}

int bias_gradient(ag_device *dev, const Shape &s, const float *partial, __nv_bfloat16 *db) {
    return reduce(dev, s, partial, (int)(s.ic * s.fh * s.fw), 1, db);
}

}  // namespace image_stage
}  // namespace ag
