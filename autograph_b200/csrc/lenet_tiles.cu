// LeNet5 inference in bf16 on the tensor cores: a CTA takes tiles of 128 images from pixels to logits.
//
// Every layer is a product whose 128 rows are the tile's images; what an image's row holds is a window of its
// activations, and the weights are laid out as the banded matrix that maps a window to a block of
// outputs:
//   conv1: 8 columns of 6 rows (48 values) -> 4 x 2 outputs x 6 channels (N = 48), three k steps that are each
//          8 columns of a row pair; six blocks make a pooled row;
//   conv2: 8 columns x 6 channels of 5 rows (240 values) -> 4 outputs of one row x 8 channels (N = 32);
//   dense: the usual matrices.
// About half of the multiplied weights are structural zeros, which the tensor cores (4096 multiply-adds a
// clock) do not mind: the FFMA form spends 11 us on 7 images per SM, this one about as long on 128.
//
// Pixels come through shared memory (the window of a k step is 32 contiguous bytes of an image's row).
// From conv1's output on, the activations live in tensor memory only, where the accumulators' readers
// (a thread per image) put them as the next product's A operand, packed in pairs:
//   columns [0, 192)   accumulators: four buffers of 48 (conv1), two of 64 at the same places as two of those
//                      each (conv2), 128 for the dense layers
//   columns [192, 480) six rows of conv1's pooled output: 24 columns for pixels 0..7, 24 for pixels 4..11
//   columns [480, 512) pooled row 0 of conv2's output; rows 1 to 3 wait in registers until conv2 has read
//                      the last of conv1's rows, and take their place
// Warps 0-3 load pixels (two row pairs ahead), 4-19 (four sets, one per small buffer) turn accumulators into
// the next operand, 20 and 21 issue.  Reading accumulators is a chain of latencies (wait, load, maximum, pack,
// store), so warps count: with two sets a tile took 33 us.  The issuing thread is chosen by elect.sync and
// what varies between its operands is made warp-uniform first: behind a lane test, or with operands from
// ordinary registers, a tcgen05.mma takes 46-93 cycles to issue (measured), here about 10; the products
// themselves take 16 to 64.
//
// 0 x infinity is not 0: a tile with a pixel or an activation that is not finite is marked and its
// images are computed again by plain loops at the end.
//
// 65,536 images: 790 us as convolutions on the FP32 pipe and dense products over the batch.
#include <cuda_bf16.h>
#include <cstdlib>
#include <type_traits>

#include "lenet_tiles.cuh"
#include "tc_ptx.cuh"

namespace ag {
namespace lenet_tiles {

typedef __nv_bfloat16 bf16;

constexpr int kImages = 128, kSets = 4, kIssuer = 4 + 4 * kSets, kThreads = 32 * (kIssuer + 2);
constexpr int kPix = 784, kPairs = 14, kRows = 12;     // row pairs of an image, pooled rows after conv1
constexpr int D1 = 128, D2 = 84, D3 = 10, D2P = 96, D3P = 16;

// The weights as shared memory holds them: K-major rows of 64 values (128 bytes, swizzled), a block of rows
// per 64 k.
constexpr int B1_BYTES = 48 * 128, B2_CHUNK = 64 * 128, B2_BYTES = 4 * B2_CHUNK;
constexpr int W1_CHUNK = D1 * 128, W1_BYTES = 4 * W1_CHUNK, W2_CHUNK = D2P * 128, W2_BYTES = 2 * W2_CHUNK;
constexpr int W3_CHUNK = D3P * 128, W3_BYTES = 2 * W3_CHUNK;
constexpr int B1_OFF = 0, B2_OFF = B1_OFF + B1_BYTES, W1_OFF = B2_OFF + B2_BYTES, W2_OFF = W1_OFF + W1_BYTES;
constexpr int W3_OFF = W2_OFF + W2_BYTES, kBlob = W3_OFF + W3_BYTES;
// Pixels: four row pairs, two to a group of three blocks of 128-byte rows.  Windows 0..3 of pair i of a group are
// the four 32-byte pieces of block i, windows 4 and 5 half i of block 2.
constexpr int IN_OFF = kBlob, IN_BLOCK = kImages * 128, IN_GROUP = 3 * IN_BLOCK;
constexpr int BAR_OFF = IN_OFF + 2 * IN_GROUP, kSmem = BAR_OFF + 256;
static_assert(kSmem <= 227 * 1024 && kBlob % 1024 == 0, "shared memory");

constexpr uint32_t MID = 192, FLAT = 480;              // tensor memory columns

// Where the k step i of the dense layers that follows pooled row 0 lies: three to a slot of conv1's rows.
__host__ __device__ constexpr uint32_t late_columns(int i) { return MID + 48 * (i / 3) + 8 * (i % 3); }
// The first hidden layer (64 columns): slots 4 and 5, which hold none of those; the second (48): slot 0.
constexpr uint32_t HIDDEN = MID + 48 * 4;

enum Bar { W_FULL = 0, IN_FULL = 3, IN_EMPTY = 7, ACC_FULL = 11, ACC_EMPTY = 15, MID_FULL = 19, D_FULL = 25, A_READY = 26,
           ROW_DONE = 27, TILE_DONE = 28, kBars = 29 };

struct Args {
    const bf16 *x;
    bf16 *y;
    int bs;
    const unsigned char *blob;
    int *bad;                        // per tile: computed again by plain loops
    Weights w;
    int *status;
};

// ------------------------------------------------------------------------------ weights
// A value of row n, column k of a block of `rows` rows per 64 k.
__device__ __forceinline__ int place(int chunk_bytes, int n, int k) {
    return (k >> 6) * chunk_bytes + n * 128 + ((((k >> 3) & 7) ^ (n & 7)) << 4) + (k & 7) * 2;
}

__global__ void __launch_bounds__(256) pack_kernel(const Weights w, unsigned char *__restrict__ blob, int *bad, int tiles) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < tiles) bad[i] = 0;
    if (i >= kBlob / 2) return;
    const bf16 *c1 = (const bf16 *)w.conv1, *c2 = (const bf16 *)w.conv2;
    int at, j = i;
    bf16 v = __float2bfloat16(0.f);
    if (j < B1_BYTES / 2) {
        // n = (pooled column, channel, dy, dx), k = (row pair, row, column)
        const int n = j >> 6, k = j & 63, cell = n & 3, dy = cell >> 1, dx = cell & 1, oc = (n >> 2) % 6, px = (n >> 2) / 6;
        const int fi = (k >> 3) - dy, fj = (k & 7) - 2 * px - dx;
        if (k < 48 && fi >= 0 && fi < 5 && fj >= 0 && fj < 5) v = c1[(oc * 5 + fi) * 5 + fj];
        at = B1_OFF + place(B1_BYTES, n, k);
    } else if ((j -= B1_BYTES / 2) < B2_BYTES / 2) {
        // n = (channel half, pooled column, channel, dx), k = (filter row, column, input channel)
        const int n = j >> 8, k = j & 255, dx = n & 1, oc = (n >> 5) * 8 + ((n >> 1) & 7), px = (n >> 4) & 1;
        const int fi = k / 48, r = k - fi * 48, ci = r % 6, fj = r / 6 - 2 * px - dx;
        if (fi < 5 && fj >= 0 && fj < 5) v = c2[((oc * 6 + ci) * 5 + fi) * 5 + fj];
        at = B2_OFF + place(B2_CHUNK, n, k);
    } else if ((j -= B2_BYTES / 2) < W1_BYTES / 2) {
        // k = (pooled row, column half, channel half, column, channel), as conv2's output is stored
        const int n = j >> 8, k = j & 255, q = k >> 6, h = (k >> 5) & 1, half = (k >> 4) & 1, px = 2 * h + ((k >> 3) & 1);
        const int oc = half * 8 + (k & 7);
        v = ((const bf16 *)w.dense[0])[(oc * 16 + q * 4 + px) * D1 + n];
        at = W1_OFF + place(W1_CHUNK, n, k);
    } else if ((j -= W1_BYTES / 2) < W2_BYTES / 2) {
        const int n = j >> 7, k = j & 127;
        if (n < D2) v = ((const bf16 *)w.dense[1])[k * D2 + n];
        at = W2_OFF + place(W2_CHUNK, n, k);
    } else {
        j -= W2_BYTES / 2;
        const int n = j >> 7, k = j & 127;
        if (n < D3 && k < D2) v = ((const bf16 *)w.dense[2])[k * D3 + n];
        at = W3_OFF + place(W3_CHUNK, n, k);
    }
    *reinterpret_cast<bf16 *>(blob + at) = v;
}

// ----------------------------------------------------------------------------------- PTX
// The same value in every lane, known as such to the compiler.
__device__ __forceinline__ uint32_t uniform(uint32_t v) { return __shfl_sync(0xffffffffu, v, 0); }

// Matrix descriptors are built from their low word (address >> 4) where they are used; the high word is
// the same for all: 1024 bytes between eight-row groups, version 1, 128-byte swizzle.
constexpr uint32_t kDescHigh = 64u | 1u << 14 | 2u << 29;

__device__ __forceinline__ void umma_ss(uint32_t d, uint32_t a_low, uint32_t b_low, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        ".reg .b64 da, db;\n"
        "mov.b64 da, {%1, %5};\n"
        "mov.b64 db, {%2, %5};\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n"
        "}\n" ::"r"(d),
        "r"(a_low), "r"(b_low), "r"(idesc), "r"(accumulate), "n"(kDescHigh)
        : "memory");
}
__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a_tmem, uint32_t b_low, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        ".reg .b64 db;\n"
        "mov.b64 db, {%2, %5};\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p;\n"
        "}\n" ::"r"(d),
        "r"(a_tmem), "r"(b_low), "r"(idesc), "r"(accumulate), "n"(kDescHigh)
        : "memory");
}
__device__ __forceinline__ void st2(uint32_t t, const uint32_t *r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(t), "r"(r[0]), "r"(r[1]) : "memory");
}
__device__ __forceinline__ void ld8(uint32_t t, uint32_t *r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(t)
                 : "memory");
}
__device__ __forceinline__ void st4(uint32_t t, const uint32_t *r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(t), "r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3])
                 : "memory");
}
__device__ __forceinline__ void st8(uint32_t t, const uint32_t *r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(t), "r"(r[0]),
                 "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Relu and maximum of a pool window, before the rounding that the layer stores with: rounding keeps
// order, so the result is the same.
__device__ __forceinline__ float pool4(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    return fmaxf(fmaxf(fmaxf(__uint_as_float(a), __uint_as_float(b)), fmaxf(__uint_as_float(c), __uint_as_float(d))), 0.f);
}
__device__ __forceinline__ uint32_t pack(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&v);
}
__device__ __forceinline__ bool not_finite(uint32_t w) {
    return (w & 0x7f80u) == 0x7f80u || (w & 0x7f800000u) == 0x7f800000u;
}

// ------------------------------------------------------------------- images by plain loops
__device__ float relu_pool(const float *v) {
    float m = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float r = __bfloat162float(__float2bfloat16(v[i]));
        if (r > m) m = r;
    }
    return m;
}
__device__ __noinline__ void plain_image(const Args &a, int b, float *s) {
    float *x = s, *p1 = x + kPix, *f = p1 + 864, *h1 = f + 256, *h2 = h1 + D1;
    const int tid = threadIdx.x;
    const bf16 *c1 = (const bf16 *)a.w.conv1, *c2 = (const bf16 *)a.w.conv2;
    __syncthreads();
    for (int i = tid; i < kPix; i += kThreads) x[i] = __bfloat162float(a.x[(int64_t)b * kPix + i]);
    __syncthreads();
    for (int i = tid; i < 864; i += kThreads) {
        const int c = i / 144, r = i % 144, y = r / 12 * 2, xx = r % 12 * 2;
        float v[4];
        for (int cell = 0; cell < 4; ++cell) {
            float sum = 0.f;
            for (int t = 0; t < 25; ++t)
                sum = fmaf(x[(y + cell / 2 + t / 5) * 28 + xx + cell % 2 + t % 5], __bfloat162float(c1[c * 25 + t]), sum);
            v[cell] = sum;
        }
        p1[i] = relu_pool(v);
    }
    __syncthreads();
    for (int i = tid; i < 256; i += kThreads) {
        const int c = i / 16, y = i % 16 / 4 * 2, xx = i % 4 * 2;
        float v[4];
        for (int cell = 0; cell < 4; ++cell) {
            float sum = 0.f;
            for (int t = 0; t < 150; ++t)
                sum = fmaf(p1[t / 25 * 144 + (y + cell / 2 + t % 25 / 5) * 12 + xx + cell % 2 + t % 5],
                           __bfloat162float(c2[c * 150 + t]), sum);
            v[cell] = sum;
        }
        f[i] = relu_pool(v);
    }
    const float *in = f;
    for (int l = 0; l < 3; ++l) {
        __syncthreads();
        const int K = l == 0 ? 256 : l == 1 ? D1 : D2, N = l == 0 ? D1 : l == 1 ? D2 : D3;
        const bf16 *w = (const bf16 *)a.w.dense[l], *bias = (const bf16 *)a.w.bias[l];
        for (int n = tid; n < N; n += kThreads) {
            float sum = 0.f;
            for (int k = 0; k < K; ++k) sum = fmaf(in[k], __bfloat162float(w[k * N + n]), sum);
            float v = __bfloat162float(__float2bfloat16(sum));
            if (bias) v = __bfloat162float(__float2bfloat16(v + __bfloat162float(bias[n])));
            if (l == 2)
                a.y[(int64_t)b * D3 + n] = __float2bfloat16(v);
            else
                (l == 0 ? h1 : h2)[n] = v >= 0.f ? v : 0.f;
        }
        in = l == 0 ? h1 : h2;
    }
}

// --------------------------------------------------------------------------------- kernel
__global__ void __launch_bounds__(kThreads, 1) tile_kernel(const __grid_constant__ Args a) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const uint32_t base = tc::smem_u32(smem);
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    int *abort_flag = reinterpret_cast<int *>(smem + BAR_OFF + kBars * 8), *tmem_at = abort_flag + 1;
    const auto bar = [&](int i) { return base + BAR_OFF + 8 * (uint32_t)i; };
    const int tiles = (a.bs + kImages - 1) / kImages;

    if (threadIdx.x == 0) {
        *abort_flag = (base & 1023u) != 0;   // the swizzled layouts start on 1024-byte boundaries
        for (int i = 0; i < kBars; ++i) {
            const bool warps4 = (i >= IN_FULL && i < IN_EMPTY) || (i >= ACC_EMPTY && i < MID_FULL);
            const bool readers = (i >= MID_FULL && i < D_FULL) || i == A_READY;
            const bool issuers = (i >= IN_EMPTY && i < ACC_FULL) || i == ROW_DONE;
            tc::mbar_init(bar(i), warps4 ? 4 : readers ? 4 * kSets : issuers ? 2 : 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kIssuer) {
        tc::tmem_alloc(tc::smem_u32(tmem_at), 512);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = uniform(*reinterpret_cast<volatile uint32_t *>(tmem_at));
    const bool start = *reinterpret_cast<volatile int *>(abort_flag) == 0;
    if (!start && threadIdx.x == 0) atomicCAS(a.status, 0, 175);
    // Waits of warp-wide code: the lanes agree on the outcome, since it decides what the warp runs next.
    const auto wait = [&](int i, uint32_t parity) {
        return __all_sync(0xffffffffu, tc::mbar_wait(bar(i), parity, abort_flag)) != 0;
    };
    const auto arrive = [&](int i) {
        if (lane == 0) tc::mbar_arrive(bar(i));
    };

    bool ok = start;
    if (warp < 4) {
        // ------------------------------------------------------------------------- pixels
        const int img = threadIdx.x;
        uint4 v[2][7];
        // row pair `pair` of this CTA's i-th tile (pairs count on into the next tiles)
        const auto load = [&](int i, int pair, uint4 (&dst)[7]) {
            if (pair >= kPairs) {
                pair -= kPairs;
                ++i;
            }
            const int64_t b = ((int64_t)blockIdx.x + (int64_t)i * gridDim.x) * kImages + img;
#pragma unroll
            for (int q = 0; q < 7; ++q)
                dst[q] = b < a.bs ? __ldg(reinterpret_cast<const uint4 *>(a.x + b * kPix + pair * 56) + q)
                                  : make_uint4(0, 0, 0, 0);
        };
        if (ok) {
            load(0, 0, v[0]);
            load(0, 1, v[1]);
        }
        uint32_t g = 0;
        int i = 0;
        for (int tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x, ++i) {
            bool bad = false;
            for (int pair = 0; ok && pair < kPairs; pair += 2) {
#pragma unroll
                for (int half = 0; half < 2; ++half, ++g) {
                    const uint32_t slot = g & 3;   // its low bit is `half`
                    if (!(ok = wait(IN_EMPTY + slot, ((g >> 2) & 1) ^ 1))) break;
                    const auto w = [&](int n) {
                        const uint4 &q = v[half][n >> 2];
                        return (n & 3) == 0 ? q.x : (n & 3) == 1 ? q.y : (n & 3) == 2 ? q.z : q.w;
                    };
                    const uint32_t group = IN_OFF + (slot >> 1) * IN_GROUP + img * 128;
#pragma unroll
                    for (int b = 0; b < 6; ++b) {
                        const uint32_t block = b < 4 ? half : 2, piece = b < 4 ? 2 * b : 4 * half + 2 * (b - 4);
#pragma unroll
                        for (int r = 0; r < 2; ++r)
                            *reinterpret_cast<uint4 *>(smem + group + block * IN_BLOCK + (((piece + r) ^ (img & 7)) << 4)) =
                                make_uint4(w(14 * r + 2 * b), w(14 * r + 2 * b + 1), w(14 * r + 2 * b + 2), w(14 * r + 2 * b + 3));
                    }
#pragma unroll
                    for (int q = 0; q < 28; ++q) bad |= not_finite(w(q));
                    load(i, pair + half + 2, v[half]);
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    arrive(IN_FULL + slot);
                }
            }
            if (bad) a.bad[tile] = 1;
        }
    } else if (warp < kIssuer) {
        // ---------------------------------------------------------- accumulators -> operands
        const int set = (warp - 4) >> 2;
        const uint32_t t = tmem + ((uint32_t)(warp & 3) << 21);   // lanes 32 * (warp % 4) ..
        const uint32_t acc = t + 48 * set;
        uint32_t phase = 0, dense = 0, rows_done = 0;
        for (int tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x) {
            uint32_t held[5][4];   // conv2's pooled rows 1 and 2, left half of row 3
            __nv_bfloat162 top = __floats2bfloat162_rn(0.f, 0.f);
            // conv2's pooled row Q: sets 0 and 1 have channels 0..7, 2 and 3 the others, each set one column
            // of each half
            const auto pooled_row = [&](auto row) {
                constexpr int Q = decltype(row)::value;
                const uint32_t from = t + 96 * (set >> 1) + 16 * (set & 1), word = 4 * (set & 1);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (!(ok = wait(ACC_FULL + set, phase))) return;
                    phase ^= 1;
                    tc::tc_fence_after();
                    uint32_t r[32], now[4];
                    uint32_t *o = Q == 0 || (Q == 3 && h == 1) ? now : held[2 * (Q - 1) + h];
                    tc::tmem_ld_32x16(from, r);
                    tc::tmem_ld_32x16(from + 32, r + 16);
                    tc::tmem_ld_wait();
                    tc::tc_fence_before();
                    __syncwarp();
                    arrive(ACC_EMPTY + set);
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        o[i] = pack(pool4(r[4 * i], r[4 * i + 1], r[16 + 4 * i], r[16 + 4 * i + 1]),
                                    pool4(r[4 * i + 2], r[4 * i + 3], r[16 + 4 * i + 2], r[16 + 4 * i + 3]));
                    if (Q == 0) st4(t + FLAT + 16 * h + 8 * (set >> 1) + word, o);
                    if (Q == 3 && h == 1) {
                        // conv2 has read the last of conv1's rows
                        if (!(ok = wait(ROW_DONE, rows_done++ & 1))) return;
                        tc::tc_fence_after();
#pragma unroll
                        for (int c = 0; c < 5; ++c) st4(t + late_columns(2 * c + (set >> 1)) + word, held[c]);
                        st4(t + late_columns(10 + (set >> 1)) + word, o);
                    }
                }
            };
            for (int p = 0; ok && p < kRows; ++p) {
                const uint32_t mid = t + MID + 48 * (p % 6);
                // conv2's last pooled row has read the slots of this row and the next
                if (p >= 6 && (p & 1) == 0) {
                    if (!(ok = wait(ROW_DONE, rows_done++ & 1))) break;
                    tc::tc_fence_after();
                }
                // conv1's blocks go round the sets
#pragma unroll 1
                for (int b = (set - 6 * p) & 3; b < 6; b += 4) {
                    if (!(ok = wait(ACC_FULL + set, phase))) break;
                    phase ^= 1;
                    tc::tc_fence_after();
                    uint32_t r[48], o[6];
#pragma unroll
                    for (int i = 0; i < 48; i += 16) tc::tmem_ld_32x16(acc + i, r + i);
                    tc::tmem_ld_wait();
                    tc::tc_fence_before();
                    __syncwarp();
                    arrive(ACC_EMPTY + set);
#pragma unroll
                    for (int i = 0; i < 6; ++i) {
                        o[i] = pack(pool4(r[8 * i], r[8 * i + 1], r[8 * i + 2], r[8 * i + 3]),
                                    pool4(r[8 * i + 4], r[8 * i + 5], r[8 * i + 6], r[8 * i + 7]));
                        top = __hmax2(top, *reinterpret_cast<const __nv_bfloat162 *>(&o[i]));
                    }
                    if (b < 4) {
                        st4(mid + 6 * b, o);
                        st2(mid + 6 * b + 4, o + 4);
                    }
                    if (b >= 2) {
                        st4(mid + 24 + 6 * (b - 2), o);
                        st2(mid + 24 + 6 * (b - 2) + 4, o + 4);
                    }
                }
                if (!ok) break;
                st_wait();
                tc::tc_fence_before();
                __syncwarp();
                arrive(MID_FULL + p % 6);
                if (p == 5)
                    pooled_row(std::integral_constant<int, 0>());
                else if (p == 7)
                    pooled_row(std::integral_constant<int, 1>());
                else if (p == 9)
                    pooled_row(std::integral_constant<int, 2>());
                else if (p == 11)
                    pooled_row(std::integral_constant<int, 3>());
            }
            if (!ok) break;
            if (not_finite(*reinterpret_cast<const uint32_t *>(&top))) a.bad[tile] = 1;
            st_wait();
            tc::tc_fence_before();
            __syncwarp();
            arrive(A_READY);
            // ---- dense layers: a quarter of the columns each
            const int b = tile * kImages + (warp & 3) * 32 + lane;
            const auto dense_value = [&](uint32_t r, const bf16 *bias, int n, int N) {
                float v = __bfloat162float(__float2bfloat16(__uint_as_float(r)));
                if (bias != nullptr && n < N) v = __bfloat162float(__float2bfloat16(v + __bfloat162float(bias[n])));
                return v;
            };
            if (!(ok = wait(D_FULL, dense++ & 1))) break;
            tc::tc_fence_after();
            {
                const bf16 *bias = (const bf16 *)a.w.bias[0];
                uint32_t r[32], o[16];
                tc::tmem_ld_32x16(t + 32 * set, r);
                tc::tmem_ld_32x16(t + 32 * set + 16, r + 16);
                tc::tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    o[i] = pack(fmaxf(dense_value(r[2 * i], bias, 32 * set + 2 * i, D1), 0.f),
                                fmaxf(dense_value(r[2 * i + 1], bias, 32 * set + 2 * i + 1, D1), 0.f));
                st8(t + HIDDEN + 16 * set, o);
                st8(t + HIDDEN + 16 * set + 8, o + 8);
            }
            st_wait();
            tc::tc_fence_before();
            __syncwarp();
            arrive(A_READY);
            if (!(ok = wait(D_FULL, dense++ & 1))) break;
            tc::tc_fence_after();
            {
                const bf16 *bias = (const bf16 *)a.w.bias[1];
                uint32_t r[24], o[12];
#pragma unroll
                for (int i = 0; i < 24; i += 8) ld8(t + 24 * set + i, r + i);
                tc::tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 12; ++i)
                    o[i] = pack(fmaxf(dense_value(r[2 * i], bias, 24 * set + 2 * i, D2), 0.f),
                                fmaxf(dense_value(r[2 * i + 1], bias, 24 * set + 2 * i + 1, D2), 0.f));
#pragma unroll
                for (int i = 0; i < 12; i += 4) st4(t + MID + 12 * set + i, o + i);
            }
            st_wait();
            tc::tc_fence_before();
            __syncwarp();
            arrive(A_READY);
            if (!(ok = wait(D_FULL, dense++ & 1))) break;
            tc::tc_fence_after();
            if (set == 0) {
                const bf16 *bias = (const bf16 *)a.w.bias[2];
                uint32_t r[16];
                tc::tmem_ld_32x16(t, r);
                tc::tmem_ld_wait();
                if (b < a.bs) {
                    uint32_t *y = reinterpret_cast<uint32_t *>(a.y + (int64_t)b * D3);
#pragma unroll
                    for (int i = 0; i < 5; ++i)
                        y[i] = pack(dense_value(r[2 * i], bias, 2 * i, D3), dense_value(r[2 * i + 1], bias, 2 * i + 1, D3));
                }
            }
            tc::tc_fence_before();
            __syncwarp();
            arrive(A_READY);
        }
    } else {
        // ---------------------------------------------------------------------- tensor cores
        // One thread of each of two warps, so a wait leads straight to the next issue: `side` 0 fills the buffers
        // of sets 0 and 1 and issues the dense layers, side 1 those of sets 2 and 3.  With one thread for
        // all, the 300 cycles from a wait to its commit, 72 times a tile, bound conv1 (28 us a tile).
        const int side = warp - kIssuer;
        const uint32_t b1 = (base + B1_OFF) >> 4, b2 = (base + B2_OFF) >> 4, w1 = (base + W1_OFF) >> 4;
        const uint32_t w2 = (base + W2_OFF) >> 4, w3 = (base + W3_OFF) >> 4;
        if (ok && tc::elect_one()) {
            const auto wait1 = [&](int i, uint32_t parity) { return tc::mbar_wait(bar(i), parity, abort_flag); };
            const int off[3] = {B1_OFF, B2_OFF, W1_OFF}, bytes[3] = {B1_BYTES, B2_BYTES, kBlob - W1_OFF};
#pragma unroll
            for (int i = 0; i < 3 && side == 0; ++i) {
                tc::mbar_arrive_expect_tx(bar(W_FULL + i), (uint32_t)bytes[i]);
                tc::bulk_load(base + off[i], a.blob + off[i], (uint32_t)bytes[i], bar(W_FULL + i));
            }
            constexpr uint32_t id48 = tc::make_idesc(false, false, 128, 48), id32 = tc::make_idesc(false, false, 128, 32);
            constexpr uint32_t id128 = tc::make_idesc(false, false, 128, D1), id96 = tc::make_idesc(false, false, 128, D2P);
            constexpr uint32_t id16 = tc::make_idesc(false, false, 128, D3P);
            uint32_t g = 0, mids = 0, ready = 0;
            uint32_t free_phase = 3;   // of this side's two ACC_EMPTY, a bit each
            bool first = true;
            for (int tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x) {
                if (first) ok = wait1(W_FULL, 0);
#pragma unroll 1
                for (int p2 = 0; ok && p2 < kRows; p2 += 2) {
#pragma unroll
                    for (int odd = 0; odd < 2; ++odd) {
                        const int p = p2 + odd;
                        // row p reads row pairs p, p + 1, p + 2
                        if (p2 == 0 && odd == 0) ok = wait1(IN_FULL + (g & 3), (g >> 2) & 1) && wait1(IN_FULL + ((g + 1) & 3), ((g + 1) >> 2) & 1);
                        ok = ok && wait1(IN_FULL + ((g + p + 2) & 3), ((g + p + 2) >> 2) & 1);
                        if (!ok) break;
                        uint32_t left[3], right[3];
#pragma unroll
                        for (int i = 0; i < 3; ++i) {
                            const uint32_t slot = (g + p + i) & 3;
                            left[i] = (base + IN_OFF + (slot >> 1) * IN_GROUP + (slot & 1) * IN_BLOCK) >> 4;
                            right[i] = (base + IN_OFF + (slot >> 1) * IN_GROUP + 2 * IN_BLOCK + (slot & 1) * 64) >> 4;
                        }
                        // blocks go round the four buffers, so this side has 0, 1, 4, 5 of one row of a pair
                        // and 2, 3 of the other
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            if (j >= 2 && odd != side) break;
                            const int b = odd == side ? (j < 2 ? j : j + 2) : 2 + j, k = j & 1;
                            if (!(ok = wait1(ACC_EMPTY + 2 * side + k, (free_phase >> k) & 1))) break;
                            free_phase ^= 1u << k;
                            tc::tc_fence_after();
                            const uint32_t d = tmem + 96 * side + 48 * k;
#pragma unroll
                            for (int i = 0; i < 3; ++i)
                                umma_ss(d, b < 4 ? left[i] + 2 * b : right[i] + 2 * (b - 4), b1 + 2 * i, id48, i > 0);
                            tc::umma_commit(bar(ACC_FULL + 2 * side + k));
                        }
                        if (!ok) break;
                        tc::umma_commit(bar(IN_EMPTY + ((g + p) & 3)));
                    }
                    if (!ok || p2 < 4) continue;
                    const int q = (p2 - 4) >> 1;
                    if (p2 == 10) {
                        tc::umma_commit(bar(IN_EMPTY + ((g + 12) & 3)));
                        tc::umma_commit(bar(IN_EMPTY + ((g + 13) & 3)));
                    }
                    if (first && q == 0 && !(ok = wait1(W_FULL + 1, 0))) break;
                    // each of the six row slots is filled twice per tile
                    for (int row = q == 0 ? 0 : p2; ok && row <= p2 + 1; ++row) ok = wait1(MID_FULL + row % 6, (mids + row / 6) & 1);
                    if (!ok) break;
                    uint32_t rows[6];
#pragma unroll
                    for (int i = 0; i < 6; ++i) rows[i] = tmem + MID + 48 * ((2 * q + i) % 6);
#pragma unroll 1
                    for (int h = 0; h < 2; ++h) {
                        // a large buffer is two small ones, read by both sets
                        if (!(ok = wait1(ACC_EMPTY + 2 * side, free_phase & 1))) break;
                        if (!(ok = wait1(ACC_EMPTY + 2 * side + 1, free_phase >> 1))) break;
                        free_phase ^= 3u;
                        tc::tc_fence_after();
                        const uint32_t d = tmem + 96 * side, w = b2 + 256 * side;
#pragma unroll
                        for (int dy = 0; dy < 2; ++dy)
#pragma unroll
                            for (int s = 0; s < 15; ++s)
                                umma_ts(d + 32 * dy, rows[dy + s / 3] + 24 * h + 8 * (s % 3),
                                        w + (s >> 2) * (B2_CHUNK / 16) + 2 * (s & 3), id32, s > 0);
                        tc::umma_commit(bar(ACC_FULL + 2 * side));
                        tc::umma_commit(bar(ACC_FULL + 2 * side + 1));
                    }
                    if (ok) tc::umma_commit(bar(ROW_DONE));
                }
                if (!ok) break;
                g += kPairs;
                mids += 2;
                if (first && !(ok = wait1(W_FULL + 2, 0))) break;
                first = false;
                if (side == 1) {   // side 0 issues the dense layers
                    ok = wait1(TILE_DONE, ready++ & 1);
                    tc::tc_fence_after();
                    continue;
                }
                // the accumulators are free when the flattened rows are complete
                if (!(ok = wait1(A_READY, ready++ & 1))) break;
                tc::tc_fence_after();
#pragma unroll
                for (int s = 0; s < 16; ++s)
                    umma_ts(tmem, tmem + (s < 4 ? FLAT + 8 * s : late_columns(s - 4)), w1 + (s >> 2) * (W1_CHUNK / 16) + 2 * (s & 3),
                            id128, s > 0);
                tc::umma_commit(bar(D_FULL));
                if (!(ok = wait1(A_READY, ready++ & 1))) break;
                tc::tc_fence_after();
#pragma unroll
                for (int s = 0; s < 8; ++s)
                    umma_ts(tmem, tmem + HIDDEN + 8 * s, w2 + (s >> 2) * (W2_CHUNK / 16) + 2 * (s & 3), id96, s > 0);
                tc::umma_commit(bar(D_FULL));
                if (!(ok = wait1(A_READY, ready++ & 1))) break;
                tc::tc_fence_after();
#pragma unroll
                for (int s = 0; s < 6; ++s)
                    umma_ts(tmem, tmem + MID + 8 * s, w3 + (s >> 2) * (W3_CHUNK / 16) + 2 * (s & 3), id16, s > 0);
                tc::umma_commit(bar(D_FULL));
                ok = wait1(A_READY, ready++ & 1);
                tc::tc_fence_after();
                if (ok) tc::mbar_arrive(bar(TILE_DONE));
            }
            if (!ok) {   // a bounded wait for the weight copies in flight
                int none = 0;
                for (int i = 0; i < 3; ++i) tc::mbar_wait_for(bar(W_FULL + i), 0, &none, 100000000ull);
                atomicCAS(a.status, 0, 176);
            }
        }
        __syncwarp();
    }
    if (!ok && start && lane == 0) atomicCAS(a.status, 0, 176);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    if (warp == kIssuer) tc::tmem_dealloc(tmem, 512);
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        if (*reinterpret_cast<volatile int *>(a.bad + tile) == 0) continue;
        for (int b = tile * kImages; b < min(a.bs, (tile + 1) * kImages); ++b)
            plain_image(a, b, reinterpret_cast<float *>(smem));
    }
}

// ----------------------------------------------------------------------------------- host
bool takes(const ag_device *dev, const void *x, const void *y, int64_t bs) {
    // From about half a tile per SM on.  Below, the FFMA kernel gives the bits of the layers run one by
    // one, which callers compare; a single wave of tiles takes as long as 1000 images there.
    if (bs < (int64_t)kImages / 2 * dev->sm_count || bs >= (1 << 30)) return false;
    const char *e = getenv("AG_LENET_TILES");   // 0: off, for comparisons
    return !(e && e[0] == '0') && (reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(y) & 3) == 0;
}

int forward(ag_device *dev, const void *x, int64_t bs, const Weights &w, void *y) {
    const int tiles = (int)ceil_div(bs, (int64_t)kImages);
    void *ws = nullptr;
    AG_TRY(workspace(dev, kBlob + (size_t)tiles * sizeof(int), &ws));
    Args a;
    a.x = (const bf16 *)x;
    a.y = (bf16 *)y;
    a.bs = (int)bs;
    a.blob = (const unsigned char *)ws;
    a.bad = (int *)((char *)ws + kBlob);
    a.w = w;
    a.status = dev->status_dev;
    const int threads = tiles > kBlob / 2 ? tiles : kBlob / 2;
    pack_kernel<<<(unsigned)ceil_div(threads, 256), 256, 0, dev->stream>>>(w, (unsigned char *)ws, a.bad, tiles);
    AG_CHECK_LAUNCH();
    static SmemAllowed allowed;
    AG_TRY(allow_smem<kSmem>(dev, tile_kernel, allowed));
    tile_kernel<<<(unsigned)(tiles < dev->sm_count ? tiles : dev->sm_count), kThreads, kSmem, dev->stream>>>(a);
    AG_CHECK_LAUNCH();
    return AG_OK;
}

}  // namespace lenet_tiles
}  // namespace ag
