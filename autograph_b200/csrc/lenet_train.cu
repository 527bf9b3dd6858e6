// LeNet5 training: the forward pass, the loss and every gradient of a group of images by one CTA that
// keeps the activations in shared memory, then one launch that turns what the CTAs left into parameter
// gradients and applies the update.
//
// Layer by layer the step was 14 launches of a few microseconds each with idle SMs in most of them (at
// 100 images the dense chain ran on 13 CTAs): 109 us of kernels for 0.17 GFLOP.  A CTA here owns G images at
// a time (1 while every image gets an SM of its own, then 2 or 4) and walks over its groups:
//   conv1 + relu + pool -> conv2 + relu + pool -> three dense layers -> softmax and its gradient ->
//   dense input gradients -> pool / relu gates -> conv2 input gradient -> both convolutions' weight
//   gradients, accumulated in registers over the CTA's groups.
// The dense weights (174 KB in f32) come into shared memory by bulk copies that land while the
// convolutions run; the next group's images are fetched into registers at the start of a group.
// A max-pool passes its gradient to one cell per window, so the weight gradients run over windows
// (value, position) instead of over pixels: a quarter of the multiply-adds.
//
// The second launch forms the dense weight gradients (products over the batch) in 32 x 32 tiles, adds the
// CTAs' convolution gradients and the row losses in a fixed order, and applies SGD to each value where it
// is produced.  Batches beyond 256 images cut the dense products along the batch and add the parts in a
// third launch.
//
// Every value is rounded to the tensor type where the separate operators store it, sums are f32; only the
// order of the sums is this kernel's own.  What bounds it: at 100 images latency (one image per SM, a
// chain of about twenty barrier-separated phases), at large batches the shared-memory return path of the
// convolution phases.
#include "dense_small_device.cuh"
#include "lenet_train.cuh"
#include "tc_ptx.cuh"

namespace ag {
namespace lenet_train {

using dense_small::load1_as;
using dense_small::load4_w_as;

constexpr int kThreads = 512;
constexpr int F = 5, IW = 28, PIX = 784;
constexpr int C1 = 6, P1 = 12, N1 = C1 * P1 * P1;    // 864 pooled values after conv1
constexpr int C2 = 16, NF = 256;                     // 16 x 4 x 4 after conv2
constexpr int D1 = 128, D2 = 84, D3 = 10;
constexpr int kPlane = 2552;                         // 150 + 2400 convolution weights, padded
// Filter banks as in the inference kernel: [channel pair][..][filter row: 5 taps x 2 channels + 2].
constexpr int W1_ROW = 12, W1_PAIR = F * W1_ROW + 4, W1_FLOATS = 3 * W1_PAIR;
constexpr int W2_ROW = 12, W2_CI = F * W2_ROW, W2_PAIR = C1 * W2_CI + 4, W2_FLOATS = 8 * W2_PAIR;
constexpr int kFramePair = 16 * 16 * 2 + 4;          // conv2's output gradient, zero-framed, channel pairs
constexpr int kFrame = 8 * kFramePair;
// Copies the weight gradients gather from, with pitches that put the lanes' words in 32 banks:
// x rows 37 apart (25 taps), pooled values by (channel, row) (30 pairs).
constexpr int X_ROW = 37, Q_PLANE = 13, Q_ROW = 6 * Q_PLANE;
constexpr int kXCopy = 2 * N1, kQCopy = kXCopy + 28 * X_ROW + 4, kGather = kQCopy + 12 * Q_ROW;

struct Args {
    const void *x;
    const uint8_t *t;
    int bs;
    float scale;                     // 1 / bs, the loss gradient's factor
    const void *w1, *w2, *d1, *d2, *d3, *b3;
    // left for the second launch: [bs][n] of every dense layer's input and output gradient, the
    // convolution gradients per CTA and the loss per image
    void *a0, *a1, *a2, *g1, *g2, *g3;
    float *planes, *row_loss;
    int *status;
};

// Shared memory of a CTA with G images, in floats.
template <class T, int G>
struct Smem {
    static constexpr int dw1 = 0;                                        // dense weights, raw T
    static constexpr int dw2 = dw1 + NF * D1 * (int)sizeof(T) / 4;
    static constexpr int dw3 = dw2 + D1 * D2 * (int)sizeof(T) / 4;
    static constexpr int w1 = dw3 + D2 * D3 * (int)sizeof(T) / 4;
    static constexpr int w2 = w1 + W1_FLOATS;
    static constexpr int x = w2 + W2_FLOATS;                             // [G][784]
    static constexpr int p1 = x + G * PIX;                               // [G][6][144]
    static constexpr int p2 = p1 + G * N1;                               // [256][G]
    static constexpr int pre1 = p2 + NF * G;                             // dense outputs before relu
    static constexpr int pre2 = pre1 + D1 * G;
    static constexpr int out = pre2 + D2 * G;
    static constexpr int g3 = out + 12 * G;
    static constexpr int g2 = g3 + 12 * G;
    static constexpr int g1 = g2 + D2 * G;
    static constexpr int g0 = g1 + D1 * G;                               // gradient at the flatten
    static constexpr int win2 = g0 + NF * G;                             // [256] (value, position)
    static constexpr int work = win2 + 2 * NF;                           // frame / slice sums / windows
    static constexpr int work_floats = 16 * G * D1 > kFrame ? 16 * G * D1 : kFrame;
    static_assert(kGather <= kFrame, "windows and copies");
    static constexpr int code1 = work + work_floats;                     // [G][864] bytes
    static constexpr int code2 = code1 + G * N1 / 4;                     // [G][256] bytes
    static constexpr int bar = code2 + G * NF / 4;
    static constexpr int floats = bar + 4;
    static_assert(floats * 4 <= 227 * 1024 - 64, "shared memory");
    static_assert(work % 4 == 0 && x % 4 == 0 && w2 % 4 == 0 && win2 % 4 == 0 && bar % 2 == 0, "alignment");
};

template <class T>
__device__ __forceinline__ float round_t(float v) {
    return to_f32(from_f32<T>(v));
}

__device__ __forceinline__ uint64_t dup2(float v) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ void fma2(uint64_t &acc, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ void unpack2(uint64_t v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
// A padded filter row of a channel pair: five (a, b) pairs.
__device__ __forceinline__ void load_row(const float *p, uint64_t (&w)[6]) {
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(p + 4 * q);
        w[2 * q] = v.x;
        w[2 * q + 1] = v.y;
    }
}

// Relu and 2x2 max of a window of stored values: the pooled value, and bits 0..1 the first maximum's
// cell, bit 2 whether relu passes the gradient there.
__device__ __forceinline__ float pool_window(float v0, float v1, float v2, float v3, uint32_t &code) {
    const float r0 = v0 >= 0.f ? v0 : 0.f, r1 = v1 >= 0.f ? v1 : 0.f;
    const float r2 = v2 >= 0.f ? v2 : 0.f, r3 = v3 >= 0.f ? v3 : 0.f;
    float m = r0, raw = v0;
    uint32_t at = 0;
    if (r1 > m) { m = r1; at = 1; raw = v1; }
    if (r2 > m) { m = r2; at = 2; raw = v2; }
    if (r3 > m) { m = r3; at = 3; raw = v3; }
    code = at | (raw >= 0.f ? 4u : 0u);
    return m;
}

// A 16-byte piece (f32) or 8-byte piece (bf16) of an image as four f32.
__device__ __forceinline__ float4 image4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ float4 image4(const __nv_bfloat16 *p) {
    const uint2 v = *reinterpret_cast<const uint2 *>(p);
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u),
                       __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
}

template <class T, int G>
__global__ void __launch_bounds__(kThreads, 1) lenet_train_kernel(const Args a) {
    using S = Smem<T, G>;
    extern __shared__ __align__(16) float smem[];
    __shared__ int s_abort;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float *s_x = smem + S::x, *s_p1 = smem + S::p1, *s_p2 = smem + S::p2, *work = smem + S::work;
    float *pre1 = smem + S::pre1, *pre2 = smem + S::pre2, *s_out = smem + S::out;
    float *g3 = smem + S::g3, *g2 = smem + S::g2, *g1 = smem + S::g1, *g0 = smem + S::g0;
    float *s_w1 = smem + S::w1, *s_w2 = smem + S::w2;
    float2 *win2 = reinterpret_cast<float2 *>(smem + S::win2);
    uint8_t *code1 = reinterpret_cast<uint8_t *>(smem + S::code1);
    uint8_t *code2 = reinterpret_cast<uint8_t *>(smem + S::code2);
    const T *dw1 = reinterpret_cast<const T *>(smem + S::dw1), *dw2 = reinterpret_cast<const T *>(smem + S::dw2);
    const T *dw3 = reinterpret_cast<const T *>(smem + S::dw3);
    const uint32_t bar = tc::smem_u32(smem + S::bar);
    const T *x = reinterpret_cast<const T *>(a.x);
    const int ngroups = (a.bs + G - 1) / G;
    // The second launch may take the SMs this one leaves free now; it waits there for this one's end.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    if (tid == kThreads - 1) {   // the dense weights start their way into shared memory
        s_abort = 0;
        tc::mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        const uint32_t n1 = NF * D1 * sizeof(T), n2 = D1 * D2 * sizeof(T), n3 = D2 * D3 * sizeof(T);
        tc::mbar_arrive_expect_tx(bar, n1 + n2 + n3);
        const void *src[3] = {a.d1, a.d2, a.d3};
        const uint32_t dst[3] = {tc::smem_u32(dw1), tc::smem_u32(dw2), tc::smem_u32(dw3)}, n[3] = {n1, n2, n3};
#pragma unroll
        for (int i = 0; i < 3; ++i) tc::bulk_load(dst[i], src[i], n[i], bar);
    }
    // a thread's piece of the group's images (G * 196 pieces of four pixels)
    auto fetch = [&](int grp, float4 (&v)[(G * 196 + kThreads - 1) / kThreads]) {
#pragma unroll
        for (int j = 0; j < (G * 196 + kThreads - 1) / kThreads; ++j) {
            const int64_t q = (int64_t)grp * (G * 196) + tid + j * kThreads;
            v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (tid + j * kThreads < G * 196 && q < (int64_t)a.bs * 196) v[j] = image4(x + 4 * q);
        }
    };
    float4 next[(G * 196 + kThreads - 1) / kThreads];
    fetch(blockIdx.x, next);
    // the label of warp g's image, fetched as early: it may come over PCIe
    auto fetch_label = [&](int grp) {
        const int b = grp * G + warp;
        return lane == 0 && warp < G && b < a.bs ? (uint32_t)a.t[b] : 0u;
    };
    uint32_t next_label = fetch_label(blockIdx.x);
    {
        const T *w1 = reinterpret_cast<const T *>(a.w1), *w2 = reinterpret_cast<const T *>(a.w2);
        for (int i = tid; i < W1_FLOATS; i += kThreads) {
            const int pair = i / W1_PAIR, r = i - pair * W1_PAIR;
            const int fi = r / W1_ROW, r2 = r - fi * W1_ROW, fj = r2 >> 1, o = r2 & 1;
            s_w1[i] = (fi < F && fj < F) ? to_f32(w1[((pair * 2 + o) * F + fi) * F + fj]) : 0.f;
        }
#pragma unroll
        for (int j = 0; j < (W2_FLOATS + kThreads - 1) / kThreads; ++j) {
            const int i = tid + j * kThreads;
            const int pair = i / W2_PAIR, r = i - pair * W2_PAIR;
            const int ci = r / W2_CI, r2 = r - ci * W2_CI, fi = r2 / W2_ROW, r3 = r2 - fi * W2_ROW;
            const int fj = r3 >> 1, o = r3 & 1;
            if (i < W2_FLOATS)
                s_w2[i] = (ci < C1 && fj < F) ? to_f32(w2[(((pair * 2 + o) * C1 + ci) * F + fi) * F + fj]) : 0.f;
        }
    }
    bool weights_here = false;
    float aw1[3] = {0.f, 0.f, 0.f}, aw2[F] = {0.f, 0.f, 0.f, 0.f, 0.f};

    for (int grp = blockIdx.x; grp < ngroups; grp += gridDim.x) {
        const int b0 = grp * G, nimg = min(G, a.bs - b0);
#pragma unroll
        for (int j = 0; j < (G * 196 + kThreads - 1) / kThreads; ++j)
            if (tid + j * kThreads < G * 196) reinterpret_cast<float4 *>(s_x)[tid + j * kThreads] = next[j];
        const uint32_t label = next_label;
        __syncthreads();
        if (grp + (int)gridDim.x < ngroups) {
            fetch(grp + gridDim.x, next);
            next_label = fetch_label(grp + gridDim.x);
        }

        // ---- conv1 + relu + pool: item = (image, 2 rows x 4 columns, channel pair)
        for (int it = tid; it < G * 216; it += kThreads) {
            const int g = it / 216, r = it - g * 216, pair = r % 3, blk = r / 3, by = blk / 6, hx = blk - by * 6;
            const float *img = s_x + g * PIX + 2 * by * IW + 4 * hx;
            uint64_t acc[2][4] = {};
            uint64_t wprev[6];
#pragma unroll
            for (int pr = 0; pr < F + 1; ++pr) {
                const float4 pa = *reinterpret_cast<const float4 *>(img + pr * IW);
                const float4 pb = *reinterpret_cast<const float4 *>(img + pr * IW + 4);
                const uint64_t pp[8] = {dup2(pa.x), dup2(pa.y), dup2(pa.z), dup2(pa.w),
                                        dup2(pb.x), dup2(pb.y), dup2(pb.z), dup2(pb.w)};
                uint64_t wcur[6];
                if (pr < F) load_row(s_w1 + pair * W1_PAIR + pr * W1_ROW, wcur);
#pragma unroll
                for (int fj = 0; fj < F; ++fj)
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        if (pr < F) fma2(acc[0][c], pp[fj + c], wcur[fj]);
                        if (pr >= 1) fma2(acc[1][c], pp[fj + c], wprev[fj]);
                    }
                if (pr < F) {
#pragma unroll
                    for (int q = 0; q < 6; ++q) wprev[q] = wcur[q];
                }
            }
            float v[2][4][2];
#pragma unroll
            for (int r2 = 0; r2 < 2; ++r2)
#pragma unroll
                for (int c = 0; c < 4; ++c) unpack2(acc[r2][c], v[r2][c][0], v[r2][c][1]);
#pragma unroll
            for (int o = 0; o < 2; ++o)
#pragma unroll
                for (int w = 0; w < 2; ++w) {
                    uint32_t code;
                    const float m = pool_window(round_t<T>(v[0][2 * w][o]), round_t<T>(v[0][2 * w + 1][o]),
                                                round_t<T>(v[1][2 * w][o]), round_t<T>(v[1][2 * w + 1][o]), code);
                    const int at = g * N1 + (pair * 2 + o) * (P1 * P1) + by * P1 + 2 * hx + w;
                    s_p1[at] = m;
                    code1[at] = (uint8_t)code;
                }
        }
        __syncthreads();

        // ---- conv2 + relu + pool: (image, 2 rows x 4 columns, channel pair) split over 8 / G adjacent
        // lanes by input channels, whose sums meet by shuffles
        {
            constexpr int LANES = 8 / G, PER = G == 1 ? 1 : G == 2 ? 2 : 3;
            const int s = tid % LANES, it = tid / LANES;
            const int g = it >> 6, r = it & 63, pair = r & 7, blk = r >> 3, by = blk >> 1, bx = blk & 1;
            const float *img = s_p1 + g * N1 + 2 * by * P1 + 4 * bx;
            uint64_t acc[2][4] = {};
#pragma unroll 1
            for (int ci = s * PER; ci < min(C1, (s + 1) * PER); ++ci) {
                uint64_t wprev[6];
#pragma unroll
                for (int pr = 0; pr < F + 1; ++pr) {
                    const float4 pa = *reinterpret_cast<const float4 *>(img + ci * (P1 * P1) + pr * P1);
                    const float4 pb = *reinterpret_cast<const float4 *>(img + ci * (P1 * P1) + pr * P1 + 4);
                    const uint64_t pp[8] = {dup2(pa.x), dup2(pa.y), dup2(pa.z), dup2(pa.w),
                                            dup2(pb.x), dup2(pb.y), dup2(pb.z), dup2(pb.w)};
                    uint64_t wcur[6];
                    if (pr < F) load_row(s_w2 + pair * W2_PAIR + ci * W2_CI + pr * W2_ROW, wcur);
#pragma unroll
                    for (int fj = 0; fj < F; ++fj)
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            if (pr < F) fma2(acc[0][c], pp[fj + c], wcur[fj]);
                            if (pr >= 1) fma2(acc[1][c], pp[fj + c], wprev[fj]);
                        }
                    if (pr < F) {
#pragma unroll
                        for (int q = 0; q < 6; ++q) wprev[q] = wcur[q];
                    }
                }
            }
            __syncwarp();
            float v[2][4][2];
#pragma unroll
            for (int r2 = 0; r2 < 2; ++r2)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    unpack2(acc[r2][c], v[r2][c][0], v[r2][c][1]);
#pragma unroll
                    for (int o = 0; o < 2; ++o)
#pragma unroll
                        for (int m = 1; m < LANES; m <<= 1)
                            v[r2][c][o] += __shfl_xor_sync(0xffffffffu, v[r2][c][o], m);
                }
            if (s == 0) {
#pragma unroll
                for (int o = 0; o < 2; ++o)
#pragma unroll
                    for (int w = 0; w < 2; ++w) {
                        uint32_t code;
                        const float m = pool_window(round_t<T>(v[0][2 * w][o]), round_t<T>(v[0][2 * w + 1][o]),
                                                    round_t<T>(v[1][2 * w][o]), round_t<T>(v[1][2 * w + 1][o]), code);
                        const int k = (pair * 2 + o) * 16 + by * 4 + 2 * bx + w;
                        s_p2[k * G + g] = m;
                        code2[g * NF + k] = (uint8_t)code;
                    }
            }
        }
        __syncthreads();
        if (!weights_here) {
            // completes for every thread or for none, so all threads take the same way out
            if (!tc::mbar_wait(bar, 0, &s_abort)) {
                if (tid == 0) atomicCAS(a.status, 0, 173);
                return;
            }
            weights_here = true;
        }

        // ---- dense 256 -> 128: (four outputs, slice of 16 inputs), then the slices in order
        {
            const int q = tid & 31, sl = tid >> 5;
            float acc[4][G] = {};
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const int k = sl * 16 + j;
                float w[4];
                load4_w_as<true>(dw1 + k * D1 + 4 * q, w);
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    const float v = s_p2[k * G + g];
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[c][g] = fmaf(v, w[c], acc[c][g]);
                }
            }
#pragma unroll
            for (int g = 0; g < G; ++g)
                *reinterpret_cast<float4 *>(work + (sl * G + g) * D1 + 4 * q) =
                    make_float4(acc[0][g], acc[1][g], acc[2][g], acc[3][g]);
        }
        __syncthreads();
        for (int i = tid; i < D1 * G; i += kThreads) {
            const int g = i / D1, n = i - g * D1;
            float s = 0.f;
#pragma unroll
            for (int sl = 0; sl < 16; ++sl) s += work[(sl * G + g) * D1 + n];
            pre1[n * G + g] = round_t<T>(s);
        }
        __syncthreads();
        // ---- dense 128 -> 84
        {
            const int q = tid % 21, sl = tid / 21;
            if (sl < 16) {
                float acc[4][G] = {};
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int k = sl * 8 + j;
                    float w[4];
                    load4_w_as<true>(dw2 + k * D2 + 4 * q, w);
#pragma unroll
                    for (int g = 0; g < G; ++g) {
                        const float p = pre1[k * G + g], v = p >= 0.f ? p : 0.f;
#pragma unroll
                        for (int c = 0; c < 4; ++c) acc[c][g] = fmaf(v, w[c], acc[c][g]);
                    }
                }
#pragma unroll
                for (int g = 0; g < G; ++g)
                    *reinterpret_cast<float4 *>(work + (sl * G + g) * D2 + 4 * q) =
                        make_float4(acc[0][g], acc[1][g], acc[2][g], acc[3][g]);
            }
        }
        __syncthreads();
        for (int i = tid; i < D2 * G; i += kThreads) {
            const int g = i / D2, n = i - g * D2;
            float s = 0.f;
#pragma unroll
            for (int sl = 0; sl < 16; ++sl) s += work[(sl * G + g) * D2 + n];
            pre2[n * G + g] = round_t<T>(s);
        }
        __syncthreads();
        // ---- dense 84 -> 10: a warp per logit
        for (int task = warp; task < D3 * G; task += kThreads / 32) {
            const int g = task / D3, n = task - g * D3;
            float s = 0.f;
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const int k = lane + 32 * j;
                if (k < D2) {
                    const float p = pre2[k * G + g];
                    s = fmaf(p >= 0.f ? p : 0.f, load1_as<true>(dw3 + k * D3 + n), s);
                }
            }
#pragma unroll
            for (int m = 16; m > 0; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
            if (lane == 0) {
                float v = round_t<T>(s);
                if (a.b3 != nullptr) v = round_t<T>(__fadd_rn(v, to_f32(reinterpret_cast<const T *>(a.b3)[n])));
                s_out[n * G + g] = v;
            }
        }
        __syncthreads();
        // ---- loss and its gradient: a thread per image (criterion.rs:84, learn/criterion.rs:299-324)
        if (lane == 0 && warp < G) {
            const int g = warp;
            const bool live = g < nimg;
            const uint32_t t = label;
            float m = -INFINITY, s = 0.f, xt = 0.f, e[D3];
#pragma unroll
            for (int i = 0; i < D3; ++i) m = fmaxf(m, s_out[i * G + g]);
#pragma unroll
            for (int i = 0; i < D3; ++i) {
                const float v = s_out[i * G + g];
                e[i] = expf(v - m);
                s += e[i];
                if ((uint32_t)i == t) xt = v;
            }
            if (live) a.row_loss[b0 + g] = logf(s) - (xt - m);
#pragma unroll
            for (int i = 0; i < D3; ++i) {
                const float d = __fmul_rn(a.scale, __fsub_rn(__fdiv_rn(e[i], s), (uint32_t)i == t ? 1.f : 0.f));
                g3[i * G + g] = live ? round_t<T>(d) : 0.f;
            }
        }
        __syncthreads();

        // ---- dense input gradients; Relu passes where its input is >= 0
        for (int i = tid; i < D2 * G; i += kThreads) {
            const int k = i / G, g = i - k * G;
            float s = 0.f;
#pragma unroll
            for (int n = 0; n < D3; ++n) s = fmaf(g3[n * G + g], load1_as<true>(dw3 + k * D3 + n), s);
            g2[i] = pre2[i] >= 0.f ? round_t<T>(s) : 0.f;
        }
        __syncthreads();
        {
            // 84 -> 128: four lanes per output, groups of four inputs each
            const int k = tid >> 2, s4 = tid & 3;
            float acc[G] = {};
            for (int n4 = s4; n4 < D2 / 4; n4 += 4) {
                float w[4];
                load4_w_as<true>(dw2 + k * D2 + 4 * n4, w);
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int g = 0; g < G; ++g) acc[g] = fmaf(g2[(4 * n4 + c) * G + g], w[c], acc[g]);
            }
            __syncwarp();
#pragma unroll
            for (int g = 0; g < G; ++g) {
                acc[g] += __shfl_xor_sync(0xffffffffu, acc[g], 1);
                acc[g] += __shfl_xor_sync(0xffffffffu, acc[g], 2);
                if (s4 == 0) g1[k * G + g] = pre1[k * G + g] >= 0.f ? round_t<T>(acc[g]) : 0.f;
            }
        }
        __syncthreads();
        {
            // 128 -> 256: a warp reads whole rows (a lane four weights) of 16 outputs; the 16 sums over
            // lanes meet in a transposing reduction that leaves one output per pair of lanes
#pragma unroll
            for (int g = 0; g < G; ++g) {
                float gv[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) gv[c] = g1[(4 * lane + c) * G + g];
                float v[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    float w[4];
                    load4_w_as<true>(dw1 + (warp * 16 + j) * D1 + 4 * lane, w);
                    v[j] = fmaf(gv[3], w[3], fmaf(gv[2], w[2], fmaf(gv[1], w[1], gv[0] * w[0])));
                }
#pragma unroll
                for (int m = 16, n = 8; m >= 2; m >>= 1, n >>= 1) {
                    const bool up = lane & m;
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (j < n) {
                            const float send = up ? v[j] : v[j + n], keep = up ? v[j + n] : v[j];
                            v[j] = keep + __shfl_xor_sync(0xffffffffu, send, m);
                        }
                }
                v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
                // lane bits 4..1 select the output: bit 4 its bit 3, and so on
                const int j = lane >> 1;
                if ((lane & 1) == 0) g0[(warp * 16 + j) * G + g] = round_t<T>(v[0]);
            }
        }
        __syncthreads();
        // ---- what the second launch multiplies
        {
            T *a0 = reinterpret_cast<T *>(a.a0), *a1 = reinterpret_cast<T *>(a.a1), *a2 = reinterpret_cast<T *>(a.a2);
            T *q1 = reinterpret_cast<T *>(a.g1), *q2 = reinterpret_cast<T *>(a.g2), *q3 = reinterpret_cast<T *>(a.g3);
            for (int i = tid; i < nimg * NF; i += kThreads)
                a0[(int64_t)b0 * NF + i] = from_f32<T>(s_p2[(i % NF) * G + i / NF]);
            for (int i = tid; i < nimg * D1; i += kThreads) {
                const int at = (i % D1) * G + i / D1;
                const float p = pre1[at];
                a1[(int64_t)b0 * D1 + i] = from_f32<T>(p >= 0.f ? p : 0.f);
                q1[(int64_t)b0 * D1 + i] = from_f32<T>(g1[at]);
            }
            for (int i = tid; i < nimg * D2; i += kThreads) {
                const int at = (i % D2) * G + i / D2;
                const float p = pre2[at];
                a2[(int64_t)b0 * D2 + i] = from_f32<T>(p >= 0.f ? p : 0.f);
                q2[(int64_t)b0 * D2 + i] = from_f32<T>(g2[at]);
            }
            for (int i = tid; i < nimg * D3; i += kThreads)
                q3[(int64_t)b0 * D3 + i] = from_f32<T>(g3[(i % D3) * G + i / D3]);
        }

        for (int g = 0; g < nimg; ++g) {
            // ---- conv2's output gradient: one cell per pool window, as a zero-framed dense array
            // (input gradient) and as (value, position) per window (weight gradient)
#pragma unroll
            for (int i = tid; i < kFrame / 4; i += kThreads)
                reinterpret_cast<float4 *>(work)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            __syncthreads();
            if (tid < NF) {
                const int co = tid >> 4, wy = (tid >> 2) & 3, wx = tid & 3;
                const uint32_t code = code2[g * NF + tid];
                const float v = (code & 4u) ? g0[tid * G + g] : 0.f;
                const int yy = 2 * wy + (int)((code >> 1) & 1u), xx = 2 * wx + (int)(code & 1u);
                work[(co >> 1) * kFramePair + ((yy + 4) * 16 + xx + 4) * 2 + (co & 1)] = v;
                win2[tid] = make_float2(v, __int_as_float(yy * Q_ROW + xx));
            }
            __syncthreads();
            // ---- conv2 input gradient: (2 rows x 12 columns, input channel), a lane per pair of output
            // channels (the halves of a packed sum), lanes added by a transposing reduction
            float dp[3];
            int dp_at = 0;
            if (tid < 288) {
                const int pair = tid & 7, r = tid >> 3, ci = r % 6, by = r / 6;
                const float *fr = work + pair * kFramePair + 2 * by * 32;
                const float *wt = s_w2 + pair * W2_PAIR + ci * W2_CI;
                uint64_t acc[2][12] = {};
                uint64_t wprev[6];
#pragma unroll
                for (int pr = 0; pr < F + 1; ++pr) {
                    uint64_t pp[16], wcur[6];
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(fr + pr * 32 + 4 * q);
                        pp[2 * q] = v.x;
                        pp[2 * q + 1] = v.y;
                    }
                    if (pr < F) load_row(wt + (F - 1 - pr) * W2_ROW, wcur);
#pragma unroll
                    for (int u = 0; u < F; ++u)
#pragma unroll
                        for (int c = 0; c < 12; ++c) {
                            if (pr < F) fma2(acc[0][c], pp[u + c], wcur[F - 1 - u]);
                            if (pr >= 1) fma2(acc[1][c], pp[u + c], wprev[F - 1 - u]);
                        }
                    if (pr < F) {
#pragma unroll
                        for (int q = 0; q < 6; ++q) wprev[q] = wcur[q];
                    }
                }
                float v[24];
#pragma unroll
                for (int i = 0; i < 24; ++i) {
                    float lo, hi;
                    unpack2(acc[i / 12][i % 12], lo, hi);
                    v[i] = lo + hi;
                }
#pragma unroll
                for (int m = 4, n = 12; m >= 1; m >>= 1, n >>= 1) {
                    const bool up = pair & m;
#pragma unroll
                    for (int j = 0; j < 12; ++j)
                        if (j < n) {
                            const float send = up ? v[j] : v[j + n], keep = up ? v[j + n] : v[j];
                            v[j] = keep + __shfl_xor_sync(0xffffffffu, send, m);
                        }
                }
#pragma unroll
                for (int j = 0; j < 3; ++j) dp[j] = round_t<T>(v[j]);
                dp_at = ci * (P1 * P1) + (2 * by + (pair >> 2)) * P1 + ((pair >> 1) & 1) * 6 + (pair & 1) * 3;
            }
            __syncthreads();   // the frame is no longer read
            // ---- conv1's output gradient per pool window, and the copies the weight gradients gather from
            float2 *win1 = reinterpret_cast<float2 *>(work);
            if (tid < 288) {
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const int at = dp_at + j, cell = at % (P1 * P1), wy = cell / P1, wx = cell - wy * P1;
                    const uint32_t code = code1[g * N1 + at];
                    const int yy = 2 * wy + (int)((code >> 1) & 1u), xx = 2 * wx + (int)(code & 1u);
                    win1[at] = make_float2((code & 4u) ? dp[j] : 0.f, __int_as_float(yy * X_ROW + xx));
                }
            } else {
                for (int i = tid - 288; i < PIX; i += kThreads - 288)
                    work[kXCopy + i / IW * X_ROW + i % IW] = s_x[g * PIX + i];
                for (int i = tid - 288; i < N1; i += kThreads - 288) {
                    const int ci = i / (P1 * P1), r = i - ci * (P1 * P1);
                    work[kQCopy + r / P1 * Q_ROW + ci * Q_PLANE + r % P1] = s_p1[g * N1 + i];
                }
            }
            __syncthreads();
            // ---- conv2 weight gradient: a warp per output channel, a lane per (input channel, filter row)
            if (lane < 30) {
                const int ci = lane / 5, fi = lane - ci * 5;
                const float *src = work + kQCopy + fi * Q_ROW + ci * Q_PLANE;
#pragma unroll
                for (int w = 0; w < 16; w += 2) {
                    const float4 e = *reinterpret_cast<const float4 *>(win2 + warp * 16 + w);
                    const float *p = src + __float_as_int(e.y), *q = src + __float_as_int(e.w);
#pragma unroll
                    for (int fj = 0; fj < F; ++fj) aw2[fj] = fmaf(e.z, q[fj], fmaf(e.x, p[fj], aw2[fj]));
                }
            }
            // ---- conv1 weight gradient: a warp per (three channels, 18 windows), a lane per tap
            if (lane < 25) {
                const float *src = work + kXCopy + lane / 5 * X_ROW + lane % 5;
                const float2 *w1 = win1 + (warp & 1) * 3 * (P1 * P1) + (warp >> 1) * 18;
#pragma unroll
                for (int w = 0; w < 18; w += 2)
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const float4 e = *reinterpret_cast<const float4 *>(w1 + c * (P1 * P1) + w);
                        aw1[c] = fmaf(e.z, src[__float_as_int(e.w)], fmaf(e.x, src[__float_as_int(e.y)], aw1[c]));
                    }
            }
            __syncthreads();
        }
    }

    // ---- this CTA's part of the convolution gradients
    float *plane = a.planes + (int64_t)blockIdx.x * kPlane;
    if (lane < 30) {
#pragma unroll
        for (int fj = 0; fj < F; ++fj) plane[150 + (warp * 30 + lane) * 5 + fj] = aw2[fj];
    }
    if (lane < 25) {
#pragma unroll
        for (int c = 0; c < 3; ++c) work[(warp >> 1) * 150 + ((warp & 1) * 3 + c) * 25 + lane] = aw1[c];
    }
    __syncthreads();
    if (tid < 150) {
        float s = 0.f;
#pragma unroll
        for (int sl = 0; sl < 8; ++sl) s += work[sl * 150 + tid];
        plane[tid] = s;
    }
}

// ------------------------------------------------------------------ gradients and update
struct Update {
    void *values, *grads, *velocity;
    int update, use_momentum;
    float lr, momentum;
};

// Stores a gradient and applies SGD in the arithmetic of ag_sgd_update / ag_sgd_update_momentum.
template <class T>
__device__ __forceinline__ void finish_value(const Update &u, int64_t at, float grad) {
    const T gt = from_f32<T>(grad);
    reinterpret_cast<T *>(u.grads)[at] = gt;
    if (!u.update) return;
    T *w = reinterpret_cast<T *>(u.values) + at;
    const float g = to_f32(gt);
    if (u.use_momentum) {
        T *v = reinterpret_cast<T *>(u.velocity) + at;
        const float vv = __fadd_rn(__fmul_rn(u.momentum, to_f32(*v)), g);
        *w = from_f32<T>(__fsub_rn(to_f32(*w), __fmul_rn(u.lr, vv)));
        *v = from_f32<T>(vv);
    } else {
        const float p = round_t<T>(__fmul_rn(round_t<T>(-u.lr), g));
        *w = from_f32<T>(__fadd_rn(p, to_f32(*w)));
    }
}

struct Finish {
    Update u;
    int64_t off[6];
    const void *in[3], *g[3];   // dense layers' inputs and output gradients, [bs][n]
    int bs, planes;
    int splits, rows_per_split; // parts of the batch of the dense products
    float *partial;             // splits > 1: [splits][kDense]
    const float *conv_planes, *row_loss;
    float *loss;
};

constexpr int kTiles1 = 8 * 4, kTiles2 = 4 * 3, kTiles3 = 3, kTiles = kTiles1 + kTiles2 + kTiles3;
constexpr int kDense = NF * D1 + D1 * D2 + D2 * D3 + D3;     // 44,370 values of the dense layers
constexpr int kConvBlocks = (2550 + 31) / 32;
constexpr int kChunk = 64, kPitch = 36;

// Blocks [0, 47 * splits): a 32 x 32 tile of a dense weight gradient over a part of the batch;
// then 80 blocks for the convolution gradients and one for the loss.
template <class T>
__global__ void __launch_bounds__(256) lenet_finish_kernel(const __grid_constant__ Finish f) {
    __shared__ __align__(16) float As[2][kChunk][kPitch], Bs[2][kChunk][kPitch];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int tid = threadIdx.x;
    int blk = blockIdx.x;
    if (blk >= kTiles * f.splits) {
        blk -= kTiles * f.splits;
        if (blk < kConvBlocks) {
            // 32 outputs, eight warps that each add every eighth CTA's part, the eight sums in order
            float *part = &As[0][0][0];
            const int lane = tid & 31, grp = tid >> 5, i = blk * 32 + lane;
            float s = 0.f;
            if (i < 2550) {
                // sixteen loads in flight: 148 planes in two rounds
                for (int z = grp; z < f.planes; z += 128) {
                    float v[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        v[j] = z + 8 * j < f.planes ? f.conv_planes[(int64_t)(z + 8 * j) * kPlane + i] : 0.f;
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (z + 8 * j < f.planes) s += v[j];
                }
            }
            part[grp * 32 + lane] = s;
            __syncthreads();
            if (grp == 0 && i < 2550) {
                s = part[lane];
#pragma unroll
                for (int q = 1; q < 8; ++q) s += part[q * 32 + lane];
                finish_value<T>(f.u, i < 150 ? f.off[0] + i : f.off[1] + i - 150, s);
            }
            return;
        }
        float *part = &As[0][0][0];
        float s = 0.f;
        for (int i = tid; i < f.bs; i += 256) s += f.row_loss[i];
        part[tid] = s;
        __syncthreads();
        for (int o = 128; o > 0; o >>= 1) {
            if (tid < o) part[tid] += part[tid + o];
            __syncthreads();
        }
        if (tid == 0) *f.loss = part[0];
        return;
    }
    const int split = blk / kTiles;
    int tile = blk - split * kTiles;
    const int layer = tile < kTiles1 ? 0 : tile < kTiles1 + kTiles2 ? 1 : 2;
    tile -= layer == 0 ? 0 : layer == 1 ? kTiles1 : kTiles1 + kTiles2;
    const int rows = layer == 0 ? NF : layer == 1 ? D1 : D2, cols = layer == 0 ? D1 : layer == 1 ? D2 : D3;
    const int tiles_n = (cols + 31) / 32, m0 = tile / tiles_n * 32, n0 = tile % tiles_n * 32;
    const T *in = reinterpret_cast<const T *>(f.in[layer]), *g = reinterpret_cast<const T *>(f.g[layer]);
    const int r0 = split * f.rows_per_split, r1 = min(f.bs, r0 + f.rows_per_split);
    const int mn = tid & 31, kb = tid >> 5;            // staging: 32 columns of batch rows kb, kb + 8, ..
    const int kg = tid >> 6, t = tid & 63, tx = t & 7, ty = t >> 3;
    const bool bias = layer == 2 && f.off[5] >= 0 && m0 == 0 && tid < 32;
    float acc[4][4] = {}, bsum = 0.f;
    // two chunks ahead: a batch of up to 128 images costs one trip to memory
    float ra[2][kChunk / 8], rb[2][kChunk / 8];
    auto load = [&](int kc, float (&va)[kChunk / 8], float (&vb)[kChunk / 8]) {
#pragma unroll
        for (int i = 0; i < kChunk / 8; ++i) {
            const int r = kc + i * 8 + kb;
            va[i] = r < r1 && m0 + mn < rows ? to_f32(in[(int64_t)r * rows + m0 + mn]) : 0.f;
            vb[i] = r < r1 && n0 + mn < cols ? to_f32(g[(int64_t)r * cols + n0 + mn]) : 0.f;
        }
    };
    load(r0, ra[0], rb[0]);
    load(r0 + kChunk, ra[1], rb[1]);
    for (int kc0 = r0; kc0 < r1; kc0 += 2 * kChunk)
#pragma unroll
    for (int buf = 0; buf < 2; ++buf) {
        const int kc = kc0 + buf * kChunk;
        if (kc >= r1) break;
#pragma unroll
        for (int i = 0; i < kChunk / 8; ++i) {
            As[buf][i * 8 + kb][mn] = ra[buf][i];
            Bs[buf][i * 8 + kb][mn] = rb[buf][i];
        }
        __syncthreads();
        if (kc + 2 * kChunk < r1) load(kc + 2 * kChunk, ra[buf], rb[buf]);
        // four groups of 64 threads, a quarter of the chunk each, 4 x 4 outputs per thread
#pragma unroll 8
        for (int k = kg * (kChunk / 4); k < (kg + 1) * (kChunk / 4); ++k) {
            const float4 a4 = *reinterpret_cast<const float4 *>(&As[buf][k][ty * 4]);
            const float4 b4 = *reinterpret_cast<const float4 *>(&Bs[buf][k][tx * 4]);
            const float av[4] = {a4.x, a4.y, a4.z, a4.w}, bv[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
        if (bias)
            for (int k = 0; k < kChunk; ++k) bsum += Bs[buf][k][tid];
    }
    __syncthreads();
    float *red = &As[0][0][0];   // [3 groups][16 values][64 threads]
    if (kg > 0) {
#pragma unroll
        for (int i = 0; i < 16; ++i) red[((kg - 1) * 16 + i) * 64 + t] = acc[i / 4][i % 4];
    }
    __syncthreads();
    const int base = layer == 0 ? 0 : layer == 1 ? NF * D1 : NF * D1 + D1 * D2;
    if (bias && tid < D3) {
        if (f.splits > 1)
            f.partial[(int64_t)split * kDense + kDense - D3 + tid] = bsum;
        else
            finish_value<T>(f.u, f.off[5] + tid, bsum);
    }
    if (kg > 0) return;
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i / 4][i % 4] += red[(q * 16 + i) * 64 + t];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int m = m0 + ty * 4 + i, n = n0 + tx * 4 + j;
            if (m >= rows || n >= cols) continue;
            if (f.splits > 1)
                f.partial[(int64_t)split * kDense + base + m * cols + n] = acc[i][j];
            else
                finish_value<T>(f.u, f.off[2 + layer] + m * cols + n, acc[i][j]);
        }
}

// The parts of the dense gradients, added in order.
template <class T>
__global__ void __launch_bounds__(256) lenet_reduce_kernel(const __grid_constant__ Finish f) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= kDense - (f.off[5] < 0 ? D3 : 0)) return;
    float s = 0.f;
#pragma unroll 4
    for (int z = 0; z < f.splits; ++z) s += f.partial[(int64_t)z * kDense + i];
    const int e1 = NF * D1, e2 = e1 + D1 * D2, e3 = e2 + D2 * D3;
    finish_value<T>(f.u, i < e1 ? f.off[2] + i : i < e2 ? f.off[3] + i - e1 : i < e3 ? f.off[4] + i - e2
                                                                                 : f.off[5] + i - e3, s);
}

// ------------------------------------------------------------------------------- host
template <class T, int G>
static int launch_pass(ag_device *dev, const Args &a, int ctas) {
    auto kernel = lenet_train_kernel<T, G>;
    constexpr int bytes = Smem<T, G>::floats * 4;
    static SmemAllowed allowed;
    AG_TRY(allow_smem<bytes>(dev, kernel, allowed));
    kernel<<<ctas, kThreads, bytes, dev->stream>>>(a);
    AG_CHECK_LAUNCH();
    return AG_OK;
}

template <class T>
static int step_typed(ag_device *dev, const Net &net, const void *x, const uint8_t *t, int bs, void *values,
                      void *grads, void *velocity, const Sgd &sgd, float *loss) {
    const T *v = reinterpret_cast<const T *>(values);
    // Images per CTA: one while every image has an SM of its own; then as many as fit shared memory,
    // which share each dense weight read.
    constexpr int GMAX = sizeof(T) == 4 ? 2 : 4;
    const int group = bs <= dev->sm_count ? 1 : bs <= 2 * dev->sm_count || GMAX == 2 ? 2 : 4;
    const int groups = (int)ceil_div(bs, group), ctas = groups < dev->sm_count ? groups : dev->sm_count;
    // Parts of the batch: the 47 tiles of the dense gradients fill the GPU from about four parts on.
    const int splits = bs <= 256 ? 1 : (int)(ceil_div(bs, 128) < 12 ? ceil_div(bs, 128) : 12);
    const int per = (int)(ceil_div(ceil_div(bs, splits), kChunk) * kChunk);

    Args a;
    a.x = x; a.t = t; a.bs = bs;
    a.scale = 1.f / (float)bs;
    a.w1 = v + net.off[0]; a.w2 = v + net.off[1];
    a.d1 = v + net.off[2]; a.d2 = v + net.off[3]; a.d3 = v + net.off[4];
    a.b3 = net.off[5] >= 0 ? v + net.off[5] : nullptr;
    Finish f;
    f.splits = (int)ceil_div(bs, per);
    const int widths[6] = {NF, D1, D2, D1, D2, D3};
    size_t at = 0, off[6];
    for (int i = 0; i < 6; ++i) {
        off[i] = at;
        at += ((size_t)bs * widths[i] * sizeof(T) + 255) / 256 * 256;
    }
    const size_t planes_at = at, rows_at = planes_at + (size_t)ctas * kPlane * 4;
    const size_t part_at = rows_at + ((size_t)bs * 4 + 255) / 256 * 256;
    void *ws = nullptr;
    AG_TRY(workspace(dev, part_at + (f.splits > 1 ? (size_t)f.splits * kDense * 4 : 0), &ws));
    char *base = (char *)ws;
    void **slots[6] = {&a.a0, &a.a1, &a.a2, &a.g1, &a.g2, &a.g3};
    for (int i = 0; i < 6; ++i) *slots[i] = base + off[i];
    a.planes = (float *)(base + planes_at);
    a.row_loss = (float *)(base + rows_at);
    a.status = dev->status_dev;
    if (group == 1)
        AG_TRY((launch_pass<T, 1>(dev, a, ctas)));
    else if (group == 2)
        AG_TRY((launch_pass<T, 2>(dev, a, ctas)));
    else
        AG_TRY((launch_pass<T, GMAX>(dev, a, ctas)));

    f.u = Update{values, grads, velocity, sgd.update ? 1 : 0, sgd.use_momentum ? 1 : 0, sgd.lr, sgd.momentum};
    for (int i = 0; i < 6; ++i) f.off[i] = net.off[i];
    f.in[0] = a.a0; f.in[1] = a.a1; f.in[2] = a.a2;
    f.g[0] = a.g1; f.g[1] = a.g2; f.g[2] = a.g3;
    f.bs = bs;
    f.planes = ctas;
    f.rows_per_split = per;
    f.partial = (float *)(base + part_at);
    f.conv_planes = a.planes;
    f.row_loss = a.row_loss;
    f.loss = loss;
    // Dependent launches: at 100 images the step is a chain of launches, each of which started 2 us after the last.
    AG_TRY(launch_dependent(dev, lenet_finish_kernel<T>, dim3((unsigned)(kTiles * f.splits + kConvBlocks + 1)), 256, 0,
                            f));
    if (f.splits > 1)
        AG_TRY(launch_dependent(dev, lenet_reduce_kernel<T>, dim3((unsigned)ceil_div(kDense, 256)), 256, 0, f));
    return AG_OK;
}

int step(ag_device *dev, ag_dtype dtype, const Net &net, const void *x, const uint8_t *t, int64_t bs,
         void *values, void *grads, void *velocity, const Sgd &sgd, float *loss) {
    AG_REQUIRE(bs > 0 && bs < (1 << 24), AG_ERR_LIMIT, "batch of %lld images", (long long)bs);
    if (dtype == AG_F32) return step_typed<float>(dev, net, x, t, (int)bs, values, grads, velocity, sgd, loss);
    return step_typed<__nv_bfloat16>(dev, net, x, t, (int)bs, values, grads, velocity, sgd, loss);
}

}  // namespace lenet_train
}  // namespace ag
