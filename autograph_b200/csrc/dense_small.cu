// Latency-oriented kernels for small dense products (m up to a few thousand
// rows, n <= 256 outputs): y[m,n] = x[m,k] . w[k,n] (+ bias) (relu), row-major.
//
// At these sizes a shared-memory-tiled GEMM runs two warps per SM through a
// chain of load -> barrier -> multiply steps and is bound by memory and
// instruction-fetch latency.  Here the threads of a CTA split the work as
// (output column, k slice): each streams its weights straight from L2 with
// coalesced loads and keeps one accumulator per row; the k slices are then
// summed in a fixed order, so the result is deterministic.  How k is sliced
// depends on (k, n) alone and every kernel that runs such a layer -- a single
// product, a chain of layers, a whole network -- adds in that order, so their
// bits agree.
#include "dense_small.cuh"
#include "dense_small_device.cuh"

namespace ag {
namespace dense_small {

// One layer of the chain's code on 8 rows per CTA: batches large enough to fill the GPU at 8 rows per CTA.
template <class T>
__global__ void __launch_bounds__(1024)
    dense_rows_kernel(const T *__restrict__ x, T *__restrict__ y, int M, const ChainStep st) {
    let_dependents_launch();
    dependency_wait();
    extern __shared__ __align__(16) float smem[];
    float *xs = smem;                             // [K][ROWS]
    float *red = smem + (size_t)st.K * ROWS;      // [slices][ROWS][np]
    const int m0 = blockIdx.x * ROWS;
    const int rows = min(ROWS, M - m0);
    for (int i = threadIdx.x; i < ROWS * st.K; i += blockDim.x) {
        const int r = i / st.K, k = i - r * st.K;    // coalesced along k
        xs[k * ROWS + r] = (r < rows) ? to_f32(x[(int64_t)(m0 + r) * st.K + k]) : 0.f;
    }
    __syncthreads();
    chain_layer<T>(st, reinterpret_cast<const T *>(st.w), xs, nullptr, red, m0, rows, true, y);
}

// A layer with at most 16 outputs (narrow_step) on its own: narrow_layer's sums, four lanes per output that add
// k = q, q + 4, ..., with the weights and R rows of x in shared memory.  Read from L2 16 at a time and on 8 rows
// per CTA, 256 x 512 x 10 took 7.8 us (32 CTAs, eight trips to L2 one after another), now 4.0; 4096 x 84 x 10 6.1 and 3.7.
template <class T>
__global__ void __launch_bounds__(256)
    dense_narrow_kernel(const T *__restrict__ x, T *__restrict__ y, int M, int R, const ChainStep st) {
    let_dependents_launch();
    dependency_wait();
    extern __shared__ __align__(16) float smem[];
    float *ws = smem, *xs = smem + st.K * st.N;   // [K][N], [R][K]
    const T *w = reinterpret_cast<const T *>(st.w), *bias = reinterpret_cast<const T *>(st.bias);
    const int m0 = blockIdx.x * R, rows = min(R, M - m0);
    const T *xr = x + (int64_t)m0 * st.K;
    const int n_w = st.K * st.N, n_x = rows * st.K;
    for (int i0 = threadIdx.x; i0 < n_w + n_x; i0 += 8 * 256) {
        T v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int i = i0 + j * 256;
            if (i < n_w) v[j] = __ldg(w + i);
            else if (i < n_w + n_x) v[j] = __ldg(xr + (i - n_w));
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (i0 + j * 256 < n_w + n_x) smem[i0 + j * 256] = to_f32(v[j]);
    }
    __syncthreads();
    const int total = rows * st.N * 4, padded = (total + 31) & ~31;   // whole warps take part in the shuffles
    for (int it = threadIdx.x; it < padded; it += 256) {
        const bool live = it < total;
        const int q = it & 3, o = live ? it >> 2 : 0, r = o / st.N, c = o - r * st.N;
        float p = 0.f;
        if (live) {
            const float *wp = ws + c, *xp = xs + r * st.K;
#pragma unroll 8
            for (int k = q; k < st.K; k += 4) p = fmaf(xp[k], wp[k * st.N], p);
        }
        p += __shfl_xor_sync(0xffffffffu, p, 1);
        p += __shfl_xor_sync(0xffffffffu, p, 2);
        if (!live || q != 0) continue;
        float v = to_f32(from_f32<T>(p));
        if (bias != nullptr) v = to_f32(from_f32<T>(__fadd_rn(v, to_f32(bias[c]))));
        if (st.relu) v = (v >= 0.f) ? v : 0.f;
        y[(int64_t)(m0 + r) * st.N + c] = from_f32<T>(v);
    }
}

// R rows x 32 columns per CTA, a warp per k slice.  Latency bound (a CTA streams kchunk weights
// per thread from L2), so a small batch is spread over rows and columns until every SM has a
// CTA instead of running 8 rows and all columns on each of a few.
template <class T, int R>
__global__ void __launch_bounds__(512)
    dense_small_kernel(const T *__restrict__ x, T *__restrict__ y, int M, const ChainStep st) {
    let_dependents_launch();
    dependency_wait();
    extern __shared__ __align__(16) float smem[];
    float *xs = smem;                          // [K][R]
    float *red = smem + (size_t)st.K * R;      // [slices][R][32]
    const T *w = reinterpret_cast<const T *>(st.w), *bias = reinterpret_cast<const T *>(st.bias);
    const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
    const int m0 = blockIdx.x * R, n = blockIdx.y * 32 + lane;
    const int k0 = slice * st.kchunk, k1 = min(st.K, k0 + st.kchunk);
    const bool live = n < st.N;
    // the first weights are on their way while x is staged
    constexpr int AHEAD = 16;
    float wv[AHEAD];
    const T *wp = w + (int64_t)k0 * st.N + n;
#pragma unroll
    for (int j = 0; j < AHEAD; ++j) wv[j] = live && k0 + j < k1 ? to_f32(wp[(int64_t)j * st.N]) : 0.f;
#pragma unroll
    for (int r = 0; r < R; ++r)
        for (int k = threadIdx.x; k < st.K; k += blockDim.x)
            xs[k * R + r] = m0 + r < M ? to_f32(x[(int64_t)(m0 + r) * st.K + k]) : 0.f;
    __syncthreads();
    float acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = 0.f;
    for (int k = k0; k < k1; k += AHEAD) {
        float cur[AHEAD];
#pragma unroll
        for (int j = 0; j < AHEAD; ++j) cur[j] = wv[j];
        wp += (int64_t)AHEAD * st.N;
#pragma unroll
        for (int j = 0; j < AHEAD; ++j)
            wv[j] = live && k + AHEAD + j < k1 ? to_f32(wp[(int64_t)j * st.N]) : 0.f;
#pragma unroll
        for (int j = 0; j < AHEAD; ++j) {
            if (k + j < k1) {
                const float *xk = xs + (k + j) * R;
#pragma unroll
                for (int r = 0; r < R; ++r) acc[r] = fmaf(xk[r], cur[j], acc[r]);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) red[(slice * R + r) * 32 + lane] = acc[r];
    __syncthreads();
    for (int i = threadIdx.x; i < R * 32; i += blockDim.x) {
        const int r = i / 32, c = blockIdx.y * 32 + (i & 31);
        if (c >= st.N || m0 + r >= M) continue;
        float s = 0.f;
        for (int sl = 0; sl < st.slices; ++sl) s += red[sl * R * 32 + i];
        float v = to_f32(from_f32<T>(s));
        if (bias != nullptr) v = to_f32(from_f32<T>(__fadd_rn(v, to_f32(bias[c]))));
        if (st.relu) v = (v >= 0.f) ? v : 0.f;
        y[(int64_t)(m0 + r) * st.N + c] = from_f32<T>(v);
    }
}

// Up to 512 inputs and 1.7e8 multiply-adds: beyond either the tensor-core engines are faster
// (602 x 861 x 163 f32: 21 us here, 13 us there; 32 x 2048 x 32: 30 and 5 us).  The limit on the
// multiply-adds keeps LeNet5's layers here up to kMostRows images (1.34e8).
bool eligible(int64_t m, int64_t k, int64_t n) {
    return m > 0 && m <= kMostRows && n > 0 && n <= 256 && k > 0 && k <= 512 && m * k * n <= 170000000;
}

bool fits_one_kernel(int64_t k, int64_t n) { return n > 0 && n <= 256 && k > 0 && k <= 2048; }

template <class T, int R>
static int launch_small(ag_device *dev, const T *x, T *y, int m, const ChainStep &st) {
    const size_t smem = ((size_t)st.K + (size_t)st.slices * 32) * R * sizeof(float);
    AG_TRY((launch_dependent(dev, dense_small_kernel<T, R>, dim3((unsigned)ceil_div(m, R), (unsigned)(st.np / 32)),
                             32 * st.slices, smem, x, y, m, st)));
    return AG_OK;
}

template <class T>
int forward(ag_device *dev, const T *x, int m, int k, const T *w, int n, const T *bias, bool relu,
            T *y) {
    ChainStep st = {};
    st.w = w; st.bias = bias;
    st.K = k; st.N = n; st.relu = relu ? 1 : 0;
    plan_step(k, n, &st.np, &st.slices, &st.kchunk);
    // Rows x columns against k: with many outputs the 8-row form's wider tiles win, with a long k the
    // spread form's larger number of loads in flight (f32 100 x 256 x 128: 7.9 us on 8 rows per CTA,
    // 4.2 us spread; 256^3 13.1 and 10.1; 384 x 145 x 135 5.9 and 6.8; bf16 256^3 13.1 and 13.9).
    if (narrow_step(st)) {
        // as many rows per CTA, up to four, as leave every SM one; 512 inputs and 16 outputs take 40 KB
        const int r = ceil_div(m, 4) >= dev->sm_count ? 4 : ceil_div(m, 2) >= dev->sm_count ? 2 : 1;
        AG_TRY((launch_dependent(dev, dense_narrow_kernel<T>, dim3((unsigned)ceil_div(m, r)), 256,
                                 sizeof(float) * (size_t)k * (n + r), x, y, m, r, st)));
        return AG_OK;
    }
    if ((int64_t)m * st.np > (sizeof(T) == 4 ? 256 : 128) * (int64_t)k) {
        const int threads = st.np * st.slices;
        const size_t smem = ((size_t)k * ROWS + (size_t)st.slices * ROWS * st.np) * sizeof(float);
        if (smem > 48 * 1024) {
            static SmemAllowed allowed;
            AG_TRY(allow_smem(dev, dense_rows_kernel<T>, allowed));
        }
        AG_TRY((launch_dependent(dev, dense_rows_kernel<T>, dim3((unsigned)ceil_div(m, ROWS)), threads, smem, x, y, m,
                                 st)));
        return AG_OK;
    }
    // the most rows per CTA (weights read once for them) that still give every SM eight warps;
    // shared memory stays below 48 KB with 512 inputs
    const int64_t warps = (int64_t)(st.np / 32) * st.slices;
    if (ceil_div(m, 4) * warps >= 8 * dev->sm_count) return launch_small<T, 4>(dev, x, y, m, st);
    if (ceil_div(m, 2) * warps >= 8 * dev->sm_count) return launch_small<T, 2>(dev, x, y, m, st);
    return launch_small<T, 1>(dev, x, y, m, st);
}

// ---------------------------------------------------------------- layer chain
template <class T>
__global__ void __launch_bounds__(1024)
    dense_chain_kernel(const T *__restrict__ x, T *__restrict__ y, const ChainParams p) {
    extern __shared__ __align__(16) float smem[];
    float *xa = smem;                              // [max_k][ROWS] current layer input
    float *xb = smem + (size_t)p.max_k * ROWS;     // next layer input
    float *red = xb + (size_t)p.max_k * ROWS;      // [slices][ROWS][np]
    const int m0 = blockIdx.x * ROWS;
    const int rows = min(ROWS, p.M - m0);
    {
        const int K = p.s[0].K;
        for (int i = threadIdx.x; i < ROWS * K; i += blockDim.x) {
            const int r = i / K, k = i - r * K;
            xa[k * ROWS + r] = (r < rows) ? to_f32(x[(int64_t)(m0 + r) * K + k]) : 0.f;
        }
    }
    __syncthreads();
    chain_layers<T>(xa, xb, red, p, m0, rows, y);
}

bool chain_eligible(int64_t m, int n_layers, const ChainLayer *layers) {
    if (n_layers < 2 || n_layers > kMaxChain) return false;
    for (int i = 0; i < n_layers; ++i) {
        if (!eligible(m, layers[i].inputs, layers[i].outputs)) return false;
        if (i > 0 && layers[i].inputs != layers[i - 1].outputs) return false;
    }
    return true;
}

template <class T>
int chain_forward(ag_device *dev, const T *x, int m, int n_layers, const ChainLayer *layers, T *y) {
    ChainParams p;
    const size_t smem = plan_chain(&p, m, n_layers, layers) * sizeof(float);
    const int threads = p.threads;
    auto kernel = dense_chain_kernel<T>;
    if (smem > 48 * 1024) {
        static SmemAllowed allowed;
        AG_TRY(allow_smem(dev, kernel, allowed));
    }
    kernel<<<(unsigned)ceil_div(m, ROWS), threads, smem, dev->stream>>>(x, y, p);
    AG_CHECK_LAUNCH();
    return AG_OK;
}

// ---------------------------------------------------------------- backward
template <class T>
__global__ void __launch_bounds__(1024)
    dense_chain_backward_kernel(const T *__restrict__ dy, const T *__restrict__ gate_last,
                                T *__restrict__ g_last, T *__restrict__ y, const ChainParams p) {
    extern __shared__ __align__(16) float smem[];
    float *xa = smem;
    float *xb = smem + (size_t)p.max_k * ROWS;
    float *red = xb + (size_t)p.max_k * ROWS;
    const int m0 = blockIdx.x * ROWS;
    const int rows = min(ROWS, p.M - m0);
    {
        const int K = p.s[0].K;
        for (int i = threadIdx.x; i < ROWS * K; i += blockDim.x) {
            const int r = i / K, k = i - r * K;
            float v = 0.f;
            if (r < rows) {
                const int64_t at = (int64_t)(m0 + r) * K + k;
                v = to_f32(dy[at]);
                if (gate_last != nullptr) {
                    if (!(to_f32(gate_last[at]) >= 0.f)) v = 0.f;
                    g_last[at] = from_f32<T>(v);
                }
            }
            xa[k * ROWS + r] = v;
        }
    }
    __syncthreads();
    chain_layers<T>(xa, xb, red, p, m0, rows, y);
}

bool chain_backward_eligible(int64_t m, int n_steps, const ChainLayer *steps) {
    if (n_steps < 1 || n_steps > kMaxChain) return false;
    for (int i = 0; i < n_steps; ++i) {
        if (!eligible(m, steps[i].inputs, steps[i].outputs)) return false;
        if (i > 0 && steps[i].inputs != steps[i - 1].outputs) return false;
    }
    return true;
}

template <class T>
int chain_backward_input(ag_device *dev, const T *dy, int m, int n_steps, const ChainLayer *steps,
                         const T *gate_last, T *g_last, T *y) {
    ChainParams p;
    const size_t smem = plan_chain(&p, m, n_steps, steps) * sizeof(float);
    auto kernel = dense_chain_backward_kernel<T>;
    if (smem > 48 * 1024) {
        static SmemAllowed allowed;
        AG_TRY(allow_smem(dev, kernel, allowed));
    }
    kernel<<<(unsigned)ceil_div(m, ROWS), p.threads, smem, dev->stream>>>(dy, gate_last, g_last, y, p);
    AG_CHECK_LAUNCH();
    return AG_OK;
}

// A 32 x 32 tile of one problem's dw per CTA of 256 threads.  The reduction runs over the
// batch in chunks of 128 rows staged whole in shared memory; the four groups of 64 threads
// each take a quarter of every chunk for the full tile (4 x 4 outputs per thread) and their
// sums are added in group order.  The CTAs of a problem's first tile row also add up the
// columns of g (the bias gradient), row after row.
constexpr int kWgChunk = 128, kWgPitch = 36;
struct WgradParams {
    WgradProblem p[kMaxChain];
    int n, M;
};

template <class T>
__global__ void __launch_bounds__(256) dense_wgrad_group_kernel(const WgradParams P) {
    __shared__ __align__(16) float As[kWgChunk][kWgPitch];
    __shared__ __align__(16) float Bs[kWgChunk][kWgPitch];
    int q = 0;
    while (q + 1 < P.n && (int)blockIdx.x >= P.p[q + 1].tile0) ++q;
    const WgradProblem pr = P.p[q];
    const int tile = blockIdx.x - pr.tile0;
    const int tm = tile / pr.tiles_n, tn = tile - tm * pr.tiles_n;
    const int m0 = tm * 32, n0 = tn * 32;
    const T *in = reinterpret_cast<const T *>(pr.in), *g = reinterpret_cast<const T *>(pr.g);
    const int tid = threadIdx.x;
    const int mn = tid & 31, kb = tid >> 5;  // staging: 32 consecutive columns of one batch row
    const int kg = tid >> 6, t = tid & 63, tx = t & 7, ty = t >> 3;
    const bool sums = pr.db != nullptr && tm == 0 && tid < 32;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    float bsum = 0.f;

    for (int kc = 0; kc < P.M; kc += kWgChunk) {
        const int chunk = min(kWgChunk, P.M - kc);
        float ra[kWgChunk / 8], rb[kWgChunk / 8];
#pragma unroll
        for (int i = 0; i < kWgChunk / 8; ++i)
            if (i * 8 < chunk) {
                const int k = i * 8 + kb;
                const bool ok = k < chunk;
                ra[i] = (ok && m0 + mn < pr.rows)
                            ? to_f32(in[(int64_t)(kc + k) * pr.rows + m0 + mn]) : 0.f;
                rb[i] = (ok && n0 + mn < pr.cols)
                            ? to_f32(g[(int64_t)(kc + k) * pr.cols + n0 + mn]) : 0.f;
            }
        if (kc > 0) __syncthreads();  // the previous chunk is no longer read
#pragma unroll
        for (int i = 0; i < kWgChunk / 8; ++i)
            if (i * 8 < chunk) {
                As[i * 8 + kb][mn] = ra[i];
                Bs[i * 8 + kb][mn] = rb[i];
            }
        __syncthreads();
        const int kp = (chunk + 7) & ~7;
        const int kq = (kp / 8 + 3) / 4 * 8;
        const int k0 = min(kp, kg * kq), k1 = min(kp, k0 + kq);
#pragma unroll 4
        for (int k = k0; k < k1; ++k) {
            const float4 a4 = *reinterpret_cast<const float4 *>(&As[k][ty * 4]);
            const float4 b4 = *reinterpret_cast<const float4 *>(&Bs[k][tx * 4]);
            const float a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        if (sums)
            for (int k = 0; k < chunk; ++k) bsum += Bs[k][tid];
    }
    __syncthreads();
    float *red = &As[0][0];  // [3 groups][16 values][64 threads]
    if (kg > 0) {
#pragma unroll
        for (int i = 0; i < 16; ++i) red[((kg - 1) * 16 + i) * 64 + t] = acc[i / 4][i % 4];
    }
    __syncthreads();
    if (sums && n0 + tid < pr.cols) reinterpret_cast<T *>(pr.db)[n0 + tid] = from_f32<T>(bsum);
    if (kg > 0) return;
#pragma unroll
    for (int gi = 0; gi < 3; ++gi)
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i / 4][i % 4] += red[(gi * 16 + i) * 64 + t];
    T *dw = reinterpret_cast<T *>(pr.dw);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= pr.rows) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n < pr.cols) dw[(int64_t)m * pr.cols + n] = from_f32<T>(acc[i][j]);
        }
    }
}

template <class T>
int chain_weight_grads(ag_device *dev, int m, int n, WgradProblem *problems) {
    WgradParams P;
    P.n = n;
    P.M = m;
    int tiles = 0;
    for (int i = 0; i < n; ++i) {
        problems[i].tile0 = tiles;
        problems[i].tiles_n = (problems[i].cols + 31) / 32;
        tiles += ((problems[i].rows + 31) / 32) * problems[i].tiles_n;
        P.p[i] = problems[i];
    }
    if (tiles == 0) return AG_OK;
    dense_wgrad_group_kernel<T><<<(unsigned)tiles, 256, 0, dev->stream>>>(P);
    AG_CHECK_LAUNCH();
    return AG_OK;
}

// C[m][n] = sum over k of A[k][m] . B[k][n], k <= kFewK, n <= NP: the weight gradient of a layer with few outputs.  A lane owns a
// column of A and all of B's, so A is read once, coalesced, and B comes from shared memory for the whole warp; the sixteen
// warps take every sixteenth k and their sums are added in warp order.
constexpr int kColWarps = 16;
template <class T, int NP>
__global__ void __launch_bounds__(kColWarps * 32)
    few_columns_kernel(const T *__restrict__ a, int64_t lda, const T *__restrict__ b, int64_t ldb, T *__restrict__ c,
                       int64_t ldc, int M, int K, int N) {
    let_dependents_launch();
    dependency_wait();
    constexpr int kFloats = kColWarps * NP * 33 > kFewK * NP ? kColWarps * NP * 33 : kFewK * NP;
    __shared__ __align__(16) float buf[kFloats];   // [k][NP] of B, then [warp][NP][33] sums
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, m = blockIdx.x * 32 + lane;
    float acc[NP];
#pragma unroll
    for (int j = 0; j < NP; ++j) acc[j] = 0.f;
    for (int i = threadIdx.x; i < K * NP; i += kColWarps * 32) {
        const int k = i / NP, j = i % NP;
        buf[i] = load_or_zero(b + (int64_t)k * ldb + j, j < N);
    }
    __syncthreads();
    for (int k0 = warp; k0 < K; k0 += 8 * kColWarps) {
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int k = k0 + u * kColWarps;
            v[u] = load_or_zero(a + (int64_t)k * lda + m, k < K && m < M);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int k = k0 + u * kColWarps;
            if (k >= K) break;   // what shared memory holds there may be anything
#pragma unroll
            for (int j = 0; j < NP; j += 4) {
                const float4 w = *reinterpret_cast<const float4 *>(buf + k * NP + j);
                acc[j] = fmaf(v[u], w.x, acc[j]);
                acc[j + 1] = fmaf(v[u], w.y, acc[j + 1]);
                acc[j + 2] = fmaf(v[u], w.z, acc[j + 2]);
                acc[j + 3] = fmaf(v[u], w.w, acc[j + 3]);
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < NP; ++j) buf[(warp * NP + j) * 33 + lane] = acc[j];
    __syncthreads();
    for (int i = threadIdx.x; i < 32 * N; i += kColWarps * 32) {
        const int r = i / N, j = i - r * N;
        if (blockIdx.x * 32 + r >= M) break;
        float s = buf[j * 33 + r];
#pragma unroll
        for (int w = 1; w < kColWarps; ++w) s += buf[(w * NP + j) * 33 + r];
        c[(int64_t)(blockIdx.x * 32 + r) * ldc + j] = from_f32<T>(s);
    }
}

template <class T>
int few_columns(ag_device *dev, int m, int k, int n, const T *a, int64_t lda, const T *b, int64_t ldb, T *c, int64_t ldc) {
    AG_REQUIRE(k <= kFewK && n <= kFewColumns, AG_ERR_LIMIT, "product has too many columns or too long a k");
    const dim3 grid((unsigned)ceil_div(m, 32));
    auto kernel = n <= 4 ? few_columns_kernel<T, 4> : n <= 8 ? few_columns_kernel<T, 8>
                : n <= 12 ? few_columns_kernel<T, 12> : few_columns_kernel<T, 16>;
    return launch_dependent(dev, kernel, grid, kColWarps * 32, 0, a, lda, b, ldb, c, ldc, m, k, n);
}
template int few_columns<float>(ag_device *, int, int, int, const float *, int64_t, const float *, int64_t, float *, int64_t);
template int few_columns<__nv_bfloat16>(ag_device *, int, int, int, const __nv_bfloat16 *, int64_t, const __nv_bfloat16 *,
                                        int64_t, __nv_bfloat16 *, int64_t);

template int chain_backward_input<float>(ag_device *, const float *, int, int, const ChainLayer *,
                                         const float *, float *, float *);
template int chain_backward_input<__nv_bfloat16>(ag_device *, const __nv_bfloat16 *, int, int,
                                                 const ChainLayer *, const __nv_bfloat16 *,
                                                 __nv_bfloat16 *, __nv_bfloat16 *);
template int chain_weight_grads<float>(ag_device *, int, int, WgradProblem *);
template int chain_weight_grads<__nv_bfloat16>(ag_device *, int, int, WgradProblem *);

template int chain_forward<float>(ag_device *, const float *, int, int, const ChainLayer *, float *);
template int chain_forward<__nv_bfloat16>(ag_device *, const __nv_bfloat16 *, int, int,
                                          const ChainLayer *, __nv_bfloat16 *);

template int forward<float>(ag_device *, const float *, int, int, const float *, int, const float *,
                            bool, float *);
template int forward<__nv_bfloat16>(ag_device *, const __nv_bfloat16 *, int, int,
                                    const __nv_bfloat16 *, int, const __nv_bfloat16 *, bool,
                                    __nv_bfloat16 *);

}  // namespace dense_small
}  // namespace ag
