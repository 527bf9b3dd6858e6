// Memory-bound operators: relu, max-pool, scaled add, bias add / bias gradient
// and the SGD updates.  Each kernel moves 16 bytes per thread per access where
// the layout allows it and is sized as a grid-stride loop over a multiple of
// the SM count.  Arithmetic is written with explicit round-to-nearest multiply
// and add (no fused multiply-add) so that results are bit-identical to the
// reference's host code, which does not contract.
#include <algorithm>

#include "common.cuh"

namespace ag {

static unsigned grid_for(int64_t items, int threads, int sms) {
    int64_t blocks = ceil_div(items, threads);
    int64_t cap = (int64_t)sms * 8;
    return (unsigned)(blocks < cap ? (blocks < 1 ? 1 : blocks) : cap);
}

// 16-byte vector of T.
template <class T>
struct Vec16 {
    static constexpr int N = 16 / sizeof(T);
    uint4 raw;
    __device__ __forceinline__ float get(int i) const;
    __device__ __forceinline__ void set(int i, float v);
};
template <>
__device__ __forceinline__ float Vec16<float>::get(int i) const {
    return __uint_as_float((&raw.x)[i]);
}
template <>
__device__ __forceinline__ void Vec16<float>::set(int i, float v) {
    (&raw.x)[i] = __float_as_uint(v);
}
template <>
__device__ __forceinline__ float Vec16<__nv_bfloat16>::get(int i) const {
    uint32_t w = (&raw.x)[i >> 1];
    return __uint_as_float((i & 1) ? (w & 0xffff0000u) : (w << 16));
}
template <>
__device__ __forceinline__ void Vec16<__nv_bfloat16>::set(int i, float v) {
    __nv_bfloat16 h = __float2bfloat16_rn(v);
    uint32_t bits = *reinterpret_cast<unsigned short *>(&h);
    uint32_t &w = (&raw.x)[i >> 1];
    w = (i & 1) ? ((w & 0x0000ffffu) | (bits << 16)) : ((w & 0xffff0000u) | bits);
}

template <class T>
static bool aligned16(const T *p) {
    return (reinterpret_cast<uintptr_t>(p) & 15) == 0;
}

// ---- generic unary / binary / ternary element-wise driver --------------------
// f(i, in0[i], in1[i]) -> out[i]; vector body when every pointer is 16-byte aligned.
template <class T, class F>
__global__ void map2_kernel(const T *a, const T *b, T *out,
                            int64_t n, bool vec, F f) {
    let_dependents_launch();
    dependency_wait();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    constexpr int V = Vec16<T>::N;
    int64_t done = 0;
    if (vec) {
        const int64_t nv = n / V;
        for (int64_t i = tid; i < nv; i += stride) {
            Vec16<T> va, vb, vo;
            va.raw = reinterpret_cast<const uint4 *>(a)[i];
            vb.raw = b ? reinterpret_cast<const uint4 *>(b)[i] : va.raw;
            vo.raw = make_uint4(0, 0, 0, 0);
#pragma unroll
            for (int j = 0; j < V; ++j) vo.set(j, f(va.get(j), vb.get(j)));
            reinterpret_cast<uint4 *>(out)[i] = vo.raw;
        }
        done = nv * V;
    }
    for (int64_t i = done + tid; i < n; i += stride) {
        float x = to_f32(a[i]);
        float y = b ? to_f32(b[i]) : x;
        out[i] = from_f32<T>(f(x, y));
    }
}

template <class T, class F>
static int map2(ag_device *dev, const T *a, const T *b, T *out, int64_t n, F f) {
    if (n == 0) return AG_OK;
    const bool vec = aligned16(a) && aligned16(out) && (b == nullptr || aligned16(b));
    const int threads = 256;
    const int64_t items = vec ? ceil_div(n, Vec16<T>::N) : n;
    AG_TRY((launch_dependent(dev, map2_kernel<T, F>,
                             dim3(grid_for(items, threads, dev->sm_count)), threads, 0, a, b, out, n, vec, f)));
    return AG_OK;
}

struct ReluF {
    __device__ __forceinline__ float operator()(float x, float) const {
        return (x >= 0.f) ? x : 0.f;
    }
};
struct ReluBackwardF {  // (x, dy)
    __device__ __forceinline__ float operator()(float x, float dy) const {
        return (x >= 0.f) ? dy : 0.f;
    }
};
template <class T>
struct ScaledAddF {  // (x, y) -> alpha*x + y in T arithmetic
    float alpha;
    __device__ __forceinline__ float operator()(float x, float y) const {
        float p = to_f32(from_f32<T>(__fmul_rn(alpha, x)));
        return __fadd_rn(p, y);
    }
};

// ---- max pool ---------------------------------------------------------------
template <class T>
__global__ void max_pool2_kernel(const T *__restrict__ x, T *__restrict__ y, int64_t planes,
                                 int ih, int iw, int oh, int ow, int h, int w, int sh, int sw) {
    const int64_t total = planes * oh * ow;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        int wid = (int)(i % ow);
        int64_t t = i / ow;
        int hid = (int)(t % oh);
        int64_t plane = t / oh;
        const T *src = x + (plane * ih + (int64_t)hid * sh) * iw + (int64_t)wid * sw;
        float m = 0.f;
        for (int fi = 0; fi < h; ++fi)
            for (int fj = 0; fj < w; ++fj) {
                float v = to_f32(src[fi * iw + fj]);
                if ((fi == 0 && fj == 0) || v > m) m = v;
            }
        y[i] = from_f32<T>(m);
    }
}

// 2x2 window, stride 2, even width, 16-byte aligned rows: each thread reads two
// 16-byte row segments and writes V/2 outputs.
template <class T>
__global__ void max_pool2_2x2_kernel(const T *__restrict__ x, T *__restrict__ y, int64_t planes,
                                     int ih, int iw, int oh, int ow) {
    let_dependents_launch();
    dependency_wait();
    constexpr int V = Vec16<T>::N;  // inputs per vector
    const int vec_per_row = iw / V;
    const int64_t total = planes * oh * vec_per_row;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        int vx = (int)(i % vec_per_row);
        int64_t t = i / vec_per_row;
        int hid = (int)(t % oh);
        int64_t plane = t / oh;
        const T *r0 = x + (plane * ih + 2 * (int64_t)hid) * iw + vx * V;
        Vec16<T> a, b;
        a.raw = *reinterpret_cast<const uint4 *>(r0);
        b.raw = *reinterpret_cast<const uint4 *>(r0 + iw);
        T *dst = y + (plane * oh + hid) * (int64_t)ow + vx * (V / 2);
#pragma unroll
        for (int j = 0; j < V / 2; ++j) {
            float m = a.get(2 * j);
            float v = a.get(2 * j + 1);
            if (v > m) m = v;
            v = b.get(2 * j);
            if (v > m) m = v;
            v = b.get(2 * j + 1);
            if (v > m) m = v;
            dst[j] = from_f32<T>(m);
        }
    }
}

// One thread per window; windows do not overlap, so no two threads touch the
// same cell.  dx holds the forward input on entry.
template <class T>
__global__ void max_pool2_backward_kernel(T *__restrict__ dx, const T *__restrict__ dy,
                                          int64_t planes, int ih, int iw, int oh, int ow, int h,
                                          int w, int sh, int sw) {  // in place only
    const int64_t total = planes * oh * ow;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        int wid = (int)(i % ow);
        int64_t t = i / ow;
        int hid = (int)(t % oh);
        int64_t plane = t / oh;
        T *win = dx + (plane * ih + (int64_t)hid * sh) * iw + (int64_t)wid * sw;
        float m = 0.f;
        int am = 0;
        for (int fi = 0; fi < h; ++fi)
            for (int fj = 0; fj < w; ++fj) {
                float v = to_f32(win[fi * iw + fj]);
                if ((fi == 0 && fj == 0) || v > m) {
                    m = v;
                    am = fi * iw + fj;
                }
                win[fi * iw + fj] = from_f32<T>(0.f);
            }
        win[am] = from_f32<T>(__fadd_rn(0.f, to_f32(dy[i])));
    }
}

// 2x2 window, stride 2, width a multiple of the vector length, 16-byte aligned rows:
// each thread owns V/2 adjacent windows, reads and rewrites two 16-byte row segments.
template <class T>
__global__ void max_pool2_backward_2x2_kernel(const T *src, T *dx, const T *__restrict__ dy,
                                              int64_t planes, int ih, int iw, int oh, int ow) {
    let_dependents_launch();
    dependency_wait();
    constexpr int V = Vec16<T>::N;
    const int vec_per_row = iw / V;
    const int64_t total = planes * oh * vec_per_row;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        int vx = (int)(i % vec_per_row);
        int64_t t = i / vec_per_row;
        int hid = (int)(t % oh);
        int64_t plane = t / oh;
        const int64_t off = (plane * ih + 2 * (int64_t)hid) * iw + vx * V;
        T *r0 = dx + off;
        const T *g = dy + (plane * oh + hid) * (int64_t)ow + vx * (V / 2);
        Vec16<T> a, b, oa, ob;
        a.raw = *reinterpret_cast<const uint4 *>(src + off);
        b.raw = *reinterpret_cast<const uint4 *>(src + off + iw);
        oa.raw = make_uint4(0, 0, 0, 0);
        ob.raw = make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int j = 0; j < V / 2; ++j) {
            // window order (0,0),(0,1),(1,0),(1,1); the first maximum wins
            float m = a.get(2 * j);
            int am = 0;
            float v = a.get(2 * j + 1);
            if (v > m) { m = v; am = 1; }
            v = b.get(2 * j);
            if (v > m) { m = v; am = 2; }
            v = b.get(2 * j + 1);
            if (v > m) { m = v; am = 3; }
            const float gv = __fadd_rn(0.f, to_f32(g[j]));
            oa.set(2 * j, am == 0 ? gv : 0.f);
            oa.set(2 * j + 1, am == 1 ? gv : 0.f);
            ob.set(2 * j, am == 2 ? gv : 0.f);
            ob.set(2 * j + 1, am == 3 ? gv : 0.f);
        }
        *reinterpret_cast<uint4 *>(r0) = oa.raw;
        *reinterpret_cast<uint4 *>(r0 + iw) = ob.raw;
    }
}

// Windows of 2x2 with stride 2 over planes of any size.  One window per thread with 64-bit divisions kept too few
// bytes in flight (bf16, 6528 planes of 36 x 36: forward 11.8 us, gradient 13.2; now 6.5 and 8.9), and odd widths
// went through shared memory (8128 planes of 55 x 55: 38.9 and 57.3; now 14.3 and 38.2).  From DRAM, replayed; the bytes
// of the two take 3.4 and 6, 9.4 and 17 us.  Forward, a thread loads all cells of W windows before it uses the first:
// as many as fill the loads in flight (16384 planes of 62 x 62 f32: 51.8 us with one, 47.3 with two, 53.1 with four;
// bf16 39.2, 40.0, 41.8; 8128 of 55 x 55 bf16 14.3, 15.1, 14.2).  The gradient takes one: it stores as much as
// it loads, and more windows a thread only cost warps (62 x 62 f32 89 to 92 us, with four 102 to 104; bf16 59, 89).  PAIR:
// even widths, rows that keep pairs aligned.
// Offsets are 32-bit: the host cuts the planes into launches of fewer than 2^32 cells.
struct PoolMap {
    int ih, iw, gh, gw;      // plane, grid of windows
    uint32_t total;          // windows of this launch
    FastDiv div_gw, div_gh;
};
template <class T, bool PAIR>
constexpr int pool_windows_per_thread() { return sizeof(T) == 4 ? 2 : PAIR ? 1 : 4; }
__device__ __forceinline__ uint32_t raw_of(__nv_bfloat16 v) { return __bfloat16_as_ushort(v); }
__device__ __forceinline__ uint32_t raw_of(float v) { return __float_as_uint(v); }
template <class T>
__device__ __forceinline__ float value_of(uint32_t raw) { return __uint_as_float(sizeof(T) == 2 ? raw << 16 : raw); }
// Two neighbouring elements at an address that is a multiple of their size (4 bytes for bf16, 8 for f32), as bits.
__device__ __forceinline__ void load_word(const __nv_bfloat16 *p, uint32_t &a, uint32_t &b) {
    const uint32_t w = *reinterpret_cast<const uint32_t *>(p);
    a = w & 0xffffu;
    b = w >> 16;
}
__device__ __forceinline__ void load_word(const float *p, uint32_t &a, uint32_t &b) {
    const uint2 w = *reinterpret_cast<const uint2 *>(p);
    a = w.x;
    b = w.y;
}
__device__ __forceinline__ void store_word(__nv_bfloat16 *p, uint32_t a, uint32_t b) { *reinterpret_cast<uint32_t *>(p) = a | b << 16; }
__device__ __forceinline__ void store_word(float *p, uint32_t a, uint32_t b) { *reinterpret_cast<uint2 *>(p) = make_uint2(a, b); }
__device__ __forceinline__ void store_cell(__nv_bfloat16 *p, uint32_t a) { *p = __ushort_as_bfloat16((unsigned short)a); }
__device__ __forceinline__ void store_cell(float *p, uint32_t a) { *p = __uint_as_float(a); }

// RELU: the window is taken over relu(x) (x >= 0 ? x : 0), i.e. Relu followed by the pool.
template <class T, bool RELU, bool PAIR>
__global__ void __launch_bounds__(256) max_pool2_2x2_window_kernel(const T *__restrict__ x, T *__restrict__ y, const PoolMap m) {
    let_dependents_launch();
    dependency_wait();
    constexpr int W = pool_windows_per_thread<T, PAIR>();
    for (uint32_t i0 = blockIdx.x * (256u * W) + threadIdx.x; i0 < m.total; i0 += gridDim.x * (256u * W)) {
        uint32_t v[W][4];
#pragma unroll
        for (int u = 0; u < W; ++u) {
            const uint32_t i = i0 + (uint32_t)u * 256u;
            if (i >= m.total) break;
            uint32_t wx, wy, t, plane;
            m.div_gw.divmod(i, t, wx);
            m.div_gh.divmod(t, plane, wy);
            const T *q = x + ((plane * (uint32_t)m.ih + 2 * wy) * (uint32_t)m.iw + 2 * wx), *q1 = q + m.iw;
            if (PAIR) {
                load_word(q, v[u][0], v[u][1]);
                load_word(q1, v[u][2], v[u][3]);
            } else {
                v[u][0] = raw_of(q[0]);
                v[u][1] = raw_of(q[1]);
                v[u][2] = raw_of(q1[0]);
                v[u][3] = raw_of(q1[1]);
            }
        }
#pragma unroll
        for (int u = 0; u < W; ++u) {
            const uint32_t i = i0 + (uint32_t)u * 256u;
            if (i >= m.total) break;
            float best = 0.f;  // window order (0,0),(0,1),(1,0),(1,1); the first maximum wins
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float c = value_of<T>(v[u][j]);
                if (RELU) c = c >= 0.f ? c : 0.f;
                if (j == 0 || c > best) best = c;
            }
            y[i] = from_f32<T>(best);
        }
    }
}

// Two neighbouring cells of a window's row, where rows start anywhere: as one word where the first cell's address
// is even, else the word of the left neighbour's second cell and this lane's first one, so that a warp's stores
// cover whole words.  Called by whole warps; lanes hold consecutive windows.  `left`: the lane below holds the
// window to the left; `right`: the lane above holds the one to the right and stores this lane's second cell.
template <class T>
__device__ __forceinline__ void store_row(T *p, uint32_t a, uint32_t b, bool row, bool second, bool left, bool right) {
    const uint32_t before = __shfl_up_sync(0xffffffffu, b, 1);
    if (!row) return;
    if (reinterpret_cast<uintptr_t>(p) % (2 * sizeof(T)) == 0) {
        if (second) store_word(p, a, b);
        else store_cell(p, a);
        return;
    }
    if (left) store_word(p - 1, before, a);
    else store_cell(p, a);
    if (second && !right) store_cell(p + 1, b);
}

// Gradient of the same: src holds the forward input, dx receives dy at the first maximum of every window and
// zero elsewhere; cells that no window covers (the last row or column of an odd plane) keep src's value.  The
// grid counts those cells' partial windows too (gw = ceil(iw / 2)).  src may be dx: a warp has read its
// window's cells before it writes them.  RELU (even planes): src is the input of a Relu whose output was
// pooled; the result is the gradient at that input (the pool's gradient gated by src >= 0, as Relu's
// backward gates it).
template <class T, bool RELU, bool PAIR>
__global__ void __launch_bounds__(256) max_pool2_backward_2x2_window_kernel(const T *src, T *dx, const T *__restrict__ dy,
                                                                            const PoolMap m, int oh, int ow) {
    let_dependents_launch();
    dependency_wait();
    const uint32_t lane = threadIdx.x % 32;
    // whole warps: i - lane is the warp's first window
    for (uint32_t i = blockIdx.x * 256u + threadIdx.x; i - lane < m.total; i += gridDim.x * 256u) {
        const bool mine = i < m.total;
        uint32_t v[4] = {}, off = 0, wx = 0, wy = 0;   // cells as they lie in memory
        bool second = true, below = true;
        float g = 0.f;
        if (mine) {
            uint32_t t, plane;
            m.div_gw.divmod(i, t, wx);
            m.div_gh.divmod(t, plane, wy);
            off = (plane * (uint32_t)m.ih + 2 * wy) * (uint32_t)m.iw + 2 * wx;
            const T *q = src + off, *q1 = q + m.iw;
            if (PAIR) {
                g = to_f32(dy[i]);
                load_word(q, v[0], v[1]);
                load_word(q1, v[2], v[3]);
            } else {
                second = (int)(2 * wx) < m.iw - 1;
                below = (int)(2 * wy) < m.ih - 1;
                v[0] = raw_of(q[0]);
                if (second) v[1] = raw_of(q[1]);
                if (below) v[2] = raw_of(q1[0]);
                if (second && below) {
                    v[3] = raw_of(q1[1]);
                    g = to_f32(dy[(plane * (uint32_t)oh + wy) * (uint32_t)ow + wx]);
                }
            }
        }
        if (second && below) {
            float c[4];
            bool pass[4] = {true, true, true, true};  // Relu lets the gradient pass
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                c[j] = value_of<T>(v[j]);
                if (RELU) {
                    pass[j] = c[j] >= 0.f;
                    c[j] = pass[j] ? c[j] : 0.f;
                }
            }
            float best = c[0];
            int am = 0;
#pragma unroll
            for (int j = 1; j < 4; ++j)
                if (c[j] > best) {
                    best = c[j];
                    am = j;
                }
            const uint32_t gv = raw_of(from_f32<T>(__fadd_rn(0.f, g)));   // one conversion, then bits
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = am == j && pass[j] ? gv : 0u;
        }
        T *d = dx + off;
        if (PAIR) {
            if (!mine) continue;
            store_word(d, v[0], v[1]);
            store_word(d + m.iw, v[2], v[3]);
        } else {
            const bool left = lane > 0 && wx > 0, right = lane < 31 && wx + 1 < (uint32_t)m.gw && i + 1 < m.total;
            store_row<T>(d, v[0], v[1], mine, second, left, right);
            store_row<T>(d + m.iw, v[2], v[3], mine && below, second, left, right);
        }
    }
}

// Calls launch(first plane, first row of windows, map, grid) for as many planes at a time as 32-bit offsets hold;
// a plane of more cells than that is cut along its rows.  gh x gw windows a plane.
template <class F>
static int for_pool_planes(ag_device *dev, int64_t planes, int64_t ih, int64_t iw, int64_t gh, int64_t gw, int per_thread, F launch) {
    constexpr int64_t kCells = (1ll << 32) - 1;
    const int64_t most = kCells / ((ih + 1) * (iw + 1));
    const int64_t at_once = most < 1 ? 1 : most, rows = most < 1 ? kCells / (2 * (iw + 1)) : gh;
    for (int64_t p = 0; p < planes; p += at_once)
        for (int64_t y = 0; y < gh; y += rows) {
            const int64_t n = std::min(at_once, planes - p), band = std::min(rows, gh - y);
            const PoolMap m{(int)(y + band == gh ? ih - 2 * y : 2 * band), (int)iw, (int)band, (int)gw,
                            (uint32_t)(n * band * gw), FastDiv((uint32_t)gw), FastDiv((uint32_t)band)};
            AG_TRY(launch(p, y, m, dim3(grid_for(ceil_div((int64_t)m.total, per_thread), 256, dev->sm_count))));
        }
    return AG_OK;
}

template <class T>
static bool pair_aligned(const T *p) {
    return reinterpret_cast<uintptr_t>(p) % (2 * sizeof(T)) == 0;
}

// Relu + pool takes pairs alone (relu_pool_check): the other form is not compiled for it.
template <class T, bool RELU, bool PAIR>
static int pool_windows_as(ag_device *dev, const T *x, T *y, int64_t planes, int64_t ih, int64_t iw, int64_t oh, int64_t ow) {
    return for_pool_planes(dev, planes, ih, iw, oh, ow, pool_windows_per_thread<T, PAIR>(),
                           [&](int64_t p, int64_t y0, const PoolMap &m, dim3 grid) {
        return launch_dependent(dev, max_pool2_2x2_window_kernel<T, RELU, PAIR>, grid, 256, 0,
                                x + (p * ih + 2 * y0) * iw,
                                y + (p * oh + y0) * ow, m);
    });
}

template <class T, bool RELU>
static int pool_windows(ag_device *dev, const T *x, T *y, int64_t planes, int64_t ih, int64_t iw, int64_t oh, int64_t ow) {
    if constexpr (!RELU)
        if ((iw & 1) != 0 || !pair_aligned(x)) return pool_windows_as<T, RELU, false>(dev, x, y, planes, ih, iw, oh, ow);
    return pool_windows_as<T, RELU, true>(dev, x, y, planes, ih, iw, oh, ow);
}

template <class T, bool RELU, bool PAIR>
static int pool_windows_backward_as(ag_device *dev, const T *x, T *dx, const T *dy, int64_t planes, int64_t ih, int64_t iw,
                                    int64_t oh, int64_t ow) {
    return for_pool_planes(dev, planes, ih, iw, (ih + 1) / 2, (iw + 1) / 2, 1,
                           [&](int64_t p, int64_t y0, const PoolMap &m, dim3 grid) {
        const int64_t at = (p * ih + 2 * y0) * iw;
        return launch_dependent(dev, max_pool2_backward_2x2_window_kernel<T, RELU, PAIR>, grid, 256, 0, x + at, dx + at,
                                dy + (p * oh + y0) * ow, m, (int)oh, (int)ow);
    });
}

template <class T, bool RELU>
static int pool_windows_backward(ag_device *dev, const T *x, T *dx, const T *dy, int64_t planes, int64_t ih, int64_t iw, int64_t oh,
                                 int64_t ow) {
    // pairs: every cell is in a window
    if constexpr (!RELU)
        if ((iw & 1) != 0 || (ih & 1) != 0 || !pair_aligned(x) || !pair_aligned(dx))
            return pool_windows_backward_as<T, RELU, false>(dev, x, dx, dy, planes, ih, iw, oh, ow);
    return pool_windows_backward_as<T, RELU, true>(dev, x, dx, dy, planes, ih, iw, oh, ow);
}

// Any non-overlapping window, any width: a CTA stages a run of whole planes in
// shared memory with 16-byte loads (the staged copy keeps the alignment of the
// global run), works on the windows there, and writes the run back with 16-byte
// stores, so the 2- and 4-byte window accesses never reach global memory.
template <class T>
__global__ void max_pool2_backward_staged_kernel(const T *src, T *dx, const T *__restrict__ dy,
                                                 int64_t planes, int ih, int iw, int oh, int ow,
                                                 int h, int w, int sh, int sw, int per_cta) {
    extern __shared__ __align__(16) unsigned char staged_raw[];
    T *s = reinterpret_cast<T *>(staged_raw);
    constexpr int V = 16 / (int)sizeof(T);
    const int plane_len = ih * iw;
    for (int64_t p0 = (int64_t)blockIdx.x * per_cta; p0 < planes;
         p0 += (int64_t)gridDim.x * per_cta) {
        const int np = (int)min((int64_t)per_cta, planes - p0);
        const int n = np * plane_len;
        const T *in = src + p0 * plane_len;
        T *base = dx + p0 * plane_len;
        // the staged copy keeps the 16-byte phase of the source run; the run is written back
        // with 16-byte stores when the destination run has the same phase (always, in place)
        const int shift = (int)((reinterpret_cast<uintptr_t>(in) & 15) / sizeof(T));
        const bool same_phase =
            shift == (int)((reinterpret_cast<uintptr_t>(base) & 15) / sizeof(T));
        const int head = min(n, (V - shift) % V);
        const int nv = (n - head) / V;
        const int tail0 = head + nv * V;
        for (int i = threadIdx.x; i < head; i += blockDim.x) s[shift + i] = in[i];
        for (int v = threadIdx.x; v < nv; v += blockDim.x)
            *reinterpret_cast<uint4 *>(s + shift + head + v * V) =
                *reinterpret_cast<const uint4 *>(in + head + v * V);
        for (int i = tail0 + threadIdx.x; i < n; i += blockDim.x) s[shift + i] = in[i];
        __syncthreads();
        const int windows = np * oh * ow;
        const T *g = dy + p0 * oh * ow;
        for (int i = threadIdx.x; i < windows; i += blockDim.x) {
            const int wid = i % ow;
            const int t = i / ow;
            const int hid = t % oh, plane = t / oh;
            T *win = s + shift + plane * plane_len + hid * sh * iw + wid * sw;
            float m = 0.f;
            int am = 0;
            for (int fi = 0; fi < h; ++fi)
                for (int fj = 0; fj < w; ++fj) {
                    const float v = to_f32(win[fi * iw + fj]);
                    if ((fi == 0 && fj == 0) || v > m) {
                        m = v;
                        am = fi * iw + fj;
                    }
                    win[fi * iw + fj] = from_f32<T>(0.f);
                }
            win[am] = from_f32<T>(__fadd_rn(0.f, to_f32(g[i])));
        }
        __syncthreads();
        if (same_phase) {
            for (int i = threadIdx.x; i < head; i += blockDim.x) base[i] = s[shift + i];
            for (int v = threadIdx.x; v < nv; v += blockDim.x)
                *reinterpret_cast<uint4 *>(base + head + v * V) =
                    *reinterpret_cast<const uint4 *>(s + shift + head + v * V);
            for (int i = tail0 + threadIdx.x; i < n; i += blockDim.x) base[i] = s[shift + i];
        } else {
            for (int i = threadIdx.x; i < n; i += blockDim.x) base[i] = s[shift + i];
        }
        __syncthreads();
    }
}

// ---- u8 images -> float ----------------------------------------------------------
// y = alpha * x in the output type (alpha rounded to T first, one rounding of the product).
// A thread converts 16 bytes when both pointers allow 16-byte accesses.
template <class T>
__global__ void scaled_cast_u8_kernel(const uint8_t *__restrict__ x, T *__restrict__ y, int64_t n,
                                      float alpha) {
    const float a = to_f32(from_f32<T>(alpha));
    const bool vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0 &&
                     (reinterpret_cast<uintptr_t>(y) & 15) == 0;
    const int64_t nvec = vec ? n / 16 : 0;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nvec; i += stride) {
        const uint4 q = reinterpret_cast<const uint4 *>(x)[i];
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
        __align__(16) T out[16];
#pragma unroll
        for (int j = 0; j < 16; ++j)
            out[j] = from_f32<T>(a * (float)((w[j >> 2] >> (8 * (j & 3))) & 0xffu));
        uint4 *dst = reinterpret_cast<uint4 *>(y + i * 16);
        const uint4 *src = reinterpret_cast<const uint4 *>(out);
#pragma unroll
        for (int j = 0; j < (int)(16 * sizeof(T) / 16); ++j) dst[j] = src[j];
    }
    for (int64_t i = nvec * 16 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        y[i] = from_f32<T>(a * (float)x[i]);
}

// ---- bias ---------------------------------------------------------------------
template <class T>
__global__ void bias_add_kernel(T *__restrict__ y, const T *__restrict__ bias, int64_t total,
                                int64_t cols, int64_t inner) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (int64_t)gridDim.x * blockDim.x) {
        int64_t c = (i / inner) % cols;
        y[i] = from_f32<T>(__fadd_rn(to_f32(y[i]), to_f32(bias[c])));
    }
}

// Bias gradient y[c] = beta*y[c] + sum over (r, i) of x[r, c, i], in two passes with a
// fixed summation order (deterministic):
//   pass 1  partial[chunk][c] over a chunk of rows, reading x coalesced
//   pass 2  y[c] = beta*y[c] + sum over chunks
// inner == 1 (Dense): threads walk the columns.  Other inner (Conv2, NCHW): warps walk
// the contiguous inner positions of one channel.
template <class T>
__global__ void bias_grad_cols_kernel(const T *__restrict__ x, float *__restrict__ partial,
                                      int64_t rows, int64_t cols, int64_t rows_per_chunk,
                                      T *__restrict__ y, float beta) {
    __shared__ float part[8][33];
    const int cx = threadIdx.x & 31, ry = threadIdx.x >> 5;  // 32 columns x 8 row lanes
    const int64_t c = (int64_t)blockIdx.x * 32 + cx;
    const int64_t r0 = (int64_t)blockIdx.y * rows_per_chunk;
    const int64_t r1 = min(rows, r0 + rows_per_chunk);
    float s = 0.f;
    if (c < cols)
        for (int64_t r = r0 + ry; r < r1; r += 8) s += to_f32(x[r * cols + c]);
    part[ry][cx] = s;
    __syncthreads();
    if (ry == 0 && c < cols) {
        float t = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) t += part[k][cx];
        if (y != nullptr) {  // a single chunk: this is the whole sum
            if (beta != 0.f) t = __fadd_rn(t, __fmul_rn(beta, to_f32(y[c])));
            y[c] = from_f32<T>(t);
        } else {
            partial[(int64_t)blockIdx.y * cols + c] = t;
        }
    }
}

// The same for wide matrices whose rows keep 16-byte alignment: a thread owns the columns of one
// 16-byte vector (4 f32 / 8 bf16) and has four rows' loads in flight before it adds them, in row
// order, to its running sums.
template <class T>
__global__ void bias_grad_cols_vec_kernel(const T *__restrict__ x, float *__restrict__ partial,
                                          int64_t rows, int64_t cols, int64_t rows_per_chunk,
                                          T *__restrict__ y, float beta) {
    constexpr int V = Vec16<T>::N;
    __shared__ float part[8][32 * V + 1];
    const int cx = threadIdx.x & 31, ry = threadIdx.x >> 5;
    const int64_t c = ((int64_t)blockIdx.x * 32 + cx) * V;
    const int64_t r0 = (int64_t)blockIdx.y * rows_per_chunk;
    const int64_t r1 = min(rows, r0 + rows_per_chunk);
    float s[V];
#pragma unroll
    for (int j = 0; j < V; ++j) s[j] = 0.f;
    if (c < cols) {
        int64_t r = r0 + ry;
        for (; r + 24 < r1; r += 32) {
            Vec16<T> v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                v[u].raw = *reinterpret_cast<const uint4 *>(x + (r + 8 * u) * cols + c);
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int j = 0; j < V; ++j) s[j] += v[u].get(j);
        }
        for (; r < r1; r += 8) {
            Vec16<T> v;
            v.raw = *reinterpret_cast<const uint4 *>(x + r * cols + c);
#pragma unroll
            for (int j = 0; j < V; ++j) s[j] += v.get(j);
        }
    }
#pragma unroll
    for (int j = 0; j < V; ++j) part[ry][cx * V + j] = s[j];
    __syncthreads();
    for (int i = threadIdx.x; i < 32 * V; i += blockDim.x) {
        const int64_t col = (int64_t)blockIdx.x * 32 * V + i;
        if (col >= cols) continue;
        float t = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) t += part[k][i];
        if (y != nullptr) {  // a single chunk: this is the whole sum
            if (beta != 0.f) t = __fadd_rn(t, __fmul_rn(beta, to_f32(y[col])));
            y[col] = from_f32<T>(t);
        } else {
            partial[(int64_t)blockIdx.y * cols + col] = t;
        }
    }
}

// One channel of planes.  The channel's rows are cut into units of kBiasVectors 16-byte vectors per lane, a unit
// per warp at a time with all its loads in flight; chunks of units spread a channel over CTAs.  A row's first and
// last elements, where the row does not start or end on 16 bytes, belong to the lanes whose vectors they would be
// part of.  One element per thread at a time took 8.2 us for 32 channels of 64 x 32 x 32 f32 and 30 for 254 x
// 55 x 55 bf16 (8.4 and 49 MB): now 7.0 and 14.8, of which the second round's two trips to L2 are about 3.
constexpr int kBiasVectors = 4;
// Sum over the CTA in thread 0: shuffles within a warp, then the warps' sums in warp order.
__device__ __forceinline__ float block_sum(float s, float *part) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    __syncthreads();
    if (threadIdx.x % 32 == 0) part[threadIdx.x / 32] = s;
    __syncthreads();
    s = part[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) s += part[w];
    return s;
}
template <class T>
__global__ void __launch_bounds__(256)
    bias_grad_planes_kernel(const T *__restrict__ x, float *__restrict__ partial, int64_t cols, int64_t inner, int64_t units,
                            int64_t units_per_chunk, int units_per_row, int *__restrict__ arrivals, T *__restrict__ y, float beta) {
    let_dependents_launch();
    dependency_wait();
    constexpr int V = Vec16<T>::N;
    __shared__ float part[8];
    __shared__ bool last;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int64_t c = blockIdx.x;
    const int64_t u0 = (int64_t)blockIdx.y * units_per_chunk, u1 = min(units, u0 + units_per_chunk);
    float s = 0.f;
    int64_t r = (u0 + warp) / units_per_row;
    int k0 = (int)(u0 + warp - r * units_per_row);
    for (int64_t u = u0 + warp; u < u1; u += 8, k0 += 8) {
        for (; k0 >= units_per_row; k0 -= units_per_row) ++r;
        const T *row = x + (r * cols + c) * inner;
        const int shift = (int)(reinterpret_cast<uintptr_t>(row) % 16 / sizeof(T));
        // vector v of the row: its elements [v * V - shift, v * V - shift + V)
        const int64_t v0 = (int64_t)k0 * (32 * kBiasVectors) + lane;
        Vec16<T> q[kBiasVectors];
        bool whole[kBiasVectors];
#pragma unroll
        for (int j = 0; j < kBiasVectors; ++j) {
            const int64_t e = (v0 + 32 * j) * V - shift;
            whole[j] = e >= 0 && e + V <= inner;
            if (whole[j]) q[j].raw = __ldg(reinterpret_cast<const uint4 *>(row + e));
        }
#pragma unroll
        for (int j = 0; j < kBiasVectors; ++j) {
            const int64_t e = (v0 + 32 * j) * V - shift;
            if (whole[j]) {
                float t = q[j].get(0);
#pragma unroll
                for (int k = 1; k < V; ++k) t += q[j].get(k);
                s += t;
            } else if (e < inner) {
                for (int k = 0; k < V; ++k)
                    if (e + k >= 0 && e + k < inner) s += to_f32(row[e + k]);
            }
        }
    }
    s = block_sum(s, part);
    if (threadIdx.x == 0) {
        partial[(int64_t)blockIdx.y * cols + c] = s;
        // the column's last chunk adds them all, chunk k in thread k % 256
        last = false;
        if (arrivals != nullptr) {
            __threadfence();
            last = atomicAdd(arrivals + c, 1) == (int)gridDim.y - 1;
            if (last) {
                arrivals[c] = 0;
                __threadfence();
            }
        }
    }
    __syncthreads();
    if (!last) return;
    s = 0.f;
    for (int k = threadIdx.x; k < (int)gridDim.y; k += 256) s += __ldcg(partial + (int64_t)k * cols + c);
    s = block_sum(s, part);
    if (threadIdx.x == 0) y[c] = from_f32<T>(beta != 0.f ? __fadd_rn(s, __fmul_rn(beta, to_f32(y[c]))) : s);
}

// Block of 32 x 8 threads: 32 consecutive columns, the chunk rows dealt round-robin to the eight
// thread rows; the eight sums are added in row order (reproducible).
template <class T>
__global__ void bias_grad_final_kernel(const float *__restrict__ partial, T *__restrict__ y,
                                       int64_t cols, int chunks, float beta) {
    __shared__ float part[8][33];
    const int64_t c = (int64_t)blockIdx.x * 32 + threadIdx.x;
    float v = 0.f;
    if (c < cols)
        for (int k = threadIdx.y; k < chunks; k += 8) v += partial[(int64_t)k * cols + c];
    part[threadIdx.y][threadIdx.x] = v;
    __syncthreads();
    if (threadIdx.y != 0 || c >= cols) return;
    v = part[0][threadIdx.x];
#pragma unroll
    for (int r = 1; r < 8; ++r) v += part[r][threadIdx.x];
    if (beta != 0.f) v = __fadd_rn(v, __fmul_rn(beta, to_f32(y[c])));
    y[c] = from_f32<T>(v);
}

template <class T>
static int bias_grad_planes(ag_device *dev, const T *x, int64_t rows, int64_t cols, int64_t inner, float beta, T *y) {
    constexpr int V = Vec16<T>::N;
    // a row may lie over one more vector than it has elements for
    const int64_t per_row = ceil_div(ceil_div(inner, V) + 1, 32 * kBiasVectors), units = rows * per_row;
    AG_REQUIRE(per_row < (1ll << 31), AG_ERR_LIMIT, "planes too large");
    // up to eight CTAs per SM, a unit or more for each of a CTA's warps, at most 1024 sums per channel
    int64_t chunks = std::min(std::min(ceil_div((int64_t)dev->sm_count * 8, cols), ceil_div(units, 8)), (int64_t)1024);
    const int64_t per_chunk = ceil_div(units > 0 ? units : 1, chunks < 1 ? 1 : chunks);
    chunks = units > 0 ? ceil_div(units, per_chunk) : 1;
    void *ws = nullptr;
    AG_TRY(workspace(dev, sizeof(float) * (size_t)chunks * (size_t)cols, &ws));
    // one launch when every column has a counter
    int *arrivals = cols < kTileCounters ? dev->tile_counters : nullptr;
    AG_TRY((launch_dependent(dev, bias_grad_planes_kernel<T>, dim3((unsigned)cols, (unsigned)chunks), 256, 0, x,
                             (float *)ws, cols, inner, units, per_chunk, (int)per_row, arrivals, y, beta)));
    if (arrivals != nullptr) return AG_OK;
    bias_grad_final_kernel<T><<<(unsigned)ceil_div(cols, 32), dim3(32, 8), 0, dev->stream>>>((const float *)ws, y, cols, (int)chunks,
                                                                                             beta);
    AG_CHECK_LAUNCH();
    return AG_OK;
}

template <class T>
static int bias_grad_run(ag_device *dev, const T *x, int64_t rows, int64_t cols, int64_t inner,
                         float beta, T *y) {
    // Wide, aligned matrices: 16-byte loads (a CTA covers 32 vectors of columns).
    constexpr int V = Vec16<T>::N;
    const bool vec = cols % V == 0 && cols >= 32 * V && rows > 1024 &&
                     (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    if (inner != 1) return bias_grad_planes<T>(dev, x, rows, cols, inner, beta, y);
    // Enough row chunks to fill the GPU (eight CTAs per SM for the vector form), at most 1024.
    int64_t col_blocks = ceil_div(cols, vec ? 32 * V : 32);
    int64_t chunks = ceil_div((int64_t)dev->sm_count * (vec ? 8 : 4), col_blocks);
    if (chunks > rows) chunks = rows;
    if (chunks > 1024) chunks = 1024;
    if (chunks < 1) chunks = 1;
    // Few rows (a Dense layer's small batch): one launch, no second pass.
    if (rows <= 1024) chunks = 1;
    const int64_t rows_per_chunk = ceil_div(rows > 0 ? rows : 1, chunks);
    chunks = rows > 0 ? ceil_div(rows, rows_per_chunk) : 1;
    if (chunks == 1) {
        bias_grad_cols_kernel<T><<<(unsigned)col_blocks, 256, 0, dev->stream>>>(
            x, nullptr, rows, cols, rows_per_chunk, y, beta);
        AG_CHECK_LAUNCH();
        return AG_OK;
    }
    void *ws = nullptr;
    AG_TRY(workspace(dev, sizeof(float) * (size_t)chunks * (size_t)cols, &ws));
    dim3 grid((unsigned)col_blocks, (unsigned)chunks);
    AG_REQUIRE(col_blocks < (1ll << 31), AG_ERR_LIMIT, "too many columns");
    if (vec)
        bias_grad_cols_vec_kernel<T><<<grid, 256, 0, dev->stream>>>(x, (float *)ws, rows, cols,
                                                                    rows_per_chunk, nullptr, 0.f);
    else
        bias_grad_cols_kernel<T><<<grid, 256, 0, dev->stream>>>(x, (float *)ws, rows, cols,
                                                                rows_per_chunk, nullptr, 0.f);
    AG_CHECK_LAUNCH();
    bias_grad_final_kernel<T><<<(unsigned)ceil_div(cols, 32), dim3(32, 8), 0, dev->stream>>>(
        (const float *)ws, y, cols, (int)chunks, beta);
    AG_CHECK_LAUNCH();
    return AG_OK;
}

// ---- SGD ------------------------------------------------------------------------
template <class T>
__global__ void sgd_momentum_kernel(T *__restrict__ w, const T *__restrict__ g, T *__restrict__ v,
                                    int64_t n, float lr, float mom) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        float vv = __fadd_rn(__fmul_rn(mom, to_f32(v[i])), to_f32(g[i]));
        float ww = __fsub_rn(to_f32(w[i]), __fmul_rn(lr, vv));
        v[i] = from_f32<T>(vv);
        w[i] = from_f32<T>(ww);
    }
}

// Any window, any width: a CTA stages a run of whole planes in shared memory with
// 16-byte loads (the staged copy keeps the alignment of the global run) and takes the
// window maxima from there; consecutive threads write consecutive outputs.
template <class T>
__global__ void max_pool2_staged_kernel(const T *__restrict__ x, T *__restrict__ y, int64_t planes,
                                        int ih, int iw, int oh, int ow, int h, int w, int sh,
                                        int sw, int per_cta) {
    extern __shared__ __align__(16) unsigned char staged_raw[];
    T *s = reinterpret_cast<T *>(staged_raw);
    constexpr int V = 16 / (int)sizeof(T);
    const int plane_len = ih * iw;
    for (int64_t p0 = (int64_t)blockIdx.x * per_cta; p0 < planes;
         p0 += (int64_t)gridDim.x * per_cta) {
        const int np = (int)min((int64_t)per_cta, planes - p0);
        const int n = np * plane_len;
        const T *base = x + p0 * plane_len;
        const int shift = (int)((reinterpret_cast<uintptr_t>(base) & 15) / sizeof(T));
        const int head = min(n, (V - shift) % V);
        const int nv = (n - head) / V;
        const int tail0 = head + nv * V;
        for (int i = threadIdx.x; i < head; i += blockDim.x) s[shift + i] = base[i];
        for (int v = threadIdx.x; v < nv; v += blockDim.x)
            *reinterpret_cast<uint4 *>(s + shift + head + v * V) =
                *reinterpret_cast<const uint4 *>(base + head + v * V);
        for (int i = tail0 + threadIdx.x; i < n; i += blockDim.x) s[shift + i] = base[i];
        __syncthreads();
        const int outs = np * oh * ow;
        T *dst = y + p0 * oh * ow;
        for (int i = threadIdx.x; i < outs; i += blockDim.x) {
            const int wid = i % ow;
            const int t = i / ow;
            const int hid = t % oh, plane = t / oh;
            const T *win = s + shift + plane * plane_len + hid * sh * iw + wid * sw;
            float m = to_f32(win[0]);
            for (int fi = 0; fi < h; ++fi)
                for (int fj = 0; fj < w; ++fj) {
                    const float v = to_f32(win[fi * iw + fj]);
                    if (v > m) m = v;  // the first maximum wins; NaNs never win after the first cell
                }
            dst[i] = from_f32<T>(m);
        }
        __syncthreads();
    }
}

template <class T>
static int pool_forward(ag_device *dev, const T *x, T *y, int64_t planes, int ih, int iw, int oh,
                        int ow, int h, int w, int sh, int sw) {
    const int threads = 256;
    constexpr int V = Vec16<T>::N;
    const int64_t plane_bytes = (int64_t)ih * iw * (int64_t)sizeof(T);
    if (h == 2 && w == 2 && sh == 2 && sw == 2 && iw % V == 0 && aligned16(x)) {
        const int64_t items = planes * oh * (iw / V);
        return launch_dependent(dev, max_pool2_2x2_kernel<T>,
                                dim3(grid_for(items, threads, dev->sm_count)), threads, 0, x, y, planes, ih,
                                iw, oh, ow);
    } else if (h == 2 && w == 2 && sh == 2 && sw == 2) {
        return pool_windows<T, false>(dev, x, y, planes, ih, iw, oh, ow);
    } else if (plane_bytes <= 40 * 1024 && planes >= dev->sm_count) {
        // a run of whole planes per CTA, about four CTAs per SM
        int per_cta = (int)((40 * 1024) / plane_bytes);
        const int64_t spread = ceil_div(planes, (int64_t)dev->sm_count * 4);
        if (per_cta > spread) per_cta = (int)(spread < 1 ? 1 : spread);
        const size_t smem = (size_t)per_cta * (size_t)plane_bytes + 16;
        const unsigned grid = (unsigned)std::min<int64_t>(ceil_div(planes, per_cta),
                                                          (int64_t)dev->sm_count * 8);
        max_pool2_staged_kernel<T><<<grid, threads, smem, dev->stream>>>(x, y, planes, ih, iw, oh, ow,
                                                                         h, w, sh, sw, per_cta);
    } else {
        const int64_t items = planes * oh * ow;
        max_pool2_kernel<T><<<grid_for(items, threads, dev->sm_count), threads, 0, dev->stream>>>(
            x, y, planes, ih, iw, oh, ow, h, w, sh, sw);
    }
    AG_CHECK_LAUNCH();
    return AG_OK;
}

}  // namespace ag

using namespace ag;

#define AG_DISPATCH_FLOAT(dtype, T, ...)            \
    do {                                            \
        if ((dtype) == AG_F32) {                    \
            using T = float;                        \
            __VA_ARGS__                             \
        } else {                                    \
            using T = __nv_bfloat16;                \
            __VA_ARGS__                             \
        }                                           \
    } while (0)

extern "C" {

int ag_scaled_cast_u8(ag_device *dev, ag_dtype dtype, float alpha, const uint8_t *x, void *y,
                      int64_t n) {
    AG_ENTER(dev);
    AG_REQUIRE(is_float_dtype(dtype), AG_ERR_DTYPE, "scaled_cast to %d unimplemented", (int)dtype);
    AG_REQUIRE(n >= 0, AG_ERR_SHAPE, "negative length");
    if (n == 0) return AG_OK;
    AG_REQUIRE(x && y, AG_ERR_INVALID, "null tensor pointer");
    const int threads = 256;
    const unsigned grid = grid_for(ceil_div(n, 16), threads, dev->sm_count);
    AG_DISPATCH_FLOAT(dtype, T,
        scaled_cast_u8_kernel<T><<<grid, threads, 0, dev->stream>>>(x, (T *)y, n, alpha););
    AG_CHECK_LAUNCH();
    return AG_OK;
}

int ag_relu(ag_device *dev, ag_dtype dtype, const void *x, void *y, int64_t n) {
    AG_ENTER(dev);
    AG_REQUIRE(is_float_dtype(dtype), AG_ERR_DTYPE, "relu %d unimplemented", (int)dtype);
    AG_REQUIRE(n >= 0, AG_ERR_SHAPE, "negative length");
    if (n == 0) return AG_OK;
    AG_REQUIRE(x && y, AG_ERR_INVALID, "null tensor pointer");
    AG_DISPATCH_FLOAT(dtype, T, return map2<T>(dev, (const T *)x, (const T *)nullptr, (T *)y, n, ReluF{}););
}

int ag_relu_backward(ag_device *dev, ag_dtype dtype, const void *x, const void *dy, void *dx,
                     int64_t n) {
    AG_ENTER(dev);
    AG_REQUIRE(is_float_dtype(dtype), AG_ERR_DTYPE, "relu_backward %d unimplemented", (int)dtype);
    AG_REQUIRE(n >= 0, AG_ERR_SHAPE, "negative length");
    if (n == 0) return AG_OK;
    AG_REQUIRE(x && dy && dx, AG_ERR_INVALID, "null tensor pointer");
    AG_DISPATCH_FLOAT(dtype, T, return map2<T>(dev, (const T *)x, (const T *)dy, (T *)dx, n, ReluBackwardF{}););
}

int ag_scaled_add(ag_device *dev, ag_dtype dtype, float alpha, const void *x, void *y, int64_t n) {
    AG_ENTER(dev);
    AG_REQUIRE(is_float_dtype(dtype), AG_ERR_DTYPE, "scaled_add %d unimplemented", (int)dtype);
    AG_REQUIRE(n >= 0, AG_ERR_SHAPE, "negative length");
    if (n == 0) return AG_OK;
    AG_REQUIRE(x && y, AG_ERR_INVALID, "null tensor pointer");
    if (dtype == AG_F32)
        return map2<float>(dev, (const float *)x, (const float *)y, (float *)y, n,
                           ScaledAddF<float>{alpha});
    // alpha is cast to the element type first (ScalarElem::scalar_cast in the reference).
    float a = __bfloat162float(__float2bfloat16_rn(alpha));
    return map2<__nv_bfloat16>(dev, (const __nv_bfloat16 *)x, (const __nv_bfloat16 *)y,
                               (__nv_bfloat16 *)y, n, ScaledAddF<__nv_bfloat16>{a});
}

int ag_max_pool2(ag_device *dev, ag_dtype dtype, const void *x, int64_t bs, int64_t c, int64_t ih,
                 int64_t iw, int32_t h, int32_t w, int32_t sh, int32_t sw, void *y) {
    AG_ENTER(dev);
    AG_REQUIRE(is_float_dtype(dtype), AG_ERR_DTYPE, "max_pool2 %d unimplemented", (int)dtype);
    AG_REQUIRE(h > 0 && w > 0 && sh > 0 && sw > 0, AG_ERR_INVALID, "bad pool options");
    AG_REQUIRE(bs >= 0 && c >= 0 && ih >= h && iw >= w, AG_ERR_SHAPE,
               "pool window [%d,%d] does not fit input [%lld,%lld]", h, w, (long long)ih,
               (long long)iw);
    AG_REQUIRE(ih < (1 << 30) && iw < (1 << 30), AG_ERR_LIMIT, "image too large");
    const int oh = (int)((ih - h) / sh + 1), ow = (int)((iw - w) / sw + 1);
    if (bs * c == 0) return AG_OK;
    AG_REQUIRE(x && y, AG_ERR_INVALID, "null tensor pointer");
    AG_DISPATCH_FLOAT(dtype, T, return pool_forward<T>(dev, (const T *)x, (T *)y, bs * c, (int)ih, (int)iw, oh, ow, h, w, sh, sw););
}

// Gradients of 2x2 windows that run faster staged than a thread per window: planes so small that half of the windows
// are partial, each with up to eight accesses of its own, and enough of them to fill the staged form's CTAs (us, windows
// and staged, from L2: bf16 131072 planes of 7 x 7 14.9, 11.3; 262144 of 3 x 3 10.4, 4.6; 131072 of 9 x 9 22.4, 17.7;
// 65536 of 11 x 11 15.5, 14.4 but from DRAM 16.5, 19.2; 16384 of 5 x 5 2.6, 2.9; 4096 of 9 x 9 2.2, 3.2;
// f32 262144 of 3 x 3 6.9, 5.4; 65536 of 3 x 3 2.8, 3.3; 262144 of 5 x 5 14.0, 14.0, from DRAM 15.2, 18.0).
static bool many_small_odd_planes(ag_dtype dtype, int64_t planes, int64_t ih, int64_t iw) {
    const int64_t windows = planes * ((ih + 1) / 2) * ((iw + 1) / 2);
    if (ih % 2 == 0 || iw % 2 == 0) return false;
    return dtype == AG_F32 ? ih * iw <= 9 && windows >= 500000 : ih * iw <= 81 && windows >= 200000;
}

// dx = max_pool2_backward(copy of x, dy); x == dx is the in-place form of the reference.
static int pool_backward(ag_device *dev, ag_dtype dtype, const void *x, void *dx, int64_t bs,
                         int64_t c, int64_t ih, int64_t iw, int32_t h, int32_t w, int32_t sh,
                         int32_t sw, const void *dy) {
    AG_ENTER(dev);
    AG_REQUIRE(is_float_dtype(dtype), AG_ERR_DTYPE, "max_pool2_backward %d unimplemented",
               (int)dtype);
    AG_REQUIRE(h > 0 && w > 0 && sh > 0 && sw > 0, AG_ERR_INVALID, "bad pool options");
    AG_REQUIRE(sh >= h && sw >= w, AG_ERR_UNSUPPORTED,
               "max_pool2_backward needs non-overlapping windows (stride >= size)");
    AG_REQUIRE(bs >= 0 && c >= 0 && ih >= h && iw >= w, AG_ERR_SHAPE,
               "pool window does not fit input");
    AG_REQUIRE(ih < (1 << 30) && iw < (1 << 30), AG_ERR_LIMIT, "image too large");
    const int oh = (int)((ih - h) / sh + 1), ow = (int)((iw - w) / sw + 1);
    const int64_t planes = bs * c;
    if (planes == 0) return AG_OK;
    AG_REQUIRE(x && dx && dy, AG_ERR_INVALID, "null tensor pointer");
    const int threads = 256;
    const int vlen = dtype == AG_F32 ? 4 : 8;
    if (h == 2 && w == 2 && sh == 2 && sw == 2 && iw % vlen == 0 &&
        (reinterpret_cast<uintptr_t>(dx) & 15) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0 &&
        ((ih & 1) == 0 || x == dx)) {  // out of place, a last row no window covers must be copied
        const unsigned grid2 = grid_for(planes * oh * (iw / vlen), threads, dev->sm_count);
        AG_DISPATCH_FLOAT(dtype, T, return launch_dependent(dev, max_pool2_backward_2x2_kernel<T>, dim3(grid2), threads,
                0, (const T *)x,
                                                            (T *)dx, (const T *)dy, planes, (int)ih, (int)iw, oh, ow););
    }
    if (h == 2 && w == 2 && sh == 2 && sw == 2 && !many_small_odd_planes(dtype, planes, ih, iw))
        AG_DISPATCH_FLOAT(dtype, T, return (pool_windows_backward<T, false>(dev, (const T *)x, (T *)dx, (const T *)dy, planes, ih, iw,
                                                                            oh, ow)););
    const int64_t plane_bytes = ih * iw * (int64_t)dtype_size(dtype);
    if (plane_bytes <= 40 * 1024) {
        // a run of whole planes per CTA, about four CTAs per SM
        int per_cta = (int)((40 * 1024) / plane_bytes);
        const int64_t spread = ceil_div(planes, (int64_t)dev->sm_count * 4);
        if (per_cta > spread) per_cta = (int)(spread < 1 ? 1 : spread);
        const size_t smem = (size_t)per_cta * (size_t)plane_bytes + 16;
        const unsigned gridp = (unsigned)std::min<int64_t>(ceil_div(planes, per_cta),
                                                           (int64_t)dev->sm_count * 8);
        AG_DISPATCH_FLOAT(dtype, T,
            max_pool2_backward_staged_kernel<T><<<gridp, threads, smem, dev->stream>>>(
                (const T *)x, (T *)dx, (const T *)dy, planes, (int)ih, (int)iw, oh, ow, h, w, sh, sw, per_cta););
        AG_CHECK_LAUNCH();
        return AG_OK;
    }
    // planes too large to stage: copy first (when out of place), then the in-place kernel
    if (x != dx)
        AG_CUDA_TRY(cudaMemcpyAsync(dx, x, (size_t)(planes * ih * iw) * dtype_size(dtype),
                                    cudaMemcpyDeviceToDevice, dev->stream));
    const unsigned grid = grid_for(planes * oh * ow, threads, dev->sm_count);
    AG_DISPATCH_FLOAT(dtype, T,
        max_pool2_backward_kernel<T><<<grid, threads, 0, dev->stream>>>(
            (T *)dx, (const T *)dy, planes, (int)ih, (int)iw, oh, ow, h, w, sh, sw););
    AG_CHECK_LAUNCH();
    return AG_OK;
}

int ag_max_pool2_backward(ag_device *dev, ag_dtype dtype, void *dx, int64_t bs, int64_t c,
                          int64_t ih, int64_t iw, int32_t h, int32_t w, int32_t sh, int32_t sw,
                          const void *dy) {
    return pool_backward(dev, dtype, dx, dx, bs, c, ih, iw, h, w, sh, sw, dy);
}

int ag_max_pool2_backward_from_input(ag_device *dev, ag_dtype dtype, const void *x, int64_t bs,
                                     int64_t c, int64_t ih, int64_t iw, int32_t h, int32_t w,
                                     int32_t sh, int32_t sw, const void *dy, void *dx) {
    return pool_backward(dev, dtype, x, dx, bs, c, ih, iw, h, w, sh, sw, dy);
}

// Relu followed by a 2x2 / stride 2 pool over planes of even height and width, and the
// gradient of the pair at the Relu's input.
static int relu_pool_check(ag_device *dev, ag_dtype dtype, int64_t bs, int64_t c, int64_t ih,
                           int64_t iw, const void *a, const void *b, const void *d) {
    AG_REQUIRE(is_float_dtype(dtype), AG_ERR_DTYPE, "relu_max_pool2 %d unimplemented", (int)dtype);
    AG_REQUIRE(bs >= 0 && c >= 0 && ih >= 2 && iw >= 2, AG_ERR_SHAPE,
               "pool window [2,2] does not fit input [%lld,%lld]", (long long)ih, (long long)iw);
    AG_REQUIRE((ih & 1) == 0 && (iw & 1) == 0, AG_ERR_UNSUPPORTED,
               "relu_max_pool2 needs even height and width");
    AG_REQUIRE(ih < (1 << 30) && iw < (1 << 30), AG_ERR_LIMIT, "image too large");
    if (bs * c == 0) return AG_OK;
    AG_REQUIRE(a && b && d, AG_ERR_INVALID, "null tensor pointer");
    const size_t pair_bytes = 2 * dtype_size(dtype);
    AG_REQUIRE(reinterpret_cast<uintptr_t>(a) % pair_bytes == 0 &&
                   reinterpret_cast<uintptr_t>(b) % pair_bytes == 0,
               AG_ERR_UNSUPPORTED, "relu_max_pool2 needs element-pair aligned tensors");
    return AG_OK;
}

int ag_relu_max_pool2_forward(ag_device *dev, ag_dtype dtype, const void *x, int64_t bs, int64_t c,
                              int64_t ih, int64_t iw, void *y) {
    AG_ENTER(dev);
    AG_TRY(relu_pool_check(dev, dtype, bs, c, ih, iw, x, x, y));
    const int64_t planes = bs * c;
    if (planes == 0) return AG_OK;
    AG_DISPATCH_FLOAT(dtype, T, return (pool_windows<T, true>(dev, (const T *)x, (T *)y, planes, ih, iw, ih / 2, iw / 2)););
}

int ag_relu_max_pool2_backward(ag_device *dev, ag_dtype dtype, const void *x, int64_t bs,
                               int64_t c, int64_t ih, int64_t iw, const void *dy, void *dx) {
    AG_ENTER(dev);
    AG_TRY(relu_pool_check(dev, dtype, bs, c, ih, iw, x, dx, dy));
    const int64_t planes = bs * c;
    if (planes == 0) return AG_OK;
    AG_DISPATCH_FLOAT(dtype, T, return (pool_windows_backward<T, true>(dev, (const T *)x, (T *)dx, (const T *)dy, planes, ih, iw, ih / 2,
                                                                       iw / 2)););
}

int ag_bias_add(ag_device *dev, ag_dtype dtype, void *y, const void *bias, int64_t rows,
                int64_t cols, int64_t inner) {
    AG_ENTER(dev);
    AG_REQUIRE(is_float_dtype(dtype), AG_ERR_DTYPE, "add_assign %d unimplemented", (int)dtype);
    AG_REQUIRE(rows >= 0 && cols >= 0 && inner >= 0, AG_ERR_SHAPE, "negative dimension");
    const int64_t total = rows * cols * inner;
    if (total == 0) return AG_OK;
    AG_REQUIRE(y && bias, AG_ERR_INVALID, "null tensor pointer");
    const int threads = 256;
    const unsigned grid = grid_for(total, threads, dev->sm_count);
    AG_DISPATCH_FLOAT(dtype, T,
        bias_add_kernel<T><<<grid, threads, 0, dev->stream>>>((T *)y, (const T *)bias, total, cols, inner););
    AG_CHECK_LAUNCH();
    return AG_OK;
}

int ag_bias_grad(ag_device *dev, ag_dtype dtype, const void *x, int64_t rows, int64_t cols,
                 int64_t inner, float beta, void *y) {
    AG_ENTER(dev);
    AG_REQUIRE(is_float_dtype(dtype), AG_ERR_DTYPE, "sum_axis %d unimplemented", (int)dtype);
    AG_REQUIRE(rows >= 0 && cols >= 0 && inner >= 0, AG_ERR_SHAPE, "negative dimension");
    if (cols == 0) return AG_OK;
    AG_REQUIRE(y && (rows * inner == 0 || x), AG_ERR_INVALID, "null tensor pointer");
    AG_REQUIRE(cols < (1ll << 31), AG_ERR_LIMIT, "too many columns");
    AG_DISPATCH_FLOAT(dtype, T, return bias_grad_run<T>(dev, (const T *)x, rows, cols, inner, beta, (T *)y););
}

int ag_sgd_update(ag_device *dev, ag_dtype dtype, void *w, const void *g, int64_t n, float lr) {
    // w = cast_T(-lr) * g + w in T arithmetic: the reference routes plain SGD through scaled_add.
    return ag_scaled_add(dev, dtype, -lr, g, w, n);
}

int ag_sgd_update_momentum(ag_device *dev, ag_dtype dtype, void *w, const void *g, void *v,
                           int64_t n, float lr, float momentum) {
    AG_ENTER(dev);
    AG_REQUIRE(is_float_dtype(dtype), AG_ERR_DTYPE, "SGD %d unimplemented", (int)dtype);
    AG_REQUIRE(n >= 0, AG_ERR_SHAPE, "negative length");
    if (n == 0) return AG_OK;
    AG_REQUIRE(w && g && v, AG_ERR_INVALID, "null tensor pointer");
    const int threads = 256;
    const unsigned grid = grid_for(n, threads, dev->sm_count);
    AG_DISPATCH_FLOAT(dtype, T,
        sgd_momentum_kernel<T><<<grid, threads, 0, dev->stream>>>((T *)w, (const T *)g, (T *)v, n, lr, momentum););
    AG_CHECK_LAUNCH();
    return AG_OK;
}

}  // extern "C"
