// Convolutions on the gathered-operand tensor-core engine, for one element type.
#pragma once

#include "conv_halo_f32.cuh"
#include "gemm_tcx_impl.cuh"

namespace ag {
namespace tcx {

static ConvMap conv_map(int64_t channels, int64_t sh, int64_t sw, int64_t gh, int64_t gw,
                        const ag_conv2_options *o, bool gradient) {
    ConvMap g;
    g.channels = (int)channels;
    g.sh = (int)sh; g.sw = (int)sw;
    g.gw = (int)gw; g.ghw = (int)(gh * gw);
    g.fh = o->filter[0]; g.fw = o->filter[1];
    g.ff = g.fh * g.fw;
    g.st_h = o->stride[0]; g.st_w = o->stride[1];
    g.pad_h = o->padding[0]; g.pad_w = o->padding[1];
    g.dil_h = o->dilation[0]; g.dil_w = o->dilation[1];
    g.gradient = gradient;
    g.always_valid = !gradient && g.pad_h == 0 && g.pad_w == 0;  // gh, gw come from the output rule
    g.ranges = (g.dil_h == 1 || g.fh == 1) && (g.dil_w == 1 || g.fw == 1) && (!gradient || (g.st_h == 1 && g.st_w == 1));
    g.row_ones = 0;
    for (int fi = 0; fi < g.fh; ++fi) g.row_ones |= 1u << (fi * g.fw & 31);
    g.div_ghw = FastDiv((uint32_t)g.ghw);
    g.div_gw = FastDiv((uint32_t)g.gw);
    g.div_fw = FastDiv((uint32_t)g.fw);
    g.div_st_h = FastDiv((uint32_t)g.st_h);
    g.div_st_w = FastDiv((uint32_t)g.st_w);
    g.cp = (g.channels + 7) / 8 * 8;
    g.div_cp = FastDiv((uint32_t)g.cp);
    return g;
}

// Eight values as pieces of the planes, `plane` pieces apart.
__device__ __forceinline__ void store_pieces(const Vec8<float> &x, uint4 *dst, int64_t plane) {
    uint32_t h[4], m[4], l[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        uint32_t hb[2], mb[2], lb[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) split3(x.v[2 * e + u], hb[u], mb[u], lb[u]);
        h[e] = upper_halves(hb[0], hb[1]);
        m[e] = upper_halves(mb[0], mb[1]);
        l[e] = upper_halves(lb[0], lb[1]);
    }
    dst[0] = make_uint4(h[0], h[1], h[2], h[3]);
    dst[plane] = make_uint4(m[0], m[1], m[2], m[3]);
    dst[2 * plane] = make_uint4(l[0], l[1], l[2], l[3]);
}
__device__ __forceinline__ void store_pieces(const Vec8<__nv_bfloat16> &x, uint4 *dst, int64_t) {
    dst[0] = make_uint4(__byte_perm(x.v[0], x.v[1], 0x5410), __byte_perm(x.v[2], x.v[3], 0x5410),
                        __byte_perm(x.v[4], x.v[5], 0x5410), __byte_perm(x.v[6], x.v[7], 0x5410));
}

// src[outer][channel * s_c][inner] into pieces of eight channels: a tensor [image][channels][hw] (inner = hw, s_c = hw) into
// [image][hw][groups], or a filter bank (rows, channels, taps) into [row][tap][groups].  A thread makes one piece; a warp
// reads neighbouring inner indices, which are whole lines of a tensor.
template <class T>
struct SplitJob {
    const T *src;
    uint4 *dst;
    int64_t plane;           // pieces per plane
    int64_t s_outer;
    int channels, inner, s_c, groups;
    uint32_t total;          // outer x groups x inner
    FastDiv div_inner, div_groups;
};
template <class T>
__global__ void __launch_bounds__(256) split_kernel(const SplitJob<T> j0, const SplitJob<T> j1) {
    let_dependents_launch(kAlwaysEarly);
    dependency_wait();
    const SplitJob<T> &j = blockIdx.y == 0 ? j0 : j1;
    for (uint32_t i = blockIdx.x * 256u + threadIdx.x; i < j.total; i += gridDim.x * 256u) {
        uint32_t t, in, outer, group;
        j.div_inner.divmod(i, t, in);
        j.div_groups.divmod(t, outer, group);
        const int c0 = (int)group * 8;
        const T *q = j.src + outer * j.s_outer + (int64_t)c0 * j.s_c + in;
        Vec8<T> x;
#pragma unroll
        for (int e = 0; e < 8; ++e, q += j.s_c) fetch(x.v[e], q, c0 + e < j.channels);
        store_pieces(x, j.dst + ((int64_t)outer * j.inner + in) * j.groups + group, j.plane);
    }
}

template <class T>
static SplitJob<T> split_job(const T *src, int64_t outer, int64_t s_outer, int64_t channels, int64_t s_c, int64_t inner) {
    SplitJob<T> j;
    j.src = src;
    j.dst = nullptr;
    j.s_outer = s_outer;
    j.channels = (int)channels;
    j.inner = (int)inner;
    j.s_c = (int)s_c;
    j.groups = (int)ceil_div(channels, 8);
    j.plane = outer * inner * j.groups;
    j.total = (uint32_t)j.plane;
    j.div_inner = FastDiv((uint32_t)inner);
    j.div_groups = FastDiv((uint32_t)j.groups);
    return j;
}
template <class T>
static int64_t split_bytes(const SplitJob<T> &j) { return j.plane * Planes<T>::N * 16; }

// Both tensors, to scratch; false without room for it.
template <class T>
static bool split_scratch(ag_device *dev, SplitJob<T> *a, SplitJob<T> *b) {
    void *ws = nullptr;
    if (staging(dev, (size_t)(split_bytes(*a) + split_bytes(*b)), &ws) != AG_OK) return false;
    a->dst = (uint4 *)ws;
    b->dst = (uint4 *)((char *)ws + split_bytes(*a));
    return true;
}
template <class T>
static int launch_split(ag_device *dev, const SplitJob<T> &a, const SplitJob<T> &b) {
    const int64_t blocks = ceil_div(a.total > b.total ? a.total : b.total, 256), cap = (int64_t)dev->sm_count * 16;
    return launch_dependent(dev, split_kernel<T>, dim3((unsigned)(blocks < cap ? blocks : cap), 2), 256, 0, a, b);
}

// Whether tensors are split once, ahead of the product of `positions` rows, the map's patches and n columns (the weight
// gradient's likewise).  Against gathering, us split and gathered, images x channels x side -> filters: f32 forward 172 x
// 32 x 16 -> 128 5x5 58 and 81, 16 x 64 x 37 -> 128 3x3 46 and 61, 52 x 32 x 37 -> 6 3x3 29 and 33, weight gradient 46 x 32 x
// 27 -> 96 5x5 59 and 80, input gradient 34 x 16 x 47 -> 128 5x5 186 and 276; bf16 forward 48 x 16 x 47 -> 128 5x5 / 2 25 and
// 42, weight gradient 171 x 64 x 42 -> 16 3x3 148 and 176, input gradient 34 x 16 x 47 -> 128 5x5 117 and 187.  The pass and
// its launch want a long patch and some work: f32 64 x 16 x 32 -> 32 3x3 (144 values) forward 27 and 24, 13 x 6 x 39 -> 32
// 16 and 12, 11 x 32 x 40 -> 6 3x3 14 and 12, input gradient 5 x 32 x 42 -> 96 20.7 and 18.3; the weight gradient's second
// tensor wants more of it (37 x 6 x 52 -> 128 5x5, 200 values, 119 and 89).  Planes beyond what stays in L2 are read again
// per tap from memory: f32 171 x 64 x 42 -> 16 (116 MB) 237 and 211.
// A pass costs some 4 us per 10 MB of planes, and an element that is not gathered saves 4e-7 us (bf16 2e-7) per 128 columns, so the
// elements that would be gathered are held against the bytes of the planes.  Few reads of each, with a stride or a filter of
// few taps, make no gain but with many columns or a long patch (forward 153 x 64 x 30 -> 6 3x3 / 2 f32 45 and 32, 107 x 32 x 47 ->
// 64 3x3 / 2 42 and 35, its weight gradient 58 and 50, 15 x 96 x 63 x 50 -> 36 1x3 37 and 31, bf16 215 x 91 x 10 x 32 -> 62 3x1 / 2x1
// 23 and 18; from 32 channels into 96 3x3 / 2 85 and 94, 19 x 47 x 42 x 51 -> 68 2x5 / 2x1 40 and 49), nor do channels that are mostly
// padding (42 x 6 x 57 -> 32 5x5 56 and 52), a short patch and little work (input gradient 49 x 45 x 25 x 30 -> 11 5x3 / 2x1 24 and
// 22).  Planes of 60 MB and more leave the L2 (40 x 72 x 57 x 57 -> 10 3x3 75 and 66).  With a dilation the pieces of a row of taps
// lie apart, most of all short ones (80 x 18 x 58 x 60 -> 31 5x3 dilated 97 and 70).  Over 617 passes of 500 drawn convolutions,
// a third of them with strides of two and a third dilated, the time is 0.861 of gathering, 0.858 if each took the faster form;
// by patch, planes and work alone it was 0.867.  Passes that take more than 1.03 of gathering's time: 20 (to 1.26) and 50 (1.51).
template <class T>
static bool split_worth(const ConvMap &g, int64_t bytes, int tensors, int64_t positions, int64_t n, int least_patch) {
    const bool f32 = sizeof(T) == 4, wide = n > 80;
    const int64_t patch = (int64_t)g.ff * g.cp, work = positions * patch * (n < 32 ? 32 : n);
    if (patch < least_patch || bytes > 80000000 || work < 300000000) return false;
    const bool padding = f32 && tensors == 1 && g.ff * g.channels < 200 && !(g.gradient && g.st_w > 1);
    if (n >= 32 && !wide && ((patch < 270 && work < 500000000) || padding)) return false;
    double least = f32 ? (wide ? 0.3 : tensors == 2 ? (n > 32 ? 0.8 : 1) : n > 32 ? 0.6 : patch < 600 ? 1 : 0.8)
                       : n >= (tensors == 1 ? 64 : 81) ? 0.9 : tensors == 1 ? 1.75 : n > 40 ? 2 : 3.5;
    if (g.dil_w > 1 && g.cp <= 24) least *= 2;
    if (tensors == 1 && bytes > 60000000 && least < 1.4) least = 1.4;
    return (double)(positions * patch * ceil_div(n, 128) * tensors) >= least * (double)bytes;
}

// The map that counts positions instead of elements.
static ConvMap of_positions(const ConvMap &g) {
    ConvMap p = g;
    p.channels = 1;
    return p;
}

// A filter bank in the order of ConvRows' k: out[row][tap * cp + c] = w[row * s_row + c * s_c + tap],
// zero for the padding channels.  Without it every 64-k step of every tile would fetch filters at a
// stride of the tap count, one sector per element.
template <class T>
__global__ void repack_kernel(const T *w, T *out, int total, int channels, int cp, int s_row, int s_c,
                              FastDiv div_k, FastDiv div_cp) {
    let_dependents_launch();
    dependency_wait();
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    if (i >= (uint32_t)total) return;
    uint32_t row, k, tap, c;
    div_k.divmod(i, row, k);
    div_cp.divmod(k, tap, c);
    out[i] = (int)c < channels ? w[(int)row * s_row + (int)c * s_c + (int)tap] : from_f32<T>(0.f);
}

inline bool plain(const ag_conv2_options *o) {
    return o->stride[0] == 1 && o->stride[1] == 1 && o->dilation[0] == 1 && o->dilation[1] == 1;
}
inline halo32::Problem input_rows(const float *w, int64_t oc, int64_t ic, const float *dy, int64_t bs, int64_t ih, int64_t iw,
                                  const ag_conv2_options *o, int64_t oh, int64_t ow) {
    const int fh = o->filter[0], fw = o->filter[1];
    return halo32::Problem{dy, w, bs, oc, oh, ow, ic, ih, iw, fh, fw, fh - 1 - o->padding[0], fw - 1 - o->padding[1],
                           (int64_t)fh * fw, ic * fh * fw, true};
}
inline halo32::Wgrad weight_rows(const float *x, int64_t bs, int64_t ic, int64_t ih, int64_t iw, const float *dy, int64_t oc,
                                 const ag_conv2_options *o, int64_t oh, int64_t ow) {
    return halo32::Wgrad{x, dy, bs, ic, ih, iw, oc, oh, ow, o->filter[0], o->filter[1], o->padding[0], o->padding[1]};
}

// f32 convolutions with stride and dilation 1 on the engine with resident filters; AG_ERR_UNSUPPORTED (nothing launched,
// no message) where that is not the one to take them.
template <class T>
static int by_halo(ag_device *dev, const ag_conv2_options *o, const halo32::Problem &p, const T *bias, bool relu, T *y) {
    if constexpr (sizeof(T) == 4) {
        if (plain(o) && halo32::takes(dev, p))
            return halo32::run(dev, p, bias, relu, y);
    }
    return AG_ERR_UNSUPPORTED;
}

// A product with the patch matrix of `map` (rows = positions, k = taps x channels) and the filter
// bank w[row * s_row + channel * s_c + tap].
template <class T>
static int patches_times_filters(ag_device *dev, const T *src, int64_t images, const ConvMap &map, int M, const T *w, int N,
                                 int s_row, int s_c, const NchwOut<T> &E) {
    const int K = map.ff * map.cp, total = N * K;
    const int64_t hw = (int64_t)map.sh * map.sw;
    SplitJob<T> x = split_job(src, images, map.channels * hw, (int64_t)map.channels, hw, hw);
    SplitJob<T> f = split_job(w, (int64_t)N, (int64_t)s_row, (int64_t)map.channels, (int64_t)s_c, (int64_t)map.ff);
    if (split_worth<T>(map, split_bytes(x), 1, M, N, 200) && split_scratch(dev, &x, &f)) {
        AG_TRY(launch_split<T>(dev, x, f));
        return gemm<T>(dev, M, N, K, SplitRows<T>{{x.dst, x.plane}, of_positions(map), x.div_groups, x.groups, {src, map, M}},
                       SplitFilters<T>{{f.dst, f.plane}, K / 8, {w, s_row, s_c, map.channels, map.div_cp}}, E);
    }
    // One wave of tiles and up to 18 k steps of an input gradient, whose neighbouring rows are neighbouring
    // filters: read in place at the copy's device time, without its launch (forward, 5 x 64 x 22 x 22 -> 128:
    // 27 us in place, 19 copied; input gradient 21.7 and 21.5; 50 steps of 128 channels 5x5 190 and 87).
    // So are they where there is no room for the copy.
    void *ws = nullptr;
    if ((s_row < s_c && K <= 18 * BK && ceil_div(M, BM) * ceil_div(N, 64) <= dev->sm_count) ||
        staging(dev, (size_t)total * sizeof(T), &ws) != AG_OK)
        return gemm<T>(dev, M, N, K, ConvRows<T>{src, map, M}, FilterRows<T>{w, s_row, s_c, map.channels, map.div_cp}, E);
    T *packed = (T *)ws;
    AG_TRY((launch_dependent(dev, repack_kernel<T>, dim3((unsigned)ceil_div(total, 256)), 256, 0, w, packed, total,
                             map.channels, map.cp, s_row, s_c, FastDiv((uint32_t)K), map.div_cp)));
    return gemm<T>(dev, M, N, K, ConvRows<T>{src, map, M}, strided<kVecK>((const T *)packed, K, 1, N), E);
}

// Whether a convolution's patches are better indexed by (channel, tap) than by (tap, channel padded to
// eight): the padding costs more than the table look-ups (6 channels: 8 / 6 of 4 instructions
// per element against 6).  The table packs an offset of at most 26 bits and a sign with the tap; a tap that
// meets the image from far into the padding is at an offset beyond the channel's plane.
static bool few_channels(const ConvMap &g) {
    const int64_t furthest = (int64_t)g.channels * g.sh * g.sw + (int64_t)(g.fh - 1) * g.dil_h * g.sw + (int64_t)(g.fw - 1) * g.dil_w;
    return g.cp * 10 > g.channels * 14 && g.channels * g.ff <= kFewPatch && furthest < (1 << 26);
}

template <class T>
int conv_forward(ag_device *dev, const T *x, int64_t bs, int64_t ic, int64_t ih, int64_t iw,
                 const T *w, int64_t oc, const T *bias, const ag_conv2_options *o, int64_t oh,
                 int64_t ow, bool relu, T *y) {
    const int M = (int)(bs * oh * ow), N = (int)oc, ff = o->filter[0] * o->filter[1];
    if constexpr (sizeof(T) == 4) {
        const halo32::Problem p{x, w, bs, ic, ih, iw, oc, oh, ow, o->filter[0], o->filter[1], o->padding[0], o->padding[1],
                                ic * ff, ff, false};
        const int status = by_halo<T>(dev, o, p, bias, relu, y);
        if (status != AG_ERR_UNSUPPORTED) return status;
    }
    NchwOut<T> E{y, bias, N, (int)(oh * ow), FastDiv((uint32_t)(oh * ow)), relu};
    const ConvMap map = conv_map(ic, ih, iw, oh, ow, o, false);
    if (few_channels(map)) {
        const int patch = (int)ic * ff;
        return gemm<T>(dev, M, N, patch, FewRows<T>{x, map, M, patch}, strided<kByRow>(w, patch, 1, N), E);
    }
    return patches_times_filters<T>(dev, x, bs, map, M, w, N, (int)ic * ff, ff, E);
}

constexpr int64_t kTapSums = 1ll << 28;   // f32 values

// dx from the products with every tap: col[c * ff + tap][position of dy] -> dx[b][c][y][x].
template <class T>
__global__ void __launch_bounds__(256)
    taps_to_image_kernel(const float *col, T *dx, ConvMap g, int grid_hw, int64_t positions,
                         int total, FastDiv div_hw, FastDiv div_w, FastDiv div_c) {
    let_dependents_launch();
    dependency_wait();
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    if (i >= (uint32_t)total) return;
    uint32_t plane, r, y, x, b, c;
    div_hw.divmod(i, plane, r);
    div_w.divmod(r, y, x);
    div_c.divmod(plane, b, c);
    const float *q = col + (int64_t)c * g.ff * positions + (int64_t)b * grid_hw;
    float s = 0.f;
    for (int fi = 0; fi < g.fh; ++fi) {
        const int ty = (int)y + g.pad_h - fi * g.dil_h;
        uint32_t oy, ry;
        g.div_st_h.divmod((uint32_t)max(ty, 0), oy, ry);
        if (ty < 0 || ry != 0 || oy >= (uint32_t)g.sh) continue;
        for (int fj = 0; fj < g.fw; ++fj) {
            const int tx = (int)x + g.pad_w - fj * g.dil_w;
            uint32_t ox, rx;
            g.div_st_w.divmod((uint32_t)max(tx, 0), ox, rx);
            if (tx < 0 || rx != 0 || ox >= (uint32_t)g.sw) continue;
            s += q[(int64_t)(fi * g.fw + fj) * positions + oy * g.sw + ox];
        }
    }
    dx[i] = from_f32<T>(s);
}

template <class T>
int conv_backward_input(ag_device *dev, const T *w, int64_t oc, int64_t ic, const T *dy, int64_t bs,
                        int64_t ih, int64_t iw, const ag_conv2_options *o, int64_t oh, int64_t ow,
                        T *dx) {
    const int ff = o->filter[0] * o->filter[1];
    const int M = (int)(bs * ih * iw), N = (int)ic;
    if constexpr (sizeof(T) == 4) {
        const halo32::Problem p = input_rows((const float *)w, oc, ic, (const float *)dy, bs, ih, iw, o, oh, ow);
        const int status = by_halo<T>(dev, o, p, nullptr, false, dx);
        if (status != AG_ERR_UNSUPPORTED) return status;
    }
    const ConvMap map = conv_map(oc, oh, ow, ih, iw, o, true);
    // With few input channels a tile of the patch form is mostly empty columns, and it gathers dy
    // once per tap.  The other order multiplies dy by the filters of every (channel, tap) and adds
    // the taps afterwards, in f32.  Compared by the time of one 128-position tile on an SM: 1.7 us per
    // 64-k step, 34 bytes per ns for the taps' trip through memory (6 channels from 128, 3x3, 132 x 40
    // x 40 f32: 277 us by patches, 92 us by taps).  Beyond 128 (channel, tap) pairs the taps no longer
    // fit L2 at the batch sizes that matter (32 channels from 128, 121 x 27 x 27: 127 and 185 us).
    const int taps_n = N * ff;
    const double by_patches = 1.7 * (double)ceil_div((int64_t)ff * map.cp, 64);
    const double by_taps = 1.7 * (double)(ceil_div(oc, 64) * ceil_div(taps_n, 128)) + 0.03 * taps_n;
    // As many images at a time as have 1 GiB of sums per tap; without room for those, by patches.
    const int64_t image = oh * ow * taps_n, at_once = image < kTapSums ? kTapSums / image : 1;
    const int64_t images = at_once < bs ? at_once : bs;
    void *ws = nullptr;
    if (taps_n <= 128 && 1.3 * by_taps < by_patches && image < (1ll << 31) &&
        staging(dev, sizeof(float) * (size_t)(images * image), &ws) == AG_OK) {
        float *col = (float *)ws;
        ag_conv2_options point = {{1, 1}, {0, 0}, {1, 1}, {1, 1}};
        for (int64_t b = 0; b < bs; b += images) {
            const int64_t n = images < bs - b ? images : bs - b, positions = n * oh * ow;
            AG_TRY(gemm<T>(dev, (int)positions, taps_n, (int)oc,
                           ConvRows<T>{dy + b * oc * oh * ow, conv_map(oc, oh, ow, oh, ow, &point, false), (int)positions},
                           strided<kByRow>(w, 1, taps_n, taps_n), StridedOut<float>{col, 1, positions, 1.f, 0.f}));
            const int total = (int)(n * ic * ih * iw);
            AG_TRY((launch_dependent(dev, taps_to_image_kernel<T>, dim3((unsigned)ceil_div(total, 256)), 256, 0, col,
                                     dx + b * ic * ih * iw, map, (int)(oh * ow), positions, total,
                                     FastDiv((uint32_t)(ih * iw)), FastDiv((uint32_t)iw), FastDiv((uint32_t)ic))));
        }
        return AG_OK;
    }
    NchwOut<T> E{dx, nullptr, N, (int)(ih * iw), FastDiv((uint32_t)(ih * iw)), false};
    return patches_times_filters<T>(dev, dy, bs, map, M, w, N, ff, (int)ic * ff, E);
}

template <class T>
int conv_backward_weight(ag_device *dev, const T *x, int64_t bs, int64_t ic, int64_t ih, int64_t iw,
                         const T *dy, int64_t oc, const ag_conv2_options *o, int64_t oh, int64_t ow,
                         float beta, T *dw) {
    if constexpr (sizeof(T) == 4) {
        const halo32::Wgrad p = weight_rows((const float *)x, bs, ic, ih, iw, (const float *)dy, oc, o, oh, ow);
        if (plain(o) && halo32::takes_wgrad(p)) {
            bool taken = false;
            AG_TRY(halo32::run_wgrad(dev, p, beta, dw, &taken));
            if (taken) return AG_OK;
        }
    }
    const ConvMap map = conv_map(ic, ih, iw, oh, ow, o, false);
    const int N = (int)oc, K = (int)(bs * oh * ow), hw = (int)(oh * ow);
    if (few_channels(map)) {
        const int patch = (int)ic * map.ff;
        return gemm<T>(dev, patch, N, K, FewCols<T>{{x, map, 0, patch}}, ChannelRows<T>{dy, N, hw, FastDiv((uint32_t)hw)},
                       StridedOut<T>{dw, 1, patch, 1.f, beta});
    }
    const int M = map.ff * map.cp;
    SplitJob<T> jx = split_job(x, bs, ic * ih * iw, ic, ih * iw, ih * iw);
    SplitJob<T> jy = split_job(dy, bs, oc * hw, oc, (int64_t)hw, (int64_t)hw);
    if (split_worth<T>(map, split_bytes(jx) + split_bytes(jy), 2, K, N, 288) && split_scratch(dev, &jx, &jy)) {
        AG_TRY(launch_split<T>(dev, jx, jy));
        return gemm<T>(dev, M, N, K, SplitCols<T>{{jx.dst, jx.plane}, of_positions(map), jx.div_groups, jx.groups, {x, map, M}},
                       SplitChannels<T>{{jy.dst, jy.plane}, jy.groups, {dy, N, hw, FastDiv((uint32_t)hw)}},
                       FilterOut<T>{dw, map.channels, map.ff, map.div_cp, map.cp, beta});
    }
    return gemm<T>(dev, M, N, K, ConvCols<T>{x, map, M}, ChannelRows<T>{dy, N, hw, FastDiv((uint32_t)hw)},
                   FilterOut<T>{dw, map.channels, map.ff, map.div_cp, map.cp, beta});
}

}  // namespace tcx
}  // namespace ag
