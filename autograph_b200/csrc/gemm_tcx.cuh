// Tensor-core tile engine with gathered operands: the counterpart of the SIMT engine in
// gemm_simt.cuh for products that are worth a tensor core but that TMA cannot feed -- f32
// operands, bf16 operands whose rows are not 16-byte aligned, and the implicit GEMMs of
// convolutions with any padding / stride / dilation.
//
// One persistent CTA per SM walks 128 x BN output tiles (and k slices).  Warp roles:
//   first warps  producers: fetch 8 consecutive k of a row at a time with plain loads, split
//                f32 values into bf16 planes, and write the 128-byte-swizzled K-major tiles
//                tcgen05.mma reads
//   EPI warps    read finished accumulators from tensor memory and store through an epilogue
//   last warp    issues tcgen05.mma
//
// f32 products.  A f32 value is written as hi + 2^-8 mid + 2^-16 lo of three bf16 values (8 + 8 + 8
// bits, the remainders exact), and a product as the six partial products down to 2^-16 of the
// leading one (Henry, Tang, Heinecke, "Leveraging the bfloat16 artificial intelligence datatype
// for higher-precision computations", 2019); what is dropped is below 2^-24 of a product, an ulp
// at most.  mid and lo are held scaled up, because bf16 ends at 2^-133: unscaled, a value below 2^-109
// lost bits (1e-36 times 1e30 kept 15 of 24), scaled, every f32 value down to 2^-149 is exact (what is
// dropped of a product with a subnormal one is below 2^-149 of the other operand).  The scales come off between groups of partial products of one size, by the shift of the accumulator
// that tcgen05.mma can do.  The tensor core adds with truncation, so an accumulator is read
// out after every 64 k and the 64-k sums are added in registers with round-to-nearest; within
// 64 k the small partial products are accumulated first, which leaves four truncating additions
// of full-size terms.  A bf16 accumulator takes 1024 k, 64 truncating additions: over all of a long k
// those add up (positive operands, k = 100,001: 6e-4 of a value, always towards zero; read out like
// this 2e-7, in the same time).  Uniform f32 operands, relative 2-norm error against an f64 product:
// k = 128 8e-8 (the FFMA kernel 1.1e-7), k = 1024 1.1e-7 (5.7e-7), k = 4096 1.7e-7 (1.2e-6).  The split of
// an infinity, or of a value that rounds up to one, is not usable: blocks of outputs with a sum
// that is infinite or NaN are left out and computed with FFMAs from the f32 operands when the
// CTA's tiles are done (redo_block).
//
// What bounds it: with BN = 128 a 64-k step is 16 MMAs that read (128 + N) x 32 bytes of shared
// memory each, about 2600 cycles; the producers convert 16 k elements in the same time.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "pair_ptx.cuh"

namespace ag {
namespace tcx {

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int ROW_BYTES = BK * 2;

// 64-k steps that one accumulator takes before it is read out and added in registers.
template <int PL>
constexpr int kAccSteps = PL == 3 ? 1 : 16;

template <class T>
struct Planes;
template <>
struct Planes<float> { static constexpr int N = 3; };
template <>
struct Planes<__nv_bfloat16> { static constexpr int N = 1; };

// Eight consecutive k of one row, as fetched.
template <class T>
struct Vec8;
template <>
struct Vec8<float> { float v[8]; };
template <>
struct Vec8<__nv_bfloat16> { uint32_t v[8]; };  // one value per register until they are packed

__device__ __forceinline__ void fetch(float &d, const float *p, bool ok) {
    d = 0.f;
    if (ok) d = __ldg(p);
}
__device__ __forceinline__ void fetch(uint32_t &d, const __nv_bfloat16 *p, bool ok) {
    d = 0u;
    if (ok) d = __ldg(reinterpret_cast<const unsigned short *>(p));
}
__device__ __forceinline__ void fetch8(Vec8<float> &d, const float *p) {
    const float4 a = __ldg(reinterpret_cast<const float4 *>(p));
    const float4 b = __ldg(reinterpret_cast<const float4 *>(p) + 1);
    d.v[0] = a.x; d.v[1] = a.y; d.v[2] = a.z; d.v[3] = a.w;
    d.v[4] = b.x; d.v[5] = b.y; d.v[6] = b.z; d.v[7] = b.w;
}
__device__ __forceinline__ void fetch8(Vec8<__nv_bfloat16> &d, const __nv_bfloat16 *p) {
    const uint4 a = __ldg(reinterpret_cast<const uint4 *>(p));
    const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        d.v[2 * j] = w[j] & 0xffffu;
        d.v[2 * j + 1] = w[j] >> 16;
    }
}

// Bits whose upper halves are hi, mid and lo of an f32 value (hi + 2^-8 mid + 2^-16 lo).  Rounding is half
// away from zero to 8 bits (the upper half of bits + 0x8000); both remainders are exact, of at most 16
// and 8 bits, and stay so times 2^8: each is at most 2^-8 of the value it is left from.
// A NaN or an infinity, or a value whose hi rounds up to one, ends in a NaN: NaN - x and
// inf - inf give the NaN 0x7fffffff, whose upper half stays a NaN in lo (only the additions of
// 0x8000 can wrap one around).  Its outputs are NaN and are recomputed.
__device__ __forceinline__ void split3(float v, uint32_t &hi, uint32_t &mid, uint32_t &lo) {
    hi = __float_as_uint(v) + 0x8000u;
    const float r = (v - __uint_as_float(hi & 0xffff0000u)) * 256.f;
    mid = __float_as_uint(r) + 0x8000u;
    lo = __float_as_uint((r - __uint_as_float(mid & 0xffff0000u)) * 256.f);
}

// Upper halves of two f32 words as one packed bf16 pair.
__device__ __forceinline__ uint32_t upper_halves(uint32_t lo, uint32_t hi) {
    return __byte_perm(lo, hi, 0x7632);
}

__device__ __forceinline__ void st_shared_v4(uint32_t dst, const uint32_t (&w)[4]) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]),
                 "r"(w[3])
                 : "memory");
}

// Writes eight k of one row into the tile's plane(s); dst = shared address of the 16-byte chunk
// in plane 0, planes `plane_bytes` apart.
__device__ __forceinline__ void put8(const Vec8<__nv_bfloat16> &x, uint32_t dst, uint32_t) {
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = __byte_perm(x.v[2 * j], x.v[2 * j + 1], 0x5410);
    st_shared_v4(dst, w);
}
__device__ __forceinline__ void put8(const Vec8<float> &x, uint32_t dst, uint32_t plane_bytes) {
    uint32_t h[4], m[4], l[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        uint32_t hb[2], mb[2], lb[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) split3(x.v[2 * j + i], hb[i], mb[i], lb[i]);
        h[j] = upper_halves(hb[0], hb[1]);
        m[j] = upper_halves(mb[0], mb[1]);
        l[j] = upper_halves(lb[0], lb[1]);
    }
    st_shared_v4(dst, h);
    st_shared_v4(dst + plane_bytes, m);
    st_shared_v4(dst + 2 * plane_bytes, l);
}

// ---------------------------------------------------------------- operands
// rows = the m or n index of the product.  How a producer warp walks an operand, and with it the
// tile's layout in shared memory, follows the memory:
enum Walk {
    kVecK,    // rows contiguous along k and 16-byte aligned: a thread fetches 8 k with vector loads,
              // eight threads a row; K-major tile
    kByRow,   // contiguous along the rows: a thread keeps one row and fetches 8 k one by one, a warp
              // 32 neighbouring rows; K-major tile
    kByK,     // contiguous along k, no alignment: a thread keeps one k and fetches 8 rows one by one,
              // a warp 32 neighbouring k; MN-major tile
    kPiecesByRow,   // pieces of 16 bytes along k: as kVecK, with a state per row
    kPiecesByK,     // pieces of 16 bytes along the rows: eight threads a k (64 rows), MN-major tile
};
constexpr bool by_rows(Walk w) { return w == kByRow || w == kPiecesByRow; }   // states belong to rows
constexpr bool mn_major(Walk w) { return w == kByK || w == kPiecesByK; }
// Concept:
//   static constexpr Walk kWalk
//   static constexpr int kTable      ints of shared memory prepared by init()
//   void begin(State &, table, int i, int end)   kByRow: row i once per tile; kByK: k = i once per
//                                    64-k step (end: rows, or the k slice's end)
//   void load(const State &, table, int row, int k, int k_end, Vec8<T> &) const
//                                    kVecK, kByRow: k .. k + 7 of `row`; kByK: row .. row + 7 at
//                                    the state's k
//   float at(int row, int k) const   one element (the recomputation of a non-finite output)
// Rows beyond `rows` are zero or not staged at all: they only reach output rows or columns that
// are not stored.

// Strided matrix: element (row, k) at p[row * s_row + k * s_k].
template <class T, Walk WALK>
struct Strided {
    static constexpr Walk kWalk = WALK;
    static constexpr int kTable = 0;
    const T *p;
    int64_t s_row, s_k;
    int rows;
    struct State { int k, ok; };
    __device__ __forceinline__ void init(int *, int, int) const {}
    __device__ __forceinline__ void begin(State &s, const int *, int i, int end) const {
        s.k = i;
        s.ok = i < end;
    }
    __device__ __forceinline__ void load(const State &s, const int *, int row, int k, int k_end,
                                         Vec8<T> &d) const {
        if (WALK == kByK) {
            const T *q = p + (int64_t)row * s_row + (int64_t)s.k * s_k;
            if (row + 8 <= rows) {
#pragma unroll
                for (int j = 0; j < 8; ++j, q += s_row) fetch(d.v[j], q, s.ok);
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j, q += s_row) fetch(d.v[j], q, s.ok && row + j < rows);
            }
            return;
        }
        const T *q = p + (int64_t)row * s_row + (int64_t)k * s_k;
        if (WALK == kVecK) {
            if (k + 8 <= k_end) {
                fetch8(d, q);
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) fetch(d.v[j], q + j, k + j < k_end);
            }
        } else if (k + 8 <= k_end) {
#pragma unroll
            for (int j = 0; j < 8; ++j, q += s_k) fetch(d.v[j], q, true);
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j, q += s_k) fetch(d.v[j], q, k + j < k_end);
        }
    }
    __device__ __forceinline__ float at(int row, int k) const {
        return to_f32(p[(int64_t)row * s_row + (int64_t)k * s_k]);
    }
};

// Geometry of a convolution seen from a grid of positions [b][gh][gw]: position (b, y, x) and
// filter tap (fi, fj) meet source element (sy, sx) of channel c of [b][channels][sh][sw].
//   forward / weight gradient: sy = y * st_h - pad_h + fi * dil_h          (source = x)
//   input gradient:            sy = (y + pad_h - fi * dil_h) / st_h, exact (source = dy)
// In both cases the source address is separable, base(position) + offset(channel, tap): for the
// input gradient (a - b) / s = floor(a / s) - floor(b / s) whenever s divides a - b.  Which taps
// are valid at a position is a bit mask of at most 32 taps.
struct ConvMap {
    int channels, sh, sw;        // source planes
    int gw, ghw;                 // position grid
    int fh, fw, ff;
    int st_h, st_w, pad_h, pad_w, dil_h, dil_w;
    bool gradient;               // input-gradient form
    bool always_valid;           // no tap of any position leaves the source
    bool ranges;                 // neighbouring taps meet neighbouring elements: valid taps are a range
    uint32_t row_ones;           // bit fi * fw of every filter row
    FastDiv div_ghw, div_gw, div_fw, div_st_h, div_st_w, div_cp;
    int cp;                      // channels rounded up to 8

    __device__ __forceinline__ int tap_offset(int tap) const {
        const int fi = (int)div_fw.div((uint32_t)tap), fj = tap - fi * fw;
        if (gradient)
            return -((int)div_st_h.div((uint32_t)(fi * dil_h)) * sw + (int)div_st_w.div((uint32_t)(fj * dil_w)));
        return fi * dil_h * sw + fj * dil_w;
    }
    // Taps of one filter row valid at grid column x, and the rows' bits (bit fi * fw) at grid row y.
    __device__ __forceinline__ uint32_t columns(int x) const {
        uint32_t cols = 0;
        for (int fj = 0; fj < fw; ++fj) {
            if (!gradient) {
                if ((unsigned)(x * st_w - pad_w + fj * dil_w) < (unsigned)sw) cols |= 1u << fj;
            } else {
                const int t = x + pad_w - fj * dil_w;
                if (t < 0) break;
                uint32_t q, rem;
                div_st_w.divmod((uint32_t)t, q, rem);
                if (rem == 0 && q < (uint32_t)sw) cols |= 1u << fj;
            }
        }
        return cols;
    }
    __device__ __forceinline__ uint32_t row_bits(int y) const {
        uint32_t bits = 0;
        for (int fi = 0; fi < fh; ++fi) {
            if (!gradient) {
                if ((unsigned)(y * st_h - pad_h + fi * dil_h) < (unsigned)sh) bits |= 1u << (fi * fw);
            } else {
                const int t = y + pad_h - fi * dil_h;
                if (t < 0) break;
                uint32_t q, rem;
                div_st_h.divmod((uint32_t)t, q, rem);
                if (rem == 0 && q < (uint32_t)sh) bits |= 1u << (fi * fw);
            }
        }
        return bits;
    }
    __device__ __forceinline__ int base_of(int b, int y, int x) const {
        const int image = b * channels * sh * sw;
        if (!gradient) return image + (y * st_h - pad_h) * sw + x * st_w - pad_w;
        return image + (int)div_st_h.div((uint32_t)(y + pad_h)) * sw + (int)div_st_w.div((uint32_t)(x + pad_w));
    }
    // Taps [lo, hi) of a filter of n whose first tap meets source coordinate t of `size`, scaled by `unit` bits.
    __device__ __forceinline__ uint32_t range_bits(int t, int n, int size, int unit) const {
        const int lo = max(0, gradient ? t - size + 1 : -t), hi = min(n, gradient ? t + 1 : size - t);
        uint32_t bits;
        // volatile: moved about freely, its operands stay in registers through the main loop of the 128-column
        // tiles (9 x 64 x 44 x 44 -> 128 5x5 f32 81 us instead of 72)
        asm volatile("bmsk.clamp.b32 %0, %1, %2;" : "=r"(bits) : "r"(lo * unit), "r"(max(hi - lo, 0) * unit));
        return bits;
    }
    // Base address of a position and its tap mask (columns < 2^fw, so the product has no carries).  A thread
    // does this once per tile (rows) or per 64-k step (columns), where the loops over taps were a quarter of
    // the weight gradient's instructions: with ranges they are two masks (16 -> 32 3x3, 64 x 32 x 32 f32: weight gradient 40.6 -> 38.3 us, input
    // gradient 34.9 -> 32.9, forward 28.7 -> 27.6; 5 x 64 x 22 x 22 -> 128 bf16 forward 15.9 -> 15.1).
    __device__ __forceinline__ void position(int pos, int &base, uint32_t &mask) const {
        uint32_t b, r, y, x;
        div_ghw.divmod((uint32_t)pos, b, r);
        div_gw.divmod(r, y, x);
        if (ranges) {
            const int ty = (int)y * st_h + (gradient ? pad_h : -pad_h), tx = (int)x * st_w + (gradient ? pad_w : -pad_w);
            base = (int)b * channels * sh * sw + ty * sw + tx;
            mask = (range_bits(ty, fh, sh, fw) & row_ones) * range_bits(tx, fw, sw, 1);
            return;
        }
        base = base_of((int)b, (int)y, (int)x);
        mask = always_valid ? 0xffffffffu : row_bits((int)y) * columns((int)x);
    }
};

// The patch index runs tap-major over channels padded to a multiple of 8, so that eight neighbouring
// indices share a tap: its check and offset are made once and the addresses step by whole planes (4
// instructions per element, where a channel-major order takes 16).
//
// Rows are positions, k = (tap, channel): the patch matrix of the forward pass and of the input
// gradient.
template <class T>
struct ConvRows {
    static constexpr Walk kWalk = kByRow;
    static constexpr int kTable = 32;
    const T *src;
    ConvMap g;
    int rows;
    struct State {
        int base;
        uint32_t mask;
    };
    __device__ __forceinline__ void init(int *table, int tid, int threads) const {
        for (int t = tid; t < g.ff; t += threads) table[t] = g.tap_offset(t);
    }
    __device__ __forceinline__ void begin(State &s, const int *, int row, int end) const {
        s.base = 0;
        s.mask = 0;
        if (row < end) g.position(row, s.base, s.mask);
    }
    __device__ __forceinline__ void load(const State &s, const int *table, int, int k, int k_end,
                                         Vec8<T> &d) const {
        uint32_t tap, c;
        g.div_cp.divmod((uint32_t)k, tap, c);
        const int plane = g.sh * g.sw;
        const bool ok = k < k_end && ((s.mask >> tap) & 1u);
        const T *q = src + (ok ? s.base + table[tap] + (int)c * plane : 0);
        if (c + 8 <= (uint32_t)g.channels) {
#pragma unroll
            for (int j = 0; j < 8; ++j, q += plane) fetch(d.v[j], q, ok);
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j, q += plane) fetch(d.v[j], q, ok && (int)c + j < g.channels);
        }
    }
    __device__ __forceinline__ float at(int row, int k) const {
        int base;
        uint32_t mask, c, tap;
        g.position(row, base, mask);
        g.div_cp.divmod((uint32_t)k, tap, c);
        if (!((mask >> tap) & 1u) || (int)c >= g.channels) return 0.f;
        return to_f32(src[base + (int)c * g.sh * g.sw + g.tap_offset((int)tap)]);
    }
};

// Rows are (tap, channel), k = positions: the transposed patch matrix of the weight gradient.
template <class T>
struct ConvCols {
    static constexpr Walk kWalk = kByK;
    static constexpr int kTable = 32;
    const T *src;
    ConvMap g;
    int rows;
    struct State {
        int base;
        uint32_t mask;
    };
    __device__ __forceinline__ void init(int *table, int tid, int threads) const {
        for (int t = tid; t < g.ff; t += threads) table[t] = g.tap_offset(t);
    }
    __device__ __forceinline__ void begin(State &s, const int *, int k, int end) const {
        s.base = 0;
        s.mask = 0;
        if (k < end) g.position(k, s.base, s.mask);
    }
    __device__ __forceinline__ void load(const State &s, const int *table, int row, int, int,
                                         Vec8<T> &d) const {
        uint32_t tap, c;
        g.div_cp.divmod((uint32_t)row, tap, c);
        const int plane = g.sh * g.sw;
        const bool ok = (s.mask >> tap) & 1u;
        const T *q = src + (ok ? s.base + table[tap] + (int)c * plane : 0);
        if (c + 8 <= (uint32_t)g.channels) {
#pragma unroll
            for (int j = 0; j < 8; ++j, q += plane) fetch(d.v[j], q, ok);
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j, q += plane) fetch(d.v[j], q, ok && (int)c + j < g.channels);
        }
    }
    __device__ __forceinline__ float at(int row, int k) const {
        int base;
        uint32_t mask, c, tap;
        g.position(k, base, mask);
        g.div_cp.divmod((uint32_t)row, tap, c);
        if (!((mask >> tap) & 1u) || (int)c >= g.channels) return 0.f;
        return to_f32(src[base + (int)c * g.sh * g.sw + g.tap_offset((int)tap)]);
    }
};

// A filter bank in the order of ConvRows' k, read where it lies: element (row, (tap, channel)) at
// w[row * s_row + channel * s_c + tap], zero for the padding channels.  Eight strided loads per chunk where the
// repacked copy is one vector, but no launch to make the copy.
template <class T>
struct FilterRows {
    static constexpr Walk kWalk = kByRow;
    static constexpr int kTable = 0;
    const T *w;
    int s_row, s_c, channels;
    FastDiv div_cp;
    struct State { const T *q; };
    __device__ __forceinline__ void init(int *, int, int) const {}
    __device__ __forceinline__ void begin(State &s, const int *, int row, int) const { s.q = w + (int64_t)row * s_row; }
    __device__ __forceinline__ void load(const State &s, const int *, int, int k, int k_end, Vec8<T> &d) const {
        uint32_t tap, c;
        div_cp.divmod((uint32_t)k, tap, c);
        const T *q = s.q + (int)c * s_c + (int)tap;
#pragma unroll
        for (int j = 0; j < 8; ++j, q += s_c) fetch(d.v[j], q, k < k_end && (int)c + j < channels);
    }
    __device__ __forceinline__ float at(int row, int k) const {
        uint32_t tap, c;
        div_cp.divmod((uint32_t)k, tap, c);
        return (int)c < channels ? to_f32(w[(int64_t)row * s_row + (int)c * s_c + (int)tap]) : 0.f;
    }
};

// Few channels: padding them to eight would multiply the patch (1 channel: by eight).  The patch index is
// the filter bank's own (channel, tap) order instead, so the filters need no repacking; a table holds
// each index's offset and tap, and an element costs 6 instructions.
constexpr int kFewPatch = 160;           // longest patch
template <class T>
struct FewRows {                         // as ConvRows
    static constexpr Walk kWalk = kByRow;
    static constexpr int kTable = kFewPatch;
    const T *src;
    ConvMap g;
    int rows, patch;                     // patch = channels * taps
    struct State {
        int base;
        uint32_t mask;
    };
    __device__ __forceinline__ int entry(int k) const {
        const int c = k / g.ff, tap = k - c * g.ff;
        return ((c * g.sh * g.sw + g.tap_offset(tap)) << 5) | tap;
    }
    __device__ __forceinline__ void init(int *table, int tid, int threads) const {
        for (int k = tid; k < patch; k += threads) table[k] = entry(k);
    }
    __device__ __forceinline__ void begin(State &s, const int *, int row, int end) const {
        s.base = 0;
        s.mask = 0;
        if (row < end) g.position(row, s.base, s.mask);
    }
    __device__ __forceinline__ void one(const State &s, const int *table, int k, bool in, decltype(Vec8<T>().v[0]) &d) const {
        const int e = in ? table[k] : 0;
        const bool ok = in && ((s.mask >> (e & 31)) & 1u);
        fetch(d, src + (ok ? s.base + (e >> 5) : 0), ok);
    }
    __device__ __forceinline__ void load(const State &s, const int *table, int, int k, int k_end, Vec8<T> &d) const {
#pragma unroll
        for (int j = 0; j < 8; ++j) one(s, table, k + j, k + j < k_end, d.v[j]);
    }
    __device__ __forceinline__ float at(int row, int k) const {
        State s;
        begin(s, nullptr, row, row + 1);
        const int e = entry(k);
        return (s.mask >> (e & 31)) & 1u ? to_f32(src[s.base + (e >> 5)]) : 0.f;
    }
};
template <class T>
struct FewCols {                         // as ConvCols: rows are (channel, tap), k = positions
    static constexpr Walk kWalk = kByK;
    static constexpr int kTable = kFewPatch;
    FewRows<T> f;                        // f.rows is not used
    using State = typename FewRows<T>::State;
    __device__ __forceinline__ void init(int *table, int tid, int threads) const { f.init(table, tid, threads); }
    __device__ __forceinline__ void begin(State &s, const int *table, int k, int end) const { f.begin(s, table, k, end); }
    __device__ __forceinline__ void load(const State &s, const int *table, int row, int, int, Vec8<T> &d) const {
#pragma unroll
        for (int j = 0; j < 8; ++j) f.one(s, table, row + j, row + j < f.patch, d.v[j]);
    }
    __device__ __forceinline__ float at(int row, int k) const { return f.at(k, row); }
};

// Rows are channels of an NCHW tensor, k = (image, position).
template <class T>
struct ChannelRows {
    static constexpr Walk kWalk = kByK;
    static constexpr int kTable = 0;
    const T *src;
    int rows, hw;
    FastDiv div_hw;
    struct State { int base, ok; };
    __device__ __forceinline__ void init(int *, int, int) const {}
    __device__ __forceinline__ void begin(State &s, const int *, int k, int end) const {
        uint32_t b, r;
        div_hw.divmod((uint32_t)k, b, r);
        s.base = (int)b * rows * hw + (int)r;
        s.ok = k < end;
    }
    __device__ __forceinline__ void load(const State &s, const int *, int row, int, int, Vec8<T> &d) const {
        const T *q = src + (s.ok ? s.base + row * hw : 0);
        if (row + 8 <= rows) {
#pragma unroll
            for (int j = 0; j < 8; ++j, q += hw) fetch(d.v[j], q, s.ok);
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j, q += hw) fetch(d.v[j], q, s.ok && row + j < rows);
        }
    }
    __device__ __forceinline__ float at(int row, int k) const {
        uint32_t b, r;
        div_hw.divmod((uint32_t)k, b, r);
        return to_f32(src[((int64_t)b * rows + row) * hw + r]);
    }
};

// The same on tensors that have been split once, [plane][image][position][cp] bf16 with the channels padded to eight (zeros):
// eight channels of a position are one 16-byte piece per plane, which cp.async brings to the tile, where the forms above
// fetch eight times and split again for every tap that meets the position.
//   int piece(State &, table, row, k, k_end)   index of the piece at (row, k), or -1 for zeros
// `from` is the form it stands for, which an output that is not finite is computed with.
constexpr bool in_pieces(Walk w) { return w == kPiecesByRow || w == kPiecesByK; }
struct Pieces {
    const uint4 *p;
    int64_t plane;                       // pieces per plane
};
template <class T>
struct SplitRows {                       // as ConvRows
    static constexpr Walk kWalk = kPiecesByRow;
    static constexpr int kTable = 32;
    Pieces src;
    ConvMap g;                           // of one channel: bases and offsets count positions
    FastDiv div_groups;
    int groups;                          // of eight channels
    ConvRows<T> from;
    struct State {
        int base;
        uint32_t mask;
    };
    __device__ __forceinline__ void init(int *table, int tid, int threads) const {
        for (int t = tid; t < g.ff; t += threads) table[t] = g.tap_offset(t);
    }
    __device__ __forceinline__ void begin(State &s, const int *, int row, int end) const {
        s.base = 0;
        s.mask = 0;
        if (row < end) g.position(row, s.base, s.mask);
    }
    __device__ __forceinline__ int piece(const State &s, const int *table, int, int k, int k_end) const {
        uint32_t tap, c;
        div_groups.divmod((uint32_t)k / 8, tap, c);
        return k < k_end && ((s.mask >> tap) & 1u) ? (s.base + table[tap]) * groups + (int)c : -1;
    }
    __device__ __forceinline__ float at(int row, int k) const { return from.at(row, k); }
};
template <class T>
struct SplitCols {                       // as ConvCols
    static constexpr Walk kWalk = kPiecesByK;
    static constexpr int kTable = 32;
    Pieces src;
    ConvMap g;
    FastDiv div_groups;
    int groups;
    ConvCols<T> from;
    struct State {
        int base;
        uint32_t mask;
    };
    __device__ __forceinline__ void init(int *table, int tid, int threads) const {
        for (int t = tid; t < g.ff; t += threads) table[t] = g.tap_offset(t);
    }
    __device__ __forceinline__ void begin(State &s, const int *, int k, int end) const {
        s.base = 0;
        s.mask = 0;
        if (k < end) g.position(k, s.base, s.mask);
    }
    __device__ __forceinline__ int piece(const State &s, const int *table, int row, int, int) const {
        uint32_t tap, c;
        div_groups.divmod((uint32_t)row / 8, tap, c);
        return (s.mask >> tap) & 1u ? (s.base + table[tap]) * groups + (int)c : -1;
    }
    __device__ __forceinline__ float at(int row, int k) const { return from.at(row, k); }
};
template <class T>
struct SplitChannels {                   // as ChannelRows
    static constexpr Walk kWalk = kPiecesByK;
    static constexpr int kTable = 0;
    Pieces src;
    int groups;
    ChannelRows<T> from;
    struct State { int base; };
    __device__ __forceinline__ void init(int *, int, int) const {}
    __device__ __forceinline__ void begin(State &s, const int *, int k, int end) const { s.base = k < end ? k * groups : -1; }
    __device__ __forceinline__ int piece(const State &s, const int *, int row, int, int) const {
        return s.base < 0 ? -1 : s.base + row / 8;
    }
    __device__ __forceinline__ float at(int row, int k) const { return from.at(row, k); }
};
template <class T>
struct SplitFilters {                    // as FilterRows: [plane][row][(tap, padded channel)]
    static constexpr Walk kWalk = kPiecesByRow;
    static constexpr int kTable = 0;
    Pieces src;
    int pitch;                           // pieces per row
    FilterRows<T> from;
    struct State { int base; };
    __device__ __forceinline__ void init(int *, int, int) const {}
    __device__ __forceinline__ void begin(State &s, const int *, int row, int) const { s.base = row * pitch; }
    __device__ __forceinline__ int piece(const State &s, const int *, int, int k, int k_end) const {
        return k < k_end ? s.base + k / 8 : -1;
    }
    __device__ __forceinline__ float at(int row, int k) const { return from.at(row, k); }
};

// 16 bytes of global memory, or zeros, to shared memory, asynchronously.
__device__ __forceinline__ void copy_piece(uint32_t dst, const uint4 *src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
template <int PL>
__device__ __forceinline__ void copy_pieces(uint32_t dst, uint32_t plane_bytes, const Pieces &src, int at) {
#pragma unroll
    for (int i = 0; i < PL; ++i) copy_piece(dst + i * plane_bytes, src.p + (at < 0 ? 0 : i * src.plane + at), at >= 0);
}

// ---------------------------------------------------------------- epilogues
// Concept: State begin(int row, int col); void store(State &, int col, float acc), which stores at the
// state's position and moves it to the next column: with a 64-bit address per element from
// scratch the stores were a third of the kernel's instructions at 48 k.
// A warp holds 32 consecutive rows of one column at a time, so the tensor written should be
// contiguous along the rows.

// C = alpha * acc + beta * C, element (row, col) at c[row * s_row + col * s_col].
template <class T>
struct StridedOut {
    static constexpr bool kLastCtaAdds = false;   // who adds k slices, see launch()
    T *c;
    int64_t s_row, s_col;
    float alpha, beta;
    struct State { T *q; };
    __device__ __forceinline__ State begin(int row, int col) const {
        return State{c + (int64_t)row * s_row + (int64_t)col * s_col};
    }
    __device__ __forceinline__ void store(State &s, int, float acc) const {
        float v = alpha * acc;
        if (beta != 0.f) v += beta * to_f32(*s.q);
        *s.q = from_f32<T>(v);
        s.q += s_col;
    }
};

// y[col][row] = relu?(round(round(acc) + bias[row])): a Dense layer with rows = outputs.
template <class T>
struct DenseOut {
    static constexpr bool kLastCtaAdds = false;
    T *c;
    int64_t s_col;
    const T *bias;
    bool relu;
    struct State { T *q; float b; };
    __device__ __forceinline__ State begin(int row, int col) const {
        return State{c + row + (int64_t)col * s_col, bias != nullptr ? to_f32(bias[row]) : 0.f};
    }
    __device__ __forceinline__ void store(State &s, int, float acc) const {
        float v = to_f32(from_f32<T>(acc));
        if (bias != nullptr) v = to_f32(from_f32<T>(__fadd_rn(v, s.b)));
        if (relu) v = (v >= 0.f) ? v : 0.f;
        *s.q = from_f32<T>(v);
        s.q += s_col;
    }
};

// Rows are (image, position), columns channels of an NCHW tensor; optional bias and relu with
// the roundings of the separate operators.
template <class T>
struct NchwOut {
    static constexpr bool kLastCtaAdds = true;
    T *y;
    const T *bias;
    int channels, hw;
    FastDiv div_hw;
    bool relu;
    struct State { T *q; };
    __device__ __forceinline__ State begin(int row, int col) const {
        uint32_t b, r;
        div_hw.divmod((uint32_t)row, b, r);
        return State{y + ((int64_t)b * channels + col) * hw + r};
    }
    __device__ __forceinline__ void store(State &s, int col, float acc) const {
        float v = to_f32(from_f32<T>(acc));
        if (bias != nullptr) v = to_f32(from_f32<T>(v + to_f32(bias[col])));
        if (relu) v = (v >= 0.f) ? v : 0.f;
        *s.q = from_f32<T>(v);
        s.q += hw;
    }
};

// Rows are (tap, padded channel), columns output channels: dw[col][channel][tap] = beta * dw + acc.
template <class T>
struct FilterOut {
    static constexpr bool kLastCtaAdds = true;
    T *dw;
    int channels, ff;
    FastDiv div_cp;
    int cp;
    float beta;
    struct State { T *q; bool padding; };
    __device__ __forceinline__ State begin(int row, int col) const {
        uint32_t tap, c;
        div_cp.divmod((uint32_t)row, tap, c);
        return State{dw + ((int64_t)col * channels + (int)c) * ff + (int)tap, (int)c >= channels};
    }
    __device__ __forceinline__ void store(State &s, int, float acc) const {
        if (!s.padding) *s.q = from_f32<T>(beta != 0.f ? acc + beta * to_f32(*s.q) : acc);
        s.q += channels * ff;
    }
};

// ------------------------------------------------------------------- kernel
// Tiles of one CTA in one launch whose blocks of outputs can be marked, a byte each.
constexpr int kMarks = 1024;
// Shared memory of redo_block: 16 k of 32 rows and 32 columns.
constexpr int kRedoK = 16, kRedoPitch = 36, kRedoFloats = 2 * kRedoK * kRedoPitch;

template <class T, int BN_>
struct Cfg {
    static constexpr int PL = Planes<T>::N;
    static constexpr int BN = BN_;
    static constexpr int EPI_WARPS = BN >= 64 ? 8 : 4;
    static constexpr int COLS = BN * 4 / EPI_WARPS;              // columns per epilogue warp
    // Sixteen producer warps hide more of the loads' latency; the 128-column epilogue
    // leaves registers for eight.
    static constexpr int PRODUCERS = BN == 128 ? 256 : 512;
    static constexpr int THREADS = PRODUCERS + EPI_WARPS * 32 + 32;
    static constexpr int A_PLANE = BM * ROW_BYTES, B_PLANE = BN * ROW_BYTES;
    static constexpr int STAGE = PL * (A_PLANE + B_PLANE);
    static constexpr int STAGES = PL == 3 ? (BN > 64 ? 2 : 3) : 4;
    static constexpr int ACC_COLS = PL == 3 ? 2 * BN : BN;       // f32: leading block + corrections
    static constexpr int TMEM = 2 * ACC_COLS < 64 ? 64 : 2 * ACC_COLS;
    static constexpr int SMEM = STAGES * STAGE + 1024 + 256 + 2 * kFewPatch * (int)sizeof(int) + (PL == 3 ? kMarks : 0);
    // A slice's sums lie behind redo_block's buffers.
    static constexpr int SUMS = PL == 3 ? (THREADS / 32 * kRedoFloats * 4 + 1023) / 1024 * 1024 : 0;
    static_assert(SUMS + BN * BM * 4 <= STAGES * STAGE, "a slice's sums fit the stages");
    static_assert(SMEM <= 227 * 1024, "shared memory");
    static_assert(TMEM <= 512 && (TMEM & (TMEM - 1)) == 0, "tensor memory columns");
    static_assert(COLS % 32 == 0 && EPI_WARPS <= 8, "blocks of 32 columns, a mark bit per epilogue warp");
    static_assert(PRODUCERS % 128 == 0, "epilogue warp e reads rows e % 4 * 32 ..");
    static_assert(THREADS / 32 * kRedoFloats * 4 <= STAGES * STAGE || PL == 1, "the stages hold redo_block's buffers");
};

struct Params {
    int M, N, K;
    int tiles_m, tiles_n, splits, k_split;  // k_split: k per slice, a multiple of BK
    int work0, work1;                       // this launch's share of the tiles x slices
    float *partial;                         // splits > 1: [splits][N][M] f32 sums
    int *arrivals;                          // not null: the CTA of a tile that finishes last adds its slices
    int cluster;                            // the CTAs of a tile's slices are a cluster, which adds them
    int *status;
};

// Which 16-byte chunks of an R x 64 operand tile a producer thread fills.  K-major tiles hold rows of
// 128 bytes (64 k), MN-major tiles 64-row atoms of 8 KiB with 128 bytes (64 rows) per k; both with
// the 128-byte swizzle.
template <Walk WALK, int R, int PRODUCERS>
struct Slots {
    static constexpr bool kEight = WALK == kVecK || WALK == kPiecesByRow || WALK == kPiecesByK;   // eight threads a row or k
    static constexpr int kAtoms = R >= 64 ? R / 64 : 1;
    // States of an operand that a thread walks with, and the one of its i-th chunk.
    static constexpr int kChunks = R * 8 / PRODUCERS < 1 ? 1 : R * 8 / PRODUCERS;
    static constexpr int kStates = WALK == kPiecesByRow ? kChunks : WALK == kPiecesByK ? (kChunks + kAtoms - 1) / kAtoms : 1;
    static constexpr __device__ __forceinline__ int state(int i) {
        return WALK == kPiecesByRow ? i : WALK == kPiecesByK ? i / kAtoms : 0;
    }
    int a, b;      // kByRow: row, chunk; kVecK, kPiecesByRow: row, chunk; kByK, kPiecesByK: k, group of 8 rows
    bool mine;
    __device__ __forceinline__ explicit Slots(int tid) {
        a = WALK == kByRow ? (tid & (R - 1)) : kEight ? (tid >> 3) : (tid & 63);
        b = WALK == kByRow ? tid / R : kEight ? (tid & 7) : (tid >> 6);
        // One value per warp, and known to be: what follows from it (tap, channel, the table's entry,
        // the bounds) is computed once per warp.  With 256 producers, who hold four chunks of each operand,
        // the same costs spills (9 x 64 x 44 x 44 -> 128 5x5 f32 72 -> 83 us).
        if (!kEight && PRODUCERS > 256) b = __shfl_sync(0xffffffffu, b, 0);
        mine = R * 8 >= PRODUCERS || tid < R * 8;
    }
    __device__ __forceinline__ int row(int i) const {
        return WALK == kByRow ? a : WALK == kPiecesByK ? (b + i % kAtoms * 8) * 8
             : WALK == kByK ? (b + i * (PRODUCERS / 64)) * 8 : a + i * (PRODUCERS / 8);
    }
    __device__ __forceinline__ int k(int i) const {
        return WALK == kByRow ? (b + i * (PRODUCERS / R)) * 8 : WALK == kPiecesByK ? a + i / kAtoms * (PRODUCERS / 8)
             : WALK == kByK ? a : b * 8;
    }
    __device__ __forceinline__ uint32_t offset(int i) const {
        if (mn_major(WALK)) {
            const int g = row(i) >> 3, kk = k(i);
            return (g >> 3) * 8192 + kk * 128 + (((g & 7) ^ (kk & 7)) << 4);
        }
        const int r = row(i), ch = k(i) >> 3;
        return r * ROW_BYTES + ((ch ^ (r & 7)) << 4);
    }
};

// The 32 x 32 outputs at (row0, col0) from the operands as they were given: sums of k0 .. k1 in order, one
// warp.  A lane has rows row0 + lane / 4 * 4 .. + 3 and columns col0 + lane % 4 * 8 .. + 7.  `buf` is the warp's
// (kRedoFloats); ROWS_A, ROWS_B: neighbouring lanes fetch neighbouring rows of the operand, else
// neighbouring k.  4096^3 f32, 0.59 ms: with a NaN in one row of A 2.3 ms (a chain of FMAs per lane in
// the epilogue, which the pipeline's bounded waits had to outlast: 31 to 42 ms), with NaNs everywhere 0.7 ms.
template <bool ROWS_A, bool ROWS_B, class AOp, class BOp>
__device__ __forceinline__ void redo_block(const AOp &A, const BOp &B, int row0, int M, int col0, int N, int k0, int k1,
                                        float *buf, float (&acc)[4][8]) {
    const int lane = threadIdx.x & 31, ty = lane >> 2, tx = lane & 3;
    float *sa = buf, *sb = buf + kRedoK * kRedoPitch;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
    for (int k = k0; k < k1; k += kRedoK) {
        __syncwarp();
#pragma unroll 1
        for (int i0 = 0; i0 < kRedoK; i0 += 8) {   // sixteen loads in flight
            float va[8], vb[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int ra = ROWS_A ? lane : 2 * (i0 + i) + (lane >> 4), ka = ROWS_A ? i0 + i : lane & 15;
                const int rb = ROWS_B ? lane : 2 * (i0 + i) + (lane >> 4), kb = ROWS_B ? i0 + i : lane & 15;
                va[i] = row0 + ra < M && k + ka < k1 ? A.at(row0 + ra, k + ka) : 0.f;
                vb[i] = col0 + rb < N && k + kb < k1 ? B.at(col0 + rb, k + kb) : 0.f;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                sa[(ROWS_A ? i0 + i : lane & 15) * kRedoPitch + (ROWS_A ? lane : 2 * (i0 + i) + (lane >> 4))] = va[i];
                sb[(ROWS_B ? i0 + i : lane & 15) * kRedoPitch + (ROWS_B ? lane : 2 * (i0 + i) + (lane >> 4))] = vb[i];
            }
        }
        __syncwarp();
        const int ks = min(kRedoK, k1 - k);
        for (int i = 0; i < ks; ++i) {
            const float4 a = *reinterpret_cast<const float4 *>(sa + i * kRedoPitch + 4 * ty);
            const float4 b0 = *reinterpret_cast<const float4 *>(sb + i * kRedoPitch + 8 * tx);
            const float4 b1 = *reinterpret_cast<const float4 *>(sb + i * kRedoPitch + 8 * tx + 4);
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 8; ++c) acc[r][c] = fmaf(av[r], bv[c], acc[r][c]);
        }
        // a sum that is a NaN stays one: a block of them is done
        if (__all_sync(0xffffffffu, isnan(acc[0][0]) || row0 + 4 * ty >= M || col0 + 8 * tx >= N)) {
            bool all = true;
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    all = all && (isnan(acc[r][c]) || row0 + 4 * ty + r >= M || col0 + 8 * tx + c >= N);
            if (__all_sync(0xffffffffu, all)) return;
        }
    }
}

// One tile's slices added in slice order, as reduce_splits_kernel adds them, and stored: four columns and
// four slices at a time, because a single SM pulls them out of L2.
template <int THREADS, class Epi>
__device__ __forceinline__ void reduce_tile(const Params &p, const Epi &E, int m0, int n0, int bn, int tid) {
    constexpr int LANES = THREADS / BM;        // threads beyond LANES * BM idle
    const int row = m0 + tid % BM, n1 = min(p.N, n0 + bn);
    if (tid >= LANES * BM || row >= p.M) return;
    const int64_t plane = (int64_t)p.M * p.N;
    for (int col = n0 + tid / BM * 4; col < n1; col += LANES * 4) {
        const float *q = p.partial + (int64_t)col * p.M + row;
        float s[4] = {0.f, 0.f, 0.f, 0.f};
        for (int z = 0; z < p.splits; z += 4) {
            float v[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    v[i][j] = z + i < p.splits && col + j < n1 ? __ldcg(q + (z + i) * plane + (int64_t)j * p.M) : 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (z + i < p.splits) s[j] += v[i][j];
        }
        typename Epi::State st = E.begin(row, col);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (col + j < n1) E.store(st, col + j, s[j]);
    }
}

// Whether CTAs of this kernel add slices themselves.  Operands of few channels have three steps of k at most, which are never
// sliced: the code for it cost their bf16 kernels spills (47 x 3 x 15 x 21 -> 121 1x3 7.0 us, 6.5 without).
template <class AOp>
constexpr bool kShortK = false;
template <class T>
constexpr bool kShortK<FewRows<T>> = true;
template <class AOp, class Epi>
constexpr bool kAddsSlices = Epi::kLastCtaAdds && !kShortK<AOp>;

// First work item of a CTA; item w is slice w / tiles of tile w % tiles, and the slices of a tile are neighbouring CTAs
// where they are a cluster.
template <bool ADDS>
__device__ __forceinline__ int first_item(const Params &p) {
    if (ADDS && p.cluster) return (int)(blockIdx.x % (unsigned)p.splits) * p.tiles_m * p.tiles_n + (int)(blockIdx.x / (unsigned)p.splits);
    return p.work0 + (int)blockIdx.x;
}

// The marked blocks of this CTA's tiles, dealt to its warps.
template <class C, class AOp, class BOp, class Epi>
__device__ __noinline__ void redo_marked(const AOp &A, const BOp &B, const Epi &E, const Params &p,
                                         const unsigned *marks, float *buf, float *sums) {
    constexpr int WARPS = C::THREADS / 32, BLOCKS = C::EPI_WARPS * C::COLS / 32;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, tiles = p.tiles_m * p.tiles_n;
    int turn = 0;
    constexpr bool ADDS = kAddsSlices<AOp, Epi>;
    for (int w = first_item<ADDS>(p), i = 0; w < p.work1; w += gridDim.x, ++i) {
        const unsigned mark = marks[i / 4] >> (i % 4 * 8) & 255u;
        const int tile = w % tiles, z = w / tiles;
        const int k_begin = z * p.k_split, k_end = min(p.K, k_begin + p.k_split);
        for (int block = 0; mark != 0 && block < BLOCKS; ++block) {
            const int e = block % C::EPI_WARPS;
            const int row0 = (tile % p.tiles_m) * BM + e % 4 * 32;
            const int col0 = (tile / p.tiles_m) * C::BN + e / 4 * C::COLS + block / C::EPI_WARPS * 32;
            if ((mark >> e & 1u) == 0 || row0 >= p.M || col0 >= p.N || turn++ % WARPS != warp) continue;
            float acc[4][8];
            redo_block<by_rows(AOp::kWalk), by_rows(BOp::kWalk)>(A, B, row0, p.M, col0, p.N, k_begin, k_end, buf, acc);
            const int row = row0 + lane / 4 * 4, col = col0 + lane % 4 * 8;
            for (int r = 0; r < 4; ++r) {
                if (row + r >= p.M || col >= p.N) break;
                typename Epi::State st = E.begin(row + r, col);
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    if (col + c >= p.N) break;
                    const float v = r == 0 ? acc[0][c] : r == 1 ? acc[1][c] : r == 2 ? acc[2][c] : acc[3][c];
                    if (ADDS && p.cluster)
                        sums[(col + c) % C::BN * BM + (row + r) % BM] = v;
                    else if (p.splits > 1)
                        p.partial[((int64_t)z * p.N + col + c) * p.M + row + r] = v;
                    else
                        E.store(st, col + c, v);
                }
            }
        }
    }
}

template <class T, int BN, class AOp, class BOp, class Epi>
__global__ void __launch_bounds__(Cfg<T, BN>::THREADS, 1)
    gemm_tcx_kernel(const __grid_constant__ AOp A, const __grid_constant__ BOp B,
                    const __grid_constant__ Epi E, const __grid_constant__ Params p) {
    using C = Cfg<T, BN>;
    constexpr int PL = C::PL, STAGES = C::STAGES, PRODUCERS = C::PRODUCERS;
    constexpr bool ADDS = kAddsSlices<AOp, Epi>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                                ~uintptr_t(1023));
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + STAGES * C::STAGE);
    uint64_t *full_bar = bars, *empty_bar = bars + STAGES;
    uint64_t *acc_full = bars + 2 * STAGES, *acc_empty = bars + 2 * STAGES + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * STAGES + 4);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    volatile int *redo = reinterpret_cast<volatile int *>(tmem_slot + 2);   // any mark
    int *table_a = reinterpret_cast<int *>(tmem_slot + 4), *table_b = table_a + kFewPatch;
    // bit e of byte i: epilogue warp e left its block of this CTA's i-th tile out
    unsigned *marks = reinterpret_cast<unsigned *>(table_b + kFewPatch);

    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    constexpr int MMA_WARP = PRODUCERS / 32 + C::EPI_WARPS;
    float *sums = reinterpret_cast<float *>(smem + C::SUMS);   // [column][row] of a slice, in stages that are not used any more

    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) {
            tc::mbar_init(tc::smem_u32(&full_bar[s]), PRODUCERS / 32);
            tc::mbar_init(tc::smem_u32(&empty_bar[s]), 1);
        }
        for (int s = 0; s < 2; ++s) {
            tc::mbar_init(tc::smem_u32(&acc_full[s]), 1);
            tc::mbar_init(tc::smem_u32(&acc_empty[s]), C::EPI_WARPS);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // The last tile's B rows beyond N are never staged: they start as zeros, so that the columns
    // nobody stores do not look like sums to compute again.
    if (PL == 3 && p.N % BN != 0) {
        for (uint32_t i = tid; i < STAGES * PL * C::B_PLANE / 16; i += C::THREADS) {
            const uint32_t st = i / (PL * C::B_PLANE / 16), off = i % (PL * C::B_PLANE / 16);
            const uint32_t zero[4] = {0, 0, 0, 0};
            st_shared_v4(tc::smem_u32(smem + st * C::STAGE + PL * C::A_PLANE) + off * 16, zero);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (PL == 3) {
        if (tid == 0) *redo = 0;
        if (tid < kMarks / 4) marks[tid] = 0;
    }
    if (warp == MMA_WARP) {
        tc::tmem_alloc(tc::smem_u32(tmem_slot), C::TMEM);
        tc::tmem_relinquish();
    }
    if (AOp::kTable) A.init(table_a, tid, C::THREADS);
    if (BOp::kTable) B.init(table_b, tid, C::THREADS);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // The k slices of a convolution (its weight gradient) on every SM let dependents launch at their end: 16 -> 32 3x3,
    // 64 x 32 x 32 f32, 40.0 us at the start, 33.8 so; with an SM left free they gain as all others do (8 x 6 x 20 x 20
    // -> 16 5x5, stride 2, f32: 12.1, at the end 12.9).
    let_dependents_launch(ADDS && p.splits > 1 ? 147u : kAlwaysEarly);
    dependency_wait();

    const int tiles = p.tiles_m * p.tiles_n;
    const int num_work = p.work1, work0 = first_item<ADDS>(p);

    if (warp < PRODUCERS / 32) {
        // ------------------------------------------------------------------ producers
        constexpr int A_PER = BM * 8 / PRODUCERS;                       // row chunks per thread
        constexpr int B_PER = BN * 8 / PRODUCERS < 1 ? 1 : BN * 8 / PRODUCERS;
        int stage = 0;
        uint32_t phase = 0;
        int in_flight = 0, oldest = 0;   // pieces: steps whose copies are under way, and the stage of the first
        const auto hand_over = [&](auto left) {
            asm volatile("cp.async.wait_group %0;" ::"n"(decltype(left)::value) : "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(tc::smem_u32(&full_bar[oldest]));
            if (++oldest == STAGES) oldest = 0;
        };
        for (int w = work0; w < num_work; w += gridDim.x) {
            const int tile = w % tiles, z = w / tiles;
            const int m0 = (tile % p.tiles_m) * BM, n0 = (tile / p.tiles_m) * BN;
            const int k_begin = z * p.k_split, k_end = min(p.K, k_begin + p.k_split);
            using LA = Slots<AOp::kWalk, BM, PRODUCERS>;
            using LB = Slots<BOp::kWalk, BN, PRODUCERS>;
            const LA la(tid);
            const LB lb(tid);
            typename AOp::State sa[LA::kStates];
            typename BOp::State sb[LB::kStates];
#pragma unroll
            for (int i = 0; i < LA::kStates; ++i)
                if (by_rows(AOp::kWalk)) A.begin(sa[i], table_a, m0 + la.row(i), p.M);
#pragma unroll
            for (int i = 0; i < LB::kStates; ++i)
                if (by_rows(BOp::kWalk)) B.begin(sb[i], table_b, n0 + lb.row(i), p.N);
            bool ok = true;
            if constexpr (in_pieces(AOp::kWalk) && in_pieces(BOp::kWalk)) {
                // A step is handed over when the copies of up to STAGES - 2 after it are under way, so that the tensor
                // cores have one while the next is waited for.
                constexpr int kAhead = STAGES > 2 ? STAGES - 2 : 0;
                for (int k0 = k_begin; k0 < k_end; k0 += BK) {
                    const int k_stop = k0 + BK <= k_end ? BK : (k_end - k0 + 15) & ~15;
                    if (!tc::mbar_wait(tc::smem_u32(&empty_bar[stage]), phase ^ 1, abort_flag)) {
                        if (lane == 0) atomicExch(p.status, 181);
                        ok = false;
                        break;
                    }
                    const uint32_t a_base = tc::smem_u32(smem + stage * C::STAGE);
                    const uint32_t b_base = a_base + PL * C::A_PLANE;
#pragma unroll
                    for (int i = 0; i < LA::kStates; ++i)
                        if (mn_major(AOp::kWalk)) A.begin(sa[i], table_a, k0 + la.k(i * LA::kAtoms), k_end);
#pragma unroll
                    for (int i = 0; i < A_PER; ++i)
                        if (m0 + la.row(i) < p.M && la.k(i) < k_stop)
                            copy_pieces<PL>(a_base + la.offset(i), C::A_PLANE, A.src,
                                            A.piece(sa[LA::state(i)], table_a, m0 + la.row(i), k0 + la.k(i), k_end));
#pragma unroll
                    for (int i = 0; i < LB::kStates; ++i)
                        if (mn_major(BOp::kWalk)) B.begin(sb[i], table_b, k0 + lb.k(i * LB::kAtoms), k_end);
#pragma unroll
                    for (int i = 0; i < B_PER; ++i)
                        if (lb.mine && n0 + lb.row(i) < p.N && lb.k(i) < k_stop)
                            copy_pieces<PL>(b_base + lb.offset(i), C::B_PLANE, B.src,
                                            B.piece(sb[LB::state(i)], table_b, n0 + lb.row(i), k0 + lb.k(i), k_end));
                    asm volatile("cp.async.commit_group;" ::: "memory");
                    if (++in_flight > kAhead) {
                        --in_flight;
                        hand_over(std::integral_constant<int, kAhead>());
                    }
                    if (++stage == STAGES) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            } else {
            for (int k0 = k_begin; k0 < k_end; k0 += BK) {
                Vec8<T> va[A_PER], vb[B_PER];
                const int k_stop = k0 + BK <= k_end ? BK : (k_end - k0 + 15) & ~15;   // what the MMAs will read
                if (AOp::kWalk == kByK) A.begin(sa[0], table_a, k0 + la.k(0), k_end);
#pragma unroll
                for (int i = 0; i < A_PER; ++i)
                    if (m0 + la.row(i) < p.M && la.k(i) < k_stop)
                        A.load(sa[0], table_a, m0 + la.row(i), k0 + la.k(i), k_end, va[i]);
                if (BOp::kWalk == kByK) B.begin(sb[0], table_b, k0 + lb.k(0), k_end);
#pragma unroll
                for (int i = 0; i < B_PER; ++i)
                    if (lb.mine && n0 + lb.row(i) < p.N && lb.k(i) < k_stop)
                        B.load(sb[0], table_b, n0 + lb.row(i), k0 + lb.k(i), k_end, vb[i]);
                if (!tc::mbar_wait(tc::smem_u32(&empty_bar[stage]), phase ^ 1, abort_flag)) {
                    if (lane == 0) atomicExch(p.status, 181);
                    ok = false;
                    break;
                }
                const uint32_t a_base = tc::smem_u32(smem + stage * C::STAGE);
                const uint32_t b_base = a_base + PL * C::A_PLANE;
#pragma unroll
                for (int i = 0; i < A_PER; ++i)
                    if (m0 + la.row(i) < p.M && la.k(i) < k_stop) put8(va[i], a_base + la.offset(i), C::A_PLANE);
#pragma unroll
                for (int i = 0; i < B_PER; ++i)
                    if (lb.mine && n0 + lb.row(i) < p.N && lb.k(i) < k_stop) put8(vb[i], b_base + lb.offset(i), C::B_PLANE);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(tc::smem_u32(&full_bar[stage]));
                if (++stage == STAGES) {
                    stage = 0;
                    phase ^= 1;
                }
            }
            }
            if (!ok) break;
        }
        if constexpr (in_pieces(AOp::kWalk) && in_pieces(BOp::kWalk)) {
            // the last steps, one after another (after a wait that expired there is nobody to hand them to)
            asm volatile("cp.async.wait_all;" ::: "memory");
            for (; in_flight > 0; --in_flight) hand_over(std::integral_constant<int, 0>());
        }
    } else if (warp == MMA_WARP) {
        // ------------------------------------------------------------------ MMA issue
        if (tc::elect_one()) {
            constexpr bool A_MN = mn_major(AOp::kWalk), B_MN = mn_major(BOp::kWalk);
            constexpr uint32_t idesc1 = tc::make_idesc(A_MN, B_MN, BM, BN);
            constexpr uint32_t idesc2 = tc::make_idesc(A_MN, B_MN, BM, PL == 3 ? 2 * BN : BN);
            // 16 k further on, and the stride between 64-row atoms
            constexpr uint32_t a_step = A_MN ? 2048 : 32, b_step = B_MN ? 2048 : 32;
            constexpr uint32_t a_lbo = A_MN ? 8192 : 0, b_lbo = B_MN ? 8192 : 0;
            int stage = 0, acc = 0;
            uint32_t phase = 0, acc_phase = 0;
            bool ok = true;
            for (int w = work0; ok && w < num_work; w += gridDim.x) {
                const int k_begin = (w / tiles) * p.k_split, k_end = min(p.K, k_begin + p.k_split);
                int taken = 0;   // steps in this accumulator
                for (int k0 = k_begin; k0 < k_end; k0 += BK) {
                    if (taken == 0) {
                        if (!tc::mbar_wait(tc::smem_u32(&acc_empty[acc]), acc_phase ^ 1, abort_flag)) {
                            atomicExch(p.status, 182);
                            ok = false;
                            break;
                        }
                    }
                    if (!tc::mbar_wait(tc::smem_u32(&full_bar[stage]), phase, abort_flag)) {
                        atomicExch(p.status, 183);
                        ok = false;
                        break;
                    }
                    tc::tc_fence_after();
                    const uint32_t d = tmem + acc * C::ACC_COLS;
                    const uint32_t a_base = tc::smem_u32(smem + stage * C::STAGE);
                    const uint32_t b_base = a_base + PL * C::A_PLANE;
                    auto da = [&](int plane, int k) {
                        return tc::make_smem_desc(a_base + plane * C::A_PLANE + k * a_step, a_lbo, 1024);
                    };
                    auto db = [&](int plane, int k) {
                        return tc::make_smem_desc(b_base + plane * C::B_PLANE + k * b_step, b_lbo, 1024);
                    };
                    const int k_steps = k0 + BK <= k_end ? BK / 16 : (k_end - k0 + 15) / 16;   // a short last step
                    if (PL == 1) {
#pragma unroll
                        for (int k = 0; k < BK / 16; ++k)
                            if (k < k_steps) tc::umma_bf16(d, da(0, k), db(0, k), idesc1, (taken > 0 || k > 0) ? 1u : 0u);
                    } else {
                        // corrections first: column block 0 collects hi.mid and mid.hi (scale 2^8), block 1
                        // hi.lo, mid.mid and lo.hi (scale 2^16); then the leading products into block 0,
                        // whose scale the first of them takes off
#pragma unroll
                        for (int k = 0; k < BK / 16; ++k) {
                            if (k >= k_steps) break;
                            tc::umma_bf16(d, da(0, k), db(1, k), idesc2, k > 0 ? 1u : 0u);   // b_mid, b_lo
                            tc::umma_bf16(d, da(1, k), db(0, k), idesc2, 1u);                // b_hi, b_mid
                            tc::umma_bf16(d + BN, da(2, k), db(0, k), idesc1, 1u);
                        }
                        tc::umma_bf16_shift8(d, da(0, 0), db(0, 0), idesc1);
#pragma unroll
                        for (int k = 1; k < BK / 16; ++k)
                            if (k < k_steps) tc::umma_bf16(d, da(0, k), db(0, k), idesc1, 1u);
                    }
                    tc::umma_commit(tc::smem_u32(&empty_bar[stage]));
                    if (++stage == STAGES) {
                        stage = 0;
                        phase ^= 1;
                    }
                    if (++taken == kAccSteps<PL> || k0 + BK >= k_end) {
                        taken = 0;
                        tc::umma_commit(tc::smem_u32(&acc_full[acc]));
                        if (++acc == 2) {
                            acc = 0;
                            acc_phase ^= 1;
                        }
                    }
                }
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ epilogue
        const int e = warp - PRODUCERS / 32;
        const int quarter = warp % 4;
        const int col_base = (e / 4) * C::COLS;
        int acc = 0;
        uint32_t acc_phase = 0;
        bool ok = true;
        for (int w = work0; ok && w < num_work; w += gridDim.x) {
            const int tile = w % tiles, z = w / tiles;
            const int m0 = (tile % p.tiles_m) * BM, n0 = (tile / p.tiles_m) * BN;
            const int k_begin = z * p.k_split, k_end = min(p.K, k_begin + p.k_split);
            const int steps = (k_end - k_begin + kAccSteps<PL> * BK - 1) / (kAccSteps<PL> * BK);
            float sum[C::COLS];
#pragma unroll
            for (int j = 0; j < C::COLS; ++j) sum[j] = 0.f;
            for (int s = 0; s < steps; ++s) {
                if (!tc::mbar_wait(tc::smem_u32(&acc_full[acc]), acc_phase, abort_flag)) {
                    if (lane == 0) atomicExch(p.status, 184);
                    ok = false;
                    break;
                }
                tc::tc_fence_after();
                const uint32_t t = tmem + acc * C::ACC_COLS + col_base + ((uint32_t)(quarter * 32) << 16);
#pragma unroll
                for (int c = 0; c < C::COLS; c += 16) {
                    uint32_t r0[16], r1[16];
                    tc::tmem_ld_32x16(t + c, r0);
                    if (PL == 3) tc::tmem_ld_32x16(t + BN + c, r1);
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        float v = __uint_as_float(r0[j]);
                        if (PL == 3) v = fmaf(__uint_as_float(r1[j]), 0x1p-16f, v);
                        sum[c + j] += v;
                    }
                }
                tc::tc_fence_before();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(tc::smem_u32(&acc_empty[acc]));
                if (++acc == 2) {
                    acc = 0;
                    acc_phase ^= 1;
                }
            }
            if (!ok) break;
            const int row = m0 + quarter * 32 + lane;
            const int col0 = n0 + col_base;
            const bool in = row < p.M;
            // a sum that is not finite: the warp's block is left for redo_block
            bool redo_it = false;
            if (PL == 3) {
                float finite = 0.f;
#pragma unroll
                for (int j = 0; j < C::COLS; ++j) finite = fmaf(sum[j], 0.f, finite);
                redo_it = __any_sync(0xffffffffu, in && !(finite == 0.f));
                if (redo_it && lane == 0) {
                    const int i = (w - work0) / gridDim.x;
                    atomicOr(marks + i / 4, 1u << (i % 4 * 8 + e));
                    *redo = 1;
                }
            }
            if (redo_it) {
            } else if (ADDS && p.cluster) {
                // the stages have been read: this CTA's products are done
                float *q = sums + col_base * BM + quarter * 32 + lane;
#pragma unroll
                for (int j = 0; j < C::COLS; ++j) q[j * BM] = sum[j];
            } else if (in && p.splits > 1) {
                float *q = p.partial + ((int64_t)z * p.N + col0) * p.M + row;
#pragma unroll
                for (int j = 0; j < C::COLS; ++j, q += p.M)
                    if (col0 + j < p.N) *q = sum[j];
            } else if (in) {
                typename Epi::State st = E.begin(row, col0);
#pragma unroll
                for (int j = 0; j < C::COLS; ++j)
                    if (col0 + j < p.N) E.store(st, col0 + j, sum[j]);
            }
            __syncwarp();  // the next tensor-memory load is a warp-wide instruction
        }
    }

    tc::tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) {
        tc::tc_fence_after();
        if (*abort_flag) {   // let MMAs in flight finish before their tensor memory is given back
            const uint64_t t0 = tc::global_timer_ns();
            while (tc::global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
        }
        tc::tmem_dealloc(tmem, C::TMEM);
    }
    if (PL == 3 && *redo && !*abort_flag) {
        redo_marked<C, AOp, BOp, Epi>(A, B, E, p, marks, reinterpret_cast<float *>(smem) + warp * kRedoFloats, sums);
        __syncthreads();
    }
    if (ADDS && p.cluster) {
        // Every CTA adds a share of the columns over the slices, in slice order as reduce_splits_kernel does.
        tc::pair::cluster_sync();
        const int tile = work0 % tiles, rank = work0 / tiles;
        const int m0 = (tile % p.tiles_m) * BM, n0 = (tile / p.tiles_m) * BN, row = tid % BM;
        const int share = (min(BN, p.N - n0) + p.splits - 1) / p.splits;
        const int first = rank * share, last = min(min(BN, p.N - n0), first + share);
        if (tid < C::THREADS / BM * BM && m0 + row < p.M)
            for (int col = first + tid / BM; col < last; col += C::THREADS / BM) {
                const uint32_t at = tc::smem_u32(sums + col * BM + row);
                float v[8], sum = 0.f;
#pragma unroll
                for (int z = 0; z < 8; ++z)
                    v[z] = z < p.splits ? __uint_as_float(tc::pair::ld_shared_cluster(tc::pair::map_to_cta(at, z))) : 0.f;
#pragma unroll
                for (int z = 0; z < 8; ++z)
                    if (z < p.splits) sum += v[z];
                typename Epi::State st = E.begin(m0 + row, n0 + col);
                E.store(st, n0 + col, sum);
            }
        tc::pair::cluster_sync();   // the others have read this CTA's sums
        return;
    }
    if (ADDS && p.arrivals != nullptr) {
        // every CTA has had one slice of one tile (grid = tiles * splits)
        const int tile = blockIdx.x % tiles;
        int *last = table_a;
        if (tid == 0) {
            __threadfence();   // the slice's sums, stored by the epilogue warps before the barrier
            const int n = atomicAdd(p.arrivals + tile, 1);
            *last = n == p.splits - 1;
            if (n == p.splits - 1) {
                p.arrivals[tile] = 0;   // for the next launch
                __threadfence();        // the other slices, for the whole CTA after the barrier
            }
        }
        __syncthreads();
        if (*last) {
            reduce_tile<C::THREADS>(p, E, (tile % p.tiles_m) * BM, (tile / p.tiles_m) * BN, BN, tid);
        }
    }
}

// out = epilogue(sum over slices in slice order).
template <class Epi>
__global__ void __launch_bounds__(256)
    reduce_splits_kernel(const float *partial, int splits, int M, int N, FastDiv div_m, Epi E) {
    dependency_wait();
    const int64_t plane = (int64_t)M * N;
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= plane) return;
    const float *q = partial + i;
    float s = 0.f;
    int z = 0;
    for (; z + 4 <= splits; z += 4) {
        const float a = q[(int64_t)z * plane], b = q[(int64_t)(z + 1) * plane],
                    c = q[(int64_t)(z + 2) * plane], d = q[(int64_t)(z + 3) * plane];
        s = s + a;
        s = s + b;
        s = s + c;
        s = s + d;
    }
    for (; z < splits; ++z) s += q[(int64_t)z * plane];
    const int col = (int)(i / M), row = (int)(i - (int64_t)col * M);
    typename Epi::State st = E.begin(row, col);
    E.store(st, col, s);
}

// --------------------------------------------------------------------- host
constexpr int kMostCluster = 8;   // what every GPU takes

// One more than the clusters of `size` CTAs that run at a time.
template <class... P>
int cluster_room(void (*kernel)(P...), int threads, int smem, int size, int *room) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)size);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)size;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    AG_CUDA_TRY(cudaOccupancyMaxActiveClusters(&n, kernel, &cfg));
    *room = n + 1;
    return AG_OK;
}

// launch_dependent with clusters of `size` CTAs.
template <class... P, class... A>
int launch_clusters(ag_device *dev, void (*kernel)(P...), int grid, int threads, int smem, int size, const A &...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = dev->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)size;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    AG_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, args...));
    AG_CHECK_LAUNCH();
    return AG_OK;
}

template <class T, int BN, class AOp, class BOp, class Epi>
int launch(ag_device *dev, const AOp &A, const BOp &B, const Epi &E, Params p) {
    using C = Cfg<T, BN>;
    p.tiles_m = (int)ceil_div(p.M, BM);
    p.tiles_n = (int)ceil_div(p.N, BN);
    const int64_t tiles = (int64_t)p.tiles_m * p.tiles_n;
    // Slices of k fill the SMs that whole tiles leave idle; at least two k steps each.
    const int steps = (int)ceil_div(p.K, BK);
    int splits = 1;
    if (tiles * 2 <= dev->sm_count && steps >= 4) {
        splits = (int)(dev->sm_count / tiles);
        if (splits > steps / 2) splits = steps / 2;
    }
    const int per = (int)ceil_div(steps, splits);
    p.k_split = per * BK;
    p.splits = (int)ceil_div(steps, per);
    p.status = dev->status_dev;
    p.partial = nullptr;
    p.arrivals = nullptr;
    auto kernel = gemm_tcx_kernel<T, BN, AOp, BOp, Epi>;
    static SmemAllowed allowed;
    AG_TRY(allow_smem<C::SMEM>(dev, kernel, allowed));
    // Convolutions of up to eight short slices: the CTAs of a tile are a cluster and add them through its shared memory, if
    // all clusters find room at once (a GPC holds two of eight CTAs).  Against the tile's last CTA, us, images x channels x
    // side -> filters: 9 x 16 x 10 -> 64 5x5 f32 forward 14.5 and 18.0, weight gradient 11.6 and 15.0, 24 x 64 x 13 -> 128 5x5
    // bf16 forward 18.8 and 21.1, weight gradient 23.6 and 28.0.  Long slices are slower so (6 x 64 x 43 -> 128 5x5 f32 weight
    // gradient, 35 steps each, 72 and 60), and so are products in a row, whose second launch overlaps the next one (464 x 256
    // x 112 bf16 8.6 and 7.2).
    p.cluster = 0;
    if (kAddsSlices<AOp, Epi> && p.splits > 1 && p.splits <= kMostCluster && per <= 16) {
        static int room_on[64][kMostCluster + 1] = {};   // clusters + 1
        int &room = room_on[dev->ordinal & 63][p.splits];
        if (room == 0) AG_TRY(cluster_room(kernel, C::THREADS, C::SMEM, p.splits, &room));
        p.cluster = tiles < room;
    }
    if (p.splits > 1 && !p.cluster) {
        void *ws = nullptr;
        AG_TRY(engine_scratch(dev, sizeof(float) * (size_t)p.splits * p.M * p.N, &ws));
        p.partial = (float *)ws;
        // Convolutions of up to eight slices: the tile's last CTA adds them.  That takes 3 us more on the device
        // than the separate kernel (512^3 f32 13.8 us against 9.9), whose launch costs 4 us on the host; a pass
        // over a small convolution's edges is ten launches that the device waits for, a product by itself
        // is not.  More slices would be a chain of round trips (37 slices: 24 us against 13).
        if (kAddsSlices<AOp, Epi> && p.splits <= 8 && tiles <= kTileCounters &&
            (int64_t)p.splits * (p.M < BM ? p.M : BM) * (p.N < BN ? p.N : BN) <= 65536)
            p.arrivals = dev->tile_counters;
    }
    if (p.cluster) {
        p.work0 = 0;
        p.work1 = (int)(tiles * p.splits);
        return launch_clusters(dev, kernel, p.work1, C::THREADS, C::SMEM, p.splits, A, B, E, p);
    }
    const int64_t work = tiles * p.splits, most = (int64_t)kMarks * dev->sm_count;
    for (int64_t w = 0; w < work; w += most) {   // one launch, but for f32 outputs of 2.4e9 values and more
        p.work0 = (int)w;
        p.work1 = (int)(C::PL == 1 || work - w < most ? work : w + most);
        const int grid = (int)(work - w < dev->sm_count ? work - w : dev->sm_count);
        AG_TRY(launch_dependent(dev, kernel, dim3((unsigned)grid), C::THREADS, C::SMEM, A, B, E, p));
        if (C::PL == 1) break;
    }
    if (p.splits > 1 && p.arrivals == nullptr) {
        AG_TRY(launch_dependent(dev, reduce_splits_kernel<Epi>, dim3((unsigned)ceil_div((int64_t)p.M * p.N, 256)), 256,
                                0,
                                (const float *)p.partial, p.splits, p.M, p.N, FastDiv((uint32_t)p.M), E));
    }
    return AG_OK;
}

// Tile width: the narrowest that holds all columns, else 128 columns when the tiles fill the GPU.
// MN-major B tiles are whole 64-row atoms.
template <class T, class AOp, class BOp, class Epi>
int gemm(ag_device *dev, int M, int N, int K, const AOp &A, const BOp &B, const Epi &E) {
    Params p = {};
    p.M = M;
    p.N = N;
    p.K = K;
    if constexpr (!mn_major(BOp::kWalk)) {
        if (N <= 32) return launch<T, 32>(dev, A, B, E, p);
    }
    const int64_t tiles = ceil_div(M, BM) * ceil_div(N, 128);
    if (N <= 64 || tiles * 2 <= dev->sm_count) return launch<T, 64>(dev, A, B, E, p);
    return launch<T, 128>(dev, A, B, E, p);
}

}  // namespace tcx
}  // namespace ag
