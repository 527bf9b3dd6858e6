// What the convolutions on matrices of pixel rows share (conv_halo_f32.cu, conv_halo_wgrad_f32.cu): operands in shared memory and the
// warps that write them.
#pragma once

#include "conv_halo_f32.cuh"
#include "gemm_tcx.cuh"

namespace ag {
namespace halo32 {

// A K- or MN-major operand of rows of RB bytes (32, 64, 128), swizzled by as much.
template <int RB>
__device__ __forceinline__ uint64_t operand(uint32_t addr) {
    constexpr uint64_t layout = RB == 32 ? 6ull : RB == 64 ? 4ull : 2ull;
    uint64_t d = (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((8 * RB) >> 4) << 32;
    d |= 1ull << 46;
    return d | layout << 61;
}

// Eight values as one 16-byte piece of each plane, `offset` bytes behind an address that is a multiple of 1024.
template <int RB>
__device__ __forceinline__ void store_pieces(const float *x, uint8_t *base, uint32_t offset, uint32_t plane_bytes) {
    uint32_t h[4], m[4], l[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        uint32_t hb[2], mb[2], lb[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) ::ag::tcx::split3(x[2 * e + u], hb[u], mb[u], lb[u]);
        h[e] = ::ag::tcx::upper_halves(hb[0], hb[1]);
        m[e] = ::ag::tcx::upper_halves(mb[0], mb[1]);
        l[e] = ::ag::tcx::upper_halves(lb[0], lb[1]);
    }
    const auto put = [&](const uint32_t (&v)[4]) {
        *reinterpret_cast<uint4 *>(base + (offset ^ (offset >> 3 & (RB - 16)))) = make_uint4(v[0], v[1], v[2], v[3]);
        offset += plane_bytes;
    };
    put(h);
    put(m);
    put(l);
}

// A tensor [image][channels][h][wd] as a matrix of rows, one per pixel of a frame of hp x wp that is zero around the image, which
// starts at (pad_h, pad_w).
struct Source {
    const float *src;
    int rows, channels, h, wd, pad_h, pad_w;
    FastDiv div_image, div_wp;   // by hp * wp, by wp
};
inline Source source(const float *src, int64_t channels, int64_t h, int64_t wd, int pad_h, int pad_w, int64_t hp, int64_t wp,
                     int64_t rows) {
    return Source{src, (int)rows, (int)channels, (int)h, (int)wd, pad_h, pad_w, FastDiv((uint32_t)(hp * wp)), FastDiv((uint32_t)wp)};
}

// 16 channels of row q; a warp reads neighbouring pixels.
__device__ __forceinline__ void load_row(const Source &s, int q, int c0, float (&v)[16]) {
    uint32_t image, at, py, px;
    s.div_image.divmod((uint32_t)q, image, at);
    s.div_wp.divmod(at, py, px);
    const int y = (int)py - s.pad_h, x = (int)px - s.pad_w;
    const bool in = (uint32_t)q < (uint32_t)s.rows && y >= 0 && y < s.h && x >= 0 && x < s.wd;
    const int64_t hw = (int64_t)s.h * s.wd;
    const float *p = s.src + (in ? ((int64_t)image * s.channels + c0) * hw + y * s.wd + x : 0);
#pragma unroll
    for (int e = 0; e < 16; ++e, p += hw) v[e] = load_or_zero(p, in && c0 + e < s.channels);
}

// The warps that fill boxes: items of 32 rows x 16 channels, dealt to them over all tiles of the CTA, so that none waits for
// another at the end of a tile.  An item's loads are issued before the one ahead of it is split.
constexpr int kFillers = 7;
struct Item {
    int at, tile, stage;
    uint32_t phase;
    __device__ __forceinline__ void forward(int by, int items, int stages) {
        for (at += by; at >= items; at -= items) {
            tile += gridDim.x;
            if (++stage == stages) {
                stage = 0;
                phase ^= 1;
            }
        }
    }
};

}  // namespace halo32
}  // namespace ag
