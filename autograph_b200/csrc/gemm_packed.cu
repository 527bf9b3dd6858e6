// Large products whose operands TMA cannot read as they are: f32 matrices, and bf16 matrices
// whose rows are not 16-byte aligned.  One pass copies both operands into bf16 planes with
// aligned rows (f32: the three planes hi, mid, lo of gemm_tcx.cuh; bf16: one), then pairs of
// CTAs multiply 256 x 256 tiles (tcgen05 cta_group::2) with the operands staged by TMA.
//
// Roles per CTA (320 threads): warp 0 = TMA producer of the CTA's own halves, warp 1 = MMA
// issuer (leader) and tensor-memory allocation, warps 2..9 = epilogue, each 32 rows x 128
// columns.  An f32 product reads the accumulator out after every 64 k and adds the 64-k sums
// in registers, a bf16 product after every 1024 (the arithmetic, and why, is described in gemm_tcx.cuh; so is
// what happens to sums that are not finite).
//
// The tile's rows run along the contiguous index of C (a row-major C is computed as
// C^T = B^T . A^T), so a warp's store is 32 consecutive elements and needs no alignment.
//
// What bounds it: the f32 form issues 24 MMAs of 256 x 256 x 16 per 64 k from two 96 KiB stages,
// the tensor pipe at the clock the power limit leaves; the copy pass moves (4 + 6) bytes per
// operand element.  f32 4096^3: 593 us (232 TFLOP/s of f32 multiply-adds, 1.39 PFLOP/s of bf16)
// in a burst, 690 us under the power cap, against 2650 - 2900 us on the FP32 pipe; bf16 4095 x 4093 x 4097: 152 us.
#include <cuda.h>

#include "gemm_packed.cuh"
#include "gemm_tcx.cuh"
#include "pair_ptx.cuh"

namespace ag {
namespace packed {

using namespace tc;
using namespace tc::pair;
using tcx::Planes;

constexpr int TILE = 256;      // per pair, both ways
constexpr int BK = 64;
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 64 + EPI_WARPS * 32;
constexpr int HALF_BYTES = 128 * BK * 2;   // 128 rows of one plane of a stage

template <int PL>
struct Cfg {
    static constexpr int STAGE = 2 * PL * HALF_BYTES;      // A half + B half of this CTA
    static constexpr int STAGES = PL == 3 ? 2 : 6;
    static constexpr int SMEM = STAGES * STAGE + 1024 + 256 + (PL == 3 ? tcx::kMarks : 0);
    static_assert(THREADS / 32 * tcx::kRedoFloats * 4 <= STAGES * STAGE, "the stages hold redo_block's buffers");
};

template <class T>
struct Params {
    int M, N, K;              // tile rows (C's contiguous index), columns, depth
    int64_t ldc;              // stride of C between columns
    float alpha, beta;
    T *C;
    // Items [0, t_full) are whole tiles, the tiles after them cut in tail_split pieces along n.
    int t_full, tail_split, num_work, group_m;
    int work0, work1;         // this launch's share of them
    int splits, kb_split;     // slices of k (whole tiles only) and 64-k steps per slice
    float *partial;           // splits > 1: [splits][N][M] f32 sums
    const T *bias;            // per row, with relu the Dense layer's epilogue
    int relu;
    // the operands as the caller gave them (redo_block)
    const T *p, *q;
    int64_t p_row, p_k, q_row, q_k;
    int *status;
};

struct Work {
    int m_blk, n_blk, n_off, n_width;
    int z, kb0, kb1;   // slice of k and its 64-k steps
};

template <class T>
__device__ __forceinline__ Work decode(int w, const Params<T> &p) {
    const int num_m = (p.M + TILE - 1) / TILE, num_n = (p.N + TILE - 1) / TILE;
    const int num_kb = (p.K + BK - 1) / BK;
    Work k;
    int tile = w;
    k.n_off = 0;
    k.n_width = TILE;
    k.z = 0;
    if (p.splits > 1) {
        k.z = w / (num_m * num_n);
        tile = w - k.z * (num_m * num_n);
    } else if (w >= p.t_full) {
        const int j = w - p.t_full;
        tile = p.t_full + j / p.tail_split;
        k.n_width = TILE / p.tail_split;
        k.n_off = (j % p.tail_split) * k.n_width;
    }
    const int group_size = p.group_m * num_n;
    const int g = tile / group_size, first_m = g * p.group_m;
    const int gm = min(num_m - first_m, p.group_m);
    const int r = tile - g * group_size;
    k.m_blk = first_m + r % gm;
    k.n_blk = r / gm;
    k.kb0 = k.z * p.kb_split;
    k.kb1 = min(num_kb, k.kb0 + p.kb_split);
    return k;
}

template <class T>
__device__ __forceinline__ void store_out(const Params<T> &p, int row, int col, float acc) {
    T *q = p.C + row + (int64_t)col * p.ldc;
    float v = p.alpha * acc;
    if (p.beta != 0.f) v += p.beta * to_f32(*q);
    if (p.bias != nullptr) v = __fadd_rn(to_f32(from_f32<T>(v)), to_f32(p.bias[row]));
    T o = from_f32<T>(v);
    if (p.relu && !(to_f32(o) >= 0.f)) o = from_f32<T>(0.f);
    *q = o;
}

// An operand as redo_block reads it.
template <class T>
struct Given {
    const T *p;
    int64_t s_row, s_k;
    __device__ __forceinline__ float at(int row, int k) const { return to_f32(p[row * s_row + k * s_k]); }
};

// The blocks that this CTA's epilogue warps left out (gemm_tcx.cuh), dealt to its warps.
template <bool A_MN, bool B_MN, class T>
__device__ __noinline__ void redo_marked(const Params<T> &p, const unsigned *marks, float *buf, int rank) {
    constexpr int WARPS = THREADS / 32;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const Given<T> A{p.p, p.p_row, p.p_k}, B{p.q, p.q_row, p.q_k};
    int turn = 0;
    for (int w = p.work0 + (int)(blockIdx.x >> 1), i = 0; w < p.work1; w += gridDim.x >> 1, ++i) {
        const unsigned mark = marks[i / 4] >> (i % 4 * 8) & 255u;
        if (mark == 0) continue;
        const Work wk = decode(w, p);
        const int width = wk.n_width / 2;
        for (int block = 0; block < EPI_WARPS * width / 32; ++block) {
            const int e = block % EPI_WARPS;   // warp 2 + e
            const int row0 = wk.m_blk * TILE + rank * 128 + (2 + e) % 4 * 32;
            const int col0 = wk.n_blk * TILE + wk.n_off + e / 4 * width + block / EPI_WARPS * 32;
            if ((mark >> e & 1u) == 0 || row0 >= p.M || col0 >= p.N || turn++ % WARPS != warp) continue;
            float acc[4][8];
            tcx::redo_block<A_MN, B_MN>(A, B, row0, p.M, col0, p.N, wk.kb0 * BK, min(p.K, wk.kb1 * BK), buf, acc);
            for (int r = 0; r < 4; ++r) {
                const int row = row0 + lane / 4 * 4 + r;
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const int col = col0 + lane % 4 * 8 + c;
                    if (row >= p.M || col >= p.N) break;
                    const float v = r == 0 ? acc[0][c] : r == 1 ? acc[1][c] : r == 2 ? acc[2][c] : acc[3][c];
                    if (p.splits > 1)
                        p.partial[((int64_t)wk.z * p.N + col) * p.M + row] = v;
                    else
                        store_out(p, row, col, v);
                }
            }
        }
    }
}

// Shared-memory layout of one operand half in a stage (rows = 128, or 64 for a tail piece of B):
//   K-major:  [plane][row][64 k], plane stride rows * 128 bytes
//   MN-major: [64-row atom][plane][64 k][64 rows], plane stride 8 KiB, atom stride PL * 8 KiB
template <int PL, bool A_MN, bool B_MN, class T>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
    gemm_packed_kernel(const __grid_constant__ CUtensorMap tmap_a,
                       const __grid_constant__ CUtensorMap tmap_b,
                       const __grid_constant__ CUtensorMap tmap_b_tail,
                       const __grid_constant__ Params<T> p) {
    constexpr int STAGES = Cfg<PL>::STAGES, STAGE = Cfg<PL>::STAGE;
    constexpr int ATOM = 64 * BK * 2;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                                ~uintptr_t(1023));
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + STAGES * STAGE);
    uint64_t *full_bar = bars;                         // leader only
    uint64_t *empty_bar = bars + STAGES;               // per CTA
    uint64_t *acc_full = bars + 2 * STAGES;            // [2] per CTA
    uint64_t *acc_empty = bars + 2 * STAGES + 2;       // [2] leader only
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * STAGES + 4);  // [2]
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 2);
    volatile int *redo = reinterpret_cast<volatile int *>(tmem_slot + 3);                // any mark
    unsigned *marks = tmem_slot + 4;   // bit e of byte i: epilogue warp e left its block of the pair's i-th item out

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const uint32_t rank = cluster_ctarank();
    const bool leader = rank == 0;
    const int work0 = p.work0 + (int)(blockIdx.x >> 1), num_pairs = gridDim.x >> 1;

    if (threadIdx.x == 0) {
        prefetch_tmap(&tmap_a);
        prefetch_tmap(&tmap_b);
        prefetch_tmap(&tmap_b_tail);
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(&full_bar[s]), 1);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(smem_u32(&acc_full[s]), 1);
            mbar_init(smem_u32(&acc_empty[s]), 2 * EPI_WARPS);
        }
        tmem_slot[0] = tmem_slot[1] = 0xffffffffu;
        *abort_flag = 0;
        *redo = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (PL == 3 && threadIdx.x < tcx::kMarks / 4) marks[threadIdx.x] = 0;
    // Both CTAs of the pair are here before either allocates: an allocation of a pair needs the other one.  With a
    // barrier of the CTA alone, and a load of a microsecond before it, one in some hundred launches of 74 pairs left a
    // CTA without an address (0xffffffe0).
    cluster_sync();
    // Tensor memory in two 256-column steps; after the first the pair compares addresses (as in
    // gemm_tc2.cu) and stops before anything could block on them if they differ.
    if (warp == 1) tmem_alloc2(smem_u32(&tmem_slot[0]), 256);
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    tc_fence_after();
    const bool ok_alloc =
        tmem_slot[0] == ld_shared_cluster(map_to_cta(smem_u32(&tmem_slot[0]), rank ^ 1u));
    cluster_sync();
    if (!ok_alloc) {
        if (threadIdx.x == 0) atomicExch(p.status, 190);
        if (warp == 1) {
            tmem_dealloc2(tmem_slot[0], 256);
            tmem_relinquish2();
        }
        return;
    }
    if (warp == 1) {
        tmem_alloc2(smem_u32(&tmem_slot[1]), 256);
        tmem_relinquish2();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_acc[2] = {tmem_slot[0], tmem_slot[1]};
    // The copy pass, this and the sum of slices each set up while their predecessor ends (us plain and so: f32 1024^3 34.9
    // and 27.2, 2048^3 92 and 86, 256 x 25088 x 512 78 and 71; bf16 4313 x 791 x 1252 43.1 and 37.7).
    let_dependents_launch();
    dependency_wait();

    if (warp == 0) {
        if (elect_one()) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int w = work0; ok && w < p.work1; w += num_pairs) {
                const Work wk = decode(w, p);
                const int half_n = wk.n_width / 2;
                const int m0 = wk.m_blk * TILE + (int)rank * 128;
                const int n0 = wk.n_blk * TILE + wk.n_off + (int)rank * half_n;
                const uint32_t tx = (uint32_t)(2 * PL * (HALF_BYTES + half_n * BK * 2));
                for (int kb = wk.kb0; kb < wk.kb1; ++kb) {
                    if (!mbar_wait(smem_u32(&empty_bar[stage]), phase ^ 1, abort_flag)) {
                        atomicExch(p.status, 191);
                        ok = false;
                        break;
                    }
                    const uint32_t local_full = smem_u32(&full_bar[stage]);
                    if (leader) mbar_arrive_expect_tx(local_full, tx);
                    const uint32_t bar = map_to_cta(local_full, 0);
                    const uint32_t a_dst = smem_u32(smem + stage * STAGE);
                    const uint32_t b_dst = a_dst + PL * HALF_BYTES;
                    if (A_MN) {
#pragma unroll
                        for (int i = 0; i < 2; ++i)
                            tma_load_3d_pair(a_dst + i * PL * ATOM, &tmap_a, bar, m0 + i * 64, kb * BK, 0);
                    } else {
                        tma_load_3d_pair(a_dst, &tmap_a, bar, kb * BK, m0, 0);
                    }
                    if (B_MN) {
                        for (int i = 0; i < half_n / 64; ++i)
                            tma_load_3d_pair(b_dst + i * PL * ATOM, &tmap_b, bar, n0 + i * 64, kb * BK, 0);
                    } else {
                        tma_load_3d_pair(b_dst, half_n == 128 ? &tmap_b : &tmap_b_tail, bar, kb * BK, n0, 0);
                    }
                    if (++stage == STAGES) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (leader && elect_one()) {
            constexpr uint32_t lbo = PL * ATOM;
            const uint32_t a_plane = A_MN ? ATOM : HALF_BYTES;
            const uint32_t a_step = A_MN ? 16 * 128 : 32, b_step = B_MN ? 16 * 128 : 32;
            int stage = 0, acc = 0;
            uint32_t phase = 0, acc_phase = 0;
            bool ok = true;
            for (int w = work0; ok && w < p.work1; w += num_pairs) {
                const Work wk = decode(w, p);
                const uint32_t idesc = make_idesc(A_MN, B_MN, TILE, wk.n_width);
                const uint32_t b_plane = B_MN ? ATOM : wk.n_width / 2 * BK * 2;
                int taken = 0;   // steps in this accumulator
                for (int kb = wk.kb0; kb < wk.kb1; ++kb) {
                    if (taken == 0) {
                        if (!mbar_wait(smem_u32(&acc_empty[acc]), acc_phase ^ 1, abort_flag)) {
                            atomicExch(p.status, 192);
                            ok = false;
                            break;
                        }
                    }
                    if (!mbar_wait(smem_u32(&full_bar[stage]), phase, abort_flag)) {
                        atomicExch(p.status, 193);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t d = tmem_acc[acc];
                    const uint32_t a_base = smem_u32(smem + stage * STAGE);
                    const uint32_t b_base = a_base + PL * HALF_BYTES;
                    auto desc_a = [&](int plane, int k) {
                        return make_smem_desc(a_base + plane * a_plane + k * a_step, A_MN ? lbo : 0, 1024);
                    };
                    auto desc_b = [&](int plane, int k) {
                        return make_smem_desc(b_base + plane * b_plane + k * b_step, B_MN ? lbo : 0, 1024);
                    };
                    auto mma = [&](int pa, int pb, int k, bool add) {
                        umma2_bf16(d, desc_a(pa, k), desc_b(pb, k), idesc, add ? 1u : 0u);
                    };
                    if (PL == 1) {
#pragma unroll
                        for (int k = 0; k < BK / 16; ++k) mma(0, 0, k, taken > 0 || k > 0);
                    } else {
                        // the smallest partial products first, the leading ones last; the first of each
                        // size takes 2^8 off the scale of what was added before
#pragma unroll
                        for (int k = 0; k < BK / 16; ++k) {
                            mma(0, 2, k, k > 0);
                            mma(2, 0, k, true);
                            mma(1, 1, k, true);
                        }
                        umma2_bf16_shift8(d, desc_a(0, 0), desc_b(1, 0), idesc);
                        mma(1, 0, 0, true);
#pragma unroll
                        for (int k = 1; k < BK / 16; ++k) {
                            mma(0, 1, k, true);
                            mma(1, 0, k, true);
                        }
                        umma2_bf16_shift8(d, desc_a(0, 0), desc_b(0, 0), idesc);
#pragma unroll
                        for (int k = 1; k < BK / 16; ++k) mma(0, 0, k, true);
                    }
                    umma2_commit_multicast(smem_u32(&empty_bar[stage]), 3);
                    if (++stage == STAGES) {
                        stage = 0;
                        phase ^= 1;
                    }
                    if (++taken == tcx::kAccSteps<PL> || kb + 1 == wk.kb1) {
                        taken = 0;
                        umma2_commit_multicast(smem_u32(&acc_full[acc]), 3);
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
        const int quarter = warp % 4, half = (warp - 2) / 4;
        int acc = 0;
        uint32_t acc_phase = 0;
        bool ok = true;
        for (int w = work0; ok && w < p.work1; w += num_pairs) {
            const Work wk = decode(w, p);
            const int width = wk.n_width / 2;   // columns of this warp: 128, or 64 of a tail piece
            float sum[128];
            const int steps = (wk.kb1 - wk.kb0 + tcx::kAccSteps<PL> - 1) / tcx::kAccSteps<PL>;
            for (int s = 0; s < steps; ++s) {
                if (!mbar_wait(smem_u32(&acc_full[acc]), acc_phase, abort_flag)) {
                    if (lane == 0) atomicExch(p.status, 194);
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t t = tmem_acc[acc] + half * width + ((uint32_t)(quarter * 32) << 16);
#pragma unroll
                for (int c = 0; c < 128; c += 32) {
                    if (c < width) {
                        uint32_t r[32];
                        tmem_ld_32x32(t + c, r);
                        tmem_ld_wait();
                        if (s == 0) {
#pragma unroll
                            for (int j = 0; j < 32; ++j) sum[c + j] = __uint_as_float(r[j]);
                        } else {
#pragma unroll
                            for (int j = 0; j < 32; ++j) sum[c + j] += __uint_as_float(r[j]);
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&acc_empty[acc]), 0));
                if (++acc == 2) {
                    acc = 0;
                    acc_phase ^= 1;
                }
            }
            if (!ok) break;
            const int row = wk.m_blk * TILE + (int)rank * 128 + quarter * 32 + lane;
            const int col0 = wk.n_blk * TILE + wk.n_off + half * width;
            bool redo_it = false;
            if (PL == 3) {
                float finite = 0.f;
#pragma unroll
                for (int c = 0; c < 128; c += 32)
                    if (c < width)
#pragma unroll
                        for (int j = 0; j < 32; ++j) finite = fmaf(sum[c + j], 0.f, finite);
                redo_it = __any_sync(0xffffffffu, row < p.M && !(finite == 0.f));
                if (redo_it && lane == 0) {
                    const int i = (w - work0) / num_pairs;
                    atomicOr(marks + i / 4, 1u << (i % 4 * 8 + warp - 2));
                    *redo = 1;
                }
            }
            float *part = p.splits > 1 ? p.partial + (int64_t)wk.z * p.M * p.N + row : nullptr;
            if (redo_it) {
            } else if (row < p.M) {
#pragma unroll
                for (int c = 0; c < 128; c += 32)
                    if (c < width) {
                        if (part != nullptr) {
#pragma unroll
                            for (int j = 0; j < 32; ++j)
                                if (col0 + c + j < p.N) part[(int64_t)(col0 + c + j) * p.M] = sum[c + j];
                        } else {
#pragma unroll
                            for (int j = 0; j < 32; ++j)
                                if (col0 + c + j < p.N) store_out(p, row, col0 + c + j, sum[c + j]);
                        }
                    }
            }
            __syncwarp();
        }
    }

    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    cluster_sync();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc2(tmem_acc[0], 256);
        tmem_dealloc2(tmem_acc[1], 256);
    }
    // the pair's MMAs, which read both CTAs' stages, are done
    if (PL == 3 && *redo && !*abort_flag)
        redo_marked<A_MN, B_MN>(p, marks, reinterpret_cast<float *>(smem) + warp * tcx::kRedoFloats, (int)rank);
}

// C from the f32 sums of the slices, added in slice order.
template <class T>
__global__ void __launch_bounds__(256) reduce_kernel(const __grid_constant__ Params<T> p, FastDiv div_m) {
    let_dependents_launch();
    dependency_wait();
    const int64_t plane = (int64_t)p.M * p.N;
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < plane; i += (int64_t)gridDim.x * 256) {
        float s = 0.f;
        for (int z = 0; z < p.splits; ++z) s += p.partial[(int64_t)z * plane + i];
        uint32_t col, row;
        div_m.divmod((uint32_t)i, col, row);
        store_out(p, (int)row, (int)col, s);
    }
}

// ---------------------------------------------------------------- copy pass
// One operand: outer x inner elements, inner contiguous, rows `stride` apart; planes of
// outer x pitch bf16 (pitch a multiple of 8; the tail of a row is zero).
template <class T>
struct PackJob {
    const T *src;
    int64_t stride, plane;
    __nv_bfloat16 *dst;
    int inner, outer, pitch;
    FastDiv div_words;
};

// blockIdx.y picks the operand, a thread moves four pairs of neighbouring elements: 4-byte stores
// that a warp makes 128 bytes of, and loads that need no alignment.  DRAM bound.
template <class T>
__global__ void __launch_bounds__(256) pack_kernel(const PackJob<T> j0, const PackJob<T> j1) {
    let_dependents_launch(kAlwaysEarly);
    dependency_wait();
    const PackJob<T> &j = blockIdx.y == 0 ? j0 : j1;
    const uint32_t words = (uint32_t)j.pitch / 2;
    const uint32_t total = words * (uint32_t)j.outer;
    for (uint32_t base = blockIdx.x * 1024u; base < total; base += gridDim.x * 1024u) {
        T x[4][2];
        uint32_t at[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            at[u] = base + u * 256 + threadIdx.x;
            uint32_t row, w;
            j.div_words.divmod(at[u], row, w);
            const T *src = j.src + (int64_t)row * j.stride;
            const int i = 2 * (int)w;
            x[u][0] = at[u] < total && i < j.inner ? src[i] : from_f32<T>(0.f);
            x[u][1] = at[u] < total && i + 1 < j.inner ? src[i + 1] : from_f32<T>(0.f);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (at[u] >= total) break;
            uint32_t *dst = reinterpret_cast<uint32_t *>(j.dst) + at[u];
            if constexpr (sizeof(T) == 4) {
                uint32_t h[2], m[2], l[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) tcx::split3(x[u][i], h[i], m[i], l[i]);
                dst[0] = tcx::upper_halves(h[0], h[1]);
                dst[j.plane / 2] = tcx::upper_halves(m[0], m[1]);
                dst[j.plane] = tcx::upper_halves(l[0], l[1]);
            } else {
                *dst = (uint32_t)__bfloat16_as_ushort(x[u][0]) |
                       ((uint32_t)__bfloat16_as_ushort(x[u][1]) << 16);
            }
        }
    }
}

// ---------------------------------------------------------------------- host
template <int PL, bool A_MN, bool B_MN, class T>
static int launch(ag_device *dev, const CUtensorMap &ta, const CUtensorMap &tb, const CUtensorMap &tt,
                  Params<T> p) {
    auto kernel = gemm_packed_kernel<PL, A_MN, B_MN, T>;
    static SmemAllowed allowed;
    AG_TRY(allow_smem<Cfg<PL>::SMEM>(dev, kernel, allowed));
    const int most = tcx::kMarks * (dev->sm_count / 2);   // one launch for up to 5e9 outputs
    for (p.work0 = 0; p.work0 < p.num_work; p.work0 = p.work1) {
        const int left = p.num_work - p.work0, n = left < most ? left : most;
        p.work1 = p.work0 + n;
        const int pairs = n < dev->sm_count / 2 ? n : dev->sm_count / 2;
        AG_TRY(launch_dependent(dev, kernel, dim3(2 * pairs), THREADS, Cfg<PL>::SMEM, ta, tb, tt, p));
    }
    return AG_OK;
}

// Map of a packed operand: {inner, outer, planes}; MN-major boxes of 64 x 64, K-major of 64 x rows.
static int packed_map(CUtensorMap *map, const __nv_bfloat16 *base, int inner, int outer, int pitch,
                      int planes, int box_outer) {
    const uint64_t dims[3] = {(uint64_t)inner, (uint64_t)outer, (uint64_t)planes};
    const uint64_t strides[2] = {(uint64_t)pitch, (uint64_t)pitch * (uint64_t)outer};
    const uint32_t box[3] = {64, (uint32_t)box_outer, (uint32_t)planes};
    return make_tmap_bf16(map, base, 3, dims, strides, box);
}

// One operand's copy; returns the bytes of its planes.
template <class T>
static int64_t plan(PackJob<T> *j, const T *src, int rows, int k, int64_t s_row, int64_t s_k) {
    const bool mn = s_k != 1;
    j->src = src;
    j->inner = mn ? rows : k;
    j->outer = mn ? k : rows;
    j->stride = mn ? s_k : s_row;
    j->pitch = (j->inner + 7) / 8 * 8;
    j->plane = (int64_t)j->pitch * j->outer;
    j->div_words = FastDiv((uint32_t)(j->pitch / 2));
    return (j->plane * Planes<T>::N * 2 + 1023) / 1024 * 1024;
}

// Planes of one launch.  Larger products are cut into blocks of rows and columns, whose operands are
// copied in turn: 24,576^3 f32 (7.2 GB of planes) runs in two blocks at the rate of 16,384^3 in one (129 ms, 34 ms).
constexpr int64_t kMostPlanes = 4ll << 30;

template <class T>
static int64_t planes(int M, int N, int K, int64_t p_k, int64_t q_k) {
    PackJob<T> j;
    return plan<T>(&j, nullptr, M, K, 1, p_k) + plan<T>(&j, nullptr, N, K, 1, q_k);
}

template <class T>
bool reserve(ag_device *dev, int M, int N, int K, int64_t p_k, int64_t q_k) {
    const int64_t all = planes<T>(M, N, K, p_k, q_k);
    // the smallest blocks there are
    if (planes<T>(M < 2 * TILE ? M : 2 * TILE - 1, N < 2 * TILE ? N : 2 * TILE - 1, K, p_k, q_k) > kMostPlanes) return false;
    // and at most one tile per pair of f32 sums of slices
    const int64_t bytes = (all < kMostPlanes ? all : kMostPlanes) + (int64_t)sizeof(float) * TILE * TILE * (dev->sm_count / 2);
    void *ws;
    return engine_scratch(dev, (size_t)bytes, &ws) == AG_OK;
}

template <class T>
int gemm(ag_device *dev, int M, int N, int K, const T *p, int64_t p_row, int64_t p_k, const T *q,
         int64_t q_row, int64_t q_k, float alpha, float beta, T *c, int64_t ldc, const T *bias,
         bool relu) {
    if (planes<T>(M, N, K, p_k, q_k) > kMostPlanes) {
        const int longer = M >= N ? M : N, h = (int)ceil_div(longer / 2, TILE) * TILE;
        if (M >= N) {
            AG_TRY(gemm<T>(dev, h, N, K, p, p_row, p_k, q, q_row, q_k, alpha, beta, c, ldc, bias, relu));
            return gemm<T>(dev, M - h, N, K, p + h * p_row, p_row, p_k, q, q_row, q_k, alpha, beta, c + h, ldc,
                           bias != nullptr ? bias + h : nullptr, relu);
        }
        AG_TRY(gemm<T>(dev, M, h, K, p, p_row, p_k, q, q_row, q_k, alpha, beta, c, ldc, bias, relu));
        return gemm<T>(dev, M, N - h, K, p, p_row, p_k, q + h * q_row, q_row, q_k, alpha, beta, c + h * ldc, ldc, bias, relu);
    }
    constexpr int PL = Planes<T>::N;
    const bool a_mn = p_k != 1, b_mn = q_k != 1;
    PackJob<T> ja, jb;
    const int64_t a_bytes = plan<T>(&ja, p, M, K, p_row, p_k), b_bytes = plan<T>(&jb, q, N, K, q_row, q_k);
    const int64_t words = (ja.plane > jb.plane ? ja.plane : jb.plane) / 2;

    Params<T> a;
    a.M = M; a.N = N; a.K = K;
    a.ldc = ldc;
    a.alpha = alpha; a.beta = beta;
    a.C = c;
    a.bias = bias;
    a.relu = relu ? 1 : 0;
    a.p = p; a.q = q;
    a.p_row = p_row; a.p_k = p_k; a.q_row = q_row; a.q_k = q_k;
    a.status = dev->status_dev;
    a.group_m = 8;
    // Tiles of a last wave that fills at most half of the pairs, or of a product with few tiles,
    // are cut in two along n.
    const int tiles = (int)(ceil_div(M, TILE) * ceil_div(N, TILE)), pairs = dev->sm_count / 2;
    const int rem = tiles % pairs;
    a.t_full = tiles;
    a.tail_split = 1;
    a.num_work = tiles;
    if (rem > 0 && 2 * rem <= pairs) {
        a.t_full = tiles - rem;
        a.tail_split = 2;
        a.num_work = a.t_full + 2 * rem;
    }
    // Fewer tiles than half of the pairs: slices of k (at least two steps each) fill the others.
    const int steps = (int)ceil_div(K, BK);
    a.splits = 1;
    a.kb_split = steps;
    a.partial = nullptr;
    if (2 * tiles <= pairs && steps >= 4 && (int64_t)M * N < (1ll << 31)) {
        int splits = pairs / tiles;
        if (splits > steps / 2) splits = steps / 2;
        a.kb_split = (int)ceil_div(steps, splits);
        a.splits = (int)ceil_div(steps, a.kb_split);
        if (a.splits > 1) a.num_work = tiles * a.splits;
    }
    const int64_t part_bytes = a.splits > 1 ? (int64_t)sizeof(float) * a.splits * M * N : 0;
    void *ws = nullptr;
    AG_TRY(engine_scratch(dev, (size_t)(a_bytes + b_bytes + part_bytes), &ws));
    ja.dst = (__nv_bfloat16 *)ws;
    jb.dst = (__nv_bfloat16 *)((char *)ws + a_bytes);
    if (a.splits > 1) a.partial = (float *)((char *)ws + a_bytes + b_bytes);

    const int64_t blocks = ceil_div(words, 1024), cap = (int64_t)dev->sm_count * 8;
    AG_TRY(launch_dependent(dev, pack_kernel<T>, dim3((unsigned)(blocks < cap ? blocks : cap), 2), 256, 0, ja, jb));

    CUtensorMap ta, tb, tt;
    AG_TRY(packed_map(&ta, ja.dst, ja.inner, ja.outer, ja.pitch, PL, a_mn ? 64 : 128));
    AG_TRY(packed_map(&tb, jb.dst, jb.inner, jb.outer, jb.pitch, PL, b_mn ? 64 : 128));
    AG_TRY(packed_map(&tt, jb.dst, jb.inner, jb.outer, jb.pitch, PL, 64));
    if (a_mn && b_mn)
        AG_TRY((launch<PL, true, true>(dev, ta, tb, tt, a)));
    else if (a_mn)
        AG_TRY((launch<PL, true, false>(dev, ta, tb, tt, a)));
    else if (b_mn)
        AG_TRY((launch<PL, false, true>(dev, ta, tb, tt, a)));
    else
        AG_TRY((launch<PL, false, false>(dev, ta, tb, tt, a)));
    if (a.splits > 1) {
        const int64_t n = ceil_div((int64_t)M * N, 256);
        AG_TRY(launch_dependent(dev, reduce_kernel<T>, dim3((unsigned)(n < cap ? n : cap)), 256, 0, a, FastDiv((uint32_t)M)));
    }
    return AG_OK;
}

template bool reserve<float>(ag_device *, int, int, int, int64_t, int64_t);
template bool reserve<__nv_bfloat16>(ag_device *, int, int, int, int64_t, int64_t);
template int gemm<float>(ag_device *, int, int, int, const float *, int64_t, int64_t, const float *,
                         int64_t, int64_t, float, float, float *, int64_t, const float *, bool);
template int gemm<__nv_bfloat16>(ag_device *, int, int, int, const __nv_bfloat16 *, int64_t, int64_t,
                                 const __nv_bfloat16 *, int64_t, int64_t, float, float, __nv_bfloat16 *,
                                 int64_t, const __nv_bfloat16 *, bool);

}  // namespace packed
}  // namespace ag
