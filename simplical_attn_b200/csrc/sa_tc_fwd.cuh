// Forward 2-simplicial attention on the sm_100a tensor cores (tcgen05 MMA, accumulators in tensor
// memory, all operands staged by TMA).  Replaces the reference's
// two_simplicial_attn_fwd_kernel (simplicial/kernels.py:11-171).
//
// Formulation.  A query i and a K2 position k = i - delta (delta in [0, w2)) form one "virtual
// row" r = (i, delta) with the operand row  A[r, :] = Q_i * (K2_k + k2_bias)  (elementwise, formed
// on chip).  Then
//     S[r, j] = A[r, :] . K1[j, :]                      tensor-core GEMM, K = D
//     P[r, j] = exp2(S * scale*log2e - m_r)             online softmax per virtual row
//     T[r, :] = sum_j P[r, j] * V1[j, :]                tensor-core GEMM, K = j
//     O_i     = sum_delta w_r * (V2_k + v2_bias) * T[r, :] / L_i        epilogue merge over delta
// so the main loop is flash attention over the K1 window with 128-row tiles of virtual rows.
//
// A block works on "units" of one or two row tiles of 128 virtual rows (128/DW consecutive queries each, DW = w2
// rounded up to a power of two, at least 4).  The row tiles stream through the same K1/V1 column tiles (128 rows each;
// the last tile of a unit is only as wide as needed, in steps of 16).
//
// Warps.  0-3 / 4-7: softmax group of row tile 0 / 1.  8-11 / 12-15: auxiliary group of row tile 0 / 1: forms the A tile
// of the next unit as soon as the tensor cores have read the current one, and merges the finished unit's delta rows,
// both out of raw Q / K2 / V2 rows that are in shared memory by then.  16: MMA issuer; its
// loop runs over the column tiles of all units without a break, so S of the next unit's first tile is computed while
// the auxiliary group reads the finished T.  18: TMA loads of K1 / V1 (one ring of 128-row buffers, K1 and V1 in
// turn).  19: TMA loads of the raw rows, a unit ahead.
//
// The row tiles work in opposite phase: while one is in its softmax the tensor cores work for the other.  Column tiles
// are 128 wide because an MMA of 128 x 64 x 16 with A in shared memory takes 48 cycles, one of 128 x 128 x 16 takes 64:
// per row tile and 128 columns 1024 cycles of MMA instead of 1280.  The exponentials take another 1024 (16 per clock
// for the multiprocessor).  A pair of row tiles takes about 5600 cycles per 128 columns, so neither unit is the limit but
// the chain S -> softmax -> P -> P.V of each row tile with its hand-overs.
// Tensor memory: S0 | S1 (128 columns each, P overwrites S in place as packed 16-bit values) | T0 | T1 (D columns).
#pragma once

#include <type_traits>

#include "sa_ptx.cuh"

namespace sa {
namespace tc {

constexpr int kRowTile = 128;          // virtual rows per row tile = tensor-memory lanes
constexpr int kColTile = 128;          // columns of one S tile = K1/V1 rows of one TMA buffer
constexpr int kColPiece = 32;          // rows of one TMA load (a tile loads only the pieces it needs)
constexpr int kNumRowTiles = 2;        // row tiles per unit, at most
constexpr int kMaxFwdStages = 6;       // K1/V1 ring depth, at most (FwdTcParams::stages)
constexpr int kFwdThreads = 640;
constexpr float kRescaleThreshold = 8.0f;   // log2 units; below it the running maximum is kept
// Registers per thread of the softmax groups, the auxiliary groups and the MMA / TMA warps (multiples of 8).
#ifndef SA_FWD_REGS_SM
#define SA_FWD_REGS_SM 96
#define SA_FWD_REGS_AUX 112
#define SA_FWD_REGS_REST 64
#endif
// A setmaxnreg increase draws on what the block was launched with (640 x 96) and never returns if that does not
// suffice.
static_assert(2 * SA_FWD_REGS_SM + 2 * SA_FWD_REGS_AUX + SA_FWD_REGS_REST <= 5 * 96, "register pool of the block");

struct FwdTcParams {
    KParams k;
    int dw_log2;          // DW = 1 << dw_log2 delta slots per query
    int row_tiles;        // row tiles per unit: 2, or 1 where that spreads a small problem over more multiprocessors
    int stages;           // depth of the ring of K1 / V1 buffers
    int num_qblocks;      // ceil(N / queries per unit)
    int num_units;        // B * H * num_qblocks
    int off_k2, off_v2, off_q;   // shared-memory offsets of the raw rows
    DeviceStatus* status;
    uint64_t wait_limit_ns;   // bound of every device-side wait
};

// Shared memory: fixed part, A tiles, ring of K1 and V1 buffers, raw K2 / V2 window rows and Q rows of a unit.
template <int HD>
struct FwdSmem {
    static constexpr int kSlabs = HD / 64;                       // 64-element slabs per tile
    static constexpr int kTileBytes = kRowTile * HD * 2;         // one [128 x HD] A tile
    static constexpr int kSlabBytes = kRowTile * 128;
    static constexpr int kStageBytes = kColTile * HD * 2;        // one [128 x HD] K1 or V1 buffer
    static constexpr int kStageSlab = kColTile * 128;
    // fixed part; byte offsets from the 1024-aligned base
    static constexpr int kMisc = 464;                            // behind the barriers: tmem base, abort flag
    static constexpr int kZero = 512;                            // a row of zeros
    static constexpr int kStats = 1024;                          // m, l: [row tile][2][128] floats
    static constexpr int kPart = kStats + kNumRowTiles * 2 * kRowTile * 4;         // partial output rows: [row tile][4 warps][HD] floats
    static constexpr int kFixed = kPart + kNumRowTiles * 4 * 128 * 4;
    static_assert(kMisc + 16 <= kZero && kZero + 256 <= kStats && kFixed % 1024 == 0, "layout of the fixed part");
    static constexpr int kA = kFixed;                            // row tiles
    static constexpr int kRing = kA + kNumRowTiles * kTileBytes; // K1 / V1 buffers
    static constexpr int kMaxBytes = 227 * 1024 - 1024;          // 1024: alignment of the base
};

inline __host__ __device__ int fwd_window_rows(int dw_log2, int row_tiles) {
    return (1 << dw_log2) + row_tiles * (kRowTile >> dw_log2) - 1;
}

// Ring depth and offsets for the problem; returns the dynamic shared memory of the launch.
template <int HD>
int fwd_smem_plan(FwdTcParams& P) {
    using L = FwdSmem<HD>;
    const int win = ((fwd_window_rows(P.dw_log2, P.row_tiles) + 7) & ~7) * 128 * L::kSlabs;
    const int qrows = ((P.row_tiles * (kRowTile >> P.dw_log2) + 7) & ~7) * 128 * L::kSlabs;
    P.stages = (L::kMaxBytes - L::kRing - 2 * win - qrows) / L::kStageBytes;      // at least 2
    if (P.stages > kMaxFwdStages) P.stages = kMaxFwdStages;
    P.off_k2 = L::kRing + P.stages * L::kStageBytes;
    P.off_v2 = P.off_k2 + win;
    P.off_q = P.off_v2 + win;
    const int total = P.off_q + qrows + 1024;
    return total > 120 * 1024 ? total : 120 * 1024;      // more than half a multiprocessor: one block each
}

// Unit -> (head, first query, column range), walked in steps of the grid without a division.
struct UnitGeom {
    int i0;            // first query
    int col_start;     // first K1/V1 buffer row the unit needs
    int ntile;         // column tiles
    int last_width;    // width of the last one, multiple of 16
};

struct UnitWalk {
    int u, qb, bh, step_q, step_b;
    __device__ __forceinline__ explicit UnitWalk(const FwdTcParams& P) {
        u = blockIdx.x;
        bh = u / P.num_qblocks;
        qb = u - bh * P.num_qblocks;
        step_b = (int)gridDim.x / P.num_qblocks;
        step_q = (int)gridDim.x - step_b * P.num_qblocks;
    }
    __device__ __forceinline__ bool valid(const FwdTcParams& P) const { return u < P.num_units; }
    __device__ __forceinline__ void next(const FwdTcParams& P) {
        u += gridDim.x;
        qb += step_q;
        bh += step_b;
        if (qb >= P.num_qblocks) {
            qb -= P.num_qblocks;
            ++bh;
        }
    }
    __device__ __forceinline__ UnitGeom geom(const FwdTcParams& P) const {
        const KParams& p = P.k;
        UnitGeom g;
        const int qpb = (P.row_tiles * kRowTile) >> P.dw_log2;
        g.i0 = qb * qpb;
        const int i_last = min(g.i0 + qpb, p.N) - 1;
        // (the pair's first query also where row tiles are single: a query's column tiles, and with them the rounding of
        // its result, do not depend on how many heads the call holds)
        const int i_pair = g.i0 & ~(((kNumRowTiles * kRowTile) >> P.dw_log2) - 1);
        g.col_start = max(0, i_pair + p.halo1 - p.w1 + 1);
        const int ncols = i_last + p.halo1 - g.col_start + 1;
        g.ntile = (ncols + kColTile - 1) / kColTile;
        g.last_width = ((ncols - (g.ntile - 1) * kColTile) + 15) & ~15;
        return g;
    }
};

// Position in a ring of `stages` buffers.
struct RingPos {
    int s = 0;
    uint32_t phase = 0;
    __device__ __forceinline__ void next(int stages) {
        if (++s == stages) {
            s = 0;
            phase ^= 1;
        }
    }
};

// BIAS = false: both biases are zero, every bias add folds away.  F16: the tensors are IEEE half instead of bf16
// (same kernels; only the element encoding and the MMA's operand format differ).
template <int HD, bool BIAS, bool F16 = false>
__global__ void __launch_bounds__(kFwdThreads, 1)
fwd_tc_kernel(const __grid_constant__ FwdTcParams P, const __grid_constant__ CUtensorMap map_k1,
              const __grid_constant__ CUtensorMap map_v1, const __grid_constant__ CUtensorMap map_q,
              const __grid_constant__ CUtensorMap map_k2, const __grid_constant__ CUtensorMap map_v2,
              __nv_bfloat16* __restrict__ o, float* __restrict__ lse) {
    using L = FwdSmem<HD>;
    using namespace ptx;
    using E = El<F16>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t smem_base = smem_u32(smem);
    const KParams& p = P.k;

    // barriers, as byte offsets from the base
    constexpr int kFull = 0;                                     // [stages] K1 / V1 buffer landed
    constexpr int kEmpty = kFull + 8 * kMaxFwdStages;            //          every row tile's MMAs have read it
    constexpr int kAReady = kEmpty + 8 * kMaxFwdStages;          // [row tile] A tile formed (auxiliary group -> MMA warp)
    constexpr int kAFree = kAReady + 16;                         //            the unit's last S MMAs have read it (MMA warp -> auxiliary group)
    constexpr int kOReady = kAFree + 16;                         //            T final (MMA warp -> auxiliary group)
    constexpr int kTFree = kOReady + 16;                         //            T read out (auxiliary group -> MMA warp)
    constexpr int kStReady = kTFree + 16;                        //            m, l of the unit stored (softmax group -> auxiliary group)
    constexpr int kStFree = kStReady + 16;                       //            m, l consumed (auxiliary group -> softmax group)
    constexpr int kSReady = kStFree + 16;                        //            S tile computed (MMA warp -> softmax group)
    constexpr int kPReady = kSReady + 16;                        //            P stored (softmax group -> MMA warp)
    constexpr int kQkFull = kPReady + 16;                        // raw Q and K2 rows landed
    constexpr int kQkFree = kQkFull + 8;                         //             ... read by the auxiliary groups
    constexpr int kV2Full = kQkFree + 8;                         // raw V2 rows landed
    constexpr int kV2Free = kV2Full + 8;                         //             ... read by the auxiliary groups
    static_assert(kV2Free + 8 <= L::kMisc, "room for the barriers");
    uint32_t* tmem_base_slot = (uint32_t*)(smem + L::kMisc);
    volatile int* abort_flag = (volatile int*)(smem + L::kMisc + 4);
    const WaitCtx wctx{smem_base + L::kMisc + 4, P.status, P.wait_limit_ns};

    const int tid = threadIdx.x;
    SA_PROF_T0(t_life);
    SA_TR_DECL();
    const int warp = tid >> 5;
    const int lane = tid & 31;

    if (tid == 0) {
        auto init = [&](int off, int n, uint32_t count) {
            for (int x = 0; x < n; ++x) mbar_init((uint64_t*)(smem + off) + x, count);
        };
        init(kFull, kMaxFwdStages, 1);
        init(kEmpty, kMaxFwdStages, P.row_tiles);
        // (barriers a 128-thread group arrives on count one elected arrival per warp)
        init(kAReady, 2, 4);
        init(kAFree, 2, 1);
        init(kOReady, 2, 1);
        init(kTFree, 2, 4);
        init(kStReady, 2, 4);
        init(kStFree, 2, 4);
        init(kSReady, 2, 1);
        init(kPReady, 2, 4);
        init(kQkFull, 1, 1);
        init(kQkFree, 1, 4 * P.row_tiles);
        init(kV2Full, 1, 1);
        init(kV2Free, 1, 4 * P.row_tiles);
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (tid >= 64 && tid < 128) *(uint32_t*)(smem + L::kZero + (tid - 64) * 4) = 0u;
    if (warp == 16) {
        tmem_alloc(tmem_base_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_base_slot;
    // S of row tile r at column 128 r, T accumulators behind them
    const uint32_t tmem_t0 = tmem_base + 256;

    const int DW = 1 << P.dw_log2;
    const int qpt = kRowTile >> P.dw_log2;          // queries per row tile
    // One arrival per warp: every lane has finished (and fenced) its own part, the warp converges, lane 0 arrives.
#define SA_FWD_ARRIVE(OFF, BASE)                   \
    do {                                           \
        __syncwarp();                              \
        if (lane == 0) mbar_arrive<(OFF)>(BASE);   \
    } while (0)

    const int win = fwd_window_rows(P.dw_log2, P.row_tiles), qrows = P.row_tiles * qpt;      // raw K2 / V2 and Q rows of a unit
    const uint32_t win_slab = ((win + 7) & ~7) * 128, q_slab = ((qrows + 7) & ~7) * 128;
    const uint32_t k2_st = smem_base + P.off_k2, v2_st = smem_base + P.off_v2, q_st = smem_base + P.off_q;

    if (warp >= 16) {
        reg_dealloc<SA_FWD_REGS_REST>();
        if (warp == 18) {
            // -------------------------------------------------------------- TMA producer of K1 / V1
            if (lane == 0) {
                prefetch_tensormap(&map_k1);
                prefetch_tensormap(&map_v1);
                RingPos g;
                for (UnitWalk w(P); w.valid(P); w.next(P)) {
                    const UnitGeom ug = w.geom(P);
                    const int b = w.bh / p.H, hk = (w.bh - b * p.H) / p.G;
                    for (int t = 0; t < ug.ntile; ++t) {
                        const int row = ug.col_start + t * kColTile;
                        const int pieces = t == ug.ntile - 1 ? (ug.last_width + kColPiece - 1) / kColPiece : kColTile / kColPiece;
#pragma unroll 1
                        for (int kv = 0; kv < 2; ++kv) {
                            const uint32_t gb = smem_base + g.s * 8;
                            mbar_wait<kEmpty>(gb, g.phase ^ 1, wctx, 1 + kv);
                            mbar_arrive_expect_tx(gb + kFull, pieces * kColPiece * 128 * L::kSlabs);
                            const uint32_t dst = smem_base + L::kRing + g.s * L::kStageBytes;
                            for (int pc = 0; pc < pieces; ++pc)
#pragma unroll
                                for (int sl = 0; sl < L::kSlabs; ++sl)
                                    tma_load_4d(dst + sl * L::kStageSlab + pc * kColPiece * 128, kv ? &map_v1 : &map_k1, gb + kFull, sl * 64,
                                                row + pc * kColPiece, hk, b);
                            g.next(P.stages);
                        }
                    }
                }
            }
            __syncwarp();
        } else if (warp == 19) {
            // -------------------------------------------------------------- TMA producer of the raw rows of a unit: Q [i0, i0 + qrows),
            // K2 / V2 [i0 + halo2 - (DW-1), + win); rows outside the tensors are filled with zeros
            if (lane == 0) {
                prefetch_tensormap(&map_q);
                prefetch_tensormap(&map_k2);
                prefetch_tensormap(&map_v2);
                auto load_qk = [&](const UnitWalk& w) {
                    const int b = w.bh / p.H, h = w.bh - b * p.H, hk = h / p.G, i0 = w.qb * qrows;
                    mbar_arrive_expect_tx(smem_base + kQkFull, (win + qrows) * 128 * L::kSlabs);
#pragma unroll
                    for (int sl = 0; sl < L::kSlabs; ++sl) {
                        tma_load_4d(q_st + sl * q_slab, &map_q, smem_base + kQkFull, sl * 64, i0, h, b);
                        tma_load_4d(k2_st + sl * win_slab, &map_k2, smem_base + kQkFull, sl * 64, i0 + p.halo2 - (DW - 1), hk, b);
                    }
                };
                auto load_v2 = [&](const UnitWalk& w) {
                    const int b = w.bh / p.H, hk = (w.bh - b * p.H) / p.G, i0 = w.qb * qrows;
                    mbar_arrive_expect_tx(smem_base + kV2Full, win * 128 * L::kSlabs);
#pragma unroll
                    for (int sl = 0; sl < L::kSlabs; ++sl)
                        tma_load_4d(v2_st + sl * win_slab, &map_v2, smem_base + kV2Full, sl * 64, i0 + p.halo2 - (DW - 1), hk, b);
                };
                // in the order the auxiliary groups consume them: form(0); form(u + 1), merge(u), for u = 0, 1, ...
                UnitWalk wq(P), wv(P);
                if (wq.valid(P)) load_qk(wq);
                if (wv.valid(P)) load_v2(wv);
                uint32_t u = 0;
                for (wq.next(P); wv.valid(P); ++u) {
                    if (wq.valid(P)) {
                        mbar_wait<kQkFree>(smem_base, u & 1, wctx, 20);      // unit u has been formed
                        load_qk(wq);
                        wq.next(P);
                    }
                    wv.next(P);
                    if (wv.valid(P)) {
                        mbar_wait<kV2Free>(smem_base, u & 1, wctx, 21);      // unit u has been merged
                        load_v2(wv);
                    }
                }
            }
            __syncwarp();
        } else if (warp == 16) {
            // -------------------------------------------------------------- MMA issuer: P.V and the next S of row tile 0, then of row
            // tile 1, and so on.  The fixed order keeps the row tiles half a period apart.  (With an issuer of its own
            // for each, their MMAs interleave, both S tiles are complete at the same time and both softmaxes run at
            // the same time while the tensor cores idle.)
            const uint32_t leader = elect_one();      // the whole warp runs the loop; one lane issues
            const int nrt = P.row_tiles;
            // S tile = A . K1^T into the columns that row tile r's last P.V MMAs read (issued before, and the tensor cores
            // run in order)
            auto issue_s = [&](int r, int buf, bool last, int width) {
                const uint32_t idesc = make_idesc(128, width, false, false, F16);
                const uint32_t da = desc_lo(smem_base + L::kA + r * L::kTileBytes, 16);
                const uint32_t db = desc_lo(smem_base + L::kRing + buf * L::kStageBytes, 16);
                static_for<HD / 16>([&](auto kk_c) {
                    constexpr int kk = decltype(kk_c)::value, off = ((kk >> 2) * L::kSlabBytes + (kk & 3) * 32) >> 4;
                    mma_ss_lo<off, off>(leader, tmem_base + r * kColTile, da, db, idesc, kk > 0);
                });
                SA_TR(0, 32 + 100 * r);
                tc_commit<kSReady>(leader, smem_base + r * 8);
                tc_commit<kEmpty>(leader, smem_base + buf * 8);
                if (last) tc_commit<kAFree>(leader, smem_base + r * 8);       // the A tile may be overwritten
            };
            RingPos g;                                // buffers are consumed in the order K1, V1, K1, V1, ...
            uint32_t n = 0, nu = 0;                   // column tiles, units so far
            UnitWalk w(P);
            UnitGeom ug = w.geom(P);
            if (w.valid(P)) {
                mbar_wait<kFull>(smem_base + g.s * 8, g.phase, wctx, 3);
                for (int r = 0; r < nrt; ++r) {
                    mbar_wait<kAReady>(smem_base + r * 8, 0, wctx, 4);
                    tc_fence_after();
                    issue_s(r, g.s, ug.ntile == 1, ug.ntile == 1 ? ug.last_width : kColTile);
                }
                g.next(P.stages);
            }
            while (w.valid(P)) {
                UnitWalk wn = w;
                wn.next(P);
                const bool more = wn.valid(P);
                const UnitGeom ng = more ? wn.geom(P) : ug;
#pragma unroll 1
                for (int t = 0; t < ug.ntile; ++t, ++n) {
                    const bool last = t == ug.ntile - 1;
                    const int ksteps = last ? ug.last_width / 16 : kColTile / 16;
                    const bool have_next = !last || more;                      // the next S tile, which may be the next unit's first
                    const bool nlast = last ? ng.ntile == 1 : t + 1 == ug.ntile - 1;
                    const int nwidth = nlast ? (last ? ng.last_width : ug.last_width) : kColTile;
                    const int vbuf = g.s;
                    const uint32_t vphase = g.phase;
                    g.next(P.stages);
                    const int kbuf = g.s;
                    const uint32_t kphase = g.phase;
                    g.next(P.stages);
                    const uint32_t idesc = make_idesc(128, HD, false, true, F16);
                    const uint32_t db = desc_lo(smem_base + L::kRing + vbuf * L::kStageBytes, L::kStageSlab);
#pragma unroll 1
                    for (int r = 0; r < nrt; ++r) {
                        const uint32_t rb = smem_base + r * 8;
                        const uint32_t tm_s = tmem_base + r * kColTile, tm_t = tmem_t0 + r * HD;
                        mbar_wait<kFull>(smem_base + vbuf * 8, vphase, wctx, 6);
                        SA_TR(0, 41 + 100 * r);
                        // the previous unit's T has been read out by the auxiliary group
                        if (t == 0 && nu > 0) mbar_wait<kTFree>(rb, (nu - 1) & 1, wctx, 10);
                        mbar_wait<kPReady>(rb, n & 1, wctx, 5);
                        SA_TR(0, 20 + 100 * r);
                        tc_fence_after();
                        static_for<8>([&](auto kk_c) {
                            constexpr int kk = decltype(kk_c)::value;
                            if (kk < ksteps) mma_ts_lo<kk * 8, kk * (2048 >> 4)>(leader, tm_t, tm_s, db, idesc, t > 0 || kk > 0);
                        });
                        SA_TR(0, 29 + 100 * r);
                        tc_commit<kEmpty>(leader, smem_base + vbuf * 8);
                        if (last) tc_commit<kOReady>(leader, rb);
                        SA_TR(0, 30 + 100 * r);
                        if (have_next) {
                            mbar_wait<kFull>(smem_base + kbuf * 8, kphase, wctx, 3);
                            SA_TR(0, 31 + 100 * r);
                            if (last) mbar_wait<kAReady>(rb, (nu + 1) & 1, wctx, 4);
                            tc_fence_after();
                            issue_s(r, kbuf, nlast, nwidth);
                        }
                        SA_TR(0, 40 + 100 * r);
                    }
                }
                w = wn;
                ug = ng;
                ++nu;
            }
        }
    } else if (warp >= 8) {
        // ------------------------------------------------------------------ auxiliary groups: operand formation ahead of the
        // softmax groups, merge over delta and output behind them
        reg_alloc<SA_FWD_REGS_AUX>();
        const int r = (warp - 8) >> 2;
        const int t = tid & 127;
        const int wq = warp & 3;
        const uint32_t rb = smem_base + r * 8;
        const float v2_bias = BIAS ? p.v2_bias : 0.f;
        // A tile of row tile r of the unit at query i0: row rho = (query rho / DW, delta rho % DW), a thread takes one
        // 16-byte chunk of every RPP-th row.  Padding (delta >= w2, K2 rows before the first) repeats the query's last row:
        // its scores and T are as finite as that row's, so that the merge's zero weight drops them.  (Zero rows would meet
        // an infinity in K1 as NaN.)
        auto form = [&](int i0) {
            constexpr int CH = HD / 8, RPP = 128 / CH;
            const int c = t % CH, row0 = t / CH;
            const uint32_t tile = smem_base + L::kA + r * L::kTileBytes + (c >> 3) * L::kSlabBytes;
            const uint32_t ksl = k2_st + (c >> 3) * win_slab, qsl = q_st + (c >> 3) * q_slab;
#pragma unroll 4
            for (int k = 0; k < 128 / RPP; ++k) {
                const int rho = row0 + k * RPP;
                const int q2 = r * qpt + (rho >> P.dw_log2), dlt = min(rho & (DW - 1), min(p.w2 - 1, max(i0 + q2 + p.halo2, 0)));
                const int wr = q2 + DW - 1 - dlt;
                const uint4 x = lds128(qsl + q2 * 128 + (((c ^ q2) & 7) << 4));
                const uint4 y = lds128(ksl + wr * 128 + (((c ^ wr) & 7) << 4));
                sts128(tile + rho * 128 + (((c ^ rho) & 7) << 4), BIAS ? mul_chunk<F16>(x, y, p.k2_bias) : mul_chunk_nobias<F16>(x, y));
            }
            fence_proxy_async_smem();
            SA_FWD_ARRIVE(kAReady, rb);
            if (lane == 0) mbar_arrive<kQkFree>(smem_base);
        };
        // O rows of row tile r of the unit at (b, h, i0).  T is read in the 16x256b form: thread t of a warp gets, of
        // 16 rows, rows t/4 and t/4 + 8 and of every 8 columns the pair 2 (t % 4).  So the sum over delta is mostly
        // within the thread; the rest (8 rows apart by lane) is a halving exchange that leaves a thread with one
        // column pair of 64 columns: 14 shuffles per 64 columns and query, and V2 comes from shared memory without
        // bank conflicts.  (One row per thread needs 62 shuffles, and its V2 loads touch 32 lines each.)
        // CLS: 2 for DW >= 32 (a warp's rows are one query's), 1 for DW = 16, 0 for 8 and 4.
        auto merge = [&](auto cls_c, uint32_t nu, int b, int h, int i0) {
            constexpr int CLS = decltype(cls_c)::value;
            const uint32_t st = smem_base + L::kStats + r * 2 * kRowTile * 4;       // m | l
            mbar_wait<kStReady>(rb, nu & 1, wctx, 12);
            // the rows of this row's query: this warp's, or (DW > 32) those of DW / 32 warps, 32 at a time
            float mq = -INFINITY, lq = 0.f, m_own = -INFINITY;
            const int wpq = DW > 32 ? DW >> 5 : 1;
            auto stat = [&](int rr, float& m, float& l) {          // m = -inf for a row that is not valid
                const int i = i0 + (rr >> P.dw_log2), dlt = rr & (DW - 1);
                m = lds_f32(st + rr * 4);
                l = lds_f32(st + (kRowTile + rr) * 4);
                if (i >= p.N || dlt >= p.w2 || i + p.halo2 - dlt < 0) m = -INFINITY;
            };
            float l_own = 0.f;
            stat(t, m_own, l_own);
            mq = m_own;
            if (CLS == 2 && wpq > 1)
                for (int k = 0; k < wpq; ++k) {
                    float mm, ll;
                    stat((t & ~(DW - 1)) + lane + 32 * k, mm, ll);
                    mq = fmaxf(mq, mm);
                }
            const int sft0 = CLS == 2 ? 16 : CLS == 1 ? 8 : DW >> 1;
#pragma unroll
            for (int sft = sft0; sft >= 1; sft >>= 1) mq = fmaxf(mq, __shfl_xor_sync(0xffffffffu, mq, sft));
            const float e_own = m_own > -INFINITY ? ex2(m_own - mq) : 0.f;
            if (CLS == 2 && wpq > 1) {
                for (int k = 0; k < wpq; ++k) {
                    float mm, ll;
                    stat((t & ~(DW - 1)) + lane + 32 * k, mm, ll);
                    lq += mm > -INFINITY ? ex2(mm - mq) * ll : 0.f;
                }
            } else {
                lq = e_own * l_own;
            }
            SA_FWD_ARRIVE(kStFree, rb);           // m, l of this unit are no longer needed
#pragma unroll
            for (int sft = sft0; sft >= 1; sft >>= 1) lq += __shfl_xor_sync(0xffffffffu, lq, sft);
            const float wrow = m_own > -INFINITY ? e_own / lq : 0.f;
            {
                const int i = i0 + (t >> P.dw_log2);
                if ((t & (DW - 1)) == 0 && i < p.N) lse[((long)b * p.H + h) * p.N + i] = (mq + log2f(lq)) * kLn2;
            }
            // this thread's four rows: weight, swizzled V2 row (rows that are not valid: the zero row), slab pitch
            float wk[4];
            uint32_t va[4], sl[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int rl = (lane >> 2) + 8 * k, rr = 32 * wq + rl;
                wk[k] = __shfl_sync(0xffffffffu, wrow, rl);
                const int q2 = rr >> P.dw_log2, dlt = rr & (DW - 1), wr = r * qpt + q2 + DW - 1 - dlt;
                const bool ok = i0 + q2 < p.N && dlt < p.w2 && i0 + q2 + p.halo2 >= dlt;
                va[k] = (ok ? v2_st + wr * 128 + ((wr & 7) << 4) : smem_base + L::kZero) + (lane & 3) * 4;
                sl[k] = ok ? win_slab : 0u;
            }
            mbar_wait<kV2Full>(smem_base, nu & 1, wctx, 15);
            mbar_wait<kOReady>(rb, nu & 1, wctx, 9);
            if (wq == 0) SA_TR(2 + r, 64);
            tc_fence_after();
            const uint32_t t_addr = tmem_t0 + r * HD + ((uint32_t)(32 * wq) << 16);
            __nv_bfloat16* const obase = o + b * p.o.b + h * p.o.h;
            const uint32_t part = smem_base + L::kPart + r * (4 * HD * 4);
            // columns [64 ch, + 64) of the query that holds row rl0 (row within the warp) of this warp, from acc
            auto reduce_store = [&](float (&acc)[16], int ch, int rl0) {
                const int i = i0 + ((32 * wq + rl0) >> P.dw_log2);
                __nv_bfloat16* const orow = obase + (long)i * p.o.n + 64 * ch;
                auto halve = [&](int s, auto n_c) {
                    constexpr int N = decltype(n_c)::value;
                    const bool upper = (lane & s) != 0;
#pragma unroll
                    for (int e = 0; e < N; ++e) {
                        const float send = upper ? acc[e] : acc[e + N], keep = upper ? acc[e + N] : acc[e];
                        acc[e] = keep + __shfl_xor_sync(0xffffffffu, send, s);
                    }
                };
                if (CLS > 0 || P.dw_log2 == 3) {
                    halve(16, std::integral_constant<int, 8>{});
                    halve(8, std::integral_constant<int, 4>{});
                    halve(4, std::integral_constant<int, 2>{});
                    if (CLS == 2 && P.dw_log2 >= 6)
                        asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(part + (wq * HD + 64 * ch + 2 * lane) * 4), "f"(acc[0]), "f"(acc[1]) : "memory");
                    else if (i < p.N)
                        *(uint32_t*)(orow + 2 * lane) = E::pack(acc[0], acc[1]);
                } else {
                    // four rows to a query: lanes t/4 = 0..3 and 4..7 hold different ones
                    halve(8, std::integral_constant<int, 8>{});
                    halve(4, std::integral_constant<int, 4>{});
                    const int col = 16 * ((lane >> 2) & 3) + 2 * (lane & 3);
                    if (i < p.N) {
                        *(uint32_t*)(orow + col) = E::pack(acc[0], acc[1]);
                        *(uint32_t*)(orow + col + 8) = E::pack(acc[2], acc[3]);
                    }
                }
#pragma unroll
                for (int e = 0; e < 16; ++e) acc[e] = 0.f;
            };
            float acc[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) acc[e] = 0.f;
#pragma unroll 1
            for (int ch = 0; ch < HD / 64; ++ch) {
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    uint32_t tv[32];
                    tmem_ld_16x256_x8(t_addr + (hf << 20) + 64 * ch, tv);
                    tmem_wait_ld();
                    if (hf == 1 && ch == HD / 64 - 1) {       // T has been read: the next unit's first P.V may overwrite it
                        tc_fence_before();
                        SA_FWD_ARRIVE(kTFree, rb);
                    }
#pragma unroll
                    for (int a = 0; a < 2; ++a) {
                        const int k = 2 * hf + a;
                        const float2 w2v = make_float2(wk[k], wk[k]);
                        const uint32_t vaddr = va[k] + ch * sl[k];
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const uint32_t w = lds32(vaddr ^ (j << 4));
                            float2 x2 = make_float2(E::lo(w), E::hi(w));
                            if (BIAS) x2 = __fadd2_rn(x2, make_float2(v2_bias, v2_bias));
                            const float2 tw = __fmul2_rn(make_float2(__uint_as_float(tv[4 * j + 2 * a]), __uint_as_float(tv[4 * j + 2 * a + 1])), w2v);
                            const float2 s2 = __ffma2_rn(tw, x2, make_float2(acc[2 * j], acc[2 * j + 1]));
                            acc[2 * j] = s2.x;
                            acc[2 * j + 1] = s2.y;
                        }
                        if (CLS == 0) reduce_store(acc, ch, 8 * k + (P.dw_log2 == 2 ? (lane >> 4) * 4 : 0));
                    }
                    if (CLS == 1) reduce_store(acc, ch, 16 * hf);
                }
                if (CLS == 2) reduce_store(acc, ch, 0);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive<kV2Free>(smem_base);
            if (CLS == 2 && P.dw_log2 >= 6) {
                // a query spans DW / 32 warps: add their partial rows
                named_barrier_sync(1 + r, 128);
                for (int idx = t; idx < qpt * HD; idx += 128) {
                    const int q2 = idx / HD, col = idx % HD, i = i0 + q2;
                    float sum = 0.f;
                    for (int w = 0; w < wpq; ++w) sum += lds_f32(part + ((q2 * wpq + w) * HD + col) * 4);
                    if (i < p.N) E::st(obase + (long)i * p.o.n + col, sum);
                }
                named_barrier_sync(1 + r, 128);
            }
        };

        if (r < P.row_tiles) {
            UnitWalk w(P);                // the unit to merge; the one to form is the next
            uint32_t nu = 0;
            if (w.valid(P)) {
                mbar_wait<kQkFull>(smem_base, 0, wctx, 16);
                form(w.qb * qrows);
            }
            while (w.valid(P)) {
                UnitWalk wn = w;
                wn.next(P);
                if (wn.valid(P)) {
                    // ---- the next unit's A tile, as soon as this unit's last S MMAs have read the current one
                    mbar_wait<kQkFull>(smem_base, (nu + 1) & 1, wctx, 16);
                    mbar_wait<kAFree>(rb, nu & 1, wctx, 11);
                    if (wq == 0) SA_TR(2 + r, 50);
                    form(wn.qb * qrows);
                    if (wq == 0) SA_TR(2 + r, 52);
                }
                // ---- merge of this unit
                const int b = w.bh / p.H, h = w.bh - b * p.H, i0 = w.qb * qrows + r * qpt;
                if (wq == 0) SA_TR(2 + r, 60);
                if (P.dw_log2 >= 5) merge(std::integral_constant<int, 2>{}, nu, b, h, i0);
                else if (P.dw_log2 == 4) merge(std::integral_constant<int, 1>{}, nu, b, h, i0);
                else merge(std::integral_constant<int, 0>{}, nu, b, h, i0);
                if (wq == 0) SA_TR(2 + r, 66);
                w = wn;
                ++nu;
            }
        }
    } else {
        // ------------------------------------------------------------------ softmax groups
        reg_alloc<SA_FWD_REGS_SM>();
        const int r = warp >> 2;                     // row tile
        const int row = tid & 127;                   // virtual row = tensor-memory lane
        const uint32_t lane_addr = (uint32_t)(row & ~31) << 16;
        const float c2 = p.scale * kLog2e;
        const uint32_t s_addr = tmem_base + r * kColTile + lane_addr;
        const uint32_t t_addr = tmem_t0 + r * HD + lane_addr;
        const uint32_t rb = smem_base + r * 8;
        uint32_t n = 0, nu = 0;                      // column tiles, units so far
        UnitWalk w(P);
        if (r >= P.row_tiles) w.u = P.num_units;
        for (; w.valid(P); w.next(P), ++nu) {
            const UnitGeom ug = w.geom(P);
            // valid buffer rows of this query: [jlo, jhi].  Padding rows (delta >= w2, a K2 row before the buffer, a query past
            // the end) run along, and the merge drops them.
            const int jhi = ug.i0 + r * qpt + (row >> P.dw_log2) + p.halo1 - ug.col_start;
            const int jlo = max(-ug.col_start, jhi - p.w1 + 1);
            float m = -INFINITY, l = 0.f;
            for (int t = 0; t < ug.ntile; ++t, ++n) {
                const int width = t == ug.ntile - 1 ? ug.last_width : kColTile;
                const int lo = jlo - t * kColTile, hi = min(jhi - t * kColTile, width - 1);        // valid tile-relative columns [lo, hi]
                mbar_wait<kSReady>(rb, n & 1, wctx, 8);
                SA_TR(4 + r, 70);
                tc_fence_after();
                // One column tile of up to NC columns.  The scores are read twice, once for the maximum and once, 16 columns
                // ahead, for the exponentials: keeping 64 of them in registers spilled even at 128 registers.
                auto softmax = [&](auto nc_c, auto masked_c) {
                    constexpr int NC = decltype(nc_c)::value;
                    constexpr bool MASKED = decltype(masked_c)::value;
                    // masked scores (whatever the buffer holds there) become -inf
                    auto mask = [&](auto& x, int c0, auto n_c) {
                        if constexpr (MASKED) {
                            constexpr int N = decltype(n_c)::value;
                            const int a = max(lo - c0, 0), z = min(hi - c0, N - 1);
                            const uint32_t bits = z >= a ? (~0u >> (31 - (z - a))) << a : 0u;
#pragma unroll
                            for (int e = 0; e < N; ++e) x[e] = (bits & (1u << e)) ? x[e] : 0xff800000u;
                        }
                    };
                    float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
                    {
                        uint32_t v[2][32];
                        tmem_ld32(s_addr, v[0]);
#pragma unroll
                        for (int c = 0; c < NC / 32; ++c) {
                            tmem_wait_ld();
                            if (c + 1 < NC / 32) tmem_ld32(s_addr + 32 * (c + 1), v[(c + 1) & 1]);
                            mask(v[c & 1], 32 * c, std::integral_constant<int, 32>{});
#pragma unroll
                            for (int e = 0; e < 32; e += 8)
#pragma unroll
                                for (int y = 0; y < 4; ++y)
                                    mx[y] = max3(mx[y], __uint_as_float(v[c & 1][e + y]), __uint_as_float(v[c & 1][e + 4 + y]));
                        }
                    }
                    uint32_t v[2][16];
                    tmem_ld16(s_addr, v[0]);            // (in flight under what follows)
                    const float tmax = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * c2;      // -inf stays -inf (c2 > 0)
                    // Running maximum, lazily updated.  When it moves, l and T are scaled down (T is at rest: this tile's S
                    // was issued behind the previous tile's P.V MMAs).
                    if (tmax > m + kRescaleThreshold || m == -INFINITY) {
                        const float factor = m > -INFINITY ? ex2(m - tmax) : 1.f;
                        l *= factor;
                        m = tmax;
                        mx[0] = factor;
                    } else {
                        mx[0] = 1.f;
                    }
                    if (__any_sync(0xffffffffu, mx[0] != 1.f)) {
#pragma unroll 1
                        for (int c0 = 0; c0 < HD; c0 += 16) {
                            uint32_t tv[16];
                            tmem_ld16(t_addr + c0, tv);
                            tmem_wait_ld();
#pragma unroll
                            for (int e = 0; e < 16; ++e) tv[e] = __float_as_uint(__uint_as_float(tv[e]) * mx[0]);
                            tmem_st16(t_addr + c0, tv);
                        }
                    }
                    // P = exp2(S*c2 - m): packed two-wide fp32 arithmetic, one FMA and one add per pair of columns
                    const float nms = m == -INFINITY ? 0.f : -m;
                    float2 ls = make_float2(0.f, 0.f);
                    const float2 c2v = make_float2(c2, c2), nm = make_float2(nms, nms);
#pragma unroll
                    for (int c = 0; c < NC / 16; ++c) {
                        tmem_wait_ld();
                        // (packed columns [8c, 8c + 8) overwrite S columns that are in registers or used up by now)
                        if (c + 1 < NC / 16) tmem_ld16(s_addr + 16 * (c + 1), v[(c + 1) & 1]);
                        mask(v[c & 1], 16 * c, std::integral_constant<int, 16>{});
                        uint32_t pk[8];
#pragma unroll
                        for (int e = 0; e < 16; e += 2) {
                            const float2 y = __ffma2_rn(make_float2(__uint_as_float(v[c & 1][e]), __uint_as_float(v[c & 1][e + 1])), c2v, nm);
                            const float2 pe = make_float2(ex2(y.x), ex2(y.y));
                            ls = __fadd2_rn(ls, pe);
                            pk[e >> 1] = E::pack(pe.x, pe.y);
                        }
                        tmem_st8(s_addr + 8 * c, pk);
                    }
                    tmem_wait_st();
                    tc_fence_before();
                    SA_FWD_ARRIVE(kPReady, rb);
                    l += ls.x + ls.y;
                };
                // a tile is "full" when every column is inside every row's window: no masks needed
                const bool full = width == kColTile && __all_sync(0xffffffffu, lo <= 0 && hi >= kColTile - 1);
                if (full) softmax(std::integral_constant<int, 128>{}, std::false_type{});
                else if (width > 64) softmax(std::integral_constant<int, 128>{}, std::true_type{});
                else if (width > 32) softmax(std::integral_constant<int, 64>{}, std::true_type{});
                else softmax(std::integral_constant<int, 32>{}, std::true_type{});
                SA_TR(4 + r, 72);
            }
            // ---- hand the row statistics to the auxiliary group (once it has consumed the previous unit's)
            if (nu > 0) mbar_wait<kStFree>(rb, (nu - 1) & 1, wctx, 13);
            const uint32_t st_out = smem_base + L::kStats + r * (2 * kRowTile * 4) + row * 4;
            sts_f32(st_out, m);
            sts_f32(st_out + kRowTile * 4, l);
            SA_FWD_ARRIVE(kStReady, rb);
            SA_TR(4 + r, 74);
        }
    }
    // ---------------------------------------------------------------------- teardown
    tc_fence_before();
    __syncthreads();
    SA_PROF_LIFE(t_life);
    if (warp == 16) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

#undef SA_FWD_ARRIVE

}  // namespace tc
}  // namespace sa
