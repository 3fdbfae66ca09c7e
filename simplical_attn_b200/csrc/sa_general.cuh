// General 2-simplicial attention kernels: CUDA-core fp32 arithmetic for any dtype, head dim
// (<= 256) and window.  Every output element is written exactly once, in a fixed order, without atomics.
//
// They cover what the tensor-core kernels do not (fp32 tensors, head dims other than 64/128, unaligned rows,
// very wide K2 windows) and are the on-device cross-check of the tensor-core kernels.
//
// The arithmetic restates the reference's definition (simplicial/reference.py:39-74) with an
// online maximum, and, for the backward, the derivative the reference's backward kernels
// implement (simplicial/kernels.py:175-382 for dQ/dK1/dV1, :386-566 for dK2/dV2).
//
// A block works on tiles of 64 virtual rows (query i, K2 row k) with operand rows A = Q_i * (K2_k + bias) * scale and
// C = dO_i * (V2_k + bias) against tiles of K1/V1 rows, all in shared memory as fp32; a thread holds 4 rows by up to 4
// columns of the score tile and 4 rows by D/16 columns of the accumulators, so an operand read from shared memory is
// used four times.  Large problems are bound by the FMA pipes and shared-memory reads at about equal shares, small ones
// by the latency of a block's chain of loads.  All kernels of a forward and backward together take 141 us for fp32
// B1 N256 H2 D64 w 64/16 and 463 us for bf16 B2 N512 H4 D32 w 32/32; by a warp per output row (sa_general_rows.cuh) 846 and
// 1448 us.  Short windows, which would leave most of a tile empty, go there.
#pragma once

#include <cooperative_groups.h>

#include <type_traits>

#include "sa_common.cuh"
#include "sa_general_rows.cuh"

namespace sa {
namespace general {

constexpr int kThreads = 256;        // 16 x 16
constexpr int kRows = 64;            // virtual rows of a tile
constexpr int kMaxOwners = 16;       // queries (K2 rows) whose virtual rows a tile holds, at most
constexpr int kColRows = 32;         // K1/V1 rows a block of the dK1/dV1 kernel owns

// Shared memory for head dims up to DP: row pitch DP + 4 floats, so that 16-byte reads of consecutive rows fall into
// different banks.
template <int DP>
struct Shape {
    static constexpr int kCols = DP <= 128 ? 64 : 32;       // K1/V1 rows of a tile
    static constexpr int kPitch = DP + 4;
    static constexpr int kPPitch = kCols + 4;
    static constexpr int kUnroll = DP <= 128 ? 16 : 8;      // global loads in flight per thread
    static constexpr int kDpt = DP / 16;                    // accumulator columns per thread and row
    static constexpr int kVec = kDpt < 4 ? kDpt : 4;        // ... in groups of kVec consecutive ones, 16 kVec apart
    static constexpr int kRowTile = kRows * kPitch;         // floats
    static constexpr int kColTile = kCols * kPitch;
    static constexpr int kPTile = kRows * kPPitch;
    static constexpr int kStats = 8 * kRows + 4 * kMaxOwners;
    static constexpr int kFwdBytes = (kRowTile + 2 * kColTile + kPTile + kStats) * 4;
    static constexpr int kBwdBytes = (2 * kRowTile + 2 * kColTile + 2 * kPTile + kStats) * 4;
    static constexpr int kColPPitch = kColRows + 4;
    static constexpr int kColBytes = (2 * kRowTile + 2 * kColRows * kPitch + 2 * kRows * kColPPitch + kStats) * 4;
    static_assert(kBwdBytes <= 227 * 1024 && kColBytes <= 227 * 1024, "shared memory of a block");
};

__device__ __forceinline__ bool not_finite(float x) { return !(fabsf(x) < INFINITY); }

template <int N>
__device__ __forceinline__ void lds_vec(const float* p, float (&v)[N]) {
    if constexpr (N == 4) {
        const float4 t = *(const float4*)p;
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else {
        const float2 t = *(const float2*)p;
        v[0] = t.x; v[1] = t.y;
    }
}

// Rows [r0, r0 + count) of x (row stride xs) -> dst, fp32, zeros behind `avail` rows and behind D.  True if a value is
// not finite.
template <typename T, int DP>
__device__ __forceinline__ bool load_rows(float* dst, const T* __restrict__ x, int64_t xs, int r0, int count, int avail, int D) {
    bool bad = false;
#pragma unroll Shape<DP>::kUnroll
    for (int idx = threadIdx.x; idx < count * DP; idx += kThreads) {
        const int r = idx / DP, d = idx % DP;
        const float v = r < avail && d < D ? to_f<T>(x[(int64_t)(r0 + r) * xs + d]) : 0.f;
        bad |= not_finite(v);
        dst[r * Shape<DP>::kPitch + d] = v;
    }
    return bad;
}

// The operand rows of a tile: dst[r] = (x[ri[r]] * mult) * (y[rk[r]] + bias), zeros where ri[r] < 0.  (In this order, as in
// sa_general_rows.cuh: a scale that brings large inputs into range acts before they are multiplied with each other.)
template <typename T, int DP>
__device__ __forceinline__ void form_rows(float* dst, const int* ri, const int* rk, const T* __restrict__ x, int64_t xs,
                                          const T* __restrict__ y, int64_t ys, float bias, float mult, int D) {
#pragma unroll Shape<DP>::kUnroll
    for (int idx = threadIdx.x; idx < kRows * DP; idx += kThreads) {
        const int r = idx / DP, d = idx % DP;
        float v = 0.f;
        if (ri[r] >= 0 && d < D) v = to_f<T>(x[(int64_t)ri[r] * xs + d]) * mult * (to_f<T>(y[(int64_t)rk[r] * ys + d]) + bias);
        dst[r * Shape<DP>::kPitch + d] = v;
    }
}

// Delta = dO . O and LSE of every row of a tile, four threads to a row.  head_of(r, 0 | 1 | 2): offset of the row's
// head in o, d_o and lse.
template <typename T, typename F>
__device__ __forceinline__ void row_stats(float* delta, float* L, const int* ri, const T* __restrict__ o, int64_t os,
                                          const T* __restrict__ d_o, int64_t dos, const float* __restrict__ lse, int D, F head_of) {
    const int r = threadIdx.x >> 2, part = threadIdx.x & 3;
    float s = 0.f;
    const int i = ri[r];
    if (i >= 0) {
        const T* orow = o + head_of(r, 0) + (int64_t)i * os;
        const T* drow = d_o + head_of(r, 1) + (int64_t)i * dos;
        for (int d0 = part; d0 < D; d0 += 32) {          // (in blocks, as in `product`)
            float t = 0.f;
#pragma unroll
            for (int d = d0; d < d0 + 32; d += 4)
                if (d < D) t = fmaf(to_f<T>(drow[d]), to_f<T>(orow[d]), t);
            s += t;
        }
    }
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    if (part == 0) {
        delta[r] = s;
        L[r] = i >= 0 ? lse[head_of(r, 2) + i] : 0.f;
    }
}

// s[a][c] = X[4 ty + a] . Y[tx + 16 c], summed in blocks of 16 products: a single chain over the head dim made the error of
// dQ and dK2 against 64 bits larger than the row kernels' (fp32 D128 w 100/40: 6.6e-7 and 6.9e-7 against 5.6e-7 and 6.1e-7).
// UNROLL blocks are unrolled: more than one spills where NC is 4.
template <int DP, int NC, int UNROLL = 1>
__device__ __forceinline__ void product(const float* X, const float* Y, int ty, int tx, float (&s)[4][NC]) {
    constexpr int P = Shape<DP>::kPitch;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int c = 0; c < NC; ++c) s[a][c] = 0.f;
#pragma unroll UNROLL
    for (int d0 = 0; d0 < DP; d0 += 16) {
        float t[4][NC];
#pragma unroll
        for (int d = d0; d < d0 + 16; d += 4) {
            float x[4][4];
#pragma unroll
            for (int a = 0; a < 4; ++a) lds_vec<4>(X + (4 * ty + a) * P + d, x[a]);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                float y[4];
                lds_vec<4>(Y + (tx + 16 * c) * P + d, y);
#pragma unroll
                for (int a = 0; a < 4; ++a)
#pragma unroll
                    for (int e = 0; e < 4; ++e) t[a][c] = d == d0 && e == 0 ? x[a][e] * y[e] : fmaf(x[a][e], y[e], t[a][c]);
            }
        }
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int c = 0; c < NC; ++c) s[a][c] += t[a][c];
    }
}

// acc[a][.] += sum over j < n of W[4 ty + a][j] Y[j][.].  CHECK: Y holds values that are not finite; a row that does not
// see column j (W = 0 there) must not meet them.
template <int DP, bool CHECK>
__device__ __forceinline__ void accumulate(float (&acc)[4][Shape<DP>::kDpt], const float* W, const float* Y, int n, int ty, int tx,
                                           const int (&lo)[4], const int (&hi)[4]) {
    using S = Shape<DP>;
    constexpr int V = S::kVec, NV = S::kDpt / V;
#pragma unroll 2
    for (int j = 0; j < n; j += 4) {
        float w[4][4];
#pragma unroll
        for (int a = 0; a < 4; ++a) lds_vec<4>(W + (4 * ty + a) * S::kPPitch + j, w[a]);
#pragma unroll
        for (int jj = 0; jj < 4; ++jj)
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                float y[V];
                lds_vec<V>(Y + (j + jj) * S::kPitch + tx * V + 16 * V * v, y);
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    if (CHECK && (j + jj < lo[a] || j + jj > hi[a])) continue;
#pragma unroll
                    for (int e = 0; e < V; ++e) acc[a][V * v + e] = fmaf(w[a][jj], y[e], acc[a][V * v + e]);
                }
            }
    }
}

// W[4 ty + a][.] = acc * (x[idx[row]] + bias) * mult, zeros where ri < 0.
template <typename T, int DP>
__device__ __forceinline__ void scale_out(float* W, const float (&acc)[4][Shape<DP>::kDpt], const int* ri, const int* idx,
                                          const T* __restrict__ x, int64_t xs, float bias, float mult, int D, int ty, int tx) {
    using S = Shape<DP>;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int r = 4 * ty + a;
#pragma unroll
        for (int e = 0; e < S::kDpt; ++e) {
            const int d = (e / S::kVec) * 16 * S::kVec + tx * S::kVec + e % S::kVec;
            W[r * S::kPitch + d] = ri[r] >= 0 && d < D ? acc[a][e] * ((to_f<T>(x[(int64_t)idx[r] * xs + d]) + bias) * mult) : 0.f;
        }
    }
}

// Calls f with the number of 16-column groups that hold n columns.
template <int MAX, typename F>
__device__ __forceinline__ void with_groups(int n, F&& f) {
    if constexpr (MAX == 1) {
        f(std::integral_constant<int, 1>{});
    } else {
        if (n > 16 * (MAX - 1)) f(std::integral_constant<int, MAX>{});
        else with_groups<MAX - 1>(n, static_cast<F&&>(f));
    }
}

// Columns of the K1/V1 row tile at j0 that query i sees, relative to j0.
__device__ __forceinline__ void window(const KParams& p, int i, int j0, int& lo, int& hi) {
    hi = i < 0 ? -1 : i + p.halo1 - j0;
    lo = i < 0 ? 0 : max(0, i + p.halo1 - p.w1 + 1) - j0;
}

// Forward.  A block owns `owners` consecutive queries of one head (as many as fit 64 rows of w2 each; one, in several
// passes over 64 K2 rows, where w2 > 64).
template <typename T, int DP>
__global__ void __launch_bounds__(kThreads)
fwd_kernel(KParams p, int owners, const T* __restrict__ q, const T* __restrict__ k1, const T* __restrict__ k2,
           const T* __restrict__ v1, const T* __restrict__ v2, T* __restrict__ o, float* __restrict__ lse) {
    using S = Shape<DP>;
    extern __shared__ __align__(16) float sm[];
    float *As = sm, *Ks = As + S::kRowTile, *Vs = Ks + S::kColTile, *Ps = Vs + S::kColTile, *st = Ps + S::kPTile;
    int *ri = (int*)st, *rk = ri + kRows;
    float *row_m = st + 2 * kRows, *row_l = row_m + kRows, *own_m = row_l + kRows, *own_l = own_m + kMaxOwners, *own_f = own_l + kMaxOwners;
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const int nblk = (p.N + owners - 1) / owners;
    const int i0 = (int)(blockIdx.x % nblk) * owners, h = (int)(blockIdx.x / nblk % p.H), b = (int)(blockIdx.x / nblk / p.H);
    const int hk = h / p.G;
    const T* qh = q + b * p.q.b + h * p.q.h;
    const T* k1h = k1 + b * p.k1.b + hk * p.k1.h;
    const T* v1h = v1 + b * p.v1.b + hk * p.v1.h;
    const T* k2h = k2 + b * p.k2.b + hk * p.k2.h;
    const T* v2h = v2 + b * p.v2.b + hk * p.v2.h;
    const int per = min(p.w2, kRows);                   // rows of one owner in a tile
    const int i_last = min(i0 + owners, p.N) - 1;
    const int j_lo = max(0, i0 + p.halo1 - p.w1 + 1), j_hi = i_last + p.halo1;
    float out[DP / 16];                                 // sum over K2 rows, element tid + 256 x of [owners][DP]
#pragma unroll
    for (int x = 0; x < DP / 16; ++x) out[x] = 0.f;
    if (tid < kMaxOwners) { own_m[tid] = -INFINITY; own_l[tid] = 0.f; }
    for (int d0 = 0; d0 < p.w2; d0 += kRows) {
        __syncthreads();
        if (tid < kRows) {
            const int own = tid / per, dlt = d0 + tid % per, i = i0 + own, kb = i + p.halo2 - dlt;
            const bool ok = own < owners && i < p.N && dlt < p.w2 && kb >= 0;
            ri[tid] = ok ? i : -1;
            rk[tid] = kb;
        }
        __syncthreads();
        form_rows<T, DP>(As, ri, rk, qh, p.q.n, k2h, p.k2.n, p.k2_bias, p.scale, p.D);
        float m[4], l[4], t[4][S::kDpt];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            m[a] = -INFINITY;
            l[a] = 0.f;
#pragma unroll
            for (int e = 0; e < S::kDpt; ++e) t[a][e] = 0.f;
        }
        for (int j0 = j_lo; j0 <= j_hi; j0 += S::kCols) {
            const int n = min(j_hi - j0 + 1, S::kCols);
            const int n16 = (n + 15) & ~15;             // columns computed
            __syncthreads();
            load_rows<T, DP>(Ks, k1h, p.k1.n, j0, n16, n, p.D);
            const bool bad = load_rows<T, DP>(Vs, v1h, p.v1.n, j0, n16, n, p.D);
            const bool check = __syncthreads_or(bad);
            int lo[4], hi[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) window(p, ri[4 * ty + a], j0, lo[a], hi[a]);
            with_groups<S::kCols / 16>(n, [&](auto nc) {
                constexpr int NC = decltype(nc)::value;
                float s[4][NC];
                product<DP, NC>(As, Ks, ty, tx, s);
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    float mx = m[a];
#pragma unroll
                    for (int c = 0; c < NC; ++c)
                        if (tx + 16 * c >= lo[a] && tx + 16 * c <= hi[a]) mx = fmaxf(mx, s[a][c]);
#pragma unroll
                    for (int x = 8; x >= 1; x >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
                    const float corr = mx == m[a] ? 1.f : __expf(m[a] - mx);      // m = -inf gives 0
                    m[a] = mx;
                    l[a] *= corr;
#pragma unroll
                    for (int e = 0; e < S::kDpt; ++e) t[a][e] *= corr;
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        const float pv = tx + 16 * c >= lo[a] && tx + 16 * c <= hi[a] ? __expf(s[a][c] - mx) : 0.f;
                        l[a] += pv;
                        Ps[(4 * ty + a) * S::kPPitch + tx + 16 * c] = pv;
                    }
                }
            });
            __syncwarp();                               // a warp reads back the rows it wrote
            if (check) accumulate<DP, true>(t, Ps, Vs, n16, ty, tx, lo, hi);
            else accumulate<DP, false>(t, Ps, Vs, n16, ty, tx, lo, hi);
        }
#pragma unroll
        for (int a = 0; a < 4; ++a) {
#pragma unroll
            for (int x = 8; x >= 1; x >>= 1) l[a] += __shfl_xor_sync(0xffffffffu, l[a], x);
            if (tx == 0) {
                row_m[4 * ty + a] = m[a];
                row_l[4 * ty + a] = l[a];
            }
        }
        __syncthreads();                                // (A is no longer read)
        float* W = As;
        scale_out<T, DP>(W, t, ri, rk, v2h, p.v2.n, p.v2_bias, 1.f, p.D, ty, tx);
        if (tid < owners) {
            float mq = own_m[tid], lq = own_l[tid];
            for (int r = tid * per; r < (tid + 1) * per; ++r)
                if (ri[r] >= 0) mq = fmaxf(mq, row_m[r]);
            const float f = own_m[tid] == mq ? 1.f : __expf(own_m[tid] - mq);      // -inf gives 0
            lq *= f;
            for (int r = tid * per; r < (tid + 1) * per; ++r) {
                const float e = ri[r] >= 0 ? __expf(row_m[r] - mq) : 0.f;
                lq += e * row_l[r];
                row_m[r] = e;                           // from here on the row's weight
            }
            own_m[tid] = mq;
            own_l[tid] = lq;
            own_f[tid] = f;
        }
        __syncthreads();
#pragma unroll
        for (int x = 0; x < DP / 16; ++x) {
            const int own = (tid + kThreads * x) / DP, d = (tid + kThreads * x) % DP;
            if (own < owners) {
                float a = out[x] * own_f[own];
                for (int r = own * per; r < (own + 1) * per; ++r)
                    if (ri[r] >= 0) a = fmaf(row_m[r], W[r * S::kPitch + d], a);
                out[x] = a;
            }
        }
    }
#pragma unroll
    for (int x = 0; x < DP / 16; ++x) {
        const int own = (tid + kThreads * x) / DP, d = (tid + kThreads * x) % DP;
        if (own < owners && i0 + own < p.N && d < p.D)
            o[b * p.o.b + (int64_t)(i0 + own) * p.o.n + h * p.o.h + d] = from_f<T>(out[x] * (1.f / own_l[own]));
    }
    if (tid < owners && i0 + tid < p.N) lse[((long)b * p.H + h) * p.N + i0 + tid] = own_m[tid] + logf(own_l[tid]);
}

// dQ (KV2 = false): a block owns `owners` queries of one head.  dK2 and dV2 (KV2 = true): `owners` K2 rows of one KV
// head, summed over the group's query heads.  Tiles as in the forward.
template <typename T, int DP, bool KV2>
__global__ void __launch_bounds__(kThreads)
bwd_row_kernel(KParams p, int owners, const T* __restrict__ q, const T* __restrict__ k1, const T* __restrict__ k2,
               const T* __restrict__ v1, const T* __restrict__ v2, const T* __restrict__ o, const float* __restrict__ lse,
               const T* __restrict__ d_o, T* __restrict__ dq, T* __restrict__ dk2, T* __restrict__ dv2) {
    using S = Shape<DP>;
    extern __shared__ __align__(16) float sm[];
    float *As = sm, *Cs = As + S::kRowTile, *Ks = Cs + S::kRowTile, *Vs = Ks + S::kColTile;
    float *Ps = Vs + S::kColTile, *Ds = Ps + S::kPTile, *st = Ds + S::kPTile;
    int *ri = (int*)st, *rk = ri + kRows;
    float *delta = st + 2 * kRows, *L = delta + kRows;
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const int n_own = KV2 ? p.n2 : p.N, heads = KV2 ? p.Hkv : p.H;
    const int nblk = (n_own + owners - 1) / owners;
    const int x0 = (int)(blockIdx.x % nblk) * owners, hb = (int)(blockIdx.x / nblk % heads), b = (int)(blockIdx.x / nblk / heads);
    const int hk = KV2 ? hb : hb / p.G;
    const T* k1h = k1 + b * p.k1.b + hk * p.k1.h;
    const T* v1h = v1 + b * p.v1.b + hk * p.v1.h;
    const T* k2h = k2 + b * p.k2.b + hk * p.k2.h;
    const T* v2h = v2 + b * p.v2.b + hk * p.v2.h;
    const int per = min(p.w2, kRows);
    float outg[DP / 16], outu[KV2 ? DP / 16 : 1];
#pragma unroll
    for (int x = 0; x < DP / 16; ++x) {
        outg[x] = 0.f;
        if (KV2) outu[x] = 0.f;
    }
    for (int hq = 0; hq < (KV2 ? p.G : 1); ++hq) {
        const int h = KV2 ? hk * p.G + hq : hb;
        const T* qh = q + b * p.q.b + h * p.q.h;
        const T* doh = d_o + b * p.d_o.b + h * p.d_o.h;
        for (int d0 = 0; d0 < p.w2; d0 += kRows) {
            // queries of the tile's rows
            const int d1 = min(d0 + kRows, p.w2) - 1;
            const int i_lo = KV2 ? max(0, x0 - p.halo2 + d0) : x0;
            const int i_hi = min(p.N - 1, KV2 ? min(x0 + owners, n_own) - 1 - p.halo2 + d1 : x0 + owners - 1);
            if (i_hi < i_lo) continue;                  // (the same for the whole block)
            __syncthreads();
            if (tid < kRows) {
                const int own = tid / per, dlt = d0 + tid % per;
                const int kb = KV2 ? x0 + own : x0 + own + p.halo2 - dlt, i = KV2 ? kb - p.halo2 + dlt : x0 + own;
                const bool ok = own < owners && i >= 0 && i < p.N && dlt < p.w2 && kb >= 0 && kb < p.n2;
                ri[tid] = ok ? i : -1;
                rk[tid] = kb;
            }
            __syncthreads();
            form_rows<T, DP>(As, ri, rk, qh, p.q.n, k2h, p.k2.n, p.k2_bias, p.scale, p.D);
            form_rows<T, DP>(Cs, ri, rk, doh, p.d_o.n, v2h, p.v2.n, p.v2_bias, 1.f, p.D);
            row_stats<T>(delta, L, ri, o, p.o.n, d_o, p.d_o.n, lse, p.D, [&](int, int what) -> int64_t {
                return what == 0 ? b * p.o.b + h * p.o.h : what == 1 ? b * p.d_o.b + h * p.d_o.h : ((int64_t)b * p.H + h) * p.N;
            });
            float g[4][S::kDpt], u[KV2 ? 4 : 1][S::kDpt];
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int e = 0; e < S::kDpt; ++e) {
                    g[a][e] = 0.f;
                    if (KV2) u[a][e] = 0.f;
                }
            const int j_lo = max(0, i_lo + p.halo1 - p.w1 + 1), j_hi = i_hi + p.halo1;
            for (int j0 = j_lo; j0 <= j_hi; j0 += S::kCols) {
                const int n = min(j_hi - j0 + 1, S::kCols);
                const int n16 = (n + 15) & ~15;
                __syncthreads();
                bool bad = load_rows<T, DP>(Ks, k1h, p.k1.n, j0, n16, n, p.D);
                bad |= load_rows<T, DP>(Vs, v1h, p.v1.n, j0, n16, n, p.D);
                const bool check = __syncthreads_or(bad);
                int lo[4], hi[4];
#pragma unroll
                for (int a = 0; a < 4; ++a) window(p, ri[4 * ty + a], j0, lo[a], hi[a]);
                with_groups<S::kCols / 16>(n, [&](auto nc) {
                    constexpr int NC = decltype(nc)::value;
                    float s[4][NC], dp[4][NC];
                    product<DP, NC>(As, Ks, ty, tx, s);
                    product<DP, NC>(Cs, Vs, ty, tx, dp);
#pragma unroll
                    for (int a = 0; a < 4; ++a) {
                        const float la = L[4 * ty + a], de = delta[4 * ty + a];
#pragma unroll
                        for (int c = 0; c < NC; ++c) {
                            const bool ok = tx + 16 * c >= lo[a] && tx + 16 * c <= hi[a];
                            const float pv = ok ? __expf(s[a][c] - la) : 0.f;
                            if (KV2) Ps[(4 * ty + a) * S::kPPitch + tx + 16 * c] = pv;
                            Ds[(4 * ty + a) * S::kPPitch + tx + 16 * c] = ok ? pv * (dp[a][c] - de) : 0.f;
                        }
                    }
                });
                __syncwarp();                           // a warp reads back the rows it wrote
                if (check) accumulate<DP, true>(g, Ds, Ks, n16, ty, tx, lo, hi);
                else accumulate<DP, false>(g, Ds, Ks, n16, ty, tx, lo, hi);
                if constexpr (KV2) {
                    if (check) accumulate<DP, true>(u, Ps, Vs, n16, ty, tx, lo, hi);
                    else accumulate<DP, false>(u, Ps, Vs, n16, ty, tx, lo, hi);
                }
            }
            __syncthreads();                            // (A and C are no longer read)
            if constexpr (KV2) {
                scale_out<T, DP>(As, g, ri, ri, qh, p.q.n, 0.f, p.scale, p.D, ty, tx);
                scale_out<T, DP>(Cs, u, ri, ri, doh, p.d_o.n, 0.f, 1.f, p.D, ty, tx);
            } else {
                scale_out<T, DP>(As, g, ri, rk, k2h, p.k2.n, p.k2_bias, p.scale, p.D, ty, tx);
            }
            __syncthreads();
#pragma unroll
            for (int x = 0; x < DP / 16; ++x) {
                const int own = (tid + kThreads * x) / DP, d = (tid + kThreads * x) % DP;
                if (own < owners)
                    for (int r = own * per; r < (own + 1) * per; ++r) {
                        outg[x] += As[r * S::kPitch + d];
                        if (KV2) outu[x] += Cs[r * S::kPitch + d];
                    }
            }
        }
    }
#pragma unroll
    for (int x = 0; x < DP / 16; ++x) {
        const int own = (tid + kThreads * x) / DP, d = (tid + kThreads * x) % DP, r = x0 + own;
        if (own < owners && r < n_own && d < p.D) {
            if constexpr (KV2) {
                if (dk2) dk2[b * p.dk2.b + (int64_t)r * p.dk2.n + hb * p.dk2.h + d] = from_f<T>(outg[x]);
                if (dv2) dv2[b * p.dv2.b + (int64_t)r * p.dv2.n + hb * p.dv2.h + d] = from_f<T>(outu[x]);
            } else {
                dq[b * p.dq.b + (int64_t)r * p.dq.n + hb * p.dq.h + d] = from_f<T>(outg[x]);
            }
        }
    }
}

// dK1 and dV1.  A cluster owns 32 K1/V1 rows of one KV head; its blocks take the tiles of 64 virtual rows that see them
// (every query head of the group) in turn and add up their sums through distributed shared memory, in a fixed order.
template <typename T, int DP>
__global__ void __launch_bounds__(kThreads)
bwd_col_kernel(KParams p, const T* __restrict__ q, const T* __restrict__ k1, const T* __restrict__ k2, const T* __restrict__ v1,
               const T* __restrict__ v2, const T* __restrict__ o, const float* __restrict__ lse, const T* __restrict__ d_o,
               T* __restrict__ dk1, T* __restrict__ dv1) {
    using S = Shape<DP>;
    constexpr int PP = S::kColPPitch, V = S::kVec, NV = S::kDpt / V, NC = kColRows / 16;
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int nrank = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    extern __shared__ __align__(16) float sm[];
    float *As = sm, *Cs = As + S::kRowTile, *Ks = Cs + S::kRowTile, *Vs = Ks + kColRows * S::kPitch;
    float *Ps = Vs + kColRows * S::kPitch, *Ds = Ps + kRows * PP, *st = Ds + kRows * PP;
    int *ri = (int*)st, *rk = ri + kRows, *rh = rk + kRows;
    float *delta = st + 3 * kRows, *L = delta + kRows;
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const int item = (int)(blockIdx.x / nrank), njt = (p.n1 + kColRows - 1) / kColRows;
    const int j0 = (item % njt) * kColRows, hk = item / njt % p.Hkv, b = item / njt / p.Hkv;
    const int nj = min(kColRows, p.n1 - j0);
    const T* k2h = k2 + b * p.k2.b + hk * p.k2.h;
    const T* v2h = v2 + b * p.v2.b + hk * p.v2.h;
    load_rows<T, DP>(Ks, k1 + b * p.k1.b + hk * p.k1.h, p.k1.n, j0, kColRows, nj, p.D);
    load_rows<T, DP>(Vs, v1 + b * p.v1.b + hk * p.v1.h, p.v1.n, j0, kColRows, nj, p.D);
    float ak[2][S::kDpt], av[2][S::kDpt];               // rows 2 ty, 2 ty + 1 of dK1, dV1
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int e = 0; e < S::kDpt; ++e) ak[a][e] = av[a][e] = 0.f;
    const int i_lo = max(0, j0 - p.halo1), i_hi = min(p.N - 1, j0 + nj - 1 - p.halo1 + p.w1 - 1);
    const int ni = max(0, i_hi - i_lo + 1);
    const long total = (long)p.G * ni * p.w2;           // virtual rows, numbered (head, query, delta)
    for (long v0 = (long)rank * kRows; v0 < total; v0 += (long)nrank * kRows) {
        __syncthreads();
        if (tid < kRows) {
            const long v = v0 + tid;
            const int dlt = (int)(v % p.w2), i = i_lo + (int)(v / p.w2 % ni), hq = (int)(v / p.w2 / ni), kb = i + p.halo2 - dlt;
            ri[tid] = v < total && kb >= 0 ? i : -1;
            rk[tid] = kb;
            rh[tid] = hk * p.G + (v < total ? hq : 0);
        }
        __syncthreads();
        // (as form_rows, with a head for every row)
        bool bad = false;
#pragma unroll 8
        for (int idx = tid; idx < kRows * DP; idx += kThreads) {
            const int r = idx / DP, d = idx % DP, i = ri[r], h = rh[r];
            float a = 0.f, c = 0.f;
            if (i >= 0 && d < p.D) {
                a = to_f<T>(q[b * p.q.b + h * p.q.h + (int64_t)i * p.q.n + d]) * p.scale * (to_f<T>(k2h[(int64_t)rk[r] * p.k2.n + d]) + p.k2_bias);
                c = to_f<T>(d_o[b * p.d_o.b + h * p.d_o.h + (int64_t)i * p.d_o.n + d]) * (to_f<T>(v2h[(int64_t)rk[r] * p.v2.n + d]) + p.v2_bias);
            }
            bad |= not_finite(a) || not_finite(c);
            As[r * S::kPitch + d] = a;
            Cs[r * S::kPitch + d] = c;
        }
        row_stats<T>(delta, L, ri, o, p.o.n, d_o, p.d_o.n, lse, p.D, [&](int r, int what) -> int64_t {
            const int h = rh[r];
            return what == 0 ? b * p.o.b + h * p.o.h : what == 1 ? b * p.d_o.b + h * p.d_o.h : ((int64_t)b * p.H + h) * p.N;
        });
        const bool check = __syncthreads_or(bad);
        float s[4][NC], dp[4][NC];
        product<DP, NC, 4>(As, Ks, ty, tx, s);
        product<DP, NC, 4>(Cs, Vs, ty, tx, dp);
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            int lo, hi;
            window(p, ri[4 * ty + a], j0, lo, hi);
            const float la = L[4 * ty + a], de = delta[4 * ty + a];
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const bool ok = tx + 16 * c >= lo && tx + 16 * c <= hi;
                const float pv = ok ? __expf(s[a][c] - la) : 0.f;
                Ps[(4 * ty + a) * PP + tx + 16 * c] = pv;
                Ds[(4 * ty + a) * PP + tx + 16 * c] = ok ? pv * (dp[a][c] - de) : 0.f;
            }
        }
        __syncthreads();
        auto add = [&](auto check_c) {
            constexpr bool CHECK = decltype(check_c)::value;
#pragma unroll 4
            for (int r = 0; r < kRows; ++r) {
                float w[2], z[2];
                lds_vec<2>(Ps + r * PP + 2 * ty, w);
                lds_vec<2>(Ds + r * PP + 2 * ty, z);
                int lo = 0, hi = kColRows;
                if (CHECK) window(p, ri[r], j0, lo, hi);
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    float x[V], y[V];
                    lds_vec<V>(As + r * S::kPitch + tx * V + 16 * V * v, x);
                    lds_vec<V>(Cs + r * S::kPitch + tx * V + 16 * V * v, y);
#pragma unroll
                    for (int a = 0; a < 2; ++a) {
                        if (CHECK && (2 * ty + a < lo || 2 * ty + a > hi)) continue;      // (as in accumulate)
#pragma unroll
                        for (int e = 0; e < V; ++e) {
                            ak[a][V * v + e] = fmaf(z[a], x[e], ak[a][V * v + e]);
                            av[a][V * v + e] = fmaf(w[a], y[e], av[a][V * v + e]);
                        }
                    }
                }
            }
        };
        if (check) add(std::true_type{});
        else add(std::false_type{});
    }
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int e = 0; e < S::kDpt; ++e) {
            const int d = (e / V) * 16 * V + tx * V + e % V;
            As[(2 * ty + a) * S::kPitch + d] = ak[a][e];
            Cs[(2 * ty + a) * S::kPitch + d] = av[a][e];
        }
    cluster.sync();
    const int rows = kColRows / nrank;                  // this block's share of the 32 rows
    for (int idx = tid; idx < rows * DP; idx += kThreads) {
        const int j = rank * rows + idx / DP, d = idx % DP;
        float a = 0.f, c = 0.f;
        for (int x = 0; x < nrank; ++x) {
            a += cluster.map_shared_rank(As, x)[j * S::kPitch + d];
            c += cluster.map_shared_rank(Cs, x)[j * S::kPitch + d];
        }
        if (j < nj && d < p.D) {
            if (dk1) dk1[b * p.dk1.b + (int64_t)(j0 + j) * p.dk1.n + hk * p.dk1.h + d] = from_f<T>(a);
            if (dv1) dv1[b * p.dv1.b + (int64_t)(j0 + j) * p.dv1.n + hk * p.dv1.h + d] = from_f<T>(c);
        }
    }
    cluster.sync();                                     // the other blocks may still read this one's sums
}

// Consecutive owners whose virtual rows fill a tile; a problem too small to give every multiprocessor a block is cut
// finer.
inline int owners_per_block(const KParams& p, long n_own, long heads, int sm_count) {
    int n = kRows / p.w2 < 1 ? 1 : kRows / p.w2 > kMaxOwners ? kMaxOwners : kRows / p.w2;
    while (n > 1 && (long)p.B * heads * ((n_own + n - 1) / n) < sm_count) n = (n + 1) / 2;
    return n;
}

// Blocks of a cluster of the dK1/dV1 kernel: enough of them for every multiprocessor, as long as each has tiles to work on.
inline long col_tiles(const KParams& p) {
    return ((long)p.G * (p.w1 + kColRows < p.N ? p.w1 + kColRows : p.N) * p.w2 + kRows - 1) / kRows;
}
inline int col_cluster(const KParams& p, int sm_count) {
    const long items = (long)p.B * p.Hkv * ((p.n1 + kColRows - 1) / kColRows), tiles = col_tiles(p);
    int nrank = 1;
    while (nrank < 8 && items * nrank * 2 <= 2L * sm_count && nrank * 2 <= tiles) nrank *= 2;
    return nrank;
}

// Tiles or a warp per output row: the smaller of two estimates, in us, with constants measured on a B200 over 637 problems
// (head dims 8 ... 256, windows 1 ... 1024 / 1 ... 160, sequences of 1 ... 4096 rows, among them 200 of the usual sizes): the
// faster of the two kernels within 5 % in 95 % of them, at worst 0.59 of its speed (short launches).
//   rows:  0.14 R + max(wait (pairs + o outer) of the longest row, pair R (pairs + o outer) of the mean row), with R output
//          rows (warps) per multiprocessor, a row's (j, k) pairs and outer steps (K2 rows, or for dK1/dV1 queries);
//   tiles: max(first, blocks per multiprocessor) x (passes x (tile + group x 16-column groups)), for dK1/dV1
//          (tile + group x tiles), where `first` is what a launch of few blocks takes.
// Long windows always go by tiles: no warp per row was measured to be the faster one there, and the estimate does not
// hold for them (their rows no longer stay in the caches).
enum Kernel { kFwd = 0, kDq = 1, kKv1 = 2, kKv2 = 3 };
struct Cost {
    double pair[4], o, wait, tile[4], group[4];      // [4]: by padded head dim 32, 64, 128, 256
};
constexpr Cost kCost[4] = {
    {{.013, .013, .019, .030}, .48, .28, {4.3, 6.1, 19, 27}, {.72, 1.1, 2.0, 5.4}},
    {{.013, .014, .018, .032}, .71, .27, {4.1, 7.5, 21, 38}, {.93, 1.4, 2.8, 7.5}},
    {{.013, .015, .022, .079}, 1.7, .24, {3.0, 3.3, 10, 12}, {4.6, 7.8, 20, 44}},
    {{.013, .016, .021, .051}, 1.7, .25, {4.5, 13, 23, 44}, {1.3, 2.2, 4.1, 10}},
};

// K1 (K2) rows that a query sees, averaged over the queries: windows are cut at the first row that exists.
inline double mean_window(const KParams& p, int w, int halo) {
    const double n = p.N, cut = w - halo < 0 ? 0 : w - halo < p.N ? w - halo : p.N;
    return (cut * (cut + 1) / 2 + cut * halo + (n - cut) * w) / n;
}

inline bool by_rows(Kernel kernel, const KParams& p, int sm_count) {
    const Cost& c = kCost[kernel];
    const int d = p.D <= 32 ? 0 : p.D <= 64 ? 1 : p.D <= 128 ? 2 : 3;
    const int n_out = kernel == kKv1 ? p.n1 : kernel == kKv2 ? p.n2 : p.N;
    const double heads = kernel < kKv1 ? p.H : p.Hkv, group = kernel < kKv1 ? 1 : p.G;
    if ((double)p.w1 * p.w2 > 3300 || (kernel == kKv1 && p.w1 > 24)) return false;
    const double m1 = mean_window(p, p.w1, p.halo1), m2 = mean_window(p, p.w2, p.halo2), per = group * p.N / n_out;
    const double warps = p.B * heads * n_out / sm_count;
    const double longest = c.wait * group * ((double)p.w1 * p.w2 + c.o * (kernel == kKv1 ? p.w1 : p.w2));
    const double rows = .14 * warps + fmax(longest, c.pair[d] * warps * per * (m1 * m2 + c.o * (kernel == kKv1 ? m1 : m2)));
    double blocks, tiles;
    if (kernel == kKv1) {
        const int nrank = col_cluster(p, sm_count);
        blocks = p.B * heads * ((n_out + kColRows - 1) / kColRows) * nrank;
        tiles = c.tile[d] + c.group[d] * ((col_tiles(p) + nrank - 1) / nrank);
    } else {
        const int owners = owners_per_block(p, n_out, (long)heads, sm_count);
        const long span = p.w1 + (kernel == kKv2 ? owners + (p.w2 < kRows ? p.w2 : kRows) - 2 : owners - 1);
        blocks = p.B * heads * ((n_out + owners - 1) / owners);
        tiles = group * ((p.w2 + kRows - 1) / kRows) * (c.tile[d] + c.group[d] * (((span < p.n1 ? span : p.n1) + 15) / 16));
    }
    return rows <= fmax(d < 2 ? 1.75 : 1, blocks / sm_count) * tiles;
}

template <typename T, int DP>
cudaError_t launch_fwd_t(const KParams& p, const void* q, const void* k1, const void* k2, const void* v1,
                         const void* v2, void* o, float* lse, int sm_count, cudaStream_t st) {
    if (by_rows(kFwd, p, sm_count)) {
        row_fwd_kernel<T, DP / 32><<<row_blocks((long)p.B * p.H * p.N), kWarpsPerBlock * 32, 0, st>>>(p, (const T*)q, (const T*)k1, (const T*)k2,
                                                                                                      (const T*)v1, (const T*)v2, (T*)o, lse);
        return cudaGetLastError();
    }
    const int owners = owners_per_block(p, p.N, p.H, sm_count);
    const long blocks = (long)p.B * p.H * ((p.N + owners - 1) / owners);
    if (!allow_dynamic_smem((const void*)fwd_kernel<T, DP>, Shape<DP>::kFwdBytes)) return cudaErrorInvalidValue;
    fwd_kernel<T, DP><<<(unsigned)blocks, kThreads, Shape<DP>::kFwdBytes, st>>>(p, owners, (const T*)q, (const T*)k1, (const T*)k2,
                                                                                (const T*)v1, (const T*)v2, (T*)o, lse);
    return cudaGetLastError();
}

template <typename T, int DP>
cudaError_t launch_bwd_t(const KParams& p, const void* q, const void* k1, const void* k2, const void* v1,
                         const void* v2, const void* o, const float* lse, const void* d_o, void* dq, void* dk1,
                         void* dk2, void* dv1, void* dv2, int sm_count, cudaStream_t st) {
    using S = Shape<DP>;
    if (dq && by_rows(kDq, p, sm_count)) {
        row_dq_kernel<T, DP / 32><<<row_blocks((long)p.B * p.H * p.N), kWarpsPerBlock * 32, 0, st>>>(
            p, (const T*)q, (const T*)k1, (const T*)k2, (const T*)v1, (const T*)v2, (const T*)o, lse, (const T*)d_o, (T*)dq);
    } else if (dq) {
        const int owners = owners_per_block(p, p.N, p.H, sm_count);
        auto kern = bwd_row_kernel<T, DP, false>;
        if (!allow_dynamic_smem((const void*)kern, S::kBwdBytes)) return cudaErrorInvalidValue;
        kern<<<(unsigned)((long)p.B * p.H * ((p.N + owners - 1) / owners)), kThreads, S::kBwdBytes, st>>>(
            p, owners, (const T*)q, (const T*)k1, (const T*)k2, (const T*)v1, (const T*)v2, (const T*)o, lse, (const T*)d_o, (T*)dq,
            (T*)nullptr, (T*)nullptr);
    }
    if ((dk1 || dv1) && by_rows(kKv1, p, sm_count)) {
        row_kv1_kernel<T, DP / 32><<<row_blocks((long)p.B * p.Hkv * p.n1), kWarpsPerBlock * 32, 0, st>>>(
            p, (const T*)q, (const T*)k1, (const T*)k2, (const T*)v1, (const T*)v2, (const T*)o, lse, (const T*)d_o, (T*)dk1, (T*)dv1);
    } else if (dk1 || dv1) {
        auto kern = bwd_col_kernel<T, DP>;
        if (!allow_dynamic_smem((const void*)kern, S::kColBytes)) return cudaErrorInvalidValue;
        const long items = (long)p.B * p.Hkv * ((p.n1 + kColRows - 1) / kColRows);
        const int nrank = col_cluster(p, sm_count);
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)(items * nrank));
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = S::kColBytes;
        cfg.stream = st;
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = (unsigned)nrank;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, p, (const T*)q, (const T*)k1, (const T*)k2, (const T*)v1, (const T*)v2,
                                                 (const T*)o, lse, (const T*)d_o, (T*)dk1, (T*)dv1);
        if (e != cudaSuccess) return e;
    }
    if ((dk2 || dv2) && by_rows(kKv2, p, sm_count)) {
        row_kv2_kernel<T, DP / 32><<<row_blocks((long)p.B * p.Hkv * p.n2), kWarpsPerBlock * 32, 0, st>>>(
            p, (const T*)q, (const T*)k1, (const T*)k2, (const T*)v1, (const T*)v2, (const T*)o, lse, (const T*)d_o, (T*)dk2, (T*)dv2);
    } else if (dk2 || dv2) {
        const int owners = owners_per_block(p, p.n2, p.Hkv, sm_count);
        auto kern = bwd_row_kernel<T, DP, true>;
        if (!allow_dynamic_smem((const void*)kern, S::kBwdBytes)) return cudaErrorInvalidValue;
        kern<<<(unsigned)((long)p.B * p.Hkv * ((p.n2 + owners - 1) / owners)), kThreads, S::kBwdBytes, st>>>(
            p, owners, (const T*)q, (const T*)k1, (const T*)k2, (const T*)v1, (const T*)v2, (const T*)o, lse, (const T*)d_o,
            (T*)nullptr, (T*)dk2, (T*)dv2);
    }
    return cudaGetLastError();
}

// Dispatch on dtype and head dim (padded to 32, 64, 128 or 256).
#define SA_GENERAL_DISPATCH(FN, ...)                                                         \
    do {                                                                                     \
        const int epl = (p.D + 31) / 32;                                                     \
        const int key = dtype * 16 + (epl <= 1 ? 1 : epl <= 2 ? 2 : epl <= 4 ? 4 : 8);       \
        switch (key) {                                                                       \
            case 0 * 16 + 1: return FN<__nv_bfloat16, 32>(__VA_ARGS__);                      \
            case 0 * 16 + 2: return FN<__nv_bfloat16, 64>(__VA_ARGS__);                      \
            case 0 * 16 + 4: return FN<__nv_bfloat16, 128>(__VA_ARGS__);                     \
            case 0 * 16 + 8: return FN<__nv_bfloat16, 256>(__VA_ARGS__);                     \
            case 1 * 16 + 1: return FN<__half, 32>(__VA_ARGS__);                             \
            case 1 * 16 + 2: return FN<__half, 64>(__VA_ARGS__);                             \
            case 1 * 16 + 4: return FN<__half, 128>(__VA_ARGS__);                            \
            case 1 * 16 + 8: return FN<__half, 256>(__VA_ARGS__);                            \
            case 2 * 16 + 1: return FN<float, 32>(__VA_ARGS__);                              \
            case 2 * 16 + 2: return FN<float, 64>(__VA_ARGS__);                              \
            case 2 * 16 + 4: return FN<float, 128>(__VA_ARGS__);                             \
            case 2 * 16 + 8: return FN<float, 256>(__VA_ARGS__);                             \
            default: return cudaErrorInvalidValue;                                           \
        }                                                                                    \
    } while (0)

inline cudaError_t launch_fwd(int dtype, const KParams& p, const void* q, const void* k1, const void* k2,
                              const void* v1, const void* v2, void* o, float* lse, int sm_count, cudaStream_t st) {
    SA_GENERAL_DISPATCH(launch_fwd_t, p, q, k1, k2, v1, v2, o, lse, sm_count, st);
}

inline cudaError_t launch_bwd(int dtype, const KParams& p, const void* q, const void* k1, const void* k2,
                              const void* v1, const void* v2, const void* o, const float* lse, const void* d_o,
                              void* dq, void* dk1, void* dk2, void* dv1, void* dv2, int sm_count, cudaStream_t st) {
    SA_GENERAL_DISPATCH(launch_bwd_t, p, q, k1, k2, v1, v2, o, lse, d_o, dq, dk1, dk2, dv1, dv2, sm_count, st);
}

}  // namespace general
}  // namespace sa
