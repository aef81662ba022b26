// Device kernels of the supernodal multifrontal complex-symmetric LDL^T and
// its solves, templated on the real type R (double: complex128 factor;
// float: complex64 factor). No conjugation anywhere: the matrices are complex
// symmetric (A = A^T), so every product below is a plain transpose product.
//
// Front layout. Supernode s owns columns [first, first + w) of the
// post-ordered matrix and the sorted row structure struct_s (m rows, the
// first w being its own columns). Its front is m x m; the first w columns
// live in the panel L_s (m x w, column-major, leading dimension m, inside the
// factor storage), the trailing (m - w) x (m - w) block -- the contribution
// block CB_s -- in the CB pool. After factorization the panel holds D on its
// diagonal and the multipliers below it.
#pragma once

#include <cuda_runtime.h>

#include <cfloat>
#include <type_traits>

#include "analysis.hpp"
#include "common.cuh"
#include "i8_update.cuh"
#include "tc_update.cuh"

namespace aphi_b200 {

template <class R>
struct cx {
    R re, im;
};

template <class R>
__device__ __forceinline__ cx<R> operator*(cx<R> a, cx<R> b) {
    return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}
template <class R>
__device__ __forceinline__ cx<R> operator+(cx<R> a, cx<R> b) {
    return {a.re + b.re, a.im + b.im};
}
template <class R>
__device__ __forceinline__ cx<R> operator-(cx<R> a, cx<R> b) {
    return {a.re - b.re, a.im - b.im};
}
// a - b * c
template <class R>
__device__ __forceinline__ cx<R> fms(cx<R> a, cx<R> b, cx<R> c) {
    return {a.re - b.re * c.re + b.im * c.im, a.im - b.re * c.im - b.im * c.re};
}
// 1 / d, scaled so that neither component over- nor underflows for ordinary d.
template <class R>
__device__ __forceinline__ cx<R> crecip(cx<R> d) {
    if (fabs(d.re) >= fabs(d.im)) {
        const R r = d.im / d.re;
        const R den = d.re + d.im * r;
        return {R(1) / den, -r / den};
    }
    const R r = d.re / d.im;
    const R den = d.re * r + d.im;
    return {r / den, R(-1) / den};
}
template <class R>
__device__ __forceinline__ double cabs_d(cx<R> a) {
    return hypot(static_cast<double>(a.re), static_cast<double>(a.im));
}

struct Sched {
    const int* first;
    const int* rows;
    const long long* loff;
    const long long* cboff;
    const long long* soff;
    const int* structs;
    const long long* reloff;
    const int* rel;
    const int* child_ptr;
    const int* child_list;
    const long long* uoff;
    const Item* items;
};

inline Sched sched_of(const DeviceSchedule& d) {
    return Sched{d.first, d.rows, d.loff, d.cboff, d.soff, d.structs, d.reloff, d.rel,
                 d.child_ptr, d.child_list, d.uoff, d.items};
}

// ---------------------------------------------------------------- 64 x 64 blocks
// Blocks of L in shared memory have leading dimension kTriLd (65: column-
// strided reads fall in distinct banks).
constexpr int kTriLd = kSolveBlock + 1;
constexpr int kTriSmem = kSolveBlock * kTriLd;  // complex entries

// A block of L (rows x cols at P, leading dimension m) into shared memory T
// (leading dimension kTriLd, zeros outside the rows x cols block) by
// asynchronous copies (cp.async, zero-filled where the source size is 0), so
// the caller's own loads overlap them; the caller waits with
// triangle_wait() and a __syncthreads() before reading T.
__device__ __forceinline__ void cp_async_entry(uint32_t dst, const cx<double>* src, bool in) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16u : 0u) : "memory");
}
__device__ __forceinline__ void cp_async_entry(uint32_t dst, const cx<float>* src, bool in) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(in ? 8u : 0u) : "memory");
}
template <class R>
__device__ __forceinline__ void stage_block(cx<R>* T, const cx<R>* P, long long m, int rows, int cols) {
#pragma unroll 4
    for (int e = threadIdx.x; e < kSolveBlock * kSolveBlock; e += blockDim.x) {
        const int i = e % kSolveBlock, j = e / kSolveBlock;
        const bool in = i < rows && j < cols;
        cp_async_entry(smem_u32(T + i + j * kTriLd), in ? P + i + static_cast<long long>(j) * m : P, in);
    }
    cp_async_commit();
}
__device__ __forceinline__ void triangle_wait() { cp_async_wait<0>(); }

// ---------------------------------------------------------------- extend-add
// Item (s, c0): front columns [c0, c0 + 32) of supernode s, of which block z of
// gridDim.z takes every gridDim.z-th eight. Every entry becomes itself (L) or
// zero (CB) plus its children's contribution block entries, children in
// ascending order (a fixed summation order).
//
// Bound by memory: latency low in the tree, traffic at its top. The block turns
// two children's row maps around (front row -> child row, kEaRows rows at a
// time, in shared memory, and before it waits for the launch before it: the maps
// never change); then an entry is gathered from both, several of a thread at
// once, and written once. Scattering child by child instead (binary searches
// for the child's columns, a pass of zeros, a read and a write per entry and
// child, a barrier per child) took 28 us a launch on 8^3, where this takes 12;
// for eight matrices of 24^3 24 ms FP64, now 17.7, of about 12 that one read and
// one write of the children's blocks take; for six of 32^3 in FP32 39.5 ms,
// now 25. Three blocks a multiprocessor are best in FP64 (four 18.6 ms, two 21;
// with twice the entries in flight 19.8); in FP32 fewer entries in flight or a
// bound on the registers cost 10 %.
constexpr int kEaRows = 4096, kEaKids = 2;
static_assert(kEaKids == 2, "an entry's two maps are named");
template <class R>
__global__ void __launch_bounds__(256, sizeof(R) == 8 ? 3 : 0) k_extend_add(Sched S, long long item0, cx<R>* Lb, cx<R>* CBb,
                                                    long long lstride, long long cbstride) {
    constexpr int kUnroll = sizeof(R) == 8 ? 2 : 4;  // entries of a thread in flight
    __shared__ int row_of[kEaKids][kEaRows];  // front row r0 + i -> child row, or -1
    __shared__ int col_of[kEaKids][kEaCols];  // front column c0 + i -> child column, or -1
    pdl_start_next();
    const Item it = S.items[item0 + blockIdx.x];
    const int s = it.s, c0 = it.a;
    cx<R>* L = Lb + lstride * blockIdx.y;
    cx<R>* CB = CBb + cbstride * blockIdx.y;
    const int w = S.first[s + 1] - S.first[s];
    const int m = S.rows[s];
    const int cs = m - w;
    const int c1 = min(c0 + kEaCols, m);
    cx<R>* Ls = L + S.loff[s];
    cx<R>* CBs = CB + (cs > 0 ? S.cboff[s] : 0);
    const int t0 = S.child_ptr[s], t1 = S.child_ptr[s + 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    bool waited = false;
    for (int r0 = c0; r0 < m; r0 += kEaRows) {
        const int r1 = min(r0 + kEaRows, m);
        for (int t = t0; t == t0 || t < t1; t += kEaKids) {
            const int kids = min(kEaKids, t1 - t);
            const cx<R>* kid_cb[kEaKids];
            int kid_rows[kEaKids];
            for (int k = 0; k < kids; ++k)
                for (int i = threadIdx.x; i < r1 - r0; i += 256) row_of[k][i] = -1;
            if (threadIdx.x < kEaKids * kEaCols) col_of[threadIdx.x / kEaCols][threadIdx.x % kEaCols] = -1;
            __syncthreads();
#pragma unroll
            for (int k = 0; k < kEaKids; ++k) {
                kid_cb[k] = CB;
                kid_rows[k] = 0;
                if (k >= kids) continue;
                const int c = S.child_list[t + k];
                const int cc = S.rows[c] - (S.first[c + 1] - S.first[c]);
                if (cc <= 0) continue;
                const int* rel = S.rel + S.reloff[c];
                kid_cb[k] = CB + S.cboff[c];
                kid_rows[k] = cc;
                for (int i = threadIdx.x; i < cc; i += 256) {
                    const int r = rel[i];
                    if (r >= r0 && r < r1) row_of[k][r - r0] = i;
                    if (r >= c0 && r < c1) col_of[k][r - c0] = i;
                }
            }
            if (!waited) pdl_wait();
            waited = true;
            __syncthreads();
            for (int j = c0 + warp + 8 * blockIdx.z; j < c1; j += 8 * gridDim.z) {
                const bool in_l = j < w;
                const bool fresh = !in_l && t == t0;  // starts from zero
                const cx<R>* src[kEaKids];
                bool live[kEaKids], any = false;
#pragma unroll
                for (int k = 0; k < kEaKids; ++k) {
                    const int cj = col_of[k][j - c0];
                    live[k] = cj >= 0;
                    any |= live[k];
                    src[k] = kid_cb[k] + static_cast<long long>(max(cj, 0)) * kid_rows[k];
                }
                if (!any && !fresh) continue;
                cx<R>* dst = in_l ? Ls + static_cast<long long>(j) * m : CBs + static_cast<long long>(j - w) * cs - w;
                for (int rb = max(j, r0) + lane; rb < r1; rb += 32 * kUnroll) {
                    int at[kUnroll][kEaKids];
                    cx<R> v[kUnroll], x[kUnroll][kEaKids];
#pragma unroll
                    for (int u = 0; u < kUnroll; ++u) {
                        const int r = rb + 32 * u;
#pragma unroll
                        for (int k = 0; k < kEaKids; ++k) {
                            at[u][k] = live[k] && r < r1 ? row_of[k][r - r0] : -1;
                            if (at[u][k] >= 0) x[u][k] = src[k][at[u][k]];
                        }
                        v[u] = cx<R>{0, 0};
                        if (!fresh && max(at[u][0], at[u][1]) >= 0) v[u] = dst[r];
                    }
#pragma unroll
                    for (int u = 0; u < kUnroll; ++u) {
                        const int r = rb + 32 * u;
#pragma unroll
                        for (int k = 0; k < kEaKids; ++k)
                            if (at[u][k] >= 0) v[u] = v[u] + x[u][k];
                        if (r < r1 && (fresh || max(at[u][0], at[u][1]) >= 0)) dst[r] = v[u];
                    }
                }
            }
            __syncthreads();
        }
    }
}

// ---------------------------------------------------------------- small fronts
// 1 / d by one division where |d|^2 is far from the type's limits.
__device__ __forceinline__ cx<double> crecip_fast(cx<double> d) {
    const double n = d.re * d.re + d.im * d.im;
    if (!(n > 1e-250 && n < 1e250)) return crecip(d);
    const double r = 1.0 / n;
    return {d.re * r, -d.im * r};
}
__device__ __forceinline__ cx<float> crecip_fast(cx<float> d) {
    const float n = d.re * d.re + d.im * d.im;
    if (!(n > 1e-30f && n < 1e30f)) return crecip(d);
    const float r = 1.0f / n;
    return {d.re * r, -d.im * r};
}

// The right-looking LDL^T of the leading w columns of an m x m lower triangle F
// in shared memory (leading dimension ld, m <= 32 H), by 256 threads. The
// triangle sits in registers: lane l holds rows l + 32 h, warp v the columns
// v + 8 c, and a step needs one column of it in shared memory, which its warp
// publishes at the end of the step before. So a column costs one barrier, its
// pivot's reciprocal and a burst of independent updates. (With the triangle in
// shared memory a step's loads, one entry after the other, made it 0.8-0.9 us;
// unrolled over a block's columns instead, the code itself is fetched once a
// launch and takes as long.) The columns' registers move down as blocks of
// eight are finished, so that every register index is a constant in a short
// loop. Columns stay unscaled in F: the multipliers are F[i, j] inv[j].
// Measured per launch: 64-column diagonal blocks of 24^3 (eight FP64 entries)
// 39 us, FP32 29 us, against 24 and 19 us for each 32 columns before; one-CTA
// fronts of 8^3 29 us (52).
constexpr int kLdltThreads = 256;
template <int H, class R>
__device__ __forceinline__ void ldlt_columns(cx<R>* F, int ld, int m, int w, cx<R>* inv) {
    constexpr int C = 4 * H;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    cx<R> a[C][H];
#pragma unroll
    for (int c = 0; c < C; ++c)
#pragma unroll
        for (int h = 0; h < H; ++h) {
            const int i = lane + 32 * h, j = warp + 8 * c;
            a[c][h] = i < m && j <= i ? F[i + j * ld] : cx<R>{0, 0};
        }
    for (int k = 0; k < w; ++k) {
        const cx<R>* col = F + k * ld;
        const int base = k & ~7;
        const cx<R> r = crecip_fast(col[k]);
        if (threadIdx.x == 0) inv[k] = r;
        cx<R> x[H];
#pragma unroll
        for (int h = 0; h < H; ++h) x[h] = lane + 32 * h < m ? col[lane + 32 * h] : cx<R>{0, 0};
        // Half of the columns at a time, without branches between them: their
        // loads are in flight together (past the triangle: the last row's).
        auto update = [&](auto half) {
            constexpr int c0 = half.value * C / 2;
            cx<R> l[C / 2];
#pragma unroll
            for (int c = 0; c < C / 2; ++c) l[c] = col[min(warp + base + 8 * (c0 + c), m - 1)];
#pragma unroll
            for (int c = 0; c < C / 2; ++c) {
                l[c] = l[c] * r;
#pragma unroll
                for (int h = 0; h < H; ++h) a[c0 + c][h] = fms(a[c0 + c][h], x[h], l[c]);
            }
        };
        update(std::integral_constant<int, 0>{});
        if (base + 4 * C < m) update(std::integral_constant<int, 1>{});
        if (k + 1 < w && warp == ((k + 1) & 7)) {
            const bool same = (k & 7) != 7;  // the next column's block of eight
#pragma unroll
            for (int h = 0; h < H; ++h)
                if (lane + 32 * h < m && lane + 32 * h > k) F[lane + 32 * h + (k + 1) * ld] = same ? a[0][h] : a[1][h];
        }
        if ((k & 7) == 7)
#pragma unroll
            for (int c = 0; c + 1 < C; ++c)
#pragma unroll
                for (int h = 0; h < H; ++h) a[c][h] = a[c + 1][h];
        __syncthreads();
    }
    // What is left of the triangle: columns w ..
#pragma unroll
    for (int c = 0; c < C; ++c)
#pragma unroll
        for (int h = 0; h < H; ++h) {
            const int i = lane + 32 * h, j = warp + (w & ~7) + 8 * c;
            if (j >= w && j <= i && i < m) F[i + j * ld] = a[c][h];
        }
    __syncthreads();
}

// One CTA factorizes a whole front (m <= 96) in shared memory.
template <class R>
constexpr int small_smem(int rows) { return rows * (rows | 1) * static_cast<int>(sizeof(cx<R>)); }
template <class R>
__global__ void __launch_bounds__(kLdltThreads) k_small_front(Sched S, long long item0, cx<R>* Lb, cx<R>* CBb,
                                                     long long lstride, long long cbstride) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ cx<R> inv[96];
    pdl_start_next();
    const int s = S.items[item0 + blockIdx.x].s;
    const int w = S.first[s + 1] - S.first[s];
    const int m = S.rows[s];
    const int cs = m - w;
    const int ld = m | 1;
    cx<R>* F = reinterpret_cast<cx<R>*>(smem_raw);
    cx<R>* Ls = Lb + lstride * blockIdx.y + S.loff[s];
    cx<R>* CBs = CBb + cbstride * blockIdx.y + (cs > 0 ? S.cboff[s] : 0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    auto at = [&](int i, int j) {
        return j < w ? Ls + i + static_cast<long long>(j) * m : CBs + (i - w) + static_cast<long long>(j - w) * cs;
    };
    pdl_wait();
#pragma unroll 4
    for (int j = warp; j < m; j += nw)
        for (int i = j + lane; i < m; i += 32) F[i + j * ld] = *at(i, j);
    __syncthreads();
    if (m <= 32)
        ldlt_columns<1>(F, ld, m, w, inv);
    else if (m <= 64)
        ldlt_columns<2>(F, ld, m, w, inv);
    else
        ldlt_columns<3>(F, ld, m, w, inv);
    for (int j = warp; j < m; j += nw)
        for (int i = j + lane; i < m; i += 32) *at(i, j) = j < w && i > j ? F[i + j * ld] * inv[j] : F[i + j * ld];
}

// ---------------------------------------------------------------- blocked fronts
// A front's panels advance 64 columns a step: the step's diagonal block, the
// rows below it, then the rest of the panel's own columns.

// Step k0 of a large front: factor the kb x kb diagonal block (kb <= 64) in place.
constexpr int kDiagThreads = kLdltThreads;
template <class R>
constexpr int diag_smem() { return (kTriSmem + kStep) * static_cast<int>(sizeof(cx<R>)); }
template <class R>
__global__ void __launch_bounds__(kDiagThreads) k_diag_block(Sched S, long long item0, cx<R>* Lb, long long lstride) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cx<R>* T = reinterpret_cast<cx<R>*>(smem_raw);
    cx<R>* inv = T + kTriSmem;  // reciprocals of the pivots
    pdl_start_next();
    const Item it = S.items[item0 + blockIdx.x];
    const int s = it.s, k0 = it.a;
    const int w = S.first[s + 1] - S.first[s];
    const int m = S.rows[s];
    const int kb = min(kStep, w - k0);
    cx<R>* D = Lb + lstride * blockIdx.y + S.loff[s] + k0 + static_cast<long long>(k0) * m;
    pdl_wait();
    stage_block(T, D, m, kb, kb);
    triangle_wait();
    __syncthreads();
    if (kb <= 32)
        ldlt_columns<1>(T, kTriLd, kb, kb, inv);
    else
        ldlt_columns<2>(T, kTriLd, kb, kb, inv);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int j = warp; j < kb; j += kDiagThreads / 32)
        for (int i = j + lane; i < kb; i += 32)
            D[i + static_cast<long long>(j) * m] = i > j ? T[i + j * kTriLd] * inv[j] : T[i + j * kTriLd];
}

// Rows row0 .. row0 + 63 of the panel below the diagonal block of step k0:
// L21 = A21 L11^-T D^-1. Four neighbouring lanes take two rows, 32 apart; 16
// columns at a time, lane q of them holding four (4 u + q) of either row in
// registers: first the finished columns' products (left-looking, their values
// in shared memory), then the 16 columns' own chain, each value broadcast to
// the rows' lanes. Where rows are many, shared memory bounds it: six loads for
// eight complex multiply-adds (with a row per four lanes five for four: 24^3,
// eight FP64 entries, 75 us a launch against 63). L11 is kept as its lower triangle by blocks of 16
// columns, which leaves room for two CTAs per SM (four in FP32).
constexpr int kTrsmCols = 16, kTrsmThreads = 2 * kTrsmRows;
// Entry (row, col) of L11, row >= 16 (col / 16): block b's columns are 64 - 16 b long.
__device__ __forceinline__ int trsm_block(int b) { return kTrsmCols * (kStep * b - kTrsmCols * b * (b - 1) / 2); }
constexpr int kTrsmTri = kTrsmCols * (64 + 48 + 32 + 16);
template <class R>
constexpr int trsm_smem() { return (kTrsmTri + kStep + 48 * (kTrsmRows + 1)) * static_cast<int>(sizeof(cx<R>)); }
template <class R>
__global__ void __launch_bounds__(kTrsmThreads) k_panel_trsm(Sched S, long long item0, cx<R>* Lb,
                                                                 long long lstride) {
    static_assert(kStep == 64, "four blocks of 16 columns");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cx<R>* T = reinterpret_cast<cx<R>*>(smem_raw);
    cx<R>* Dinv = T + kTrsmTri;
    cx<R>* X = Dinv + kStep;  // [column][row]: the rows' finished columns, unscaled
    constexpr int kLdX = kTrsmRows + 1;
    pdl_start_next();
    const Item it = S.items[item0 + blockIdx.x];
    const int s = it.s, k0 = it.a, row0 = it.b;
    const int w = S.first[s + 1] - S.first[s];
    const int m = S.rows[s];
    const int kb = min(kStep, w - k0);
    cx<R>* P = Lb + lstride * blockIdx.y + S.loff[s] + static_cast<long long>(k0) * m;  // column k0 of the panel
    const int q = threadIdx.x & 3, quad = threadIdx.x & 28, r = threadIdx.x >> 2, i = row0 + r;
    constexpr int kApart = kTrsmRows / 2;
    auto load = [&](int c0, cx<R> (&x)[2][4]) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int c = c0 + 4 * u + q;
                x[h][u] = i + kApart * h < m && c < kb ? P[i + kApart * h + static_cast<long long>(c) * m] : cx<R>{0, 0};
            }
    };
    pdl_wait();
#pragma unroll 4
    for (int e = threadIdx.x; e < kStep * kStep; e += kTrsmThreads) {
        const int row = e % kStep, col = e / kStep, b = col / kTrsmCols;
        if (row < b * kTrsmCols) continue;
        const bool in = row < kb && col < kb;
        cp_async_entry(smem_u32(T + trsm_block(b) + (row - b * kTrsmCols) + (col % kTrsmCols) * (kStep - b * kTrsmCols)),
                       in ? P + k0 + row + static_cast<long long>(col) * m : P, in);
    }
    cp_async_commit();
    cx<R> x[2][4], ahead[2][4];
    load(0, ahead);
    triangle_wait();
    __syncthreads();
    if (threadIdx.x < kb) {
        const int b = threadIdx.x / kTrsmCols, c = threadIdx.x % kTrsmCols;
        Dinv[threadIdx.x] = crecip(T[trsm_block(b) + c + c * (kStep - b * kTrsmCols)]);
    }
    __syncthreads();
#pragma unroll 1
    for (int c0 = 0; c0 < kb; c0 += kTrsmCols) {
#pragma unroll
        for (int u = 0; u < 4; ++u) x[0][u] = ahead[0][u], x[1][u] = ahead[1][u];
        if (c0 + kTrsmCols < kb) load(c0 + kTrsmCols, ahead);
#pragma unroll 1
        for (int b = 0; b < c0 / kTrsmCols; ++b) {
            const int ld = kStep - b * kTrsmCols;
            const cx<R>* Tb = T + trsm_block(b) + (c0 + q - b * kTrsmCols);
            const cx<R>* Xb = X + b * kTrsmCols * kLdX + r;
#pragma unroll 4
            for (int t = 0; t < kTrsmCols; ++t) {
                const cx<R> v0 = Xb[t * kLdX], v1 = Xb[t * kLdX + kApart];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const cx<R> l = Tb[4 * u + t * ld];
                    x[0][u] = fms(x[0][u], l, v0);
                    x[1][u] = fms(x[1][u], l, v1);
                }
            }
        }
        const int ld = kStep - c0;
        const cx<R>* Tc = T + trsm_block(c0 / kTrsmCols) + q;
#pragma unroll
        for (int j = 0; j < kTrsmCols; ++j) {
            const int uj = j / 4;
            cx<R> xj[2];
#pragma unroll
            for (int h = 0; h < 2; ++h)
                xj[h] = cx<R>{__shfl_sync(0xffffffffu, x[h][uj].re, quad | (j & 3)),
                              __shfl_sync(0xffffffffu, x[h][uj].im, quad | (j & 3))};
            const cx<R>* col = Tc + j * ld;
#pragma unroll
            for (int u = uj; u < 4; ++u) {
                const cx<R> l = col[4 * u];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const cx<R> v = fms(x[h][u], l, xj[h]);
                    if (u > uj || q > (j & 3)) x[h][u] = v;
                }
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int c = c0 + 4 * u + q;
                if (c < 48) X[c * kLdX + r + kApart * h] = x[h][u];
                if (i + kApart * h < m && c < kb)
                    P[i + kApart * h + static_cast<long long>(c) * m] = x[h][u] * Dinv[c];
            }
        __syncwarp();  // the row's lanes read one another's columns
    }
}

// In-panel update tile (i0, j0) of step k0: F[i, j] -= sum_t L[i,t] D[t] L[j,t]
// over the step's kb columns t, for i >= j >= k0 + kb and j inside the
// current 128-column panel (the columns to its right get the whole panel's
// update at once when the panel is complete).
// Bound by latency and, where tiles are many, by FFMA issue: every load of a
// thread is in flight at once, the destination's behind the operands', so a
// block takes two round trips. Six entries of 32^3 in FP32 77 us a launch, eight
// of 24^3 51 us; with the operands loaded a few at a time beside their pivots
// and the destination read after the products 93 and 63. Two blocks a
// multiprocessor keep the loads in registers (three spill: 90 and 62 us).
template <class R>
__global__ void __launch_bounds__(256, sizeof(R) == 4 ? 2 : 1) k_update_panel(Sched S, long long item0, cx<R>* Lb, long long lstride) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cx<R>* As = reinterpret_cast<cx<R>*>(smem_raw);  // [kStep][kTile], scaled by D
    cx<R>* Bs = As + kStep * kTile;                  // [kStep][kTile]
    __shared__ cx<R> D[kStep];
    constexpr int kLoads = kStep * kTile / 256, kSkip = 256 / kTile;
    pdl_start_next();
    const Item it = S.items[item0 + blockIdx.x];
    const int s = it.s, k0 = it.a, i0 = it.b, j0 = it.c;
    const int w = S.first[s + 1] - S.first[s];
    const int m = S.rows[s];
    const int kb = min(kStep, w - k0);
    const int jend = min(w, (k0 / kTcPanel) * kTcPanel + kTcPanel);
    cx<R>* Ls = Lb + lstride * blockIdx.y + S.loff[s];
    const cx<R>* P = Ls + static_cast<long long>(k0) * m;
    const int r = threadIdx.x % kTile, t0 = threadIdx.x / kTile;
    const bool in_a = i0 + r < m, in_b = j0 + r < m;
    pdl_wait();
    cx<R> av[kLoads], bv[kLoads];
#pragma unroll
    for (int u = 0; u < kLoads; ++u) {
        const int t = t0 + kSkip * u;
        const cx<R>* col = P + static_cast<long long>(t) * m + r;
        av[u] = t < kb && in_a ? col[i0] : cx<R>{0, 0};
        bv[u] = t < kb && in_b ? col[j0] : cx<R>{0, 0};
    }
    if (threadIdx.x < kb) D[threadIdx.x] = P[k0 + threadIdx.x + static_cast<long long>(threadIdx.x) * m];
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kLoads; ++u) {
        const int t = t0 + kSkip * u;
        As[t * kTile + r] = t < kb ? av[u] * D[t] : cx<R>{0, 0};
        Bs[t * kTile + r] = bv[u];
    }
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    cx<R>* const dst = Ls + i0 + tx + static_cast<long long>(j0 + ty) * m;
    auto mine = [&](int a, int b) {
        const int i = i0 + tx + 16 * a, j = j0 + ty + 16 * b;
        return j < jend && i < m && i >= j;
    };
    cx<R> old[4][4];
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int a = 0; a < 4; ++a)
            old[a][b] = mine(a, b) ? dst[16 * a + static_cast<long long>(16 * b) * m] : cx<R>{0, 0};
    __syncthreads();
    cx<R> acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = cx<R>{0, 0};
#pragma unroll 2
    for (int t = 0; t < kb; ++t) {
        cx<R> x[4], y[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) x[a] = As[t * kTile + tx + 16 * a];
#pragma unroll
        for (int b = 0; b < 4; ++b) y[b] = Bs[t * kTile + ty + 16 * b];
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                acc[a][b].re += x[a].re * y[b].re - x[a].im * y[b].im;
                acc[a][b].im += x[a].re * y[b].im + x[a].im * y[b].re;
            }
    }
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int a = 0; a < 4; ++a)
            if (mine(a, b)) dst[16 * a + static_cast<long long>(16 * b) * m] = old[a][b] - acc[a][b];
}

// SIMT trailing update of a complete panel (either precision). Item
// (s, p0, i0, j0): F[i, j] -= sum_{t in panel} L[i,t] D[t] L[j,t] over the
// 128 x 64 tile at rows i0.., columns j0.. (i >= j); K is the panel width
// (<= 128), consumed 8 columns at a time through double-buffered shared
// memory, the next chunk's loads in flight while the current one is used.
// 256 threads, each an 8 x 4 block of complex accumulators (rows tx + 16a,
// columns ty + 16b): per column t a thread reads 12 shared entries for 32
// complex multiply-adds.
constexpr int kWideM = 128, kWideN = 64, kWideKC = 8;

template <class R>
constexpr int wide_smem() {
    return 2 * kWideKC * (kWideM + kWideN) * static_cast<int>(sizeof(cx<R>));
}

template <class R>
__global__ void __launch_bounds__(256) k_update_wide(Sched S, long long item0, cx<R>* Lb, cx<R>* CBb,
                                                     long long lstride, long long cbstride, int kcap, int panel) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cx<R>* As = reinterpret_cast<cx<R>*>(smem_raw);   // [2][KC][128], scaled by D
    cx<R>* Bs = As + 2 * kWideKC * kWideM;            // [2][KC][64]
    const Item it = S.items[item0 + blockIdx.x];
    const int s = it.s, p0 = it.a, i0 = it.b, j0 = it.c;
    cx<R>* L = Lb + lstride * blockIdx.y;
    cx<R>* CB = CBb + cbstride * blockIdx.y;
    const int w = S.first[s + 1] - S.first[s];
    const int m = S.rows[s];
    const int cs = m - w;
    const int K = min(kcap, w - p0);
    cx<R>* Ls = L + S.loff[s];
    cx<R>* CBs = CB + (cs > 0 ? S.cboff[s] : 0);
    const cx<R>* P = Ls + static_cast<long long>(p0) * m;
    const cx<R>* dg = Ls + p0 + static_cast<long long>(p0) * m;  // pivot t at dg[t * (m + 1)]
    const int tid = threadIdx.x;
    // Loader: A chunk entry (k = tid / 128 + 2q, r = tid % 128), q < 4; B chunk
    // entry (k = tid / 64 + 4q, r = tid % 64), q < 2.
    cx<R> pa[4], pd[4], pb[2];
    auto load = [&](int kbase) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int k = kbase + (tid >> 7) + 2 * q, r = tid & 127;
            pa[q] = cx<R>{0, 0};
            pd[q] = cx<R>{0, 0};
            if (k < K && i0 + r < m) {
                pa[q] = P[static_cast<long long>(k) * m + i0 + r];
                pd[q] = dg[static_cast<long long>(k) * (m + 1)];
            }
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int k = kbase + (tid >> 6) + 4 * q, r = tid & 63;
            pb[q] = cx<R>{0, 0};
            if (k < K && j0 + r < m) pb[q] = P[static_cast<long long>(k) * m + j0 + r];
        }
    };
    auto stash = [&](int buf) {
        cx<R>* A = As + buf * kWideKC * kWideM;
        cx<R>* B = Bs + buf * kWideKC * kWideN;
#pragma unroll
        for (int q = 0; q < 4; ++q) A[((tid >> 7) + 2 * q) * kWideM + (tid & 127)] = pa[q] * pd[q];
#pragma unroll
        for (int q = 0; q < 2; ++q) B[((tid >> 6) + 4 * q) * kWideN + (tid & 63)] = pb[q];
    };
    const int tx = tid & 15, ty = tid >> 4;
    cx<R> acc[8][4];
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = cx<R>{0, 0};
    const int nc = (K + kWideKC - 1) / kWideKC;
    load(0);
    stash(0);
    __syncthreads();
    for (int c = 0; c < nc; ++c) {
        if (c + 1 < nc) load((c + 1) * kWideKC);
        const cx<R>* A = As + (c & 1) * kWideKC * kWideM;
        const cx<R>* B = Bs + (c & 1) * kWideKC * kWideN;
#pragma unroll
        for (int k = 0; k < kWideKC; ++k) {
            cx<R> av[8], bv[4];
#pragma unroll
            for (int a = 0; a < 8; ++a) av[a] = A[k * kWideM + tx + 16 * a];
#pragma unroll
            for (int b = 0; b < 4; ++b) bv[b] = B[k * kWideN + ty + 16 * b];
#pragma unroll
            for (int a = 0; a < 8; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    acc[a][b].re += av[a].re * bv[b].re - av[a].im * bv[b].im;
                    acc[a][b].im += av[a].re * bv[b].im + av[a].im * bv[b].re;
                }
        }
        if (c + 1 < nc) stash((c + 1) & 1);
        __syncthreads();
    }
    // In-panel updates (panel != 0) stop at the current panel's last column.
    const int jcap = panel ? min(w, (p0 / kTcPanel) * kTcPanel + kTcPanel) : m;
    // Read-modify-write, one column block at a time: 8 loads, then 8 stores.
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        const int j = j0 + ty + 16 * b;
        cx<R>* dst[8];
        cx<R> old[8];
#pragma unroll
        for (int a = 0; a < 8; ++a) {
            const int i = i0 + tx + 16 * a;
            dst[a] = nullptr;
            if (j < jcap && i < m && i >= j)
                dst[a] = (j < w) ? Ls + i + static_cast<long long>(j) * m
                                 : CBs + (i - w) + static_cast<long long>(j - w) * cs;
            if (dst[a]) old[a] = *dst[a];
        }
#pragma unroll
        for (int a = 0; a < 8; ++a)
            if (dst[a]) *dst[a] = old[a] - acc[a][b];
    }
}

// FP64 update on the FP64 tensor path (DMMA, mma.sync m8n8k4): the in-panel
// updates (K = 64, too short for the INT8 tiles below), and the trailing ones
// too where the factor asks for FP64 arithmetic. Same items, tile and K (up to kcap =
// kWidePair: a group of 128-column panels) as k_update_wide. 8 warps in a 4 x 2
// grid, each a 32 x 32 complex block of the tile: 4 x 4 blocks of 8 x 8, each
// four real products (Cr += Ar Br - Ai Bi, Ci += Ar Bi + Ai Br; the minus by
// a negated copy of Ai's fragment).
//
// Operands stream global -> shared by cp.async, without a register round
// trip, through a ring of 3 chunks of 16 panel columns (2 in flight while one
// is consumed; one barrier a chunk). They are staged as complex pairs, k-major
// rows 130 / 66 entries apart, so that one quarter-warp's 16-byte fragment
// loads touch distinct banks. The panel's pivots sit beside the ring and scale
// the A fragments as they are read (L[i,k] * D[k], the same product, in the
// same order, as the other trailing updates). A k-step of 4 costs a warp 9
// shared loads for 64 DMMA.
//
// The result is subtracted with red.global.add.f64 (old + (-acc) rounds as
// old - acc does): every destination entry has exactly one writer in a launch,
// so the fire-and-forget reduction leaves the same bits as a read-modify-write
// and, like it, costs the destination's traffic once after the last MMA.
constexpr int kDmmaKC = 16, kDmmaStages = 3;
constexpr int kDmmaLdA = kWideM + 2, kDmmaLdB = kWideN + 2;
constexpr int kDmmaStage = kDmmaKC * (kDmmaLdA + kDmmaLdB);  // complex entries
constexpr int kDmmaSmem = (kWidePair + kDmmaStages * kDmmaStage) * 16;
static_assert(kDmmaSmem <= 227 * 1024, "DMMA ring exceeds shared memory");
static_assert(kTcPanel % kDmmaKC == 0 && kDmmaKC % 4 == 0, "chunks must tile the panel in k-steps of 4");

__device__ __forceinline__ void dmma884(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// 16-byte global -> shared copy; bytes = 0 fills the destination with zeros.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

__device__ __forceinline__ void red_sub(double* p, double v) {
    asm volatile("red.global.add.f64 [%0], %1;" ::"l"(p), "d"(-v) : "memory");
}

// K_DMMA_SCALE item (s, p0, r0, d): rows pe + r0 .. pe + r0 + 127 of front
// s's trailing part (pe = p0 + K) prepared for the group's INT8 tiles
// (i8_update.cuh): A = L D and B = L, each row scaled to integers and split
// into byte digits, into region d. Rows past the front and columns past K are
// zeros. A row with a component that is not finite gets a NaN scale, so that
// the entries that it reaches become NaN, as in a floating-point update.
//
// 32 rows per CTA (blockIdx.z picks them), lane = row, so every global load is
// a contiguous run of a column; a warp takes 16 columns at a time, which is
// one 16-byte row of a core matrix per digit. Two passes over the operands,
// the second served by the caches: the rows' largest components, then the
// digits. Bound by its writes (48 bytes per entry; 24^3, 8 entries: 15.6 ms
// per factorization beside 115 ms of tiles) and, on small fronts, by the
// passes' dependent round trips (11 us a launch).
template <class R, class C>
__global__ void __launch_bounds__(256, 2) k_i8_split(Sched S, long long item0, const cx<R>* Lb, long long lstride,
                                                     unsigned char* ws, long long ws_stride, int kcap) {
    using Real = I8Real<R>;
    constexpr int kWarps = 8;
    __shared__ R dre[kWidePair], dim[kWidePair], up[kWidePair];  // D 2^-h, 2^h
    __shared__ int top[2][kWarps][32];                           // largest sizes of A, B
    pdl_start_next();
    const Item it = S.items[item0 + blockIdx.x];
    const int s = it.s, p0 = it.a;
    const int w = S.first[s + 1] - S.first[s];
    const int m = S.rows[s];
    const int K = min(kcap, w - p0), pe = p0 + K;
    const int Rp = (m - pe + kTcM - 1) / kTcM * kTcM;
    const int nst = (K + kI8K - 1) / kI8K;
    unsigned char* region = ws + ws_stride * blockIdx.y + static_cast<long long>(it.d) * 256;
    const cx<R>* P = Lb + lstride * blockIdx.y + S.loff[s];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = it.b + 32 * blockIdx.z + lane;  // row within the trailing part
    const bool in = pe + r < m;
    const cx<R>* X = P + (in ? pe + r : pe) + static_cast<long long>(p0) * m;
    pdl_wait();
    for (int k = threadIdx.x; k < kWidePair; k += 256) {
        const cx<R> d = k < K ? P[(p0 + k) + static_cast<long long>(p0 + k) * m] : cx<R>{0, 0};
        const int e = max(Real::exponent(Real::size(d.re)), Real::exponent(Real::size(d.im)));
        const int h = e == 0 || e == Real::none ? 0 : (e - Real::bias) >> 1;
        const R dn = Real::pow2(Real::bias - h);
        dre[k] = d.re * dn;
        dim[k] = d.im * dn;
        up[k] = Real::pow2(Real::bias + h);
    }
    __syncthreads();
    auto load = [&](int c, cx<R> (&x)[16]) {
#pragma unroll
        for (int u = 0; u < 16; ++u)
            x[u] = in && 16 * c + u < K ? X[static_cast<long long>(16 * c + u) * m] : cx<R>{0, 0};
    };
    int ta = 0, tb = 0;
    for (int c = warp; 16 * c < K; c += kWarps) {
        cx<R> x[16];
        load(c, x);
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            const int k = 16 * c + u;
            const R ar = x[u].re * dre[k] - x[u].im * dim[k], ai = x[u].re * dim[k] + x[u].im * dre[k];
            ta = max(ta, max(Real::size(ar), Real::size(ai)));
            tb = max(tb, max(Real::size(x[u].re * up[k]), Real::size(x[u].im * up[k])));
        }
    }
    top[0][warp][lane] = ta;
    top[1][warp][lane] = tb;
    __syncthreads();
#pragma unroll
    for (int v = 0; v < kWarps; ++v) {
        ta = max(ta, top[0][v][lane]);
        tb = max(tb, top[1][v][lane]);
    }
    // Biased exponents; tiny rows share one that keeps every scale normal.
    const int ea = max(Real::exponent(ta), Real::least), eb = max(Real::exponent(tb), Real::least);
    constexpr int kBits = 8 * C::S - 2;              // |integer| <= 2^kBits
    constexpr int kTop = 4 * (2 * C::S - 1 - C::L) + Real::shift;  // half of log2 of the last kept level's weight
    const R fa = Real::pow2(2 * Real::bias - 1 + kBits - ea), fb = Real::pow2(2 * Real::bias - 1 + kBits - eb);
    if (warp == 0) {
        R* scale = reinterpret_cast<R*>(region + i8_scale_off<C>(Rp, nst));
        const R bad = Real::pow2(Real::none) - Real::pow2(Real::none);  // NaN
        scale[r] = ea >= Real::none ? bad : Real::pow2(ea + 1 - kBits + kTop);
        scale[Rp + r] = eb >= Real::none ? bad : Real::pow2(eb + 1 - kBits + kTop);
    }
    // 16 values -> digit p of each, 16 bytes, to dst + p * step.
    auto digits = [&](const R (&v)[16], R f, unsigned char* dst, int step) {
        using Int = decltype(Real::integer(R(0)));
        constexpr Int kBias = static_cast<Int>((1LL << (8 * (C::S - 1))) / 255 * 128);  // 128 in every byte but the top digit's
        static_assert(sizeof(Int) == C::S, "one byte per digit");
        unsigned out[C::S][4];
#pragma unroll
        for (int g = 0; g < 4; ++g)
#pragma unroll
            for (int h = 0; h < C::S / 4; ++h) {  // bytes 4 h .. 4 h + 3 of four numbers
                unsigned z[4];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    z[u] = static_cast<unsigned>(((Real::integer(v[4 * g + u] * f) + kBias) ^ kBias) >> (h ? 8 * sizeof(Int) - 32 : 0));
                const unsigned t0 = __byte_perm(z[0], z[1], 0x5140), t1 = __byte_perm(z[2], z[3], 0x5140);
                const unsigned t2 = __byte_perm(z[0], z[1], 0x7362), t3 = __byte_perm(z[2], z[3], 0x7362);
                // byte b = digit S - 1 - b
                out[C::S - 1 - 4 * h][g] = __byte_perm(t0, t1, 0x5410);
                out[C::S - 2 - 4 * h][g] = __byte_perm(t0, t1, 0x7632);
                out[C::S - 3 - 4 * h][g] = __byte_perm(t2, t3, 0x5410);
                out[C::S - 4 - 4 * h][g] = __byte_perm(t2, t3, 0x7632);
            }
#pragma unroll
        for (int p = 0; p < C::S; ++p)
            *reinterpret_cast<uint4*>(dst + p * step) = make_uint4(out[p][0], out[p][1], out[p][2], out[p][3]);
    };
    for (int c = warp; c < 2 * nst; c += kWarps) {
        cx<R> x[16];
        R v[16];
        load(c, x);
        unsigned char* A = region + i8_a_off<C>(nst, r, c >> 1) + i8_off(r % kTcM, c & 1);
        unsigned char* B = region + i8_b_off<C>(Rp, nst, r, c >> 1) + i8_off(r % C::Nc, c & 1);
        constexpr int kPlaneA = kTcM * kI8K, kDigitB = C::W * kI8K, kHalfB = C::Nc * kI8K;
#pragma unroll
        for (int u = 0; u < 16; ++u) v[u] = x[u].re * dre[16 * c + u] - x[u].im * dim[16 * c + u];
        digits(v, fa, A, 2 * kPlaneA);
#pragma unroll
        for (int u = 0; u < 16; ++u) v[u] = x[u].re * dim[16 * c + u] + x[u].im * dre[16 * c + u];
        digits(v, fa, A + kPlaneA, 2 * kPlaneA);
#pragma unroll
        for (int u = 0; u < 16; ++u) v[u] = x[u].re * up[16 * c + u];
        digits(v, fb, B, kDigitB);
        digits(v, fb, B + C::imageB + kHalfB, kDigitB);
#pragma unroll
        for (int u = 0; u < 16; ++u) v[u] = x[u].im * up[16 * c + u];
        digits(v, fb, B + kHalfB, kDigitB);
        digits(v, -fb, B + C::imageB, kDigitB);
    }
}

// The trailing update on prepared INT8 operands. Items (s, p0, i0, j0, d) as
// the other trailing updates': a 128 x 64 tile each, taken here as 64 / Nc
// tiles of Nc columns. Persistent: one CTA per SM (its accumulators are all
// of TMEM) walks the launch's tiles -- entries outermost, so that one
// entry's operands stay in L2 -- in three roles that run side by side:
//   warp 0, lane 0  decodes the tiles into a ring of slots and copies their
//                   operand stages (two bulk copies each) into the ring of
//                   buffers, across tile boundaries;
//   warp 1, lane 0  issues each stage's MMAs;
//   warps 2 .. 17   read the destination while the tile is computed, then the
//                   accumulators, and write the difference.
// A tile's MMAs wait until the previous tile's accumulators have been read.
// Every wait is bounded and gives up early once another role has failed.
//
// Measured, trailing updates of a factorization (the form that each replaced):
//   FP64, 32^3, two entries    178-188 ms (486, DMMA) 71-75 useful FP64 TFLOP/s
//   FP64, 24^3, eight entries  115-118 ms (292)
//   FP32, 32^3, six entries    170-176 ms (311, two TF32 pieces)
//   FP32, 24^3, six entries    30.5 ms (56)
//   FP32, 12^3, six entries    0.91 ms (1.5)
// and on 8^3 (FP64, one entry) 17 launches in 0.26 ms.
// It is the faster form from the smallest launches up, so every FP64 trailing
// update takes it unless its factor asks for FP64 arithmetic
// (aphi_factor_set_fp64_digits), and every FP32 one with tc_split 2. In FP64 an
// SM's shared memory bounds a tile: per stage the MMAs read 240 KB of digits
// and the copies write 96 KB, 2,700 cycles beside 2,304 of tensor work (K =
// 256: 22,000 cycles, then 4,000 to read the accumulators); in FP32 the MMAs
// take 11,000 cycles and the accumulators' reading 3,000.
constexpr int kI8Threads = 64 + 16 * 32;

template <class R, class C>
__global__ void __launch_bounds__(kI8Threads, 1) k_update_i8(Sched S, long long item0, int count, int entries,
                                                             cx<R>* Lb, cx<R>* CBb, long long lstride,
                                                             long long cbstride, int kcap, const unsigned char* ws,
                                                             long long ws_stride, int* err) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    constexpr int kHalves = kTcN / C::Nc, kEpWarps = kI8Threads / 32 - 2;
    // A tile as the producer decodes it, a few tiles ahead of the others.
    struct Tile {
        cx<R>* panel;   // (i0, j0) in the panel, leading dimension m
        cx<R>* cb;      // (i0, j0) in the contribution block, leading dimension cs
        const R* scale_a;  // of row i0
        const R* scale_b;  // of column j0
        int i0, j0, m, cs, cut, nst;  // cut: columns below the panel's end; nst 0: no more tiles
    };
    // A producer loads at most Stages stages beyond the oldest unfinished
    // MMAs, and those wait for the epilogue's previous tile: it is never
    // more than Stages + 2 tiles ahead of a reader.
    constexpr int kSlots = 8;
    static_assert(C::Stages + 2 < kSlots, "a tile's slot must not be rewritten before everyone has read it");
    uint64_t* full = reinterpret_cast<uint64_t*>(smem_raw + C::Stages * C::stage);
    uint64_t* empty = full + C::Stages;
    uint64_t* acc_full = empty + C::Stages;
    uint64_t* acc_empty = acc_full + 1;
    uint64_t* ready = acc_empty + 1;
    Tile* slots = reinterpret_cast<Tile*>(ready + kSlots);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(slots + kSlots);
    volatile int* state = reinterpret_cast<volatile int*>(tmem_slot + 1);  // [0] failed, [1] stages committed, [2] stages loaded
    static_assert((2 * C::Stages + 2 + kSlots) * 8 + kSlots * sizeof(Tile) + 16 <= C::extra, "barriers and slots");
    pdl_start_next();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(C::tmem));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        auto init = [](uint64_t* b, int n) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(n));
        };
        for (int b = 0; b < C::Stages; ++b) init(full + b, 1), init(empty + b, 1);
        for (int b = 0; b < kSlots; ++b) init(ready + b, 1);
        init(acc_full, 1);
        init(acc_empty, kEpWarps);
        asm volatile("fence.mbarrier_init.release.cluster;");
        state[0] = 0;
        state[1] = 0;
        state[2] = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = *tmem_slot;
    pdl_wait();
    // Tile n of this CTA once the producer has decoded it; false: failed.
    auto tile = [&](int n, Tile& t) {
        if (!mbar_wait_live(smem_u32(ready + n % kSlots), (n / kSlots) & 1, state)) return false;
        t = slots[n % kSlots];
        return true;
    };

    if (tid == 0) {
        int c = 0, n = 0;  // stages loaded, tiles decoded so far
        auto publish = [&]() {
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(ready + n % kSlots)) : "memory");
            ++n;
        };
        const long long total = static_cast<long long>(count) * kHalves * entries;
        for (long long g = blockIdx.x; g < total && !state[0]; g += gridDim.x) {
            const int entry = static_cast<int>(g / (count * kHalves));
            const int q = static_cast<int>(g - static_cast<long long>(entry) * count * kHalves);
            const Item it = S.items[item0 + q / kHalves];
            const int s = it.s, i0 = it.b, j0 = it.c + (q % kHalves) * C::Nc;
            const int m = S.rows[s];
            if (j0 >= m || i0 + kTcM <= j0) continue;  // no entry on or below the diagonal
            const int w = S.first[s + 1] - S.first[s];
            const int K = min(kcap, w - it.a), pe = it.a + K, cs = m - w;
            const int nst = (K + kI8K - 1) / kI8K;
            const int Rp = (m - pe + kTcM - 1) / kTcM * kTcM;
            const unsigned char* region = ws + ws_stride * entry + static_cast<long long>(it.d) * 256;
            const R* scale = reinterpret_cast<const R*>(region + i8_scale_off<C>(Rp, nst));
            slots[n % kSlots] = Tile{Lb + lstride * entry + S.loff[s] + i0 + static_cast<long long>(j0) * m,
                                     CBb + cbstride * entry + (cs > 0 ? S.cboff[s] : 0) + (i0 - w) +
                                         static_cast<long long>(j0 - w) * cs,
                                     scale + (i0 - pe), scale + Rp + (j0 - pe), i0, j0, m, cs, w - j0, nst};
            publish();
            const unsigned char* A = region + i8_a_off<C>(nst, i0 - pe, 0);
            const unsigned char* B = region + i8_b_off<C>(Rp, nst, j0 - pe, 0);
            for (int k = 0; k < nst; ++k, ++c) {
                const int b = c % C::Stages;
                if (c >= C::Stages && !mbar_wait_live(smem_u32(empty + b), ((c / C::Stages) - 1) & 1, state)) {
                    state[0] = 1;
                    break;
                }
                const uint32_t dst = smem_u32(smem_raw + b * C::stage), fb = smem_u32(full + b);
                mbar_expect_tx(fb, C::stage);
                bulk_g2s(dst, A + static_cast<long long>(k) * C::blockA, C::blockA, fb);
                bulk_g2s(dst + C::blockA, B + static_cast<long long>(k) * C::blockB, C::blockB, fb);
                state[2] = c + 1;
            }
        }
        slots[n % kSlots].nst = 0;
        publish();
    } else if (tid == 32) {
        int c = 0;  // stages issued so far
        Tile t;
        for (int n = 0;; ++n) {
            if (!tile(n, t) || (t.nst > 0 && n > 0 && !mbar_wait_live(smem_u32(acc_empty), (n - 1) & 1, state))) {
                state[0] = 1;
                break;
            }
            if (t.nst == 0) break;
            asm volatile("tcgen05.fence::after_thread_sync;");
            for (int k = 0; k < t.nst; ++k, ++c) {
                const int b = c % C::Stages;
                if (!mbar_wait_live(smem_u32(full + b), (c / C::Stages) & 1, state)) {
                    state[0] = 1;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;");
                i8_issue<C>(smem_u32(smem_raw + b * C::stage), tmem, k == 0);
                mma_commit(smem_u32(empty + b));
                state[1] = c + 1;
            }
            if (state[0]) break;
            mma_commit(smem_u32(acc_full));
        }
    } else if (warp >= 2) {
        constexpr int kCols = C::Nc / (kEpWarps / 4);  // columns per warp
        constexpr int kChunk = 4;                      // columns per TMEM read
        constexpr R kLargest = sizeof(R) == 8 ? static_cast<R>(DBL_MAX) : static_cast<R>(FLT_MAX);
        const int quad = warp & 3, c0 = ((warp - 2) >> 2) * kCols;
        const uint32_t lanes = static_cast<uint32_t>(quad * 32) << 16;
        const int r = quad * 32 + lane;
        Tile t;
        for (int n = 0;; ++n) {
            if (!__all_sync(0xffffffffu, tile(n, t))) {
                state[0] = 1;
                break;
            }
            if (t.nst == 0) break;
            // This thread's entries: row i0 + r, columns j0 + c0 + q up to the
            // diagonal (q <= last), those below the cut in the panel, the rest
            // in the CB.
            const int last = t.i0 + r < t.m ? min(t.m - 1, t.i0 + r) - t.j0 - c0 : -1;
            const int cut = t.cut - c0;
            cx<R>* const in_cb = t.cb + r + static_cast<long long>(c0) * t.cs;
            cx<R>* const base = cut > 0 ? t.panel + r + static_cast<long long>(c0) * t.m : in_cb;
            const long long ld = cut > 0 ? t.m : t.cs;
            const bool mixed = cut > 0 && cut < kCols;
            auto at = [&](int q) {
                return mixed && q >= cut ? in_cb + static_cast<long long>(q) * t.cs : base + q * ld;
            };
            // The destination and the scales (lane q: column q's), read while
            // the tile is computed.
            cx<R> old[kCols];
#pragma unroll
            for (int q = 0; q < kCols; ++q) old[q] = q <= last ? *at(q) : cx<R>{0, 0};
            const R sa = t.scale_a[r], sb = t.scale_b[c0 + lane % kCols];
            bool live = mbar_wait_live(smem_u32(acc_full), n & 1, state);
            live = __all_sync(0xffffffffu, live);  // the TMEM loads are warp-wide
            if (!live) {
                state[0] = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
            for (int q0 = 0; q0 < kCols; q0 += kChunk) {
                R re[kChunk], im[kChunk];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    int v[C::L][kChunk];
#pragma unroll
                    for (int l = 0; l < C::L; ++l) tmem_ld(tmem + lanes + l * C::W + h * C::Nc + c0 + q0, v[l]);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int q = 0; q < kChunk; ++q) {
                        int d[C::L];
#pragma unroll
                        for (int l = 0; l < C::L; ++l) {
                            asm volatile("" : "+r"(v[l][q]));  // not before the wait
                            d[l] = v[l][q];
                        }
                        (h ? im : re)[q] = i8_combine(d);
                    }
                }
                if (q0 + kChunk == kCols) {  // everything this warp reads has been read
                    asm volatile("tcgen05.fence::before_thread_sync;");
                    __syncwarp();
                    if (lane == 0)
                        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(acc_empty)) : "memory");
                }
#pragma unroll
                for (int q = 0; q < kChunk; ++q) {
                    R s = sa * __shfl_sync(0xffffffffu, sb, q0 + q);
                    s = s > kLargest ? kLargest : s;  // so that 0 s is 0 (a NaN stays)
                    if (q0 + q <= last)
                        *at(q0 + q) = cx<R>{fma(-re[q], s, old[q0 + q].re), fma(-im[q], s, old[q0 + q].im)};
                }
            }
        }
    }
    __syncthreads();
    // What is still in flight after a failure: the last commits, then any
    // copies that no MMA consumed.
    const bool failed = state[0] != 0;
    if (tid == 0 && failed) {
        const int committed = state[1], loaded = state[2];
        for (int c = max(0, committed - C::Stages); c < committed; ++c)
            mbar_wait(smem_u32(empty + c % C::Stages), (c / C::Stages) & 1);
        for (int c = committed; c < loaded; ++c) mbar_wait(smem_u32(full + c % C::Stages), (c / C::Stages) & 1);
        atomicExch(err, 1);
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::tmem));
}

__global__ void __launch_bounds__(256) k_update_wide_dmma(Sched S, long long item0, cx<double>* Lb,
                                                          cx<double>* CBb, long long lstride, long long cbstride,
                                                          int kcap, int panel) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cx<double>* Ds = reinterpret_cast<cx<double>*>(smem_raw);  // [kWidePair] pivots of the group's panels
    cx<double>* Ring = Ds + kWidePair;                           // [stage][A: KC x ldA | B: KC x ldB]
    pdl_start_next();
    const Item it = S.items[item0 + blockIdx.x];
    const int s = it.s, p0 = it.a, i0 = it.b, j0 = it.c;
    cx<double>* L = Lb + lstride * blockIdx.y;
    cx<double>* CB = CBb + cbstride * blockIdx.y;
    const int w = S.first[s + 1] - S.first[s];
    const int m = S.rows[s];
    const int cs = m - w;
    const int K = min(kcap, w - p0);
    cx<double>* Ls = L + S.loff[s];
    cx<double>* CBs = CB + (cs > 0 ? S.cboff[s] : 0);
    const cx<double>* P = Ls + static_cast<long long>(p0) * m;
    const cx<double>* dg = Ls + p0 + static_cast<long long>(p0) * m;
    const int tid = threadIdx.x;
    const uint32_t ring = smem_u32(Ring);
    // Chunk c: panel columns 16c.. of rows i0.. (A, 128 rows) and j0.. (B, 64).
    auto fetch = [&](int c) {
        const int kbase = c * kDmmaKC;
        const uint32_t sa = ring + (c % kDmmaStages) * kDmmaStage * 16;
        const uint32_t sb = sa + kDmmaKC * kDmmaLdA * 16;
#pragma unroll
        for (int q = 0; q < kDmmaKC * kWideM / 256; ++q) {
            const int e = tid + 256 * q, k = e / kWideM, r = e % kWideM;
            const bool in = kbase + k < K && i0 + r < m;
            cp_async16(sa + (k * kDmmaLdA + r) * 16, in ? P + static_cast<long long>(kbase + k) * m + i0 + r : P,
                       in ? 16u : 0u);
        }
#pragma unroll
        for (int q = 0; q < kDmmaKC * kWideN / 256; ++q) {
            const int e = tid + 256 * q, k = e / kWideN, r = e % kWideN;
            const bool in = kbase + k < K && j0 + r < m;
            cp_async16(sb + (k * kDmmaLdB + r) * 16, in ? P + static_cast<long long>(kbase + k) * m + j0 + r : P,
                       in ? 16u : 0u);
        }
    };
    const int warp = tid >> 5, lane = tid & 31;
    const int wm = warp & 3, wn = warp >> 2;
    const int g = lane >> 2, t4 = lane & 3;
    double cr[4][4][2], ci[4][4][2];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) cr[a][b][0] = cr[a][b][1] = ci[a][b][0] = ci[a][b][1] = 0.0;
    const int nc = (K + kDmmaKC - 1) / kDmmaKC;
    pdl_wait();
    fetch(0);
    cp_async_commit();
    if (nc > 1) fetch(1);
    cp_async_commit();
    for (int t = tid; t < kWidePair; t += 256) Ds[t] = t < K ? dg[static_cast<long long>(t) * (m + 1)] : cx<double>{0, 0};
    for (int c = 0; c < nc; ++c) {
        cp_async_wait<1>();  // this thread's copies of chunk c have landed
        __syncthreads();     // everyone's have; everyone is done with chunk c - 1
        if (c + 2 < nc) fetch(c + 2);
        cp_async_commit();
        const cx<double>* A = Ring + (c % kDmmaStages) * kDmmaStage;
        const cx<double>* B = A + kDmmaKC * kDmmaLdA;
#pragma unroll
        for (int ks = 0; ks < kDmmaKC; ks += 4) {
            cx<double> af[4], bf[4];
            const cx<double> d = Ds[c * kDmmaKC + ks + t4];
#pragma unroll
            for (int a = 0; a < 4; ++a) af[a] = A[(ks + t4) * kDmmaLdA + 32 * wm + 8 * a + g] * d;
#pragma unroll
            for (int b = 0; b < 4; ++b) bf[b] = B[(ks + t4) * kDmmaLdB + 32 * wn + 8 * b + g];
            // One real product over all 16 blocks before the next, so that
            // consecutive MMAs never feed one another.
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) dmma884(cr[a][b], af[a].re, bf[b].re);
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) dmma884(ci[a][b], af[a].re, bf[b].im);
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) dmma884(cr[a][b], -af[a].im, bf[b].im);
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) dmma884(ci[a][b], af[a].im, bf[b].re);
        }
    }
    // Thread holds C[g][2 t4 + e] of each 8 x 8 block: rows i0 + 32 wm + 8a + g,
    // columns j0 + 32 wn + 8b + 2 t4 + e. In-panel updates (panel != 0) stop
    // at the current panel's last column.
    const int jcap = panel ? min(w, (p0 / kTcPanel) * kTcPanel + kTcPanel) : m;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int i = i0 + 32 * wm + 8 * a + g;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int j = j0 + 32 * wn + 8 * (q >> 1) + 2 * t4 + (q & 1);
            if (j < jcap && i < m && i >= j) {
                cx<double>* dst = (j < w) ? Ls + i + static_cast<long long>(j) * m
                                          : CBs + (i - w) + static_cast<long long>(j - w) * cs;
                red_sub(&dst->re, cr[a][q >> 1][q & 1]);
                red_sub(&dst->im, ci[a][q >> 1][q & 1]);
            }
        }
    }
}

// Tensor-core trailing update of complete panels (FP32 factors). Item
// (s, p0, i0, j0): F[i, j] -= sum_{t in panels} L[i,t] D[t] L[j,t] over the
// 128 x 64 tile at rows i0.., columns j0.. (i >= j). K = min(kcap, w - p0):
// one panel (128) or a group of them (up to kWidePair). Split: TF32 pieces per
// operand (3, or 2 for the cheaper hh + hl + lh products). A bounded wait that
// expires sets err[0] and leaves the tile unchanged; the host reports it.
template <int Split, int Stages = kTcPlaneStages, int Group = kTcGroup>
__global__ void __launch_bounds__(kTcThreads) k_update_tc(Sched S, long long item0, cx<float>* Lb, cx<float>* CBb,
                                                          long long lstride, long long cbstride, int kcap, int* err) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const Item it = S.items[item0 + blockIdx.x];
    const int s = it.s, p0 = it.a, i0 = it.b, j0 = it.c;
    cx<float>* L = Lb + lstride * blockIdx.y;
    cx<float>* CB = CBb + cbstride * blockIdx.y;
    const int w = S.first[s + 1] - S.first[s];
    const int m = S.rows[s];
    const int cs = m - w;
    const int K = min(kcap, w - p0);
    cx<float>* Ls = L + S.loff[s];
    cx<float>* CBs = CB + (cs > 0 ? S.cboff[s] : 0);
    const float2* P = reinterpret_cast<const float2*>(Ls + static_cast<long long>(p0) * m);
    const float2* dk = reinterpret_cast<const float2*>(Ls + p0 + static_cast<long long>(p0) * m);
    // Read-modify-write of 16 entries of row i: all loads first, so their
    // latencies overlap, then the stores.
    const bool ok = tc_tile<Split, Stages, Group>(smem_raw, P, m, m, K, i0, j0, dk, static_cast<long long>(m) + 1,
                            [&](int r, int c0, const float(&re)[16], const float(&im)[16]) {
                                const int i = i0 + r;
                                if (i >= m) return;
                                float2* dst[16];
                                float2 old[16];
#pragma unroll
                                for (int c = 0; c < 16; ++c) {
                                    const int j = j0 + c0 + c;
                                    dst[c] = nullptr;
                                    if (j < m && i >= j)
                                        dst[c] = reinterpret_cast<float2*>(
                                            (j < w) ? Ls + i + static_cast<long long>(j) * m
                                                    : CBs + (i - w) + static_cast<long long>(j - w) * cs);
                                    if (dst[c]) old[c] = *dst[c];
                                }
#pragma unroll
                                for (int c = 0; c < 16; ++c)
                                    if (dst[c]) *dst[c] = make_float2(old[c].x - re[c], old[c].y - im[c]);
                            });
    if (!ok && threadIdx.x == 0) atomicExch(err, 1);
}

// K_TC_SPLIT item (s, p0, r0, d): rows pe + r0 .. pe + r0 + 127 of front s's
// trailing part (pe = p0 + K, the group's K columns from p0) split into the
// pre-split tile's planes, stage by stage: A = L D (the pivots on the panel
// diagonal, the same product tc_split forms) and B = L, each as hi + lo TF32
// pieces (hi = round(x), lo = round(x - hi)); B also as -Bi. The region
// (workspace offset d) holds the A blocks (128 rows) and the B blocks (64
// rows) in the layout tc_tile_presplit reads (pre_a_off, pre_b_off), each
// plane in the canonical K-major core-matrix layout; rows past the front and
// columns past K are zeros. One thread per row; blockIdx.z picks 8 of the
// stages, so the rows' loads of those 64 columns are all in flight at once.
__global__ void __launch_bounds__(kTcThreads) k_tc_split(Sched S, long long item0, const cx<float>* Lb,
                                                         long long lstride, unsigned char* ws, long long ws_stride,
                                                         int kcap) {
    constexpr int kStagesPerCta = 8;  // blockIdx.z: this CTA's stages c0 .. c0 + 7 (64 columns)
    __shared__ cx<float> piv[kStagesPerCta * kTcK];
    const Item it = S.items[item0 + blockIdx.x];
    const int s = it.s, p0 = it.a, r0 = it.b;
    const int w = S.first[s + 1] - S.first[s];
    const int m = S.rows[s];
    const int K = min(kcap, w - p0), pe = p0 + K;
    const int R = (m - pe + kTcM - 1) / kTcM * kTcM;
    const int nst = (K + kTcK - 1) / kTcK;
    const int c0 = blockIdx.z * kStagesPerCta;
    if (c0 >= nst) return;  // the whole CTA: no barrier follows for it
    unsigned char* region = ws + ws_stride * blockIdx.y + static_cast<long long>(it.d) * 256;
    const cx<float>* P = Lb + lstride * blockIdx.y + S.loff[s];
    if (threadIdx.x < kStagesPerCta * kTcK) {
        const int k = c0 * kTcK + threadIdx.x;
        piv[threadIdx.x] = k < K ? P[(p0 + k) + static_cast<long long>(p0 + k) * m] : cx<float>{0.f, 0.f};
    }
    const int r = r0 + threadIdx.x;  // row within the trailing part
    const int row = pe + r;
    const bool in = row < m;
    // The CTA's 64 columns of this row, every load in flight before use.
    cx<float> v[kStagesPerCta * kTcK];
#pragma unroll
    for (int u = 0; u < kStagesPerCta * kTcK; ++u) {
        const int k = c0 * kTcK + u;
        v[u] = in && k < K ? P[row + static_cast<long long>(p0 + k) * m] : cx<float>{0.f, 0.f};
    }
    __syncthreads();
    const uint32_t oa = plane_off(r & 127, 0), ob = plane_off(r & 63, 0);
#pragma unroll
    for (int cc = 0; cc < kStagesPerCta; ++cc) {
        const int c = c0 + cc;
        if (c >= nst) break;
        unsigned char* A = region + pre_a_off(R, nst, r, c);
        unsigned char* B = region + pre_b_off(R, nst, r, c);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float ar[4], ai[4], br[4], bi[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const cx<float> x = v[cc * kTcK + 4 * h + q];
                const cx<float> d = piv[cc * kTcK + 4 * h + q];
                ar[q] = x.re * d.re - x.im * d.im;
                ai[q] = x.re * d.im + x.im * d.re;
                br[q] = x.re;
                bi[q] = x.im;
            }
            // A: re hi, re lo, im hi, im lo; B per piece: -Bi, Br, Bi
            split_store4<2>(A, kTcPlaneA, oa + h * 128, ar);
            split_store4<2>(A + 2 * kTcPlaneA, kTcPlaneA, oa + h * 128, ai);
            split_store4<2>(B + kTcPlaneB, 3 * kTcPlaneB, ob + h * 128, br);
            split_store4<2, true>(B + 2 * kTcPlaneB, 3 * kTcPlaneB, ob + h * 128, bi, B);
        }
    }
}

// The tensor-core trailing update on pre-split operands (K_UPDATE_TC with
// the two-piece split): item (s, p0, i0, j0, d), the front's planes in the
// workspace region d written by the launch's k_tc_split. Same tile and
// epilogue as k_update_tc.
template <int Group, int Stages>
__global__ void __launch_bounds__(kTcThreads) k_update_tc_presplit(Sched S, long long item0, cx<float>* Lb,
                                                                   cx<float>* CBb, long long lstride,
                                                                   long long cbstride, int kcap,
                                                                   const unsigned char* ws, long long ws_stride,
                                                                   int* err) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const Item it = S.items[item0 + blockIdx.x];
    const int s = it.s, p0 = it.a, i0 = it.b, j0 = it.c;
    cx<float>* L = Lb + lstride * blockIdx.y;
    cx<float>* CB = CBb + cbstride * blockIdx.y;
    const int w = S.first[s + 1] - S.first[s];
    const int m = S.rows[s];
    const int cs = m - w;
    const int K = min(kcap, w - p0), pe = p0 + K;
    const int R = (m - pe + kTcM - 1) / kTcM * kTcM;
    const int nst = (K + kTcK - 1) / kTcK;
    cx<float>* Ls = L + S.loff[s];
    cx<float>* CBs = CB + (cs > 0 ? S.cboff[s] : 0);
    const unsigned char* region = ws + ws_stride * blockIdx.y + static_cast<long long>(it.d) * 256;
    const bool ok = tc_tile_presplit<Group, Stages>(smem_raw, region, R, nst, i0 - pe, j0 - pe,
                                            [&](int r, int c0, const float(&re)[16], const float(&im)[16]) {
                                                const int i = i0 + r;
                                                if (i >= m) return;
                                                float2* dst[16];
                                                float2 old[16];
#pragma unroll
                                                for (int c = 0; c < 16; ++c) {
                                                    const int j = j0 + c0 + c;
                                                    dst[c] = nullptr;
                                                    if (j < m && i >= j)
                                                        dst[c] = reinterpret_cast<float2*>(
                                                            (j < w) ? Ls + i + static_cast<long long>(j) * m
                                                                    : CBs + (i - w) + static_cast<long long>(j - w) * cs);
                                                    if (dst[c]) old[c] = *dst[c];
                                                }
#pragma unroll
                                                for (int c = 0; c < 16; ++c)
                                                    if (dst[c]) *dst[c] = make_float2(old[c].x - re[c], old[c].y - im[c]);
                                            });
    if (!ok && threadIdx.x == 0) atomicExch(err, 1);
}

// ---------------------------------------------------------------- solves
// y, U: per batch entry, nrhs vectors of length n (post-ordered numbering) and
// upool (update vectors, one segment of m - w entries per supernode). A
// kernel handles nr <= 8 right-hand sides starting at rhs k0.
//
// Forward (L y = b), per level bottom-up: gather the children's update
// vectors into the front vector (y at the pivot rows, U_s below), then per
// 64-column block: solve the block's unit triangle, update the rows below.
// Backward (L^T x = D^-1 y), per level top-down, blocks last to first: partial
// sums of L[rows below, block]^T x over row chunks, then one CTA adds them
// in chunk order, scales by D^-1 and solves the block's triangle.


struct SolveArgs {
    int n;
    int nrhs;      // vectors per batch entry in y / U
    int k0, nr;    // the rhs handled by this pass
    long long upool;
    int max_parts;
    const int* entries;  // grid.y -> batch entry (the entries still being solved); null: grid.y is the entry
    int ny;              // grid.y of the solve launches (0: the factor's batch)
    int* counters;       // fused plans: arrival counters, ns per grid row, zero between launches
    int ns;              // supernodes
};

__device__ __forceinline__ int solve_entry(const SolveArgs& a) {
    return a.entries ? a.entries[blockIdx.y] : static_cast<int>(blockIdx.y);
}

__device__ __forceinline__ long long vec_at(const SolveArgs& a, int b, int k) {
    return static_cast<long long>(b) * a.nrhs + (a.k0 + k);
}

// Loads of values that other CTAs of the same launch wrote (through L2, not
// a possibly stale L1 line).
__device__ __forceinline__ cx<double> ld_l2(const cx<double>* p) {
    const double2 v = __ldcg(reinterpret_cast<const double2*>(p));
    return cx<double>{v.x, v.y};
}
__device__ __forceinline__ cx<float> ld_l2(const cx<float>* p) {
    const float2 v = __ldcg(reinterpret_cast<const float2*>(p));
    return cx<float>{v.x, v.y};
}

// The fused solve kernels' hand-over: every CTA working on supernode s in
// this launch counts itself in, after a fence that publishes its writes; the
// one that arrives last (count == expected) resets the counter for the next
// launch and returns true. No CTA waits for another.
__device__ __forceinline__ bool last_to_arrive(int* counter, int expected) {
    __shared__ int last;
    __syncthreads();  // the CTA's writes ordered before thread 0's fence
    if (threadIdx.x == 0) {
        __threadfence();  // ... which publishes them before the arrival
        const int prev = atomicAdd(counter, 1);
        last = prev == expected - 1;
        if (last) {
            *counter = 0;
            __threadfence();  // the other CTAs' published writes before this CTA reads them
        }
    }
    __syncthreads();
    return last;
}

// A triangle's panel entries (jb x jb at P, leading dimension m) towards L2,
// ahead of the CTA that will stage them: one prefetch per 128-byte line.
template <class R>
__device__ __forceinline__ void prefetch_triangle(const cx<R>* P, long long m, int jb) {
    constexpr int kPerLine = 128 / sizeof(cx<R>);
    const int lines = (jb + kPerLine - 1) / kPerLine;
    for (int e = threadIdx.x; e < lines * jb; e += blockDim.x) {
        const int i = (e % lines) * kPerLine, j = e / lines;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(P + i + static_cast<long long>(j) * m));
    }
}

__device__ __forceinline__ int solve_nblocks(const Sched& S, int s) {
    return (S.first[s + 1] - S.first[s] + kSolveBlock - 1) / kSolveBlock;
}

// Shared memory of the solve kernels that hold a 64 x 64 block of L, with
// leading dimension kTriLd (65: column-strided reads fall in distinct banks),
// and for the backward triangle the partial-sum reduction's kRedGroups
// sub-sums per (column, rhs).
constexpr int kRedGroups = 8;
constexpr int kBwdDiagThreads = 512;
constexpr int red_smem(int nr) { return kRedGroups * kSolveBlock * nr; }  // complex entries
constexpr int kGatherRows = 512;                   // front rows per gather CTA

// Forward triangle of block blk of supernode s: y[blk] = L_bb^-1 y[blk] for
// the pass's rhs, one warp per rhs, L_bb staged in shared memory (smem:
// kTriSmem entries; fwd_triangle_stage first). Lane l holds rows l and l + 32
// in registers; step j broadcasts y_j from its owner lane and every lane below
// updates its rows, y_i = y_i - L_ij y_j, in ascending j. Every thread of the
// CTA calls it.
template <class R>
__device__ __forceinline__ void fwd_triangle_stage(const Sched& S, int eb, const cx<R>* Lb, long long lstride, int s,
                                                   int blk, unsigned char* smem) {
    const int j0 = blk * kSolveBlock, m = S.rows[s];
    const int jb = min(kSolveBlock, S.first[s + 1] - S.first[s] - j0);
    stage_block(reinterpret_cast<cx<R>*>(smem), Lb + lstride * eb + S.loff[s] + j0 + static_cast<long long>(j0) * m, m,
                jb, jb);
}
template <class R>
__device__ void fwd_triangle(const Sched& S, const SolveArgs& a, int eb, cx<R>* yb, int s, int blk,
                             unsigned char* smem) {
    static_assert(kSolveBlock == 64, "two rows per lane");
    const cx<R>* T = reinterpret_cast<const cx<R>*>(smem);
    const int j0 = blk * kSolveBlock;
    const int f = S.first[s];
    const int jb = min(kSolveBlock, S.first[s + 1] - f - j0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    cx<R>* y = yb + vec_at(a, eb, warp) * a.n + f + j0;
    cx<R> y0{0, 0}, y1{0, 0};
    if (warp < a.nr) {
        if (lane < jb) y0 = ld_l2(y + lane);
        if (lane + 32 < jb) y1 = ld_l2(y + lane + 32);
    }
    triangle_wait();
    __syncthreads();
    if (warp < a.nr) {
        const int j1 = min(jb, 32);
#pragma unroll 4
        for (int j = 0; j < j1; ++j) {
            cx<R> yj;
            yj.re = __shfl_sync(0xffffffffu, y0.re, j);
            yj.im = __shfl_sync(0xffffffffu, y0.im, j);
            const cx<R> l0 = T[lane + j * kTriLd], l1 = T[lane + 32 + j * kTriLd];
            if (lane > j) y0 = fms(y0, l0, yj);
            if (lane + 32 < jb) y1 = fms(y1, l1, yj);
        }
#pragma unroll 4
        for (int j = 32; j < jb; ++j) {
            cx<R> yj;
            yj.re = __shfl_sync(0xffffffffu, y1.re, j & 31);
            yj.im = __shfl_sync(0xffffffffu, y1.im, j & 31);
            const cx<R> l1 = T[lane + 32 + j * kTriLd];
            if (lane + 32 > j && lane + 32 < jb) y1 = fms(y1, l1, yj);
        }
        if (lane < jb) y[lane] = y0;
        if (lane + 32 < jb) y[lane + 32] = y1;
    }
}

// Item (s), blockIdx.z: the children's update vectors added into rows
// 512 z .. of supernode s's front vector (y at its pivot rows, its own update
// segment U_s below), children in order, every rhs of the pass at once. A CTA
// reads each child's map whole and takes the entries in its rows. Fused: the
// front's first CTA then solves the supernode's first block (dynamic shared
// memory kTriSmem entries).
template <class R, bool Fused>
__global__ void __launch_bounds__(256) k_fwd_gather(Sched S, long long item0, SolveArgs a, const cx<R>* Lb,
                                                    long long lstride, cx<R>* yb, cx<R>* Ub) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    pdl_start_next();
    const int eb = solve_entry(a);
    const int s = S.items[item0 + blockIdx.x].s;
    const int w = S.first[s + 1] - S.first[s];
    const int m = S.rows[s];
    const int f = S.first[s];
    const int r0 = blockIdx.z * kGatherRows, r1 = min(r0 + kGatherRows, m);
    const bool triangle = Fused && blockIdx.z == 0 && w > 0;
    if constexpr (Fused)
        if (triangle) fwd_triangle_stage<R>(S, eb, Lb, lstride, s, 0, smem_raw);
    pdl_wait();
    if (r0 < m) {
        cx<R>* const y = yb + vec_at(a, eb, 0) * a.n + f;
        cx<R>* const U = Ub + vec_at(a, eb, 0) * a.upool;
        cx<R>* const Us = U + S.uoff[s];
        for (int i = max(r0, w) + threadIdx.x; i < r1; i += blockDim.x)
            for (int k = 0; k < a.nr; ++k) Us[k * a.upool + i - w] = cx<R>{0, 0};
        __syncthreads();
        for (int t = S.child_ptr[s]; t < S.child_ptr[s + 1]; ++t) {
            const int c = S.child_list[t];
            const int cc = S.rows[c] - (S.first[c + 1] - S.first[c]);
            const int* rel = S.rel + S.reloff[c];
            const cx<R>* Uc = U + S.uoff[c];
#pragma unroll 4
            for (int i = threadIdx.x; i < cc; i += blockDim.x) {
                const int p = rel[i];
                if (p < r0 || p >= r1) continue;
                cx<R>* dst = p < w ? y + p : Us + (p - w);
                const long long step = p < w ? a.n : a.upool;
                for (int k = 0; k < a.nr; ++k) dst[k * step] = dst[k * step] + Uc[k * a.upool + i];
            }
            __syncthreads();
        }
    }
    if constexpr (Fused) {
        if (!triangle) return;
        __threadfence();
        __syncthreads();
        fwd_triangle<R>(S, a, eb, yb, s, 0, smem_raw);
    }
}

// Item (s, blk): y[blk] = L_bb^-1 y[blk] (the split plan's triangle launch).
template <class R>
__global__ void __launch_bounds__(256) k_fwd_diag(Sched S, long long item0, SolveArgs a, const cx<R>* Lb,
                                                  long long lstride, cx<R>* yb) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    pdl_start_next();
    const Item it = S.items[item0 + blockIdx.x];
    const int eb = solve_entry(a);
    fwd_triangle_stage<R>(S, eb, Lb, lstride, it.s, it.a, smem_raw);
    pdl_wait();
    fwd_triangle<R>(S, a, eb, yb, it.s, it.a, smem_raw);
}

// Item (s, blk, row0): rows row0 .. row0 + kSolveRows - 1 of the supernode
// minus L[rows, blk] y[blk]. Four threads per row, each over 16 of the
// block's columns, all 16 loads in flight before the launch before has
// finished; the four column-ordered sub-sums are added in order, rhs k by the
// row's thread k % 4. Fused: the last of the block's CTAs then solves block
// blk + 1 (counters: one per supernode and grid row; dynamic shared memory
// kTriSmem entries).
template <class R, bool Fused>
__global__ void __launch_bounds__(256) k_fwd_update(Sched S, long long item0, SolveArgs a, const cx<R>* Lb,
                                                    long long lstride, cx<R>* yb, cx<R>* Ub) {
    static_assert(kSolveRows * 4 == 256 && kSolveBlock == 64, "four 16-column quarters per row");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ cx<R> ys[8][kSolveBlock];
    __shared__ cx<R> red[4][8][kSolveRows];  // the quarters' sub-sums
    pdl_start_next();
    const int eb = solve_entry(a);
    const Item it = S.items[item0 + blockIdx.x];
    const int s = it.s, j0 = it.a * kSolveBlock, row0 = it.b;
    const int w = S.first[s + 1] - S.first[s];
    const int m = S.rows[s];
    const int f = S.first[s];
    const int jb = min(kSolveBlock, w - j0);
    const int t = threadIdx.x % kSolveRows, qt = threadIdx.x / kSolveRows;
    const int r = row0 + t;
    const int c0 = 16 * qt, nc = min(16, jb - c0);
    cx<R> l[16];
    {
        const bool live = r < m && nc > 0;
        const cx<R>* P = Lb + lstride * eb + S.loff[s] + (live ? r : 0) + static_cast<long long>(j0 + c0) * m;
#pragma unroll
        for (int u = 0; u < 16; ++u) l[u] = live && u < nc ? P[static_cast<long long>(u) * m] : cx<R>{0, 0};
    }
    if constexpr (Fused) {
        const int jn = j0 + kSolveBlock;  // the next block, which this launch's last CTA solves
        if (row0 == j0 + jb && jn < w)
            prefetch_triangle(Lb + lstride * eb + S.loff[s] + jn + static_cast<long long>(jn) * m, m,
                              min(kSolveBlock, w - jn));
    }
    pdl_wait();
    // The destinations, read now (only this CTA writes these rows in this launch).
    auto at = [&](int k) {
        return r < w ? yb + vec_at(a, eb, k) * a.n + f + r : Ub + vec_at(a, eb, k) * a.upool + S.uoff[s] + (r - w);
    };
    cx<R> old[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) old[h] = r < m && qt + 4 * h < a.nr ? *at(qt + 4 * h) : cx<R>{0, 0};
    for (int e = threadIdx.x; e < kSolveBlock * a.nr; e += blockDim.x) {
        const int j = e % kSolveBlock, k = e / kSolveBlock;
        if (j < jb) ys[k][j] = yb[vec_at(a, eb, k) * a.n + f + j0 + j];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        if (k >= a.nr) break;
        cx<R> acc{0, 0};
        if (r < m && nc > 0) {
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                if (u >= nc) break;
                acc = acc + l[u] * ys[k][c0 + u];
            }
        }
        red[qt][k][t] = acc;
    }
    __syncthreads();
    if (r < m) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int k = qt + 4 * h;
            if (k < a.nr) *at(k) = old[h] - (((red[0][k][t] + red[1][k][t]) + red[2][k][t]) + red[3][k][t]);
        }
    }
    if constexpr (Fused) {
        const int below = j0 + jb;
        const int chunks = (m - below + kSolveRows - 1) / kSolveRows;
        if (last_to_arrive(a.counters + static_cast<long long>(blockIdx.y) * a.ns + s, chunks) &&
            it.a + 1 < solve_nblocks(S, s)) {
            fwd_triangle_stage<R>(S, eb, Lb, lstride, s, it.a + 1, smem_raw);
            fwd_triangle<R>(S, a, eb, yb, s, it.a + 1, smem_raw);
        }
    }
}

// Backward triangle of block blk of supernode s: x[blk] = L_bb^-T (D^-1
// y[blk] - sum of the partials in slots p0 .. p0 + np - 1) for the pass's
// rhs (smem: kTriSmem + red_smem(nr) entries, L_bb already being staged at its
// start). The partials are summed by kRedGroups threads per (column, rhs),
// each over every kRedGroups-th slot in slot order, the sub-sums then added in
// order. The triangle: one warp per rhs, lane l holding rows l and l + 32;
// step j (descending) broadcasts x_j from its owner lane and every lane above
// updates its rows, z_t = z_t - L_jt x_j. Every thread of the CTA calls it.
template <class R>
__device__ void bwd_triangle(const Sched& S, const SolveArgs& a, int eb, cx<R>* yb, const cx<R>* partb, int s,
                             int blk, int p0, int np, unsigned char* smem) {
    static_assert(kSolveBlock == 64, "two rows per lane");
    const cx<R>* T = reinterpret_cast<const cx<R>*>(smem);
    cx<R>* red = reinterpret_cast<cx<R>*>(smem) + kTriSmem;  // [group][rhs][column]
    const int j0 = blk * kSolveBlock;
    const int f = S.first[s];
    const int jb = min(kSolveBlock, S.first[s + 1] - f - j0);
    const cx<R>* part = partb + (static_cast<long long>(eb) * a.max_parts + p0) * (kSolveBlock * 8);
    for (int e = threadIdx.x; e < kRedGroups * kSolveBlock * a.nr; e += blockDim.x) {
        const int j = e % kSolveBlock, k = e / kSolveBlock % a.nr, g = e / kSolveBlock / a.nr;
        cx<R> sum{0, 0};
        if (j < jb) {
            const cx<R>* pj = part + k * kSolveBlock + j;
            constexpr int kU = 16, kSlot = kSolveBlock * 8;  // loads in flight per thread
            int q = g;
            for (; q + kRedGroups * (kU - 1) < np; q += kRedGroups * kU) {
                cx<R> v[kU];
#pragma unroll
                for (int u = 0; u < kU; ++u) v[u] = ld_l2(pj + static_cast<long long>(q + kRedGroups * u) * kSlot);
#pragma unroll
                for (int u = 0; u < kU; ++u) sum = sum + v[u];
            }
            if (q < np) {  // the rest, predicated, in flight too
                cx<R> v[kU];
#pragma unroll
                for (int u = 0; u < kU; ++u)
                    if (q + kRedGroups * u < np) v[u] = ld_l2(pj + static_cast<long long>(q + kRedGroups * u) * kSlot);
#pragma unroll
                for (int u = 0; u < kU; ++u)
                    if (q + kRedGroups * u < np) sum = sum + v[u];
            }
        }
        red[e] = sum;  // (g, k, j)
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    cx<R>* y = yb + vec_at(a, eb, warp) * a.n + f + j0;
    cx<R> z[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) z[h] = warp < a.nr && lane + 32 * h < jb ? ld_l2(y + lane + 32 * h) : cx<R>{0, 0};
    triangle_wait();
    __syncthreads();
    if (warp < a.nr) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int j = lane + 32 * h;
            if (j < jb) {
                const cx<R>* rj = red + warp * kSolveBlock + j;
                cx<R> sum = rj[0];
#pragma unroll
                for (int g = 1; g < kRedGroups; ++g) sum = sum + rj[g * kSolveBlock * a.nr];
                z[h] = z[h] * crecip(T[j * (kTriLd + 1)]) - sum;
            }
        }
#pragma unroll 4
        for (int j = jb - 1; j >= 32; --j) {
            cx<R> xj;
            xj.re = __shfl_sync(0xffffffffu, z[1].re, j & 31);
            xj.im = __shfl_sync(0xffffffffu, z[1].im, j & 31);
            const cx<R> l0 = T[j + lane * kTriLd], l1 = T[j + (lane + 32) * kTriLd];
            z[0] = fms(z[0], l0, xj);
            if (lane + 32 < j) z[1] = fms(z[1], l1, xj);
        }
#pragma unroll 4
        for (int j = min(jb, 32) - 1; j >= 0; --j) {
            cx<R> xj;
            xj.re = __shfl_sync(0xffffffffu, z[0].re, j);
            xj.im = __shfl_sync(0xffffffffu, z[0].im, j);
            const cx<R> l0 = T[j + lane * kTriLd];
            if (lane < j) z[0] = fms(z[0], l0, xj);
        }
        if (lane < jb) y[lane] = z[0];
        if (lane + 32 < jb) y[lane + 32] = z[1];
    }
}

// Item (s, blk, row0, slot[, p0]): partial[slot][k][j] = sum over rows
// row0 .. row0 + kSolveRows - 1 (below the block) of L[row, j0 + j] x_k[row]
// (an empty chunk, row0 = m, gives zeros). The rows' block of L is staged in
// shared memory before the launch before has finished; four threads per
// column, each over 16 of the rows in order for every rhs, the four sub-sums
// added in order. (One warp per eight columns with a butterfly per column and
// rhs took 52 us a launch for eight right-hand sides.) Fused: the last of the
// block's CTAs then reduces the block's partials (slots p0 ..) and solves the
// block (counters: one per supernode and grid row). Dynamic shared memory:
// kTriSmem entries, and red_smem(nr) more when fused.
template <class R, bool Fused>
__global__ void __launch_bounds__(256) k_bwd_update(Sched S, long long item0, SolveArgs a, const cx<R>* Lb,
                                                    long long lstride, cx<R>* yb, cx<R>* partb) {
    static_assert(kSolveRows == 64 && kSolveBlock == 64, "four 16-row quarters per column");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ cx<R> xs[8][kSolveRows];
    cx<R>* T = reinterpret_cast<cx<R>*>(smem_raw);
    pdl_start_next();
    const int eb = solve_entry(a);
    const Item it = S.items[item0 + blockIdx.x];
    const int s = it.s, j0 = it.a * kSolveBlock, row0 = it.b, slot = it.c;
    const int w = S.first[s + 1] - S.first[s];
    const int m = S.rows[s];
    const int f = S.first[s];
    const int jb = min(kSolveBlock, w - j0);
    const int nrows = max(0, min(kSolveRows, m - row0));
    const int* st = S.structs + S.soff[s];
    const cx<R>* P = Lb + lstride * eb + S.loff[s] + static_cast<long long>(j0) * m;
    stage_block(T, P + row0, m, nrows, jb);
    if constexpr (Fused) {
        if (row0 == j0 + jb)  // the block's triangle, which this launch's last CTA stages
            prefetch_triangle(P + j0, m, jb);
    }
    const int t = threadIdx.x % kSolveRows, qt = threadIdx.x / kSolveRows;
    const int g = t < nrows ? (row0 + t < w ? f + row0 + t : st[row0 + t]) : 0;
    pdl_wait();
    for (int k = qt; k < a.nr; k += 4)
        if (t < nrows) xs[k][t] = yb[vec_at(a, eb, k) * a.n + g];
    triangle_wait();
    __syncthreads();
    const int j = t;  // this thread's column
    cx<R> l[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) l[u] = T[16 * qt + u + j * kTriLd];
    __syncthreads();  // T becomes the quarters' sub-sums
    cx<R>* red = T;   // [quarter][rhs][column]
    static_assert(4 * 8 * kSolveBlock <= kTriSmem, "the sub-sums fit the block's memory");
    const int nq = min(16, nrows - 16 * qt);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        if (k >= a.nr) break;
        cx<R> acc{0, 0};
#pragma unroll
        for (int u = 0; u < 16; ++u)
            if (u < nq) acc = acc + l[u] * xs[k][16 * qt + u];
        red[(qt * 8 + k) * kSolveBlock + j] = acc;
    }
    __syncthreads();
    cx<R>* part = partb + (static_cast<long long>(eb) * a.max_parts + slot) * (kSolveBlock * 8);
    if (j < jb)
        for (int k = qt; k < a.nr; k += 4) {
            const cx<R>* rk = red + k * kSolveBlock + j;
            part[k * kSolveBlock + j] =
                ((rk[0] + rk[8 * kSolveBlock]) + rk[16 * kSolveBlock]) + rk[24 * kSolveBlock];
        }
    if constexpr (Fused) {
        const int below = j0 + jb;
        const int chunks = max(1, (m - below + kSolveRows - 1) / kSolveRows);
        if (last_to_arrive(a.counters + static_cast<long long>(blockIdx.y) * a.ns + s, chunks)) {
            stage_block(T, P + j0, m, jb, jb);
            bwd_triangle<R>(S, a, eb, yb, partb, s, it.a, it.d, chunks, smem_raw);
        }
    }
}

// Item (s, blk, first_slot, nslots): x[blk] = L_bb^-T (D^-1 y[blk] - sum of
// partials) (the split plan's triangle launch).
template <class R>
__global__ void __launch_bounds__(kBwdDiagThreads) k_bwd_diag(Sched S, long long item0, SolveArgs a, const cx<R>* Lb,
                                                              long long lstride, cx<R>* yb, const cx<R>* partb) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    pdl_start_next();
    const Item it = S.items[item0 + blockIdx.x];
    const int eb = solve_entry(a);
    const int j0 = it.a * kSolveBlock, m = S.rows[it.s];
    const int jb = min(kSolveBlock, S.first[it.s + 1] - S.first[it.s] - j0);
    stage_block(reinterpret_cast<cx<R>*>(smem_raw),
                Lb + lstride * eb + S.loff[it.s] + j0 + static_cast<long long>(j0) * m, m, jb, jb);
    pdl_wait();
    bwd_triangle<R>(S, a, eb, yb, partb, it.s, it.a, it.b, it.c, smem_raw);
}

}  // namespace aphi_b200
