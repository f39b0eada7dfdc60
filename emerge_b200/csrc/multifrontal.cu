// Multifrontal sparse LU of the sweep system on the device, the direct solve that replaces the
// reference's SolverSuperLU (src/emerge/_emerge/solver.py:535-572).  It factors the equilibrated
// D^-1/2 K D^-1/2 (D = |diag K|) with complex64 fronts, or complex128 fronts after
// emfem_mf_set_precision(lu, 128); the factor store is complex64 either way.
//
// The symbolic structure (nested-dissection tree, front DOF lists, extend-add maps, assembly lists) is
// built on the host (emerge_b200/direct.py) and uploaded once per mesh.  The numeric factorization runs
// level by level over the tree (all fronts of one height at once):
//   1. every front of the level is zeroed and gets its own entries of the scaled K (FP64 -> front
//      precision) and the Schur complements of its children (extend-add, one child slot after the other:
//      no atomics);
//   2. the first e columns of every front are eliminated in steps of 32: LU with partial pivoting inside
//      the 32 x 32 diagonal block (diag_kernel, one CTA of eight warps per front, also forming the explicit
//      inverses of its L and U), the block row (row swaps + L^-1) and block column (U^-1) of the panel
//      (panel_kernel), the update of the rest of the 128-column outer block (strip_kernel), and once per outer
//      block the rank-128 update of the trailing matrix (trail_kernel: tiles of 128 x 64 or 64 x 64,
//      8 x 4 or 4 x 4 complex accumulators per thread), every kernel batched over the level's fronts;
//   3. the factor columns, the U block row and the Schur complement are copied out of the level
//      workspace (compact_kernel): factors to the factor store (rounded to complex64), the Schur
//      complement to the update store (front precision) until the parent's level consumes it;
//   4. the 256 x 256 diagonal blocks are kept as the inverses of their L and U (block_inverse_kernel), so
//      that the solves have no 32-step chains.  The inverses are formed, stored and applied in FP64: their
//      entries grow (rows are not exchanged across steps), and products with them cancel.
// Pivoting stays inside each 32-row diagonal block (rows are never exchanged across blocks), so row swaps
// touch only the block row; the step's inverse of L holds them for the solves.  A pivot smaller than 1e-6 of its block's
// largest entry is raised to that floor and counted: the factorization is a preconditioner under an FP64
// Krylov iteration, which removes such perturbations.
//
// Solves (M^-1 r for S right-hand sides, FP64 in and out, FP32 inside but for the products with the block
// inverses, scaled by D^-1/2 on the way in and out) run the same tree: forward in level order (gather of the right-hand side and the children's
// update rows, then per 256 own rows the product with the block inverse and the update of the rows below),
// backward in reverse (U12 product with the solved boundary, then per 256 own rows, from the last).
#include "emfem_internal.cuh"

#include <algorithm>
#include <map>
#include <vector>

namespace emfem {

constexpr int MF_NB = 32;          // pivot block / elimination step
constexpr int MF_SB = 256;         // solve block
constexpr int MF_TILE = 64;        // trailing-update tile
constexpr long long MF_CHUNK = 4096;
constexpr int MF_MAX_FRONT = 46340; // n^2 must fit an int32 local offset

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ void cfma(float2& c, float2 a, float2 b) {
    c.x = fmaf(a.x, b.x, fmaf(-a.y, b.y, c.x));
    c.y = fmaf(a.x, b.y, fmaf(a.y, b.x, c.y));
}
__device__ __forceinline__ void cfms(float2& c, float2 a, float2 b) {   // c -= a b
    c.x = fmaf(-a.x, b.x, fmaf(a.y, b.y, c.x));
    c.y = fmaf(-a.x, b.y, fmaf(-a.y, b.x, c.y));
}
__device__ __forceinline__ float cabs2(float2 a) { return a.x * a.x + a.y * a.y; }

// 8-byte asynchronous global -> shared copies: a thread issues all of its copies before waiting once,
// so a staging loop costs one memory round trip instead of one per element
__device__ __forceinline__ void cp_async8(void* dst_smem, const void* src) {
    unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ float2 cinv(float2 a) {
    float d = 1.0f / cabs2(a);
    return make_float2(a.x * d, -a.y * d);
}

// The same operations in double precision (factorizations computed in complex128)
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ void cfma(double2& c, double2 a, double2 b) {
    c.x = fma(a.x, b.x, fma(-a.y, b.y, c.x));
    c.y = fma(a.x, b.y, fma(a.y, b.x, c.y));
}
__device__ __forceinline__ void cfms(double2& c, double2 a, double2 b) {
    c.x = fma(-a.x, b.x, fma(a.y, b.y, c.x));
    c.y = fma(-a.x, b.y, fma(-a.y, b.x, c.y));
}
__device__ __forceinline__ double cabs2(double2 a) { return a.x * a.x + a.y * a.y; }
__device__ __forceinline__ double2 cinv(double2 a) {
    double d = 1.0 / cabs2(a);
    return make_double2(a.x * d, -a.y * d);
}

// complex64 / complex128 element helpers for the templated factorization kernels
template <typename T> struct CxT;
template <> struct CxT<float2> {
    typedef float R;
    __device__ static float2 make(double x, double y) { return make_float2((float)x, (float)y); }
};
template <> struct CxT<double2> {
    typedef double R;
    __device__ static double2 make(double x, double y) { return make_double2(x, y); }
};
__device__ __forceinline__ float2 to_c64(float2 v) { return v; }
__device__ __forceinline__ float2 to_c64(double2 v) { return make_float2((float)v.x, (float)v.y); }
__device__ __forceinline__ void cp_async16(void* dst_smem, const void* src) {
    unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_c(float2* dst_smem, const float2* src) { cp_async8(dst_smem, src); }
__device__ __forceinline__ void cp_async_c(double2* dst_smem, const double2* src) { cp_async16(dst_smem, src); }

struct FrontMeta {        // per front, device
    int e, b, n, parent;
    int child[2];
    long long fdof, ea, asm0, asm1;   // offsets into fdof / ea / asm arrays
    long long fact, inv;              // factor store offset (float2), inverse store offset (double2)
    long long ws, upd;                // level workspace (float2) / update store (float2) offsets
    long long wv, y;                  // solve buffers: the front's rows of w, its own rows of y
};

// Stores of a front, 256 own columns [k0, k0 + w) at a time.
// Factor store (complex64): per block w columns of the n - w rows outside its diagonal block, after all blocks
// the e x b block row of U.
__host__ __device__ __forceinline__ long long mf_fact_block(int n, int k0) { return (long long)k0 * (n - MF_SB); }
__host__ __device__ inline long long mf_fact_rows_cols(int n, int e) {       // entries of the columns of all blocks
    const int last = e / MF_SB * MF_SB, w = e - last;
    return mf_fact_block(n, last) + (long long)w * (n - w);
}
// Inverse store (complex128): per block w columns of w + 32 entries.  Column c of the 32-column step j holds rows
// [0, 32 j + 32) of the inverse of U, then from entry 32 j + 32 on rows 32 j and up of the inverse of L (with the
// steps' row exchanges), so row r of the latter is entry r + 32.
__host__ __device__ __forceinline__ long long mf_inv_block(int k0) { return (long long)k0 * (MF_SB + MF_NB); }
__host__ __device__ inline long long mf_inv_entries(int e) {
    const int last = e / MF_SB * MF_SB, w = e - last;
    return mf_inv_block(last) + (long long)w * (w + MF_NB);
}

// ---------------------------------------------------------------- factorization kernels
// Symmetric diagonal equilibration: the factorization runs on D^-1/2 K D^-1/2 with D = |diag K|, so every
// pivot candidate is measured against unit diagonals.  Without it the gradient-type DOFs of the
// second-order basis (curl-curl column exactly zero, diagonal -k0^2 B_jj only) carry legitimate pivots
// far below the curl-curl scale at low frequency, and the 32-row pivot floor would perturb them.
// The scale of a DOF is set by the front that eliminates it, from its diagonal assembly entry.
__global__ void mf_scale_kernel(const int* __restrict__ lst, const FrontMeta* __restrict__ fm,
                                const double2* __restrict__ K, const int* __restrict__ slot, const int* __restrict__ off,
                                const int* __restrict__ fdof, double* __restrict__ scale) {
    const FrontMeta& f = fm[lst[blockIdx.y]];
    long long k0 = f.asm0 + (long long)blockIdx.x * MF_CHUNK;
    long long k1 = min(k0 + MF_CHUNK, f.asm1);
    const int n = f.n;
    for (long long k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
        const int o = off[k], li = o % n;
        if (li != o / n || li >= f.e) continue;
        double2 v = K[slot[k]];
        double a = fabs(v.x) + fabs(v.y);          // |.|_1 of the diagonal: scale only, no accuracy rides on it
        scale[fdof[f.fdof + li]] = a > 0.0 ? rsqrt(a) : 1.0;
    }
}

// Factorization kernels are templated on the workspace element T: float2 (complex64 fronts) or double2
// (complex128 fronts).  The factor store that the solves read is complex64 in both cases; a complex128
// factorization rounds its factors once, at compaction, so the rounding error does not compound through
// the Schur-complement chain.
template <typename T>
__global__ void mf_asm_kernel(const int* __restrict__ lst, const FrontMeta* __restrict__ fm,
                              const double2* __restrict__ K, const int* __restrict__ slot, const int* __restrict__ off,
                              const int* __restrict__ fdof, const double* __restrict__ scale, T* __restrict__ ws) {
    const FrontMeta& f = fm[lst[blockIdx.y]];
    long long k0 = f.asm0 + (long long)blockIdx.x * MF_CHUNK;
    long long k1 = min(k0 + MF_CHUNK, f.asm1);
    T* W = ws + f.ws;
    const int n = f.n;
    const int* D = fdof + f.fdof;
    for (long long k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
        const int o = off[k];
        double2 v = K[slot[k]];
        double sc = scale[D[o % n]] * scale[D[o / n]];
        W[o] = CxT<T>::make(v.x * sc, v.y * sc);
    }
}

// Extend-add of one child slot: a warp per column of the child's Schur complement (walking flat entries spent
// its time on 64-bit divisions: 290 us a launch on the 82 944-tet cavity, 260 now).
template <typename T>
__global__ void __launch_bounds__(256) mf_ea_kernel(const int* __restrict__ lst, const FrontMeta* __restrict__ fm, int cslot,
                                                    const int* __restrict__ ea, const T* __restrict__ upd, T* __restrict__ ws) {
    const FrontMeta& f = fm[lst[blockIdx.y]];
    const int c = f.child[cslot];
    if (c < 0) return;
    const FrontMeta& g = fm[c];
    const int nb = g.b, j = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (j >= nb) return;
    const int* map = ea + g.ea;
    const T* U = upd + g.upd + (long long)j * nb;
    T* W = ws + f.ws + (long long)map[j] * f.n;
    for (int i0 = threadIdx.x & 31; i0 < nb; i0 += 128) {
        T u[4], w[4];
        int r[4];
#pragma unroll
        for (int q = 0; q < 4; q++) r[q] = i0 + 32 * q < nb ? map[i0 + 32 * q] : -1;
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (r[q] >= 0) { u[q] = U[i0 + 32 * q]; w[q] = W[r[q]]; }
#pragma unroll
        for (int q = 0; q < 4; q++)            // a column's rows are distinct
            if (r[q] >= 0) { w[q].x += u[q].x; w[q].y += u[q].y; W[r[q]] = w[q]; }
    }
}

// Index order of non-negative values as unsigned words, for the pivot search (redux instructions).
__device__ __forceinline__ unsigned mf_max_key(float v, unsigned all, bool in) {
    const unsigned k = in ? __float_as_uint(v) : 0u;
    const unsigned mx = __reduce_max_sync(all, k);          // every lane takes part, candidate or not
    return __ballot_sync(all, in && k == mx);
}
__device__ __forceinline__ unsigned mf_max_key(double v, unsigned all, bool in) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const unsigned hi = in ? (unsigned)(b >> 32) : 0u;
    const unsigned mh = __reduce_max_sync(all, hi);
    const bool top = in && hi == mh;
    const unsigned lo = top ? (unsigned)b : 0u;
    const unsigned ml = __reduce_max_sync(all, lo);
    return __ballot_sync(all, top && lo == ml);
}
__device__ __forceinline__ float mf_shfl(float v, int l) { return __shfl_sync(0xffffffffu, v, l); }
__device__ __forceinline__ double mf_shfl(double v, int l) { return __shfl_sync(0xffffffffu, v, l); }

// LU with partial pivoting of the 32 x 32 diagonal block at step k, plus the explicit inverses of its
// unit-lower L and upper U.  One CTA per front: a serial step of every front's chain, bound by latency.  The block
// lives in shared memory by columns, warp w owning columns w, w + 8, ..; every warp finds the pivot of column j
// by itself (two or three redux instructions), rows keep their place and exchange their positions in `pos`, and
// one barrier a step passes the updated columns on.  Warps 0-3 then form the inverse of L and 4-7 that of U,
// eight columns per warp with a row per lane (32 steps of shuffles, no barrier).  Rolled loops: a warp with
// the block in registers needs straight-line code that the instruction cache cannot hold (45 us a step on the
// 82 944-tet cavity, as one warp in shared memory 64 us; now 20, complex128 27).  The inverses go to the diagonal
// blocks of the inverse store, read by the panel and block inverse kernels and by the solves.
template <typename T>
__global__ void __launch_bounds__(256) mf_diag_kernel(const int* __restrict__ lst, const FrontMeta* __restrict__ fm, int k,
                                                      T* __restrict__ ws, double2* __restrict__ inv,
                                                      int* __restrict__ nperturbed) {
    typedef typename CxT<T>::R R;
    __shared__ T D[MF_NB][MF_NB + 1];            // [column][row]: the block, then U
    __shared__ T L[MF_NB][MF_NB + 1];            // [column][row]: the multipliers
    __shared__ T dinv[MF_NB];
    __shared__ int sq[MF_NB];
    const FrontMeta& f = fm[lst[blockIdx.x]];
    if (k >= f.e) return;
    const unsigned all = 0xffffffffu;
    const int kb = min(MF_NB, f.e - k);
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    const long long ld = f.n;
    T* W = ws + f.ws + k + (long long)k * ld;
    const T zero = CxT<T>::make(0.0, 0.0);
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int c = wl + 8 * q;
        D[c][lane] = (lane < kb && c < kb) ? W[lane + (long long)c * ld] : zero;
        L[c][lane] = zero;
    }
    __syncthreads();
    R bmax = 0;
#pragma unroll
    for (int c = 0; c < MF_NB; c++) bmax = max(bmax, cabs2(D[c][lane]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) bmax = max(bmax, __shfl_xor_sync(all, bmax, o));
    const R floor2 = max(bmax, (R)1e-30) * (R)1e-12;      // (1e-6 of the block's largest entry)^2
    __syncthreads();                              // every warp has the same floor before any column changes
    int pos = lane, pert = 0;
    for (int j = 0; j < kb; j++) {
        // pivot: largest |row[j]| among the rows at positions >= j (ties: smallest position)
        const T aj = D[j][lane];
        const unsigned cand = mf_max_key(cabs2(aj), all, pos >= j && pos < kb);
        const unsigned key = (cand >> lane) & 1 ? (unsigned)pos : 64u;
        const int br = (int)__reduce_min_sync(all, key);
        const int bl = __ffs(__ballot_sync(all, pos == br)) - 1;
        pos = pos == br ? j : (pos == j ? br : pos);
        T d;
        d.x = mf_shfl(aj.x, bl);
        d.y = mf_shfl(aj.y, bl);
        if (cabs2(d) < floor2) {
            const R v = sqrt(cabs2(d)), fl = sqrt(floor2);
            d = v > 0 ? CxT<T>::make(d.x / v * fl, d.y / v * fl) : CxT<T>::make(fl, 0.0);
            pert++;
        }
        const T pinv = cinv(d);
        const bool low = pos > j && pos < kb;
        const T l = low ? cmul(aj, pinv) : zero;
        if (wl == 0) {
            L[j][lane] = l;
            if (lane == bl) dinv[j] = pinv;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int c = wl + 8 * q;
            if (c > j) {
                const T u = D[c][bl];
                if (low) cfms(D[c][lane], l, u);
            }
        }
        __syncthreads();                          // column j + 1 is up to date for every warp; column j is read
        if (lane == bl && wl == (j & 7)) D[j][lane] = d;          // the pivot as used
    }
    if (threadIdx.x == 0 && pert) atomicAdd(nperturbed, pert);
    if (wl == 0) sq[pos] = lane;
    __syncthreads();
    // rows in pivot order: entry (position i, column c) is L below the diagonal, D on and above it
    const int src = sq[lane];
    T row[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int c = wl + 8 * q;
        row[q] = lane > c ? L[c][src] : D[c][src];
        if (lane < kb && c < kb) W[lane + (long long)c * ld] = row[q];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int c = wl + 8 * q;
        D[c][lane] = row[q];
    }
    __syncthreads();
    const bool upper = wl >= 4;
    const int c0 = (wl & 3) * 8;
    T x[8];
#pragma unroll
    for (int q = 0; q < 8; q++) x[q] = CxT<T>::make(lane == c0 + q && lane < kb ? 1.0 : 0.0, 0.0);
    if (!upper) {
        for (int t = 0; t < kb; t++) {
            const T m = lane > t ? D[t][lane] : zero;
#pragma unroll
            for (int q = 0; q < 8; q++) {
                T v;
                v.x = mf_shfl(x[q].x, t);
                v.y = mf_shfl(x[q].y, t);
                cfms(x[q], m, v);
            }
        }
    } else {
        for (int t = kb - 1; t >= 0; t--) {
            const T m = lane < t ? D[t][lane] : zero, di = dinv[t];
#pragma unroll
            for (int q = 0; q < 8; q++) {
                T v;
                v.x = mf_shfl(x[q].x, t);
                v.y = mf_shfl(x[q].y, t);
                v = cmul(v, di);
                if (lane == t) x[q] = v;
                cfms(x[q], m, v);
            }
        }
    }
    // Linv P and Uinv.  The block's row swaps are folded into the inverse of L: position i holds row sq[i], so column
    // sq[c] of Linv P is column c of Linv.
    const int k0 = k / MF_SB * MF_SB, kl = k - k0, ldi = min(MF_SB, f.e - k0) + MF_NB;
    double2* I = inv + f.inv + mf_inv_block(k0) + (long long)kl * ldi + kl + (upper ? 0 : MF_NB) + lane;
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const int c = upper ? c0 + q : sq[c0 + q];
        if (lane < kb && c < kb) I[(long long)c * ldi] = make_double2(x[q].x, x[q].y);
    }
}

// Block row (columns >= k + kb): row swaps and L^-1; block column (rows >= k + kb): times U^-1.  A CTA takes a
// tile of TW columns (the first nt of grid.x) or rows, staged in shared memory with coalesced loads, as a
// small product with the 32 x 32 inverse, 2 x TW / 16 results per thread.  One row or column per thread
// read the block row with a stride of the front and ran on a fraction of the SMs: 58 us a step on the
// 82 944-tet cavity, 21 now.
template <typename T, int TW>
__global__ void __launch_bounds__(256) mf_panel_kernel(const int* __restrict__ lst, const FrontMeta* __restrict__ fm, int k,
                                                       int nt, T* __restrict__ ws, const double2* __restrict__ inv) {
    __shared__ T A[MF_NB][MF_NB + 1];                // inverse: [t][i] (block row) or [t][c] (block column)
    __shared__ T V[MF_NB][TW + 1];                   // tile: [t][column] or [t][row]
    const FrontMeta& f = fm[lst[blockIdx.y]];
    if (k >= f.e) return;
    const int kb = min(MF_NB, f.e - k), m = f.n - k - kb;
    const bool rowblk = (int)blockIdx.x < nt;
    const int x0 = ((int)blockIdx.x - (rowblk ? 0 : nt)) * TW;
    if (x0 >= m) return;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const long long ld = f.n;
    T* W = ws + f.ws;
    const T zero = CxT<T>::make(0.0, 0.0);
    const int k0 = k / MF_SB * MF_SB, kl = k - k0, ldi = min(MF_SB, f.e - k0) + MF_NB;
    const double2* I = inv + f.inv + mf_inv_block(k0) + (long long)kl * ldi + kl + (rowblk ? MF_NB : 0);
    constexpr int NJ = TW / 16;
    for (int q = tid; q < MF_NB * MF_NB; q += 256) {
        const int i = q % MF_NB, c = q / MF_NB;                // entry (i, c) of the step's inverse
        T v = zero;
        if (i < kb && c < kb) { const double2 d = I[i + c * ldi]; v = CxT<T>::make(d.x, d.y); }
        if (rowblk) A[c][i] = v; else A[i][c] = v;
    }
    if (rowblk) {
        T* C = W + k + (long long)(k + kb + x0) * ld;      // kb rows x (up to) TW columns
        for (int q = tid; q < MF_NB * TW; q += 256) {
            const int t = q % MF_NB, c = q / MF_NB;
            V[t][c] = (t < kb && x0 + c < m) ? C[t + c * ld] : zero;
        }
        __syncthreads();
        T o[2][NJ];
#pragma unroll
        for (int j = 0; j < NJ; j++) o[0][j] = o[1][j] = zero;
#pragma unroll 8
        for (int t = 0; t < MF_NB; t++) {
            const T a0 = A[t][tx], a1 = A[t][tx + 16];
#pragma unroll
            for (int j = 0; j < NJ; j++) {
                const T v = V[t][ty + 16 * j];
                cfma(o[0][j], a0, v);                 // (Linv P) times the column
                cfma(o[1][j], a1, v);
            }
        }
#pragma unroll
        for (int j = 0; j < NJ; j++) {
            const int c = ty + 16 * j;
            if (x0 + c >= m) continue;
            if (tx < kb) C[tx + c * ld] = o[0][j];
            if (tx + 16 < kb) C[tx + 16 + c * ld] = o[1][j];
        }
    } else {
        T* C = W + (k + kb + x0) + (long long)k * ld;      // (up to) TW rows x kb columns
        for (int q = tid; q < MF_NB * TW; q += 256) {
            const int r = q % TW, t = q / TW;
            V[t][r] = (t < kb && x0 + r < m) ? C[r + t * ld] : zero;
        }
        __syncthreads();
        T o[2][NJ];
#pragma unroll
        for (int j = 0; j < NJ; j++) o[0][j] = o[1][j] = zero;
#pragma unroll 8
        for (int t = 0; t < MF_NB; t++) {
            const T a0 = A[t][ty], a1 = A[t][ty + 16];
#pragma unroll
            for (int j = 0; j < NJ; j++) {
                const T v = V[t][tx + 16 * j];
                cfma(o[0][j], v, a0);
                cfma(o[1][j], v, a1);
            }
        }
#pragma unroll
        for (int j = 0; j < NJ; j++) {
            const int r = tx + 16 * j;
            if (x0 + r >= m) continue;
            if (ty < kb) C[r + ty * ld] = o[0][j];
            if (ty + 16 < kb) C[r + (ty + 16) * ld] = o[1][j];
        }
    }
}

// Update C -= A B of one tile of TM x 64 entries: A = W[rows, ka .. ka + kw), B = W[ka .. ka + kw, columns).
// 256 threads, TM / 16 x 4 accumulators each; the k extent runs in stages of KS columns, NSTG of them in
// flight by asynchronous copies, and the tile's C entries come straight into the accumulators meanwhile.
// Every entry is updated in ascending k, so how the k extent is cut into calls does not change a bit.
template <typename T> struct MfTile { static constexpr int KS = sizeof(T) == sizeof(float2) ? 16 : 8, NSTG = 3; };
template <typename T, int TM>
struct MfTileSmem {
    T a[MfTile<T>::NSTG][MfTile<T>::KS][TM + 1];
    T b[MfTile<T>::NSTG][MfTile<T>::KS][MF_TILE + 1];
};
template <typename T, int TM>
__device__ __forceinline__ void mf_tile_update(MfTileSmem<T, TM>& sm, T* W, int ld, int r0, int r1, int c0, int c1, int ka, int kw) {
    constexpr int KS = MfTile<T>::KS, NSTG = MfTile<T>::NSTG, NI = TM / 16;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const T zero = CxT<T>::make(0.0, 0.0);
    const int nst = (kw + KS - 1) / KS;
    const int ar = tid % TM, ak = tid / TM, bk = tid % KS, bc = tid / KS;       // the thread's share of a stage
    const T* A = W + r0 + ar + (long long)(ka + ak) * ld;
    const T* B = W + ka + bk + (long long)(c0 + bc) * ld;
    auto stage = [&](int st) {
        if (st < nst) {
            const int k0 = st * KS, slot = st % NSTG;
            const T* pa = A + (long long)k0 * ld;
#pragma unroll
            for (int u = 0; u < KS * TM / 256; u++) {
                const int kk = ak + u * (256 / TM);
                if (k0 + kk < kw && r0 + ar < r1) cp_async_c(&sm.a[slot][kk][ar], pa + (long long)(u * (256 / TM)) * ld);
                else sm.a[slot][kk][ar] = zero;
            }
            const T* pb = B + k0;
#pragma unroll
            for (int u = 0; u < KS * MF_TILE / 256; u++) {
                const int cc = bc + u * (256 / KS);
                if (k0 + bk < kw && c0 + cc < c1) cp_async_c(&sm.b[slot][bk][cc], pb + (long long)(u * (256 / KS)) * ld);
                else sm.b[slot][bk][cc] = zero;
            }
        }
        cp_async_commit();
    };
#pragma unroll
    for (int st = 0; st < NSTG - 1; st++) stage(st);
    T acc[NI][4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int c = c0 + ty + 16 * j;
#pragma unroll
        for (int i = 0; i < NI; i++) {
            const int r = r0 + tx + 16 * i;
            acc[i][j] = (r < r1 && c < c1) ? W[r + (long long)c * ld] : zero;
        }
    }
    for (int st = 0; st < nst; st++) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(NSTG - 2) : "memory");
        __syncthreads();                       // stage st has landed, stage st - 1 is consumed
        stage(st + NSTG - 1);
        const int slot = st % NSTG;
#pragma unroll
        for (int kk = 0; kk < KS; kk++) {
            T av[NI], bv[4];
#pragma unroll
            for (int i = 0; i < NI; i++) av[i] = sm.a[slot][kk][tx + 16 * i];
#pragma unroll
            for (int j = 0; j < 4; j++) bv[j] = sm.b[slot][kk][ty + 16 * j];
#pragma unroll
            for (int i = 0; i < NI; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) cfms(acc[i][j], av[i], bv[j]);
        }
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int c = c0 + ty + 16 * j;
        if (c >= c1) continue;
#pragma unroll
        for (int i = 0; i < NI; i++) {
            const int r = r0 + tx + 16 * i;
            if (r < r1) W[r + (long long)c * ld] = acc[i][j];
        }
    }
}

// The trailing update is cut in two: eliminating a step of 32 columns updates only the columns and rows of
// its outer block (MF_OB columns), which the block's next steps need, and the rest of the front is updated
// once per outer block with rank MF_OB.  C is then read and written once per MF_OB eliminated columns
// instead of once per 32: with rank 32 a tile moved 96 KB for a million flops, a quarter of DRAM's rate at half
// of the FMA pipe's, and the tiles' pipeline never filled.  Same sums in the same order.
constexpr int MF_OB = 128;

// Step k: strips of the outer block [ks, ke): columns [k + kb, ke) of all rows below k + kb (tiles x < nr), and
// rows [k + kb, ke) of the columns from ke on.
template <typename T>
__global__ void __launch_bounds__(256) mf_strip_kernel(const int* __restrict__ lst, const FrontMeta* __restrict__ fm, int k,
                                                       int ob, int nr, T* __restrict__ ws) {
    extern __shared__ __align__(16) unsigned char mf_smem[];
    MfTileSmem<T, 64>& sm = *reinterpret_cast<MfTileSmem<T, 64>*>(mf_smem);
    const FrontMeta& f = fm[lst[blockIdx.y]];
    const int k1 = k + MF_NB, ke = min(ob + MF_OB, f.e);
    if (k1 >= ke) return;                        // the outer block's last step: nothing left inside it
    const int half = blockIdx.x & 1, t = blockIdx.x >> 1;      // the strip is at most 96 wide: two tiles
    const bool cols = t < nr;
    const int along = (cols ? k1 : ke) + (cols ? t : t - nr) * 64, across = k1 + half * 64;
    if (along >= f.n || across >= ke) return;
    if (cols) mf_tile_update<T, 64>(sm, ws + f.ws, f.n, along, f.n, across, ke, k, MF_NB);
    else mf_tile_update<T, 64>(sm, ws + f.ws, f.n, across, ke, along, f.n, k, MF_NB);
}

// Rank-(ke - ob) update of everything below and right of the outer block [ob, ke)
template <typename T, int TM>
__global__ void __launch_bounds__(256, TM > 64 || sizeof(T) > 8 ? 2 : 3) mf_trail_kernel(const int* __restrict__ lst, const FrontMeta* __restrict__ fm,
                                                                         int ob, T* __restrict__ ws) {
    extern __shared__ __align__(16) unsigned char mf_smem[];
    MfTileSmem<T, TM>& sm = *reinterpret_cast<MfTileSmem<T, TM>*>(mf_smem);
    const FrontMeta& f = fm[lst[blockIdx.y]];
    if (ob >= f.e) return;
    const int ke = min(ob + MF_OB, f.e), m = f.n - ke;
    const int nr = (m + TM - 1) / TM, nc = (m + MF_TILE - 1) / MF_TILE;
    if ((int)blockIdx.x >= nr * nc) return;
    const int ti = blockIdx.x % nr, tj = blockIdx.x / nr;
    mf_tile_update<T, TM>(sm, ws + f.ws, f.n, ke + ti * TM, f.n, ke + tj * MF_TILE, f.n, ob, ke - ob);
}

// Factor columns (their rows outside the 256-blocks) and U block row (e x b), rounded to complex64, and the Schur
// complement (b x b, workspace precision) out of the workspace.
// (a warp per column: walking flat entries spent its time on 64-bit divisions, 611 us a launch on the 82 944-tet
// cavity, 469 now)
template <typename T>
__global__ void __launch_bounds__(256) mf_compact_kernel(const int* __restrict__ lst, const FrontMeta* __restrict__ fm,
                                                         const T* __restrict__ ws, float2* __restrict__ fact, T* __restrict__ upd) {
    const FrontMeta& f = fm[lst[blockIdx.y]];
    const int n = f.n, e = f.e, j = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (j >= n) return;
    const T* W = ws + f.ws + (long long)j * n;
    float2* F = fact + f.fact;
    if (j < e) {
        const int k0 = j / MF_SB * MF_SB, w = min(MF_SB, e - k0);
        F += mf_fact_block(n, k0) + (long long)(j - k0) * (n - w);
#pragma unroll 4
        for (int i = lane; i < k0; i += 32) F[i] = to_c64(W[i]);
#pragma unroll 4
        for (int i = k0 + lane; i < n - w; i += 32) F[i] = to_c64(W[i + w]);
        return;
    }
    F += mf_fact_rows_cols(n, e) + (long long)(j - e) * e;
#pragma unroll 4
    for (int i = lane; i < e; i += 32) F[i] = to_c64(W[i]);
    T* U = upd + f.upd + (long long)(j - e) * f.b;
#pragma unroll 4
    for (int i = lane; i < f.b; i += 32) U[i] = W[e + i];
}

// Inverses of the 256 x 256 diagonal blocks of L and U, below and above the steps' 32 x 32 inverses in the inverse store.
// With the step's inverses A_j = Linv_j P_j (mf_diag_kernel) on the diagonal, block column j of the inverse
// of the block-lower L is G_jj = A_j, G_ij = -A_i sum_{j <= t < i} L_it G_tj; that of U is H_jj = Uinv_j,
// H_ij = -Uinv_i sum_{i < t <= j} U_it H_tj.  One CTA per (block column, L or U, 256-block, front): the
// columns are independent, so nothing is serial but the at most 8 steps of one column.  FP64 for both front
// precisions: a product with G is then as accurate as the 32-step substitution with L (complex64 inverses
// were not: residual of one application 1.0e-4 -> 1.0e-3 on a 750-tet cavity, 0.12 -> 2.9 on a 3 696-tet
// substrate at 1 GHz).
constexpr int MF_NBB = MF_SB / MF_NB;
struct MfInvSmem {
    double2 x[MF_NBB][MF_NB][MF_NB + 1];       // the column's blocks, [block][row][column]
    double2 a[MF_NB][MF_NB + 1];
    double2 s[MF_NB][MF_NB + 1];
};
template <typename T>
__global__ void __launch_bounds__(256) mf_block_inverse_kernel(const int* __restrict__ lst, const FrontMeta* __restrict__ fm,
                                                               const T* __restrict__ ws, double2* __restrict__ inv) {
    extern __shared__ __align__(16) unsigned char mf_smem[];
    MfInvSmem& sm = *reinterpret_cast<MfInvSmem*>(mf_smem);
    const FrontMeta& f = fm[lst[blockIdx.z]];
    const int k0 = blockIdx.y * MF_SB;
    if (k0 >= f.e) return;
    const int rows = min(MF_SB, f.e - k0), ns = (rows + MF_NB - 1) / MF_NB;
    const int j = blockIdx.x >> 1;
    const bool upper = blockIdx.x & 1;
    if (j >= ns || (upper ? j == 0 : j == ns - 1)) return;       // no off-diagonal block in this column
    const long long n = f.n;
    const T* W = ws + f.ws + k0 + (long long)k0 * n;
    double2* I = inv + f.inv + mf_inv_block(k0) + (upper ? 0 : MF_NB);
    const int ldi = rows + MF_NB;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;   // thread: rows tx, tx + 16, columns ty, ty + 16
    const double2 zero = make_double2(0.0, 0.0);
    auto block = [&](int i, int q) {                             // entry q of the inverse of step i
        const int r = i * MF_NB + q % MF_NB, c = i * MF_NB + q / MF_NB;
        return r < rows && c < rows ? I[r + (long long)c * ldi] : zero;
    };
    for (int t = tid; t < MF_NB * MF_NB; t += 256) sm.x[j][t % MF_NB][t / MF_NB] = block(j, t);
    __syncthreads();
    const int step = upper ? -1 : 1;
    for (int i = j + step; upper ? i >= 0 : i < ns; i += step) {
        double2 acc[2][2] = {{zero, zero}, {zero, zero}};
        for (int t = j; t != i; t += step) {
            for (int q = tid; q < MF_NB * MF_NB; q += 256) {
                const int r = q % MF_NB, c = q / MF_NB;
                double2 v = zero;
                if (i * MF_NB + r < rows && t * MF_NB + c < rows) {
                    const T l = W[i * MF_NB + r + (long long)(t * MF_NB + c) * n];
                    v = make_double2(l.x, l.y);
                }
                sm.a[r][c] = v;
            }
            __syncthreads();
#pragma unroll 8
            for (int k = 0; k < MF_NB; k++) {
                const double2 a0 = sm.a[tx][k], a1 = sm.a[tx + 16][k], b0 = sm.x[t][k][ty], b1 = sm.x[t][k][ty + 16];
                cfma(acc[0][0], a0, b0); cfma(acc[0][1], a0, b1); cfma(acc[1][0], a1, b0); cfma(acc[1][1], a1, b1);
            }
            __syncthreads();
        }
#pragma unroll
        for (int p = 0; p < 2; p++)
#pragma unroll
            for (int q = 0; q < 2; q++) sm.s[tx + 16 * p][ty + 16 * q] = acc[p][q];
        for (int q = tid; q < MF_NB * MF_NB; q += 256) sm.a[q % MF_NB][q / MF_NB] = block(i, q);
        __syncthreads();
        double2 o[2][2] = {{zero, zero}, {zero, zero}};
#pragma unroll 8
        for (int k = 0; k < MF_NB; k++) {
            const double2 a0 = sm.a[tx][k], a1 = sm.a[tx + 16][k], b0 = sm.s[k][ty], b1 = sm.s[k][ty + 16];
            cfms(o[0][0], a0, b0); cfms(o[0][1], a0, b1); cfms(o[1][0], a1, b0); cfms(o[1][1], a1, b1);
        }
#pragma unroll
        for (int p = 0; p < 2; p++)
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const int r = tx + 16 * p, c = ty + 16 * q;
                sm.x[i][r][c] = o[p][q];
                if (i * MF_NB + r < rows && j * MF_NB + c < rows)
                    I[i * MF_NB + r + (long long)(j * MF_NB + c) * ldi] = o[p][q];
            }
        __syncthreads();
    }
}

// ---------------------------------------------------------------- assembly lists on the device
// Every CSR entry (r, c) of the free rows and columns belongs to the front that eliminates the earlier of
// r and c; its local row/column is the DOF's own index there, or e + its index among the front's boundary
// DOFs (sorted by elimination position: binary search).
__device__ __forceinline__ int mf_local(const FrontMeta& f, int v, int d, int p, const int* __restrict__ fpos,
                                        const long long* __restrict__ own0, const int* __restrict__ fdof,
                                        const int* __restrict__ pos) {
    if (fpos[p] == v) return (int)(p - own0[v]);
    int lo = f.e, hi = f.n - 1;
    const int* D = fdof + f.fdof;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (pos[D[mid]] < p) lo = mid + 1; else hi = mid;
    }
    return (lo < f.n && D[lo] == d) ? lo : -1;
}

__global__ void mf_list_count_kernel(long long n, const int* __restrict__ indptr, const int* __restrict__ indices,
                                     const int* __restrict__ pos, const int* __restrict__ fpos, int* __restrict__ cnt) {
    long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const int pr = pos[r];
    if (pr < 0) return;
    for (int k = indptr[r]; k < indptr[r + 1]; k++) {
        const int pc = pos[indices[k]];
        if (pc < 0) continue;
        atomicAdd(&cnt[fpos[min(pr, pc)]], 1);
    }
}

__global__ void mf_list_fill_kernel(long long n, const int* __restrict__ indptr, const int* __restrict__ indices,
                                    const int* __restrict__ pos, const int* __restrict__ fpos,
                                    const long long* __restrict__ own0, const FrontMeta* __restrict__ fm,
                                    const int* __restrict__ fdof, const int* __restrict__ base, int* __restrict__ cur,
                                    int* __restrict__ slot, int* __restrict__ off, int* __restrict__ status) {
    long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const int pr = pos[r];
    if (pr < 0) return;
    for (int k = indptr[r]; k < indptr[r + 1]; k++) {
        const int c = indices[k];
        const int pc = pos[c];
        if (pc < 0) continue;
        const int v = fpos[min(pr, pc)];
        const FrontMeta& f = fm[v];
        const int li = mf_local(f, v, (int)r, pr, fpos, own0, fdof, pos);
        const int lj = mf_local(f, v, c, pc, fpos, own0, fdof, pos);
        const int q = base[v] + atomicAdd(&cur[v], 1);
        if (li < 0 || lj < 0) {
            flag(status, DEV_BAD_INDEX);
            slot[q] = k;
            off[q] = 0;
            continue;
        }
        slot[q] = k;
        off[q] = li + lj * f.n;
    }
}

// ---------------------------------------------------------------- solve kernels
// Rows of the two children's fronts that each front row receives (absolute rows of w, -1: none), built once:
// the children's boundary rows are their update vectors.
__global__ void mf_child_rows_kernel(int v0, int nf, const FrontMeta* __restrict__ fm, const int* __restrict__ ea,
                                     int* __restrict__ cmap, long long rows) {
    const int v = v0 + blockIdx.y;
    if (v >= nf) return;
    const FrontMeta& g = fm[v];
    if (g.parent < 0) return;
    const FrontMeta& f = fm[g.parent];
    int* M = cmap + (f.child[0] == v ? 0 : rows) + f.wv;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < g.b; i += gridDim.x * blockDim.x)
        M[ea[g.ea + i]] = (int)(g.wv + g.e + i);
}

// The kernels of an application are a chain of some 250 short dependent launches, so each is launched before its
// predecessor has ended (programmatic stream serialization): it loads what the factorization left (maps and the
// first factor columns), waits for the predecessor, and only then touches the vectors, past L1, which may hold lines
// from before the predecessor's stores.  Every block waits, also one with nothing to do: a kernel that ended
// earlier would let its successor pass the one before.
__device__ __forceinline__ void mf_chain_start() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void mf_chain_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ float2 mf_vec(const float2* p) {
    float2 v;
    asm volatile("ld.global.cg.v2.f32 {%0, %1}, [%2];\n" : "=f"(v.x), "=f"(v.y) : "l"(p) : "memory");
    return v;
}
template <typename... P, typename... A>
static void mf_chain(void (*kernel)(P...), dim3 grid, cudaStream_t s, A... args) {
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = dim3(256);
    c.stream = s;
    c.attrs = &at;
    c.numAttrs = 1;
    cudaLaunchKernelEx(&c, kernel, P(args)...);
}

// w (the front's rows, S per row): own rows from the right-hand side, plus both children's update rows
__global__ void mf_fwd_gather_kernel(const int* __restrict__ lst, const FrontMeta* __restrict__ fm, int S,
                                     const int* __restrict__ fdof, const double* __restrict__ scale,
                                     const int* __restrict__ cmap, long long rows, MfCols cols, const double2* __restrict__ rhs,
                                     float2* __restrict__ w) {
    mf_chain_start();
    const FrontMeta& f = fm[lst[blockIdx.y]];
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)f.n * S) { mf_chain_wait(); return; }
    const int i = (int)(idx / S), s = (int)(idx % S);
    const int a = cmap[f.wv + i], b = cmap[rows + f.wv + i];
    float2 v = make_float2(0.f, 0.f);
    if (i < f.e) {
        const int d = fdof[f.fdof + i];
        const double2 r = rhs[(long long)d * cols.ld + (cols.count == cols.ld ? s : cols.m[s])];
        const double sc = scale[d];
        v = make_float2((float)(r.x * sc), (float)(r.y * sc));
    }
    mf_chain_wait();
    if (a >= 0) { const float2 u = mf_vec(w + (long long)a * S + s); v.x += u.x; v.y += u.y; }
    if (b >= 0) { const float2 u = mf_vec(w + (long long)b * S + s); v.x += u.x; v.y += u.y; }
    w[f.wv * S + idx] = v;
}

// One product of a solve: t[r] = sum_{c in [c0, c1)} M[r, c] x[c] for a tile of 32 RPL rows and NS right-hand
// sides.  Each of the 8 warps takes every 8th column, lane rl holding rows rl + 32 i, so that a warp reads
// 256 RPL contiguous bytes of a column; the columns' x values (S per row) are staged in shared memory, 256
// columns at a time, and the warps' sums meet there in a fixed order.  It streams the factors once; what
// bounds it is how many of a stage's columns are in flight (the loop is unrolled 8 deep).
constexpr int MF_KC = MF_SB;
template <int NS>
struct MfProdSmem {
    alignas(16) float2 x[MF_KC][NS];
    float2 red[8][NS < 4 ? NS : 4][64];
};

// Columns [c0, c0 + nc) of x into shared memory: XOf(c) points at column c's values, ns of them real
template <int NS, typename XOf>
__device__ __forceinline__ void mf_stage_x(MfProdSmem<NS>& sm, int c0, int nc, int ns, XOf xof) {
    for (int t = threadIdx.x; t < nc * NS; t += 256) {
        const int c = t / NS, q = t % NS;
        sm.x[c][q] = q < ns ? mf_vec(xof(c0 + c) + q) : make_float2(0.f, 0.f);
    }
}

// acc += staged columns [0, nc) times M: MAt(i, c) is entry (row rl + 32 i of the tile, staged column c).  A warp
// takes every eighth column, U of them at once with the columns past the end masked: a plain unrolled loop runs
// its remainder one load latency per column
template <int RPL, int U, typename MAt>
__device__ __forceinline__ void mf_load(float2 (*mv)[RPL], int c0, int nc, MAt mat) {
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
        for (int i = 0; i < RPL; i++) mv[u][i] = c0 + 8 * u < nc ? mat(i, c0 + 8 * u) : make_float2(0.f, 0.f);
}
// mv: this warp's first columns, loaded
template <int NS, int RPL, int U, typename MAt>
__device__ __forceinline__ void mf_accumulate(const MfProdSmem<NS>& sm, float2 (*acc)[NS], float2 (*mv)[RPL], int nc, MAt mat) {
    for (int c0 = threadIdx.x >> 5; c0 < nc;) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int c = c0 + 8 * u;
            if (c >= nc) break;              // the same for the whole warp
            if constexpr (NS > 1) {          // two right-hand sides per 16-byte read
#pragma unroll
                for (int q = 0; q < NS; q += 2) {
                    const float4 xv = *reinterpret_cast<const float4*>(&sm.x[c][q]);
#pragma unroll
                    for (int i = 0; i < RPL; i++) {
                        cfma(acc[i][q], mv[u][i], make_float2(xv.x, xv.y));
                        cfma(acc[i][q + 1], mv[u][i], make_float2(xv.z, xv.w));
                    }
                }
            } else {
#pragma unroll
                for (int i = 0; i < RPL; i++) cfma(acc[i][0], mv[u][i], sm.x[c][0]);
            }
        }
        c0 += 8 * U;
        if (c0 < nc) mf_load<RPL, U>(mv, c0, nc, mat);
    }
}

// The warps' sums in order, Out(row of the tile, right-hand side, value)
template <int NS, int RPL, typename Out>
__device__ __forceinline__ void mf_finish(MfProdSmem<NS>& sm, float2 (*acc)[NS], int ns, Out out) {
    const int rl = threadIdx.x & 31, g = threadIdx.x >> 5;
    constexpr int QB = NS < 4 ? NS : 4;
#pragma unroll
    for (int q0 = 0; q0 < NS; q0 += QB) {
        if (q0) __syncthreads();
#pragma unroll
        for (int i = 0; i < RPL; i++)
#pragma unroll
            for (int q = 0; q < QB; q++) sm.red[g][q][rl + 32 * i] = acc[i][q0 + q];
        __syncthreads();
        for (int t = threadIdx.x; t < 32 * RPL * QB; t += 256) {
            const int q = t / (32 * RPL), r = t % (32 * RPL);
            if (q0 + q >= ns) continue;
            float2 v = make_float2(0.f, 0.f);
#pragma unroll
            for (int gg = 0; gg < 8; gg++) { v.x += sm.red[gg][q][r].x; v.y += sm.red[gg][q][r].y; }
            out(r, q0 + q, v);
        }
    }
}

template <int NS, int RPL, typename XOf, typename MAt, typename Out>
__device__ __forceinline__ void mf_product(MfProdSmem<NS>& sm, int c0, int c1, int ns, XOf xof, MAt mat, Out out) {
    float2 acc[RPL][NS] = {};
    if (c0 >= c1) mf_chain_wait();
    for (int cb = c0; cb < c1; cb += MF_KC) {
        const int nc = min(MF_KC, c1 - cb);
        auto at = [&](int i, int c) { return mat(i, cb + c); };
        float2 mv[8][RPL];
        mf_load<RPL, 8>(mv, threadIdx.x >> 5, nc, at);
        if (cb == c0) mf_chain_wait();
        else __syncthreads();
        mf_stage_x(sm, cb, nc, ns, xof);
        __syncthreads();
        mf_accumulate<NS, RPL, 8>(sm, acc, mv, nc, at);
    }
    mf_finish<NS, RPL>(sm, acc, ns, out);
}

// Products with the block inverses, FP64 inside (inverse entries and sums; x and the result are complex64): 32 rows per
// CTA, a warp takes every eighth of the nc columns, 16 of them in flight.  M: entry (the CTA's first row, first
// column), XOf(c) points at column c's x values, Out(row of the tile, right-hand side, value).  Latency bounds it at
// the few-front levels: the FP64 multiply-adds of an application to 8 columns take 60 us at 24 576 tets.
template <int NS>
struct MfTriSmem {
    double2 x[MF_SB][NS];
    double2 red[8][NS < 4 ? NS : 4][MF_NB];
};
template <int NS, typename XOf, typename Out>
__device__ __forceinline__ void mf_tri_product(MfTriSmem<NS>& sm, const double2* M, int ldm, int nr, int nc, int ns, XOf xof, Out out) {
    constexpr int U = 16, QB = NS < 4 ? NS : 4;
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
    const double2 zero = make_double2(0.0, 0.0);
    double2 acc[NS], mv[U];
#pragma unroll
    for (int q = 0; q < NS; q++) acc[q] = zero;
    auto load = [&](int c0) {
#pragma unroll
        for (int u = 0; u < U; u++) mv[u] = lane < nr && c0 + 8 * u < nc ? M[lane + (long long)(c0 + 8 * u) * ldm] : zero;
    };
    load(g);
    mf_chain_wait();
    for (int t = threadIdx.x; t < nc * NS; t += 256) {
        const int c = t / NS, q = t % NS;
        const float2 v = q < ns ? mf_vec(xof(c) + q) : make_float2(0.f, 0.f);
        sm.x[c][q] = make_double2(v.x, v.y);
    }
    __syncthreads();
    for (int c0 = g; c0 < nc;) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int c = c0 + 8 * u;
            if (c >= nc) break;              // the same for the whole warp
#pragma unroll
            for (int q = 0; q < NS; q++) cfma(acc[q], mv[u], sm.x[c][q]);
        }
        c0 += 8 * U;
        if (c0 < nc) load(c0);
    }
#pragma unroll
    for (int q0 = 0; q0 < NS; q0 += QB) {    // the warps' sums in order
        if (q0) __syncthreads();
#pragma unroll
        for (int q = 0; q < QB; q++) sm.red[g][q][lane] = acc[q0 + q];
        __syncthreads();
        for (int t = threadIdx.x; t < MF_NB * QB; t += 256) {
            const int q = t / MF_NB, r = t % MF_NB;
            if (q0 + q >= ns || r >= nr) continue;
            double2 v = zero;
#pragma unroll
            for (int gg = 0; gg < 8; gg++) { v.x += sm.red[gg][q][r].x; v.y += sm.red[gg][q][r].y; }
            out(r, q0 + q, make_float2((float)v.x, (float)v.y));
        }
    }
}

// y[k0 .. k1) = G w[k0 .. k1), G the inverse of the 256-block of L
template <int NS>
__global__ void __launch_bounds__(256) mf_fwd_tri_kernel(const int* __restrict__ lst, const FrontMeta* __restrict__ fm,
                                                         int S, int k0, const double2* __restrict__ inv,
                                                         const float2* __restrict__ w, float2* __restrict__ y) {
    __shared__ MfTriSmem<NS> sm;
    mf_chain_start();
    const FrontMeta& f = fm[lst[blockIdx.y]];
    const int r0 = k0 + blockIdx.x * MF_NB;
    if (r0 >= f.e) { mf_chain_wait(); return; }
    const int s0 = blockIdx.z * NS, ns = min(NS, S - s0), nr = min(MF_NB, f.e - r0), ldi = min(MF_SB, f.e - k0) + MF_NB;
    const float2* X = w + (f.wv + k0) * S + s0;
    float2* Y = y + (f.y + r0) * S + s0;
    mf_tri_product<NS>(sm, inv + f.inv + mf_inv_block(k0) + (r0 - k0) + MF_NB, ldi, nr, r0 - k0 + nr, ns,
                       [&](int c) { return X + (long long)c * S; },
                       [&](int t, int q, float2 v) { Y[(long long)t * S + q] = v; });
}

// rows [k1, n): w[r] -= L[r, k0:k1] y[k0:k1]
template <int NS, int RPL>
__global__ void __launch_bounds__(256, NS * RPL > 16 ? 2 : 3) mf_fwd_update_kernel(const int* __restrict__ lst, const FrontMeta* __restrict__ fm,
                                                            int S, int k0, const float2* __restrict__ fact,
                                                            const float2* __restrict__ y, float2* __restrict__ w) {
    __shared__ MfProdSmem<NS> sm;
    mf_chain_start();
    const FrontMeta& f = fm[lst[blockIdx.y]];
    if (k0 >= f.e) { mf_chain_wait(); return; }
    const int k1 = min(k0 + MF_SB, f.e);
    const int r0 = k1 + blockIdx.x * 32 * RPL;
    if (r0 >= f.n) { mf_chain_wait(); return; }
    const int s0 = blockIdx.z * NS, ns = min(NS, S - s0), r = r0 + (threadIdx.x & 31);
    const long long n = f.n, ldf = n - (k1 - k0);
    const float2* F = fact + f.fact + mf_fact_block(f.n, k0) + r - (k1 - k0);         // column c of the block at c ldf
    const float2* X = y + f.y * S + s0;
    float2* W = w + f.wv * S + s0;
    mf_product<NS, RPL>(sm, k0, k1, ns, [&](int c) { return X + (long long)c * S; },
                        [&](int i, int c) { return r + 32 * i < n ? F[32 * i + (c - k0) * ldf] : make_float2(0.f, 0.f); },
                        [&](int t, int q, float2 v) {
                            if (r0 + t >= n) return;
                            float2* p = W + (long long)(r0 + t) * S + q;
                            const float2 o = mf_vec(p);
                            *p = make_float2(o.x - v.x, o.y - v.y);
                        });
}

// own rows: y[r] -= U12[r, :] x_bnd (U12 is e x b, column-major with ld e; x_bnd = the solved x of the boundary
// DOFs).  Levels of few fronts split the columns over nsplit CTAs of cw columns; their sums go to part and
// mf_bwd_bnd_sum_kernel subtracts them in order.
template <int NS, int RPL>
__global__ void __launch_bounds__(256, NS * RPL > 16 ? 2 : 3) mf_bwd_bnd_kernel(const int* __restrict__ lst, const FrontMeta* __restrict__ fm, int S,
                                                         int nrt, int nsplit, int cw, long long y0, long long yl,
                                                         const float2* __restrict__ fact, const int* __restrict__ fdof,
                                                         const float2* __restrict__ xs, float2* __restrict__ y,
                                                         float2* __restrict__ part) {
    __shared__ MfProdSmem<NS> sm;
    mf_chain_start();
    const FrontMeta& f = fm[lst[blockIdx.y]];
    const int r0 = (blockIdx.x % nrt) * 32 * RPL, sp = blockIdx.x / nrt;
    if (f.b == 0 || r0 >= f.e) { mf_chain_wait(); return; }
    const int s0 = blockIdx.z * NS, ns = min(NS, S - s0), r = r0 + (threadIdx.x & 31);
    const long long e = f.e;
    const float2* M = fact + f.fact + mf_fact_rows_cols(f.n, f.e) + r;
    const int* d = fdof + f.fdof + e;
    const float2* X = xs + s0;
    const int c0 = min(sp * cw, f.b), c1 = nsplit > 1 ? min(c0 + cw, f.b) : f.b;
    float2* Y = nsplit > 1 ? part + ((long long)sp * yl + f.y - y0) * S + s0 : y + f.y * S + s0;
    mf_product<NS, RPL>(sm, c0, c1, ns, [&](int c) { return X + (long long)d[c] * S; },
                        [&](int i, int c) { return r + 32 * i < e ? M[32 * i + c * e] : make_float2(0.f, 0.f); },
                        [&](int t, int q, float2 v) {
                            if (r0 + t >= e) return;
                            float2* p = Y + (long long)(r0 + t) * S + q;
                            if (nsplit > 1) { *p = v; return; }
                            const float2 o = mf_vec(p);
                            *p = make_float2(o.x - v.x, o.y - v.y);
                        });
}

__global__ void mf_bwd_bnd_sum_kernel(const int* __restrict__ lst, const FrontMeta* __restrict__ fm, int S, int nsplit,
                                      long long y0, long long yl, const float2* __restrict__ part, float2* __restrict__ y) {
    mf_chain_start();
    const FrontMeta& f = fm[lst[blockIdx.y]];
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    mf_chain_wait();
    if (f.b == 0 || idx >= (long long)f.e * S) return;
    float2 t = make_float2(0.f, 0.f);
    for (int sp = 0; sp < nsplit; sp++) {
        const float2 v = mf_vec(part + ((long long)sp * yl + f.y - y0) * S + idx);
        t.x += v.x;
        t.y += v.y;
    }
    float2* p = y + f.y * S + idx;
    const float2 o = mf_vec(p);
    *p = make_float2(o.x - t.x, o.y - t.y);
}

// x[k0 .. k1) = H y[k0 .. k1), H the inverse of the 256-block of U, into the solution (DOF order)
template <int NS>
__global__ void __launch_bounds__(256) mf_bwd_tri_kernel(const int* __restrict__ lst, const FrontMeta* __restrict__ fm,
                                                         int S, int k0, const double2* __restrict__ inv,
                                                         const int* __restrict__ fdof, const float2* __restrict__ y,
                                                         float2* __restrict__ xs) {
    __shared__ MfTriSmem<NS> sm;
    mf_chain_start();
    const FrontMeta& f = fm[lst[blockIdx.y]];
    const int r0 = k0 + blockIdx.x * MF_NB;
    if (r0 >= f.e) { mf_chain_wait(); return; }
    const int s0 = blockIdx.z * NS, ns = min(NS, S - s0), nr = min(MF_NB, f.e - r0), ldi = min(MF_SB, f.e - k0) + MF_NB;
    const float2* X = y + (f.y + r0) * S + s0;
    const int* d = fdof + f.fdof + r0;
    mf_tri_product<NS>(sm, inv + f.inv + mf_inv_block(k0) + (r0 - k0) + (long long)(r0 - k0) * ldi, ldi, nr,
                       min(k0 + MF_SB, f.e) - r0, ns, [&](int c) { return X + (long long)c * S; },
                       [&](int t, int q, float2 v) { xs[(long long)d[t] * S + s0 + q] = v; });
}

// rows [0, k0): y[r] -= U[r, k0:k1] x[k0:k1]
template <int NS, int RPL>
__global__ void __launch_bounds__(256, NS * RPL > 16 ? 2 : 3) mf_bwd_update_kernel(const int* __restrict__ lst, const FrontMeta* __restrict__ fm,
                                                            int S, int k0, const float2* __restrict__ fact,
                                                            const int* __restrict__ fdof, const float2* __restrict__ xs,
                                                            float2* __restrict__ y) {
    __shared__ MfProdSmem<NS> sm;
    mf_chain_start();
    const FrontMeta& f = fm[lst[blockIdx.y]];
    if (k0 >= f.e) { mf_chain_wait(); return; }
    const int k1 = min(k0 + MF_SB, f.e), r0 = blockIdx.x * 32 * RPL;      // k0 is a multiple of 256: whole tiles
    const int s0 = blockIdx.z * NS, ns = min(NS, S - s0), r = r0 + (threadIdx.x & 31);
    const long long ldf = f.n - (k1 - k0);
    const float2* F = fact + f.fact + mf_fact_block(f.n, k0) + r;         // column c of the block at c ldf
    const float2* X = xs + s0;
    const int* d = fdof + f.fdof;
    float2* Y = y + f.y * S + s0;
    mf_product<NS, RPL>(sm, k0, k1, ns, [&](int c) { return X + (long long)d[c] * S; },
                        [&](int i, int c) { return F[32 * i + (c - k0) * ldf]; },
                        [&](int t, int q, float2 v) {
                            float2* p = Y + (long long)(r0 + t) * S + q;
                            const float2 o = mf_vec(p);
                            *p = make_float2(o.x - v.x, o.y - v.y);
                        });
}

__global__ void mf_fill_kernel(long long n, double v, double* __restrict__ x) {
    long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (g < n) x[g] = v;
}

// x = D^-1/2 (scaled solution), zero outside every front
__global__ void mf_out_kernel(long long n, int S, const uint8_t* __restrict__ freed, const double* __restrict__ scale,
                              const float2* __restrict__ xs, MfCols cols, double2* __restrict__ x) {
    long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n * S) return;
    const long long i = g / S;
    const int s = (int)(g % S);
    const bool in = freed[i];
    const float2 v = in ? xs[g] : make_float2(0.f, 0.f);
    const double sc = scale[i];
    x[i * cols.ld + (cols.count == cols.ld ? s : cols.m[s])] = in ? make_double2((double)v.x * sc, (double)v.y * sc) : make_double2(0.0, 0.0);
}

}  // namespace emfem

using namespace emfem;

struct emfem_mf_s {
    Handle* h = nullptr;
    long long n = 0;
    int nf = 0;
    std::vector<FrontMeta> meta;                  // host copy
    std::vector<std::vector<int>> levels;         // fronts per level
    std::vector<long long> lvl_off;               // offsets of each level's list in d_lst
    std::vector<int> lvl_max_e, lvl_max_n;
    std::vector<long long> lvl_max_asm, lvl_max_b;
    FrontMeta* d_meta = nullptr;
    int* d_lst = nullptr;
    int* d_fdof = nullptr;
    int* d_ea = nullptr;
    int* d_slot = nullptr;
    int* d_off = nullptr;
    uint8_t* d_free = nullptr;                    // 1 where a DOF belongs to some front
    double* d_scale = nullptr;                    // equilibration D^-1/2 of the current factorization
    float2* fact = nullptr;
    double2* inv = nullptr;                       // block inverses
    void* ws = nullptr;                           // level workspace, complex64 or (wide) complex128
    void* upd = nullptr;                          // update store, same precision as ws
    bool wide = false;                            // fronts factored in complex128
    int* d_npert = nullptr;
    long long fact_n = 0, inv_n = 0, ws_n = 0, upd_n = 0;
    long long wv_n = 0, y_n = 0;                  // solve buffer rows
    std::vector<long long> lvl_y0, lvl_yl;        // per level: first row of y and rows of y (its fronts' own rows)
    std::vector<int> lvl_max_ob;                  // per level: largest boundary
    std::vector<int> lvl_split;                   // per level: CTAs that share a boundary product
    long long part_n = 0;                         // split U12 partials: max over levels of CTAs x own rows
    int* d_cmap = nullptr;                        // children's update row of every front row, two slots
    float2* spart = nullptr;                      // (part_n, S) partial sums of the split backward products
    // solve buffers for the current S
    int S = 0;
    float2 *sw = nullptr, *sy = nullptr, *sx = nullptr;
    double flops = 0.0;
    bool unowned = false;                         // a front's boundary holds DOFs that no front eliminates (zero there)
    bool factored = false;
    bool lists = false;                           // assembly lists present (given or built)
    std::vector<int> h_pos, h_fpos;               // host copies used to build the lists on the device
    std::vector<long long> h_own0;
};

static void mf_free(emfem_mf_s* m) {
    void* ps[] = {m->d_meta, m->d_lst, m->d_fdof, m->d_ea, m->d_slot, m->d_off, m->d_free, m->d_scale, m->fact, m->inv,
                  m->ws, m->upd, m->d_npert, m->d_cmap, m->sw, m->sy, m->sx, m->spart};
    for (void* p : ps)
        if (p) cudaFree(p);
}

static inline unsigned nblk(long long items, long long per) {
    long long g = (items + per - 1) / per;
    return (unsigned)std::max(1LL, g);
}

static int mf_reserve(emfem_mf_s* m, int S) {
    if (m->S >= S) return EMFEM_OK;
    void* ps[] = {m->sw, m->sy, m->sx, m->spart};
    for (void* p : ps)
        if (p) cudaFree(p);
    m->sw = m->sy = m->sx = m->spart = nullptr;
    m->S = 0;
    if (m->part_n > 0) EMFEM_CUDA(cudaMalloc(&m->spart, sizeof(float2) * m->part_n * S));
    EMFEM_CUDA(cudaMalloc(&m->sw, sizeof(float2) * std::max(1LL, m->wv_n) * S));
    EMFEM_CUDA(cudaMalloc(&m->sy, sizeof(float2) * std::max(1LL, m->y_n) * S));
    EMFEM_CUDA(cudaMalloc(&m->sx, sizeof(float2) * m->n * S));
    m->S = S;
    return EMFEM_OK;
}

namespace emfem {
int mf_reserved(const emfem_mf_s* m) { return m ? m->S : 0; }

// Tiles of 64 rows where they give every SM four CTAs, else of 32.
static bool mf_wide_tiles(long long rows, int ny, unsigned sz) { return (rows + 63) / 64 * ny * sz >= 4 * 148; }

// Forward and backward pass over the tree, NS right-hand sides per CTA.
template <int NS>
static int mf_sweep_tree(emfem_mf_s* m, const MfCols& cols, const double2* r, cudaStream_t s) {
    const int S = cols.count;
    const int nl = (int)m->levels.size();
    constexpr int NT = NS < 8 ? NS : 8;          // right-hand sides per CTA of the block-inverse products (48 KB of staging)
    const unsigned sz = (unsigned)((S + NS - 1) / NS), szt = (unsigned)((S + NT - 1) / NT);
    bool first = true;
    for (int L = 0; L < nl; L++) {
        const int nfl = (int)m->levels[L].size();
        const long long maxn = m->lvl_max_n[L];
        const int maxe = m->lvl_max_e[L];
        for (int y0 = 0; y0 < nfl; y0 += 65535) {
            const int ny = std::min(65535, nfl - y0);
            const int* lst = m->d_lst + m->lvl_off[L] + y0;
            // the first launch waits for all before it: the right-hand side and, after a factorization, the factors
            const dim3 gg(nblk(maxn * S, 256), ny);
            if (first)
                mf_fwd_gather_kernel<<<gg, 256, 0, s>>>(lst, m->d_meta, S, m->d_fdof, m->d_scale, m->d_cmap, m->wv_n, cols, r, m->sw);
            else
                mf_chain(mf_fwd_gather_kernel, gg, s, lst, m->d_meta, S, m->d_fdof, m->d_scale, m->d_cmap, m->wv_n, cols, r, m->sw);
            first = false;
            for (int k0 = 0; k0 < maxe; k0 += MF_SB) {
                const unsigned nt = nblk(std::min(MF_SB, maxe - k0), MF_NB);
                mf_chain(mf_fwd_tri_kernel<NT>, dim3(nt, ny, szt), s, lst, m->d_meta, S, k0, m->inv, m->sw, m->sy);
                const long long rows = maxn - k0;            // rows [k1, n) of a front: at most n - k0
                if (mf_wide_tiles(rows, ny, sz))
                    mf_chain(mf_fwd_update_kernel<NS, 2>, dim3(nblk(rows, 64), ny, sz), s, lst, m->d_meta, S, k0, m->fact, m->sy, m->sw);
                else
                    mf_chain(mf_fwd_update_kernel<NS, 1>, dim3(nblk(rows, 32), ny, sz), s, lst, m->d_meta, S, k0, m->fact, m->sy, m->sw);
            }
        }
        EMFEM_LAUNCH("multifrontal forward");
    }
    for (int L = nl - 1; L >= 0; L--) {
        const int nfl = (int)m->levels[L].size();
        const int maxe = m->lvl_max_e[L], nsplit = m->lvl_split[L];
        const int cw = (int)nblk(nblk(m->lvl_max_ob[L], nsplit), MF_KC) * MF_KC;
        for (int y0 = 0; y0 < nfl; y0 += 65535) {
            const int ny = std::min(65535, nfl - y0);
            const int* lst = m->d_lst + m->lvl_off[L] + y0;
            if (m->lvl_max_ob[L] > 0) {
                if (mf_wide_tiles(maxe, ny * nsplit, sz)) {
                    const int nrt = (int)nblk(maxe, 64);
                    mf_chain(mf_bwd_bnd_kernel<NS, 2>, dim3(nrt * nsplit, ny, sz), s, lst, m->d_meta, S, nrt, nsplit, cw,
                             m->lvl_y0[L], m->lvl_yl[L], m->fact, m->d_fdof, m->sx, m->sy, m->spart);
                } else {
                    const int nrt = (int)nblk(maxe, 32);
                    mf_chain(mf_bwd_bnd_kernel<NS, 1>, dim3(nrt * nsplit, ny, sz), s, lst, m->d_meta, S, nrt, nsplit, cw,
                             m->lvl_y0[L], m->lvl_yl[L], m->fact, m->d_fdof, m->sx, m->sy, m->spart);
                }
                if (nsplit > 1)
                    mf_chain(mf_bwd_bnd_sum_kernel, dim3(nblk((long long)maxe * S, 256), ny), s, lst, m->d_meta, S, nsplit,
                             m->lvl_y0[L], m->lvl_yl[L], m->spart, m->sy);
            }
            for (int k0 = (maxe - 1) / MF_SB * MF_SB; maxe > 0 && k0 >= 0; k0 -= MF_SB) {
                const unsigned nt = nblk(std::min(MF_SB, maxe - k0), MF_NB);
                mf_chain(mf_bwd_tri_kernel<NT>, dim3(nt, ny, szt), s, lst, m->d_meta, S, k0, m->inv, m->d_fdof, m->sy, m->sx);
                if (k0 == 0) continue;
                if (mf_wide_tiles(k0, ny, sz))
                    mf_chain(mf_bwd_update_kernel<NS, 2>, dim3(k0 / 64, ny, sz), s, lst, m->d_meta, S, k0, m->fact,
                             m->d_fdof, m->sx, m->sy);
                else
                    mf_chain(mf_bwd_update_kernel<NS, 1>, dim3(k0 / 32, ny, sz), s, lst, m->d_meta, S, k0, m->fact,
                             m->d_fdof, m->sx, m->sy);
            }
        }
        EMFEM_LAUNCH("multifrontal backward");
    }
    return EMFEM_OK;
}

// M^-1 r for columns of an (n, ld) FP64 batch, DOF-major -> the same columns of x (FP64), zero on DOFs outside every
// front.  The width that the columns are taken at changes no sum.
int mf_apply(emfem_mf_s* m, const MfCols& cols, const double2* r, double2* x, cudaStream_t s) {
    const int S = cols.count;
    EMFEM_REQUIRE(m->factored, "emfem_mf: solve before a successful factorization");
    if (m->S < S) {
        set_error("emfem_mf: %d right-hand sides exceed the reserved %d (emfem_mf_reserve)", S, m->S);
        return EMFEM_ERR_INVALID_ARG;
    }
    // the solution of every eliminated DOF is written before it is read; a boundary DOF that none eliminates reads zero
    if (m->unowned) EMFEM_CUDA(cudaMemsetAsync(m->sx, 0, sizeof(float2) * m->n * S, s));
    EMFEM_TRY(S >= 16 ? mf_sweep_tree<16>(m, cols, r, s) : S > 4 ? mf_sweep_tree<8>(m, cols, r, s)
              : S > 2 ? mf_sweep_tree<4>(m, cols, r, s) : S == 2 ? mf_sweep_tree<2>(m, cols, r, s) : mf_sweep_tree<1>(m, cols, r, s));
    mf_out_kernel<<<grid_for(m->n * S, 256), 256, 0, s>>>(m->n, S, m->d_free, m->d_scale, m->sx, cols, x);
    EMFEM_LAUNCH("mf_out_kernel");
    return EMFEM_OK;
}
}  // namespace emfem

// Tiles of 128 rows (8 x 4 accumulators: fewer shared-memory reads per multiply-add) where they still give every
// SM four of them, else of 64; complex128 accumulators of that size would not fit the registers.
static bool mf_tall_tiles(long long mt, int ny) {
    return (mt + 127) / 128 * ((mt + 63) / 64) * ny >= 4 * 148;
}

// The level loop of one factorization, fronts in workspace precision T.
template <typename T>
static int mf_factor_levels(emfem_mf_s* m, const double2* K_vals, cudaStream_t s) {
    T* ws = (T*)m->ws;
    T* upd = (T*)m->upd;
    int rc = EMFEM_OK;
    const int nl = (int)m->levels.size();
    for (int L = 0; L < nl && rc == EMFEM_OK; L++) {
        const int nfl = (int)m->levels[L].size();
        long long wsz = 0;
        for (int v : m->levels[L]) wsz += (long long)m->meta[v].n * m->meta[v].n;
        rc = check_cuda(cudaMemsetAsync(ws, 0, sizeof(T) * wsz, s), "cudaMemsetAsync");
        for (int y0 = 0; y0 < nfl && rc == EMFEM_OK; y0 += 65535) {
            const int ny = std::min(65535, nfl - y0);
            const int* lst = m->d_lst + m->lvl_off[L] + y0;
            long long maxn = m->lvl_max_n[L], maxb = m->lvl_max_b[L];
            mf_asm_kernel<T><<<dim3(nblk(m->lvl_max_asm[L], MF_CHUNK), ny), 256, 0, s>>>(
                lst, m->d_meta, K_vals, m->d_slot, m->d_off, m->d_fdof, m->d_scale, ws);
            for (int c = 0; c < 2; c++)
                mf_ea_kernel<T><<<dim3(nblk(maxb, 8), ny), 256, 0, s>>>(lst, m->d_meta, c, m->d_ea, upd, ws);
            const int maxe = m->lvl_max_e[L];
            for (int k = 0; k < maxe; k += MF_NB) {
                const int ob = k / MF_OB * MF_OB;
                mf_diag_kernel<T><<<ny, 256, 0, s>>>(lst, m->d_meta, k, ws, m->inv, m->d_npert);
                const long long mm = std::max(1LL, maxn - k - 1);
                constexpr int TW = sizeof(T) == sizeof(float2) ? 64 : 32;     // tiles within static shared memory
                const unsigned npt = nblk(mm, TW);
                mf_panel_kernel<T, TW><<<dim3(2 * npt, ny), 256, 0, s>>>(lst, m->d_meta, k, (int)npt, ws, m->inv);
                if (k + MF_NB < std::min(ob + MF_OB, maxe)) {
                    const unsigned nr = nblk(mm, 64);
                    mf_strip_kernel<T><<<dim3(4 * nr, ny), 256, sizeof(MfTileSmem<T, 64>), s>>>(lst, m->d_meta, k, ob, (int)nr, ws);
                    continue;
                }
                // fronts of the level that ended inside the outer block are updated with their own rank here too
                const long long mt = std::max(1LL, maxn - ob - 1), nc = (mt + MF_TILE - 1) / MF_TILE;
                bool tall = false;
                if constexpr (sizeof(T) == sizeof(float2)) {
                    tall = mf_tall_tiles(mt, ny);
                    if (tall)
                    mf_trail_kernel<T, 128><<<dim3((unsigned)((mt + 127) / 128 * nc), ny), 256, sizeof(MfTileSmem<T, 128>), s>>>(
                        lst, m->d_meta, ob, ws);
                }
                if (!tall)
                    mf_trail_kernel<T, 64><<<dim3((unsigned)(nc * nc), ny), 256, sizeof(MfTileSmem<T, 64>), s>>>(lst, m->d_meta,
                                                                                                               ob, ws);
            }
            mf_compact_kernel<T><<<dim3(nblk(maxn, 8), ny), 256, 0, s>>>(lst, m->d_meta, ws, m->fact, upd);
            if (m->lvl_max_e[L] > MF_NB) {
                const int nbb = std::min(MF_NBB, (int)nblk(m->lvl_max_e[L], MF_NB));
                mf_block_inverse_kernel<T><<<dim3(2 * nbb, nblk(m->lvl_max_e[L], MF_SB), ny), 256, sizeof(MfInvSmem), s>>>(
                    lst, m->d_meta, ws, m->inv);
            }
            rc = check_cuda(cudaGetLastError(), "multifrontal factor level");
        }
    }
    return rc;
}


extern "C" {

int emfem_mf_create(emfem_handle h, int64_t n, int n_fronts, const int32_t* e, const int32_t* b, const int32_t* parent,
                    const int32_t* level, const int64_t* fdof_ptr, const int32_t* fdof, const int32_t* ea,
                    const int64_t* asm_ptr, const int32_t* asm_slot, const int32_t* asm_off, emfem_mf* out) {
    EMFEM_REQUIRE(h && n > 0 && n_fronts > 0 && e && b && parent && level && fdof_ptr && fdof && ea && out,
                  "emfem_mf_create: bad argument");
    EMFEM_REQUIRE((asm_ptr && asm_slot && asm_off) || (!asm_ptr && !asm_slot && !asm_off),
                  "emfem_mf_create: give all three assembly arrays or none (then emfem_mf_build_lists)");
    auto* m = new emfem_mf_s();
    m->h = &h->h;
    m->n = n;
    m->nf = n_fronts;
    m->meta.resize(n_fronts);
    int nl = 0;
    long long tot_fdof = 0;
    for (int v = 0; v < n_fronts; v++) {
        if (e[v] < 0 || b[v] < 0 || e[v] + b[v] > MF_MAX_FRONT || level[v] < 0 || parent[v] >= n_fronts ||
            (parent[v] >= 0 && parent[v] <= v) || fdof_ptr[v + 1] - fdof_ptr[v] != (long long)e[v] + b[v]) {
            delete m;
            set_error("emfem_mf_create: front %d is inconsistent (e %d, b %d, parent %d)", v, e[v], b[v], parent[v]);
            return EMFEM_ERR_INVALID_ARG;
        }
        nl = std::max(nl, level[v] + 1);
        tot_fdof += e[v] + b[v];
    }
    m->levels.assign(nl, {});
    for (int v = 0; v < n_fronts; v++) m->levels[level[v]].push_back(v);
    // offsets
    long long fact = 0, inv = 0, eao = 0;
    for (int v = 0; v < n_fronts; v++) {
        FrontMeta& f = m->meta[v];
        f.e = e[v]; f.b = b[v]; f.n = e[v] + b[v]; f.parent = parent[v];
        f.child[0] = f.child[1] = -1;
        f.fdof = fdof_ptr[v];
        f.ea = eao; eao += b[v];
        f.asm0 = asm_ptr ? asm_ptr[v] : 0; f.asm1 = asm_ptr ? asm_ptr[v + 1] : 0;
        f.fact = fact; fact += mf_fact_rows_cols(f.n, f.e) + (long long)f.e * f.b;
        f.inv = inv; inv += mf_inv_entries(f.e);
    }
    for (int v = 0; v < n_fronts; v++) {
        int p = parent[v];
        if (p < 0) continue;
        FrontMeta& f = m->meta[p];
        if (f.child[0] < 0) f.child[0] = v;
        else if (f.child[1] < 0) f.child[1] = v;
        else { delete m; set_error("emfem_mf_create: front %d has more than two children", p); return EMFEM_ERR_INVALID_ARG; }
        if (level[p] <= level[v]) { delete m; set_error("emfem_mf_create: parent below child"); return EMFEM_ERR_INVALID_ARG; }
    }
    // per-level workspace and solve-buffer offsets; update store by first-fit over the level schedule
    long long ws_max = 0;
    std::map<long long, long long> freel;   // offset -> size
    long long upd_top = 0;
    auto alloc = [&](long long sz) -> long long {
        for (auto it = freel.begin(); it != freel.end(); ++it) {
            if (it->second >= sz) {
                long long o = it->first, rem = it->second - sz;
                freel.erase(it);
                if (rem > 0) freel[o + sz] = rem;
                return o;
            }
        }
        long long o = upd_top;
        upd_top += sz;
        return o;
    };
    auto release = [&](long long o, long long sz) {
        if (sz <= 0) return;
        auto it = freel.emplace(o, sz).first;
        auto nx = std::next(it);
        if (nx != freel.end() && it->first + it->second == nx->first) { it->second += nx->second; freel.erase(nx); }
        if (it != freel.begin()) {
            auto pv = std::prev(it);
            if (pv->first + pv->second == it->first) { pv->second += it->second; freel.erase(it); }
        }
    };
    long long wv = 0, yo = 0;
    m->lvl_max_e.assign(nl, 0); m->lvl_max_n.assign(nl, 0); m->lvl_max_asm.assign(nl, 0); m->lvl_max_b.assign(nl, 0);
    m->lvl_y0.assign(nl, 0); m->lvl_yl.assign(nl, 0); m->lvl_max_ob.assign(nl, 0); m->lvl_split.assign(nl, 1);
    for (int L = 0; L < nl; L++) {
        long long wso = 0;
        m->lvl_y0[L] = yo;
        for (int v : m->levels[L]) {
            FrontMeta& f = m->meta[v];
            f.ws = wso; wso += (long long)f.n * f.n;
            f.wv = wv; wv += f.n;
            f.y = yo; yo += f.e;
            m->lvl_max_e[L] = std::max(m->lvl_max_e[L], f.e);
            m->lvl_max_n[L] = std::max(m->lvl_max_n[L], f.n);
            m->lvl_max_asm[L] = std::max(m->lvl_max_asm[L], f.asm1 - f.asm0);
            long long cb = 0;
            for (int c : f.child) if (c >= 0) cb = std::max<long long>(cb, m->meta[c].b);
            m->lvl_max_b[L] = std::max(m->lvl_max_b[L], cb);
            m->lvl_max_ob[L] = std::max(m->lvl_max_ob[L], f.b);
        }
        ws_max = std::max(ws_max, wso);
        m->lvl_yl[L] = yo - m->lvl_y0[L];
        // levels of few fronts (the top of the tree) split their boundary products until every SM has four CTAs
        const long long tiles = (m->lvl_max_e[L] + 31) / 32 * (long long)m->levels[L].size();
        const long long most = (m->lvl_max_ob[L] + MF_KC - 1) / MF_KC;
        if (tiles > 0) m->lvl_split[L] = (int)std::max(1LL, std::min(most, (4 * 148 + tiles - 1) / tiles));
        if (m->lvl_split[L] > 1) m->part_n = std::max(m->part_n, m->lvl_split[L] * m->lvl_yl[L]);
        // the level's fronts get their update blocks; their children's are freed once the level assembled
        for (int v : m->levels[L]) {
            FrontMeta& f = m->meta[v];
            f.upd = alloc((long long)f.b * f.b);
        }
        for (int v : m->levels[L])
            for (int c : m->meta[v].child)
                if (c >= 0) release(m->meta[c].upd, (long long)m->meta[c].b * m->meta[c].b);
    }
    m->fact_n = fact; m->inv_n = inv; m->ws_n = ws_max; m->upd_n = upd_top;
    m->wv_n = wv; m->y_n = yo;
    if (wv >= (1LL << 31)) { delete m; set_error("emfem_mf_create: %lld front rows exceed int32", wv); return EMFEM_ERR_INVALID_ARG; }
    for (int v = 0; v < n_fronts; v++) {
        double E = e[v], B = b[v];
        m->flops += 8.0 * (E * E * E / 3 + E * E * B + E * B * B);
    }
    // device arrays
    std::vector<int> lst;
    m->lvl_off.resize(nl);
    for (int L = 0; L < nl; L++) {
        m->lvl_off[L] = (long long)lst.size();
        lst.insert(lst.end(), m->levels[L].begin(), m->levels[L].end());
    }
    std::vector<uint8_t> freed(n, 0);
    for (int v = 0; v < n_fronts; v++)
        for (int i = 0; i < e[v]; i++) {
            int d = fdof[fdof_ptr[v] + i];
            if (d < 0 || d >= n) { delete m; set_error("emfem_mf_create: DOF %d out of range", d); return EMFEM_ERR_INVALID_ARG; }
            freed[d] = 1;
        }
    for (int v = 0; v < n_fronts && !m->unowned; v++)
        for (int i = e[v]; i < e[v] + b[v]; i++) {
            const int d = fdof[fdof_ptr[v] + i];
            if (d < 0 || d >= n || !freed[d]) { m->unowned = true; break; }
        }
    long long nasm = asm_ptr ? asm_ptr[n_fronts] : 0;
    m->lists = asm_ptr != nullptr;
    // elimination position of every DOF, the front of every position, each front's first position
    m->h_pos.assign(n, -1);
    m->h_fpos.reserve((size_t)std::max<long long>(1, n));
    m->h_own0.resize(n_fronts);
    for (int v = 0; v < n_fronts; v++) {
        m->h_own0[v] = (long long)m->h_fpos.size();
        for (int i = 0; i < e[v]; i++) {
            m->h_pos[fdof[fdof_ptr[v] + i]] = (int)m->h_fpos.size();
            m->h_fpos.push_back(v);
        }
    }
    int rc = EMFEM_OK;
    auto up = [&](void** dst, const void* src, size_t bytes) {
        if (rc != EMFEM_OK) return;
        rc = check_cuda(cudaMalloc(dst, std::max<size_t>(bytes, 16)), "cudaMalloc");
        if (rc == EMFEM_OK && bytes) rc = check_cuda(cudaMemcpy(*dst, src, bytes, cudaMemcpyHostToDevice), "cudaMemcpy");
    };
    up((void**)&m->d_meta, m->meta.data(), sizeof(FrontMeta) * n_fronts);
    up((void**)&m->d_lst, lst.data(), sizeof(int) * lst.size());
    up((void**)&m->d_fdof, fdof, sizeof(int) * tot_fdof);
    up((void**)&m->d_ea, ea, sizeof(int) * eao);
    up((void**)&m->d_slot, asm_slot, sizeof(int) * nasm);
    up((void**)&m->d_off, asm_off, sizeof(int) * nasm);
    up((void**)&m->d_free, freed.data(), n);
    auto mk = [&](void** dst, size_t bytes) {
        if (rc != EMFEM_OK) return;
        rc = check_cuda(cudaMalloc(dst, std::max<size_t>(bytes, 16)), "cudaMalloc");
    };
    mk((void**)&m->fact, sizeof(float2) * fact);
    mk((void**)&m->inv, sizeof(double2) * inv);
    mk((void**)&m->ws, sizeof(float2) * ws_max);
    mk((void**)&m->upd, sizeof(float2) * upd_top);
    mk((void**)&m->d_npert, sizeof(int));
    mk((void**)&m->d_scale, sizeof(double) * n);
    mk((void**)&m->d_cmap, sizeof(int) * 2 * wv);
    if (rc != EMFEM_OK) { mf_free(m); delete m; return rc; }
    rc = check_cuda(cudaFuncSetAttribute(mf_block_inverse_kernel<float2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)sizeof(MfInvSmem)), "cudaFuncSetAttribute");
    if (rc == EMFEM_OK)
        rc = check_cuda(cudaFuncSetAttribute(mf_block_inverse_kernel<double2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sizeof(MfInvSmem)), "cudaFuncSetAttribute");
    if (rc == EMFEM_OK)
        rc = check_cuda(cudaFuncSetAttribute(mf_strip_kernel<float2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sizeof(MfTileSmem<float2, 64>)), "cudaFuncSetAttribute");
    if (rc == EMFEM_OK)
        rc = check_cuda(cudaFuncSetAttribute(mf_strip_kernel<double2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sizeof(MfTileSmem<double2, 64>)), "cudaFuncSetAttribute");
    if (rc == EMFEM_OK)
        rc = check_cuda(cudaFuncSetAttribute(mf_trail_kernel<float2, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sizeof(MfTileSmem<float2, 64>)), "cudaFuncSetAttribute");
    if (rc == EMFEM_OK)
        rc = check_cuda(cudaFuncSetAttribute(mf_trail_kernel<float2, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sizeof(MfTileSmem<float2, 128>)), "cudaFuncSetAttribute");
    if (rc == EMFEM_OK)
        rc = check_cuda(cudaFuncSetAttribute(mf_trail_kernel<double2, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sizeof(MfTileSmem<double2, 64>)), "cudaFuncSetAttribute");
    if (rc == EMFEM_OK) rc = check_cuda(cudaMemsetAsync(m->d_cmap, 0xff, sizeof(int) * 2 * wv, h->h.stream), "cudaMemsetAsync");
    if (rc == EMFEM_OK) {
        for (int v0 = 0; v0 < n_fronts; v0 += 65535)
            mf_child_rows_kernel<<<dim3(4, std::min(65535, n_fronts - v0)), 256, 0, h->h.stream>>>(v0, n_fronts, m->d_meta,
                                                                                                   m->d_ea, m->d_cmap, wv);
        rc = check_cuda(cudaGetLastError(), "mf_child_rows_kernel");
    }
    if (rc != EMFEM_OK) { mf_free(m); delete m; return rc; }
    *out = m;
    return EMFEM_OK;
}

int emfem_mf_info(emfem_mf m, size_t* device_bytes, double* flops, int* n_levels) {
    EMFEM_REQUIRE(m, "emfem_mf_info: bad handle");
    if (device_bytes)
        *device_bytes = sizeof(float2) * m->fact_n + sizeof(double2) * m->inv_n + (m->wide ? sizeof(double2) : sizeof(float2)) *
                        (m->ws_n + m->upd_n) + sizeof(int) * 2 * m->wv_n +
                        sizeof(double) * m->n;
    if (flops) *flops = m->flops;
    if (n_levels) *n_levels = (int)m->levels.size();
    return EMFEM_OK;
}

int emfem_mf_set_precision(emfem_mf m, int bits) {
    EMFEM_REQUIRE(m && (bits == 64 || bits == 128), "emfem_mf_set_precision: bits must be 64 or 128");
    const bool wide = bits == 128;
    if (wide == m->wide) return EMFEM_OK;
    int prev = 0;
    EMFEM_CUDA(cudaGetDevice(&prev));
    if (prev != m->h->device) EMFEM_CUDA(cudaSetDevice(m->h->device));
    EMFEM_CUDA(cudaStreamSynchronize(m->h->stream));
    void* ps[] = {m->ws, m->upd};
    for (void* p : ps)
        if (p) cudaFree(p);
    m->ws = m->upd = nullptr;
    m->factored = false;
    const size_t el = wide ? sizeof(double2) : sizeof(float2);
    int rc = check_cuda(cudaMalloc(&m->ws, el * std::max(1LL, m->ws_n)), "cudaMalloc");
    if (rc == EMFEM_OK) rc = check_cuda(cudaMalloc(&m->upd, el * std::max(1LL, m->upd_n)), "cudaMalloc");
    if (rc == EMFEM_OK) {
        m->wide = wide;
    } else {
        // leave a usable complex64 handle behind when the complex128 workspace does not fit
        void* qs[] = {m->ws, m->upd};
        for (void* p : qs)
            if (p) cudaFree(p);
        m->ws = m->upd = nullptr;
        m->wide = false;
        if (cudaMalloc(&m->ws, sizeof(float2) * std::max(1LL, m->ws_n)) != cudaSuccess ||
            cudaMalloc(&m->upd, sizeof(float2) * std::max(1LL, m->upd_n)) != cudaSuccess)
            set_error("emfem_mf_set_precision: the complex64 workspace could not be restored either");
    }
    if (prev != m->h->device) cudaSetDevice(prev);
    return rc;
}

int emfem_mf_factor(emfem_mf m, const void* K_vals, int* n_perturbed) {
    EMFEM_REQUIRE(m && K_vals, "emfem_mf_factor: bad argument");
    EMFEM_REQUIRE(m->lists, "emfem_mf_factor: no assembly lists (emfem_mf_build_lists)");
    cudaStream_t s = m->h->stream;
    int prev = 0;
    EMFEM_CUDA(cudaGetDevice(&prev));
    if (prev != m->h->device) EMFEM_CUDA(cudaSetDevice(m->h->device));
    int rc = EMFEM_OK;
    m->factored = false;
    rc = check_cuda(cudaMemsetAsync(m->d_npert, 0, sizeof(int), s), "cudaMemsetAsync");
    const int nl = (int)m->levels.size();
    // equilibration first: a front's boundary DOFs take their scale from the ancestors that eliminate them
    if (rc == EMFEM_OK) {
        mf_fill_kernel<<<grid_for(m->n, 256), 256, 0, s>>>(m->n, 1.0, m->d_scale);
        for (int L = 0; L < nl; L++)
            for (int y0 = 0; y0 < (int)m->levels[L].size(); y0 += 65535) {
                const int ny = std::min(65535, (int)m->levels[L].size() - y0);
                mf_scale_kernel<<<dim3(nblk(m->lvl_max_asm[L], MF_CHUNK), ny), 256, 0, s>>>(
                    m->d_lst + m->lvl_off[L] + y0, m->d_meta, (const double2*)K_vals, m->d_slot, m->d_off, m->d_fdof,
                    m->d_scale);
            }
        rc = check_cuda(cudaGetLastError(), "multifrontal equilibration");
    }
    if (rc == EMFEM_OK)
        rc = m->wide ? mf_factor_levels<double2>(m, (const double2*)K_vals, s)
                     : mf_factor_levels<float2>(m, (const double2*)K_vals, s);
    int np = 0;
    if (rc == EMFEM_OK) rc = check_cuda(cudaMemcpyAsync(&np, m->d_npert, sizeof(int), cudaMemcpyDeviceToHost, s), "copy");
    if (rc == EMFEM_OK) rc = check_cuda(cudaStreamSynchronize(s), "sync");
    if (rc == EMFEM_OK) {
        m->factored = true;
        if (n_perturbed) *n_perturbed = np;
    }
    if (prev != m->h->device) cudaSetDevice(prev);
    return rc;
}

int emfem_mf_build_lists(emfem_mf m, int64_t nnz, const int32_t* indptr, const int32_t* indices) {
    EMFEM_REQUIRE(m && indptr && indices && nnz > 0 && nnz < (1LL << 31), "emfem_mf_build_lists: bad argument");
    EMFEM_REQUIRE(!m->lists, "emfem_mf_build_lists: the lists exist already");
    cudaStream_t s = m->h->stream;
    const long long n = m->n;
    const int nf = m->nf;
    int *d_pos = nullptr, *d_fpos = nullptr, *cnt = nullptr, *base = nullptr, *cur = nullptr, *scratch = nullptr;
    long long* d_own0 = nullptr;
    int rc = EMFEM_OK;
    std::vector<int> hb(nf + 1);
#define LTRY(x) do { rc = (x); if (rc != EMFEM_OK) goto done; } while (0)
    LTRY(check_cuda(cudaMalloc(&d_pos, sizeof(int) * n), "cudaMalloc"));
    LTRY(check_cuda(cudaMalloc(&d_fpos, sizeof(int) * std::max<size_t>(1, m->h_fpos.size())), "cudaMalloc"));
    LTRY(check_cuda(cudaMalloc(&d_own0, sizeof(long long) * nf), "cudaMalloc"));
    LTRY(check_cuda(cudaMalloc(&cnt, sizeof(int) * nf), "cudaMalloc"));
    LTRY(check_cuda(cudaMalloc(&base, sizeof(int) * (nf + 1)), "cudaMalloc"));
    LTRY(check_cuda(cudaMalloc(&cur, sizeof(int) * nf), "cudaMalloc"));
    LTRY(check_cuda(cudaMalloc(&scratch, sizeof(int) * scan_scratch_ints(nf)), "cudaMalloc"));
    LTRY(check_cuda(cudaMemcpyAsync(d_pos, m->h_pos.data(), sizeof(int) * n, cudaMemcpyHostToDevice, s), "copy"));
    LTRY(check_cuda(cudaMemcpyAsync(d_fpos, m->h_fpos.data(), sizeof(int) * m->h_fpos.size(), cudaMemcpyHostToDevice, s), "copy"));
    LTRY(check_cuda(cudaMemcpyAsync(d_own0, m->h_own0.data(), sizeof(long long) * nf, cudaMemcpyHostToDevice, s), "copy"));
    LTRY(check_cuda(cudaMemsetAsync(cnt, 0, sizeof(int) * nf, s), "memset"));
    LTRY(check_cuda(cudaMemsetAsync(cur, 0, sizeof(int) * nf, s), "memset"));
    LTRY(check_cuda(cudaMemsetAsync(m->h->dev_status, 0, sizeof(int), s), "memset"));
    mf_list_count_kernel<<<grid_for(n, 256), 256, 0, s>>>(n, indptr, indices, d_pos, d_fpos, cnt);
    LTRY(check_cuda(cudaGetLastError(), "mf_list_count_kernel"));
    LTRY(exclusive_scan_i32(m->h, cnt, base, nf, scratch));
    LTRY(check_cuda(cudaMemcpyAsync(hb.data(), base, sizeof(int) * (nf + 1), cudaMemcpyDeviceToHost, s), "copy"));
    LTRY(check_cuda(cudaStreamSynchronize(s), "sync"));
    LTRY(check_cuda(cudaMalloc(&m->d_slot, sizeof(int) * std::max(1, hb[nf])), "cudaMalloc"));
    LTRY(check_cuda(cudaMalloc(&m->d_off, sizeof(int) * std::max(1, hb[nf])), "cudaMalloc"));
    mf_list_fill_kernel<<<grid_for(n, 256), 256, 0, s>>>(n, indptr, indices, d_pos, d_fpos, d_own0, m->d_meta, m->d_fdof,
                                                          base, cur, m->d_slot, m->d_off, m->h->dev_status);
    LTRY(check_cuda(cudaGetLastError(), "mf_list_fill_kernel"));
    for (int v = 0; v < nf; v++) {
        m->meta[v].asm0 = hb[v];
        m->meta[v].asm1 = hb[v + 1];
    }
    for (size_t L = 0; L < m->levels.size(); L++) {
        long long mx = 0;
        for (int v : m->levels[L]) mx = std::max<long long>(mx, hb[v + 1] - hb[v]);
        m->lvl_max_asm[L] = mx;
    }
    LTRY(check_cuda(cudaMemcpyAsync(m->d_meta, m->meta.data(), sizeof(FrontMeta) * nf, cudaMemcpyHostToDevice, s), "copy"));
    {
        int st = 0;
        LTRY(check_cuda(cudaMemcpyAsync(&st, m->h->dev_status, sizeof(int), cudaMemcpyDeviceToHost, s), "copy"));
        LTRY(check_cuda(cudaStreamSynchronize(s), "sync"));
        if (st & DEV_BAD_INDEX) {
            cudaMemsetAsync(m->h->dev_status, 0, sizeof(int), s);
            set_error("emfem_mf_build_lists: a CSR entry's DOF is in neither the own nor the boundary set of its front");
            rc = EMFEM_ERR_DEVICE_CHECK;
            goto done;
        }
    }
    m->lists = true;
done:
    cudaFree(d_pos); cudaFree(d_fpos); cudaFree(d_own0); cudaFree(cnt); cudaFree(base); cudaFree(cur); cudaFree(scratch);
    return rc;
#undef LTRY
}

int emfem_mf_reserve(emfem_mf m, int nrhs) {
    EMFEM_REQUIRE(m && nrhs >= 1 && nrhs <= 256, "emfem_mf_reserve: bad argument");
    return mf_reserve(m, nrhs);
}

int emfem_mf_solve(emfem_mf m, int nrhs, const void* b, void* x) {
    EMFEM_REQUIRE(m && b && x && nrhs >= 1, "emfem_mf_solve: bad argument");
    EMFEM_TRY(mf_reserve(m, nrhs));
    return mf_apply(m, MfCols{nrhs, nrhs, {}}, (const double2*)b, (double2*)x, m->h->stream);
}

int emfem_mf_destroy(emfem_mf m) {
    if (!m) return EMFEM_OK;
    cudaStreamSynchronize(m->h->stream);
    mf_free(m);
    delete m;
    return EMFEM_OK;
}

}  // extern "C"
