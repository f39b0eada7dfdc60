// Frequency-sweep operator and batched Krylov solvers (COCG and BiCGStab).
//
// Replaces the per-frequency direct solve (SolverSuperLU, src/emerge/_emerge/solver.py:535-572,
// through SolveRoutine.solve :1241-1326) for the systems K_f = E - k0_f^2 B + sum_p gamma_{f,p} R_p
// that Assembler.assemble_freq_matrix builds (ASM/assembler.py:255, :314-350).  All systems of a
// batch share one CSR pattern; vectors are DOF-major (n, S) so one pass over the pattern's column
// indices and E/B values serves every system, and the S entries of a gathered column are
// contiguous.  PEC elimination (SolveRoutine's A[ids, ids], solver.py:1266-1269) is a free-DOF
// mask: eliminated rows produce 0 and eliminated entries of every Krylov vector stay 0.
//
// Methods.  COCG (van der Vorst & Melissen 1990) is CG with the unconjugated form x^T y and is
// exact for complex-symmetric A.  The reference's mass matrix is not symmetric: its face-face
// block uses coefficient tables whose index lists differ between (i, j) and (j, i)
// (ASM/curlcurl.py:348-357, e.g. VBCDE = VOLUME_COEFF_CACHE[B,C,D,F]), about 0.5 % of ||B||, and
// COCG stalls near 1e-5 on it.  The default is therefore right-preconditioned BiCGStab
// (van der Vorst 1992), the general-matrix member of the same BiCG family, with the same batched
// operator and preconditioner.  Every reduction is a fixed-order tree and the host decides by iteration
// counts alone, so runs are bit-reproducible.  Iterations run in CUDA-graph chunks with all scalars on
// the device; the host reads the per-system states between chunks.
#include "emfem_internal.cuh"

#include <vector>
#include <algorithm>
#include <cmath>

namespace emfem {

template <typename R> struct V2;
template <> struct V2<double> { typedef double2 T; };
template <> struct V2<float> { typedef float2 T; };

template <typename R, typename T = typename V2<R>::T>
__device__ __forceinline__ T mk2(R x, R y) { T v; v.x = x; v.y = y; return v; }

constexpr int VB = 256;  // threads per block for vector/SpMV kernels

// relative tolerance of each FP32 inner solve in the mixed-precision refinement (compile-time)
#ifndef EMFEM_INNER_TOL
#define EMFEM_INNER_TOL 1e-4
#endif

struct SysState;

struct OpArgs {
    long long n;
    int S;                          // padded systems (power of two, divides VB)
    const int* indptr;
    const int* indices;
    const void* E;                  // value arrays (precision of the kernel)
    const void* B;                  // may be null
    const double* k0sq;             // [S]
    const int* patch_of_row;        // [n], -1 or index into patch rows
    const int* patch_rowptr;
    const int* patch_cols;
    const void* patch_vals;         // complex of kernel precision
    const int* patch_port;
    int n_ports;
    const double* gamma;            // [S][n_ports] complex (interleaved)
    const uint8_t* mask;            // [n]
    // grouped systems (emfem_krylov_solve_grouped): group of every DOF pair i < hh, or null.  Row i
    // (or i - hh) of system column s then belongs to system pg[i] * S + s of the per-system arrays.
    const int* pg;
    long long hh;
    // inside a Krylov iteration: the per-system state; rows of systems that are no longer active are
    // skipped (their scalars are zero, so these vectors are not used again).  Null elsewhere.
    const SysState* skip;
};

__device__ __forceinline__ bool sys_active(const SysState* st, int sy);

__device__ __forceinline__ int sys_of_row(const int* pg, long long hh, long long i, int S, int s) {
    return pg ? pg[i < hh ? i : i - hh] * S + s : s;
}

template <typename T>
__device__ __forceinline__ double2 dotu(T a, T b) {  // a^T b contribution (unconjugated)
    return make_double2((double)a.x * b.x - (double)a.y * b.y, (double)a.x * b.y + (double)a.y * b.x);
}
template <typename T>
__device__ __forceinline__ double2 dotc(T a, T b) {  // conj(a) b
    return make_double2((double)a.x * b.x + (double)a.y * b.y, (double)a.x * b.y - (double)a.y * b.x);
}
template <typename T>
__device__ __forceinline__ double nrm2(T a) { return (double)a.x * a.x + (double)a.y * a.y; }

enum DotMode { DOT_NONE = 0, DOT_XY = 1, DOT_CONJW_Y = 2, DOT_CONJY_W_YY = 3 };

// DOF pairs (i, i + n/2) per partial of the dot products below, for a batch of S systems.  They depend on the width
// that the batch began with only (`cut` below): a mesh's groups of pairs (multiples of 256) are cut alike alone and
// inside a grouped solve, and a batch that is narrowed while it runs keeps its cut.
__host__ __device__ constexpr int spmv_pairs(int S) { return S >= 16 ? 16 : 8; }
__host__ __device__ constexpr int vec_pairs(int S) { return S >= 16 ? 512 / S : VB / S; }

// Fixed-order tree reduction of two components per thread.  A thread holds slot (threadIdx.x / S) of system
// threadIdx.x % S; VB / cut slots make one partial, so a block writes cut / S of the nb partials of every system, at
// partial[(c * S + s) * nb + p] for component c: the partials of one system are contiguous.
__device__ __forceinline__ void block_store2(double2 v0, double2 v1, int ncomp, int S, int cut, long long nb, double2* partial) {
    __shared__ double2 r0[VB], r1[VB];
    const int W = VB / cut, slot = threadIdx.x / S, w = slot % W, s = threadIdx.x % S;
    r0[threadIdx.x] = v0;
    r1[threadIdx.x] = v1;
    __syncthreads();
    for (int off = W / 2; off > 0; off >>= 1) {
        if (w < off) {
            const int o = threadIdx.x + off * S;
            r0[threadIdx.x].x += r0[o].x; r0[threadIdx.x].y += r0[o].y;
            r1[threadIdx.x].x += r1[o].x; r1[threadIdx.x].y += r1[o].y;
        }
        __syncthreads();
    }
    const long long p = (long long)blockIdx.x * (cut / S) + slot / W;
    if (w == 0 && p < nb) {
        partial[s * nb + p] = r0[threadIdx.x];
        if (ncomp > 1) partial[(S + s) * nb + p] = r1[threadIdx.x];
    }
}

// y = A x for all systems, a warp per DOF pair (rows i and i + n/2); optional dot-product epilogue (DotMode).
// The operator values (E, B, Robin patch) are always FP64 and every row is accumulated in FP64;
// R is the precision of the Krylov vectors only (FP32 in the mixed-precision inner solve), so the
// inner iterations see the exact operator and only the vectors are rounded.  Rounding E and B to
// FP32 separately would lose the cancellation in E - k0^2 B near resonances.
//
// The latency of the gathers of x bounds it (16 S bytes per nonzero against 36 of the matrix).  The rows of a
// pair have the same columns (they belong to one mesh entity), so the warp gathers each x once for both (a
// CSR without that structure gathers the second row's too).  L lanes hold different systems, NR of them
// per lane, and the 32 / L groups of lanes take every (32 / L)-th entry, so that a read of a matrix entry
// serves NR systems and a batch of one system still has 32 entries in flight.  Entries travel by asynchronous
// copies, DEPTH stages of 32 / L entries deep: as many bytes in flight held in registers leave too few
// warps (115 against 75 us at S = 32 with one entry a stage; 8 stages cost the second block of an SM, and
// one system, whose row is three stages, is fastest with 2).  E - k0^2 B is formed per entry (2 + 4
// multiply-adds per system instead of 8).
// Measured (one launch, us, before: a thread per row and system): 6 000-tet guide, S = 1 / 4 / 16 / 32:
// 37 / 30 / 69 / 98 -> 14 / 18 / 40 / 64; 82 944-tet cavity: 283 / 379 / 1058 / 1340 -> 205 / 254 / 483 / 793
// (the last at 0.9 TB/s of matrix and 6.4 TB/s of gathered x; FP64 multiply-adds are half of its time).

// Sum over the lane groups, halving the values a lane holds while it can: afterwards a lane holds row
// (lane & 16) and max(1, 2 NR L / 32) systems of the lane, the first of them the returned one.
template <int L, int NR>
__device__ __forceinline__ int pair_reduce(double2* v, int lane) {
    int r0 = 0;
    int cnt = 2 * NR;
#pragma unroll
    for (int off = 16; off >= L; off >>= 1) {
        if (cnt > 1) {
            const int half = cnt / 2;
            const bool up = lane & off;
#pragma unroll
            for (int i = 0; i < NR; i++)
                if (i < half) {
                    double2 send = up ? v[i] : v[i + half], keep = up ? v[i + half] : v[i];
                    keep.x += __shfl_xor_sync(0xffffffffu, send.x, off);
                    keep.y += __shfl_xor_sync(0xffffffffu, send.y, off);
                    v[i] = keep;
                }
            if (off < 16 && up) r0 += half;
            cnt = half;
        } else {
            v[0].x += __shfl_xor_sync(0xffffffffu, v[0].x, off);
            v[0].y += __shfl_xor_sync(0xffffffffu, v[0].y, off);
        }
    }
    return r0;
}

__device__ __forceinline__ void cp_async16z(void* dst, const void* src, bool ok) {   // zero fill when !ok
    unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    int n = ok ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async8z(void* dst, const void* src, bool ok) {
    unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    int n = ok ? 8 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(n) : "memory");
}

// Pipeline stages of a warp: UE entries per lane group each, their x values and the two rows' E and B.  More entries
// a stage spread its bookkeeping (which took the issue slots of the narrow batches), more shared memory a warp
// costs resident warps.  Measured on the 6 000- and 82 944-tet meshes, us for one entry in four stages / two entries /
// four entries in two stages: S = 4 22.9 290 / 18.4 254 (three stages) / 19.1 286; S = 8 37.6 467 / 27.2 341 (three) /
// 24.0 305; S = 16 50.7 613 / 39.6 483 (three) / 40.4 532; S = 32 74.2 921 / 64.2 793 (three) / 86.7 1099.
template <typename R, int L, int NR, bool HASB>
struct SpmvStage {
    static constexpr bool FOUR = L == 8 && NR == 1;
    static constexpr int UE = L == 1 ? 1 : FOUR ? 4 : 2;
    static constexpr int GE = 32 / L * UE;
    static constexpr int DEPTH = L <= 2 || FOUR ? 2 : 3;
    typename V2<R>::T x[GE][L * NR];
    double2 eb[HASB ? 4 : 2][GE];            // E row 0, E row 1, B row 0, B row 1
};

template <typename R, int L, int NR, bool HASB, int NT>
__global__ void __launch_bounds__(NT, NT > VB ? 1 : NR == 1 ? 4 : NR == 2 ? 3 : 2) spmv_kernel(
    OpArgs a, const typename V2<R>::T* __restrict__ x, typename V2<R>::T* __restrict__ y, double2* __restrict__ partial,
    int dotmode, const typename V2<R>::T* __restrict__ w, int ppb) {
    typedef typename V2<R>::T T;
    typedef SpmvStage<R, L, NR, HASB> Stage;
    constexpr int G = 32 / L;                       // entry groups of a warp
    constexpr int NV = 2 * NR > G ? 2 * NR / G : 1; // values of a lane after the reduction
    constexpr int D = Stage::DEPTH, UE = Stage::UE, GE = Stage::GE, CPC = 32 / GE;   // CPC stages per 32 indices
    constexpr int XC = L * NR * (int)sizeof(T) / 16;      // 16-byte chunks of an entry's x values (0: 8 bytes)
    extern __shared__ __align__(16) unsigned char spmv_sm[];
    const int S = a.S;
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    Stage* st = reinterpret_cast<Stage*>(spmv_sm) + wl * D;
    const int g = lane / L, sl = lane % L, sb = blockIdx.y * (L * NR), s0 = sb + sl;
    const long long hh = (a.n + 1) / 2;
    const double2* __restrict__ Ev = (const double2*)a.E;
    const double2* __restrict__ Bv = (const double2*)a.B;
    double2 c0[NV];
    double c1[NV], c2[NV];
#pragma unroll
    for (int q = 0; q < NV; q++) { c0[q] = make_double2(0.0, 0.0); c1[q] = c2[q] = 0.0; }
    double2 acc[2 * NR];
    long long late = -1;                            // NT > VB: row whose dot products wait for those of warp wl - 8
    auto dots = [&](long long row, int r0) {
#pragma unroll
        for (int q = 0; q < NV; q++) {
            const long long o = row * S + s0 + (r0 + q) * L;
            const double yr = acc[q].x, yi = acc[q].y;
            if (dotmode == DOT_XY) {
                const T xi = x[o];
                const double a0 = xi.x, a1 = xi.y;
                c0[q].x = fma(a0, yr, fma(-a1, yi, c0[q].x));
                c0[q].y = fma(a0, yi, fma(a1, yr, c0[q].y));
            } else if (dotmode == DOT_CONJW_Y) {
                const T wi = w[o];
                const double a0 = wi.x, a1 = wi.y;
                c0[q].x = fma(a0, yr, fma(a1, yi, c0[q].x));
                c0[q].y = fma(a0, yi, fma(-a1, yr, c0[q].y));
            } else if (dotmode == DOT_CONJY_W_YY) {
                const T wi = w[o];
                const double a0 = wi.x, a1 = wi.y;
                c0[q].x = fma(a0, yr, fma(a1, yi, c0[q].x));
                c0[q].y = fma(a1, yr, fma(-a0, yi, c0[q].y));
                c1[q] = fma(yr, yr, fma(yi, yi, c1[q]));
                c2[q] = fma(a0, a0, fma(a1, a1, c2[q]));
            }
        }
    };
    for (int pw = wl; pw < ppb; pw += NT / 32) {
        const long long i = (long long)blockIdx.x * ppb + pw;
        if (i >= hh) break;
        const int base = a.pg ? a.pg[i] * S : 0;
        if (a.skip) {
            bool act = false;
#pragma unroll
            for (int r = 0; r < NR; r++) act |= sys_active(a.skip, base + s0 + r * L);
            if (!__any_sync(0xffffffffu, act)) continue;
        }
        const long long i1 = i + hh < a.n ? i + hh : i;      // odd n: the last pair has one row
        const bool two = i1 != i;
        const bool f0 = a.mask[i] != 0, f1 = two && a.mask[i1] != 0;
        const int j0 = a.indptr[i], j1 = a.indptr[i1];
        const int n0 = f0 ? a.indptr[i + 1] - j0 : 0, n1 = f1 ? a.indptr[i1 + 1] - j1 : 0;
        double k2[NR];
        if (HASB) {
#pragma unroll
            for (int r = 0; r < NR; r++) k2[r] = a.k0sq[base + s0 + r * L];
        }
#pragma unroll
        for (int q = 0; q < 2 * NR; q++) acc[q] = make_double2(0.0, 0.0);
        const int nm = n0 > n1 ? n0 : n1;
        const int nst = (nm + GE - 1) / GE;
        // 32 column indices of each row per coalesced load, the next ones in flight while these are used
        int ia = -1, ib = -1;
        int ia2 = lane < n0 ? a.indices[j0 + lane] : -1, ib2 = lane < n1 ? a.indices[j1 + lane] : -1;
        bool paired = true;                          // the rows' columns agree so far
        auto issue = [&](int t) {
            if (t < nst) {
                if (t % CPC == 0) {
                    ia = ia2; ib = ib2;
                    const int kn = t * GE + 32 + lane;
                    ia2 = kn < n0 ? a.indices[j0 + kn] : -1;
                    ib2 = kn < n1 ? a.indices[j1 + kn] : -1;
                    paired = paired && __all_sync(0xffffffffu, ia == ib);
                }
                Stage& sg = st[t % D];
                const int kc = (t % CPC) * GE;       // first entry of the stage inside the 32 of the chunk
                if (XC > 0) {
#pragma unroll
                    for (int q = 0; q < (GE * XC + 31) / 32; q++) {
                        const int ch = lane + 32 * q, en = ch / (XC > 0 ? XC : 1), c = __shfl_sync(0xffffffffu, ia, (kc + en) & 31);
                        if (GE * XC >= 32 || ch < GE * XC)
                            cp_async16z(reinterpret_cast<char*>(&sg.x[0][0]) + 16 * ch,
                                        reinterpret_cast<const char*>(x + (long long)(c < 0 ? 0 : c) * S + sb) + 16 * (ch % (XC > 0 ? XC : 1)), c >= 0);
                    }
                } else {
                    const int c = __shfl_sync(0xffffffffu, ia, (kc + lane) & 31);
                    if (lane < GE) cp_async8z(&sg.x[lane][0], x + (long long)(c < 0 ? 0 : c) * S, c >= 0);
                }
                constexpr int NE = (HASB ? 4 : 2) * GE;
#pragma unroll
                for (int q = 0; q < (NE + 31) / 32; q++) {
                    const int e = lane + 32 * q, which = e / GE, kk = t * GE + e % GE;
                    if (NE % 32 == 0 || e < NE) {
                        const bool second = which & 1;
                        const bool ok = kk < (second ? n1 : n0);
                        const double2* src = (which & 2 ? Bv : Ev) + (second ? j1 : j0) + (ok ? kk : 0);
                        cp_async16z(&sg.eb[which][e % GE], src, ok);
                    }
                }
            }
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        };
#pragma unroll
        for (int t = 0; t < D - 1; t++) issue(t);
        for (int t = 0; t < nst; t++) {
            issue(t + D - 1);
            asm volatile("cp.async.wait_group %0;\n" ::"n"(D - 1) : "memory");
            __syncwarp();
            const Stage& sg = st[t % D];
#pragma unroll
            for (int u = 0; u < UE; u++) {
                const int en = u * G + g;
                T xa[NR];
#pragma unroll
                for (int r = 0; r < NR; r++) xa[r] = sg.x[en][sl + r * L];
                const double2 e0 = sg.eb[0][en], e1 = sg.eb[1][en];
                double2 b0, b1;
                if (HASB) { b0 = sg.eb[2][en]; b1 = sg.eb[3][en]; }
#pragma unroll
                for (int r = 0; r < NR; r++) {
                    const double xr = xa[r].x, xi = xa[r].y;
                    const double kr = HASB ? fma(-k2[r], b0.x, e0.x) : e0.x;
                    const double ki = HASB ? fma(-k2[r], b0.y, e0.y) : e0.y;
                    acc[r].x = fma(kr, xr, fma(-ki, xi, acc[r].x));
                    acc[r].y = fma(kr, xi, fma(ki, xr, acc[r].y));
                }
                if (!paired) {                           // the second row's own columns
                    const int kk = t * GE + en;
                    const int cb = kk < n1 ? a.indices[j1 + kk] : -1;
                    const T* xc = x + (long long)(cb >= 0 ? cb : 0) * S + s0;
#pragma unroll
                    for (int r = 0; r < NR; r++) xa[r] = cb >= 0 ? xc[r * L] : mk2<R>(0, 0);
                }
#pragma unroll
                for (int r = 0; r < NR; r++) {
                    const double xr = xa[r].x, xi = xa[r].y;
                    const double kr = HASB ? fma(-k2[r], b1.x, e1.x) : e1.x;
                    const double ki = HASB ? fma(-k2[r], b1.y, e1.y) : e1.y;
                    acc[NR + r].x = fma(kr, xr, fma(-ki, xi, acc[NR + r].x));
                    acc[NR + r].y = fma(kr, xi, fma(ki, xr, acc[NR + r].y));
                }
            }
            __syncwarp();
        }
        if (a.patch_of_row) {
            const double2* Pv = (const double2*)a.patch_vals;
#pragma unroll
            for (int half = 0; half < 2; half++) {
                const int pr = (half ? f1 : f0) ? a.patch_of_row[half ? i1 : i] : -1;
                if (pr < 0) continue;
                const int je = a.patch_rowptr[pr + 1];
                for (int j = a.patch_rowptr[pr] + g; j < je; j += G) {
                    const int q = a.patch_port[j];
                    if ((unsigned)q >= (unsigned)a.n_ports) continue;        // a port this call has no gamma for
                    const double2 v = Pv[j];
                    const T* xc = x + (long long)a.patch_cols[j] * S + s0;
#pragma unroll
                    for (int r = 0; r < NR; r++) {
                        const T xv = xc[r * L];
                        const double* gm = a.gamma + 2 * ((base + s0 + r * L) * a.n_ports + q);
                        const double kr = fma(gm[0], v.x, -(gm[1] * v.y)), ki = fma(gm[0], v.y, gm[1] * v.x);
                        acc[half * NR + r].x = fma(kr, (double)xv.x, fma(-ki, (double)xv.y, acc[half * NR + r].x));
                        acc[half * NR + r].y = fma(kr, (double)xv.y, fma(ki, (double)xv.x, acc[half * NR + r].y));
                    }
                }
            }
        }
        const int r0 = pair_reduce<L, NR>(acc, lane);
        const bool hi = lane & 16;
        // (sums are written out as fma: every instantiation then rounds alike, which a narrowed batch relies on)
        // lane groups that hold copies of a value already written by another group have a bit of L..8 set
        const bool own = NR > 1 || (lane & 15 & ~(L - 1)) == 0;
        if (own && (two || !hi)) {
            const long long row = hi ? i1 : i;
#pragma unroll
            for (int q = 0; q < NV; q++) {
                const long long o = row * S + s0 + (r0 + q) * L;
                const double yr = acc[q].x, yi = acc[q].y;
                y[o] = mk2<R>((R)yr, (R)yi);
            }
            if (NT > VB && wl >= VB / 32) late = row;
            else dots(row, r0);
        }
    }
    if (dotmode == DOT_NONE) return;
    // per warp and system: row 0 + row 1, then the warps in order
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();                                 // the stages are free: the warps' sums take their place
    typedef double2 WarpSums[L * NR];
    WarpSums* r0s = reinterpret_cast<WarpSums*>(spmv_sm);
    WarpSums* r1s = r0s + VB / 32;
    const int rr0 = NR > 1 && L == 8 && (lane & 8) ? NR / 2 : 0;
    if (NT > VB) {
        // warp w takes over the sums of warp w - 8, as if it had done that warp's pair before its own
        double2* c0s = reinterpret_cast<double2*>(spmv_sm) + threadIdx.x % VB;
        double2* c1s = c0s + NV * VB;
        if (wl < VB / 32) {
#pragma unroll
            for (int q = 0; q < NV; q++) { c0s[q * VB] = c0[q]; c1s[q * VB] = make_double2(c1[q], c2[q]); }
        }
        __syncthreads();
        if (wl >= VB / 32) {
#pragma unroll
            for (int q = 0; q < NV; q++) { c0[q] = c0s[q * VB]; c1[q] = c1s[q * VB].x; c2[q] = c1s[q * VB].y; }
            if (late >= 0) dots(late, rr0);
        }
        __syncthreads();
    }
    const int wo = NT > VB ? wl - VB / 32 : wl;      // the warp's place in the sums (negative: taken over)
#pragma unroll
    for (int q = 0; q < NV; q++) {
        c0[q].x += __shfl_xor_sync(0xffffffffu, c0[q].x, 16);
        c0[q].y += __shfl_xor_sync(0xffffffffu, c0[q].y, 16);
        c1[q] += __shfl_xor_sync(0xffffffffu, c1[q], 16);
        c2[q] += __shfl_xor_sync(0xffffffffu, c2[q], 16);
        if ((NR > 1 || (lane & 15 & ~(L - 1)) == 0) && !(lane & 16) && wo >= 0) {
            r0s[wo][lane % L + (rr0 + q) * L] = c0[q];
            r1s[wo][lane % L + (rr0 + q) * L] = make_double2(c1[q], c2[q]);
        }
    }
    __syncthreads();
    if (threadIdx.x < L * NR) {
        double2 t0 = make_double2(0.0, 0.0), t1 = t0;
#pragma unroll
        for (int q = 0; q < VB / 32; q++) {
            t0.x += r0s[q][threadIdx.x].x; t0.y += r0s[q][threadIdx.x].y;
            t1.x += r1s[q][threadIdx.x].x; t1.y += r1s[q][threadIdx.x].y;
        }
        const long long nb = gridDim.x;
        const int s = blockIdx.y * (L * NR) + threadIdx.x;
        partial[s * nb + blockIdx.x] = t0;
        if (dotmode == DOT_CONJY_W_YY) {
            partial[(S + s) * nb + blockIdx.x] = make_double2(t1.x, 0.0);
            partial[(2 * S + s) * nb + blockIdx.x] = make_double2(t1.y, 0.0);
        }
    }
}

static unsigned spmv_blocks(long long n, int S) { return grid_for((n + 1) / 2, spmv_pairs(S)); }
static unsigned vec_blocks(long long h, int S) { return grid_for(h, vec_pairs(S)); }

template <typename R, bool HASB>
static void launch_spmv_b(const OpArgs& a, const typename V2<R>::T* x, typename V2<R>::T* y, double2* partial, int dotmode,
                          const typename V2<R>::T* w, int cut, cudaStream_t s) {
    const int ppb = spmv_pairs(cut);
    dim3 grid(spmv_blocks(a.n, cut), a.S > 32 ? a.S / 32 : 1);
#define EMFEM_SPMV(L, NR, NT)                                                                                  \
    do {                                                                                                       \
        constexpr size_t sm = sizeof(SpmvStage<R, L, NR, HASB>) * SpmvStage<R, L, NR, HASB>::DEPTH * (NT / 32); \
        if (sm > 48 * 1024)                                                                                    \
            cudaFuncSetAttribute(spmv_kernel<R, L, NR, HASB, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm); \
        spmv_kernel<R, L, NR, HASB, NT><<<grid, NT, sm, s>>>(a, x, y, partial, dotmode, w, ppb);               \
    } while (0)
    // 16 pairs a block are two a warp; where the blocks do not fill the SMs, 16 warps take one each, with the same sums
    // (an iteration at 32 systems, 2 774 / 4 316 DOFs: 58.4 / 60.6 us with 8 warps, 49.0 / 50.3 with 16; a thread per row
    // and system took 51.0 / 57.2)
    const bool small = (long long)grid.x * grid.y <= 148;
    switch (a.S) {
    case 1: EMFEM_SPMV(1, 1, VB); break;
    case 2: EMFEM_SPMV(2, 1, VB); break;
    case 4: EMFEM_SPMV(4, 1, VB); break;
    case 8: EMFEM_SPMV(8, 1, VB); break;
    case 16: if (small) EMFEM_SPMV(8, 2, 512); else EMFEM_SPMV(8, 2, VB); break;
    default: if (small) EMFEM_SPMV(8, 4, 512); else EMFEM_SPMV(8, 4, VB); break;
    }
#undef EMFEM_SPMV
}
template <typename R>
static void launch_spmv(const OpArgs& a, const typename V2<R>::T* x, typename V2<R>::T* y, double2* partial, int dotmode,
                        const typename V2<R>::T* w, int cut, cudaStream_t s) {
    if (a.B) launch_spmv_b<R, true>(a, x, y, partial, dotmode, w, cut, s);
    else launch_spmv_b<R, false>(a, x, y, partial, dotmode, w, cut, s);
}

// y[row] += sum_q gamma_q R_q x on the patch rows (a warp per patch row, lanes over (entry group, system)):
// the Robin terms of an SpMV that keeps no row -> patch row map.
__global__ void __launch_bounds__(VB) patch_rows_kernel(long long np, const int* __restrict__ rows, OpArgs a,
                                                        const double2* __restrict__ x, double2* __restrict__ y) {
    const int lane = threadIdx.x & 31;
    const long long p = ((long long)blockIdx.x * VB + threadIdx.x) >> 5;
    if (p >= np) return;
    const long long row = rows[p];
    if (!a.mask[row]) return;
    const int S = a.S, L = S < 32 ? S : 32, g = lane / L, G = 32 / L;
    const double2* Pv = (const double2*)a.patch_vals;
    for (int s = lane % L; s < S; s += L) {
        double2 acc = make_double2(0.0, 0.0);
        for (int j = a.patch_rowptr[p] + g; j < a.patch_rowptr[p + 1]; j += G) {
            const int q = a.patch_port[j];
            if ((unsigned)q >= (unsigned)a.n_ports) continue;                // as in spmv_kernel
            const double2 v = Pv[j], xv = x[(long long)a.patch_cols[j] * S + s];
            const double* gm = a.gamma + 2 * (s * a.n_ports + q);
            const double kr = gm[0] * v.x - gm[1] * v.y, ki = gm[0] * v.y + gm[1] * v.x;
            acc.x += kr * xv.x - ki * xv.y;
            acc.y += kr * xv.y + ki * xv.x;
        }
        for (int off = 16; off >= L; off >>= 1) {
            acc.x += __shfl_xor_sync(0xffffffffu, acc.x, off);
            acc.y += __shfl_xor_sync(0xffffffffu, acc.y, off);
        }
        if (g == 0) {
            double2 v = y[row * S + s];
            y[row * S + s] = make_double2(v.x + acc.x, v.y + acc.y);
        }
    }
}

// Solver state per system (device).
struct SysState {
    double2 rho;      // COCG: r^T z;   BiCGStab: (r_hat, r)
    double2 alpha;
    double2 beta;
    double2 omega;
    double rn2;       // ||r||^2 (conjugated)
    double bn2;       // ||b||^2
    double tol2;      // tol^2 * bn2
    double rh2;       // BiCGStab: ||r_hat||^2 (shadow residual)
    int active;
    int iters;
    int status;       // 0 converged, 1 cap, 2 breakdown
    int restart;      // BiCGStab: take r_hat = r at the next p update
};

__device__ __forceinline__ bool sys_active(const SysState* st, int sy) { return st[sy].active != 0; }

__device__ __forceinline__ double2 cdiv2(double2 a, double2 b) {
    if (fabs(b.x) >= fabs(b.y)) {
        double r = b.y / b.x, d = b.x + b.y * r;
        return make_double2((a.x + a.y * r) / d, (a.y - a.x * r) / d);
    } else {
        double r = b.x / b.y, d = b.x * r + b.y;
        return make_double2((a.x * r + a.y) / d, (a.y * r - a.x) / d);
    }
}
__device__ __forceinline__ double2 cmul2(double2 a, double2 b) { return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ double cabs1(double2 a) { return fabs(a.x) + fabs(a.y); }

enum UpdateMode { UPD_INIT = 0, UPD_SET_RHO = 1, UPD_COCG_ALPHA = 2, UPD_COCG_BETA = 3,
                  UPD_BICG_ALPHA = 4, UPD_BICG_OMEGA = 5, UPD_BICG_RHO = 6 };

__device__ void stop(SysState& q, int status) {
    q.active = 0; q.status = status;
    q.alpha = make_double2(0, 0); q.omega = make_double2(0, 0); q.beta = make_double2(0, 0);
}

// One block per system: fixed-order sum of the block partials (contiguous per component and system), then
// the scalar recurrences.  Grouped systems (G > 1): block sys = g S + s sums only group g's blocks, those
// of the pairs gpair[g] .. gpair[g + 1] (ppb pairs per block of the launch that wrote the partials).
__global__ void reduce_update_kernel(const double2* __restrict__ partial, int nblocks, int S, int ncomp,
                                     SysState* st, int mode, int maxit, double tol, int nsys, int G, int ppb,
                                     const int* __restrict__ gpair) {
    __shared__ double2 red[VB / 32][3];
    __shared__ double2 sums[3];
    const int sys = blockIdx.x;
    const int s = G > 1 ? sys % S : sys;
    int b0 = 0, b1 = nblocks;
    if (G > 1) {
        b0 = gpair[sys / S] / ppb;
        b1 = gpair[sys / S + 1] / ppb;
    }
    double2 acc[3];
#pragma unroll
    for (int comp = 0; comp < 3; comp++) acc[comp] = make_double2(0, 0);
    for (int k = b0 + threadIdx.x; k < b1; k += VB) {
#pragma unroll
        for (int comp = 0; comp < 3; comp++)
            if (comp < ncomp) {
                double2 v = partial[((long long)comp * S + s) * nblocks + k];
                acc[comp].x += v.x; acc[comp].y += v.y;
            }
    }
#pragma unroll
    for (int comp = 0; comp < 3; comp++) {
        if (comp < ncomp)
            for (int off = 16; off > 0; off >>= 1) {
                acc[comp].x += __shfl_down_sync(0xffffffffu, acc[comp].x, off);
                acc[comp].y += __shfl_down_sync(0xffffffffu, acc[comp].y, off);
            }
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][comp] = acc[comp];
    }
    __syncthreads();
    if (threadIdx.x < ncomp) {
        double2 t = make_double2(0, 0);
        for (int q = 0; q < VB / 32; q++) { t.x += red[q][threadIdx.x].x; t.y += red[q][threadIdx.x].y; }
        sums[threadIdx.x] = t;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    SysState& q = st[sys];
    double2 c0 = sums[0], c1 = ncomp > 1 ? sums[1] : make_double2(0, 0);
    double c2 = ncomp > 2 ? sums[2].x : 0.0;
    switch (mode) {
    case UPD_INIT: {  // c0 = ||b||^2, c1 = ||r||^2
        SysState z;
        z.rho = z.alpha = z.beta = z.omega = make_double2(0, 0);
        z.alpha.x = 1.0; z.omega.x = 1.0;
        z.bn2 = c0.x; z.rn2 = c1.x; z.tol2 = tol * tol * c0.x;
        z.iters = 0; z.status = 0; z.restart = 0; z.rh2 = 0;
        z.active = (s < nsys) && (z.bn2 > 0) && (z.rn2 > z.tol2);
        st[sys] = z;
        break;
    }
    case UPD_SET_RHO:
        q.rho = c0;
        q.rh2 = c0.x;
        break;
    case UPD_COCG_ALPHA:
        if (!q.active) { q.alpha = make_double2(0, 0); break; }
        if (!(cabs1(c0) > 0) || !isfinite(cabs1(c0))) { stop(q, 2); break; }
        q.alpha = cdiv2(q.rho, c0);
        break;
    case UPD_COCG_BETA:
        if (!q.active) { q.beta = make_double2(0, 0); break; }
        q.rn2 = c1.x;
        q.iters += 1;
        if (q.rn2 <= q.tol2) { stop(q, 0); break; }
        if (!isfinite(q.rn2)) { stop(q, 2); break; }
        if (q.iters >= maxit) { stop(q, 1); break; }
        if (!(cabs1(q.rho) > 0)) { stop(q, 2); break; }
        q.beta = cdiv2(c0, q.rho);
        q.rho = c0;
        break;
    case UPD_BICG_ALPHA:
        q.restart = 0;
        if (!q.active) { q.alpha = make_double2(0, 0); break; }
        if (!(cabs1(c0) > 0) || !isfinite(cabs1(c0))) { stop(q, 2); break; }
        q.alpha = cdiv2(q.rho, c0);
        break;
    case UPD_BICG_OMEGA: {
        // c0 = (t, s), c1 = ||t||^2, c2 = ||s||^2.  Minimal-residual omega, enlarged when t and s are
        // nearly orthogonal (Sleijpen & van der Vorst 1995, "maintaining convergence properties of
        // BiCGstab methods in finite precision arithmetic": |cos| >= 0.7).
        if (!q.active) { q.omega = make_double2(0, 0); break; }
        if (!(c1.x > 0)) { q.omega = make_double2(0, 0); break; }
        q.omega = make_double2(c0.x / c1.x, c0.y / c1.x);
        double cosang = sqrt(c0.x * c0.x + c0.y * c0.y) / sqrt(c1.x * c2);
        if (cosang > 0 && cosang < 0.7) { double f = 0.7 / cosang; q.omega.x *= f; q.omega.y *= f; }
        break;
    }
    case UPD_BICG_RHO: {
        if (!q.active) { q.beta = make_double2(0, 0); break; }
        q.rn2 = c1.x;
        q.iters += 1;
        if (q.rn2 <= q.tol2) { stop(q, 0); break; }
        if (!isfinite(q.rn2)) { stop(q, 2); break; }
        if (q.iters >= maxit) { stop(q, 1); break; }
        if (!(cabs1(q.rho) > 0) || !(cabs1(q.omega) > 0)) { stop(q, 2); break; }
        // restart with r_hat = r when (r_hat, r) is nearly orthogonal (tol carries the threshold)
        if (sqrt(c0.x * c0.x + c0.y * c0.y) < tol * sqrt(q.rh2 * q.rn2)) {
            q.restart = 1;
            q.rho = make_double2(q.rn2, 0.0);
            q.rh2 = q.rn2;
            q.beta = make_double2(0, 0);
            break;
        }
        q.beta = cmul2(cdiv2(c0, q.rho), cdiv2(q.alpha, q.omega));
        q.rho = c0;
        break;
    }
    }
}

// Preconditioner: z = M^-1 r on DOF pairs (i, i + h); precond 0 = identity.
template <typename R>
__device__ __forceinline__ void apply_pair(int precond, const typename V2<R>::T* __restrict__ minv, int S,
                                           long long i, int s, typename V2<R>::T a, typename V2<R>::T b,
                                           typename V2<R>::T& z_lo, typename V2<R>::T& z_hi) {
    if (precond == 0) { z_lo = a; z_hi = b; return; }
    typedef typename V2<R>::T T;
    const T* m = minv + (i * S + s) * 4;
    T m00 = m[0], m01 = m[1], m10 = m[2], m11 = m[3];
    z_lo = mk2<R>(m00.x * a.x - m00.y * a.y + m01.x * b.x - m01.y * b.y, m00.x * a.y + m00.y * a.x + m01.x * b.y + m01.y * b.x);
    z_hi = mk2<R>(m10.x * a.x - m10.y * a.y + m11.x * b.x - m11.y * b.y, m10.x * a.y + m10.y * a.x + m11.x * b.y + m11.y * b.x);
}


// ---- COCG vector kernels (thread per DOF pair i < h and system s) ----
template <typename R>
__global__ void __launch_bounds__(VB) cocg_init_kernel(long long h, int S, int precond, const typename V2<R>::T* __restrict__ r,
                                                       typename V2<R>::T* __restrict__ z, typename V2<R>::T* __restrict__ p,
                                                       const typename V2<R>::T* __restrict__ minv, double2* __restrict__ partial) {
    typedef typename V2<R>::T T;
    const int s = threadIdx.x % S;
    double2 rz = make_double2(0, 0);
    for (int q = threadIdx.x / S; q < vec_pairs(S); q += VB / S) {
        const long long i = (long long)blockIdx.x * vec_pairs(S) + q;
        if (i >= h) break;
        T rl = r[i * S + s], rh = r[(i + h) * S + s], zl, zh;
        apply_pair<R>(precond, minv, S, i, s, rl, rh, zl, zh);
        z[i * S + s] = zl; z[(i + h) * S + s] = zh;
        p[i * S + s] = zl; p[(i + h) * S + s] = zh;
        double2 a = dotu(rl, zl), b = dotu(rh, zh);
        rz.x += a.x + b.x; rz.y += a.y + b.y;
    }
    block_store2(rz, rz, 1, S, S, gridDim.x, partial);
}

template <typename R>
__global__ void __launch_bounds__(VB) cocg_update_kernel(long long h, int S, int precond, const int* __restrict__ pg,
                                                         const SysState* __restrict__ st,
                                                         typename V2<R>::T* __restrict__ x, typename V2<R>::T* __restrict__ r,
                                                         typename V2<R>::T* __restrict__ z, const typename V2<R>::T* __restrict__ p,
                                                         const typename V2<R>::T* __restrict__ q, const typename V2<R>::T* __restrict__ minv,
                                                         double2* __restrict__ partial) {
    typedef typename V2<R>::T T;
    const int s = threadIdx.x % S;
    double2 rz = make_double2(0, 0), rr = make_double2(0, 0);
    for (int qp = threadIdx.x / S; qp < vec_pairs(S); qp += VB / S) {
        const long long i = (long long)blockIdx.x * vec_pairs(S) + qp;
        if (i >= h) break;
        const int sy = sys_of_row(pg, h, i, S, s);
        if (!st[sy].active) continue;
        double2 al = st[sy].alpha;
        R ar = (R)al.x, ai = (R)al.y;
        T rv2[2];
#pragma unroll
        for (int half = 0; half < 2; half++) {
            long long k = (i + half * h) * S + s;
            T pv = p[k], qv = q[k], xv = x[k], rv = r[k];
            xv.x += ar * pv.x - ai * pv.y; xv.y += ar * pv.y + ai * pv.x;
            rv.x -= ar * qv.x - ai * qv.y; rv.y -= ar * qv.y + ai * qv.x;
            x[k] = xv; r[k] = rv; rv2[half] = rv;
        }
        T zl, zh;
        apply_pair<R>(precond, minv, S, i, s, rv2[0], rv2[1], zl, zh);
        z[i * S + s] = zl; z[(i + h) * S + s] = zh;
        double2 a = dotu(rv2[0], zl), b = dotu(rv2[1], zh);
        rz.x += a.x + b.x; rz.y += a.y + b.y;
        rr.x += nrm2(rv2[0]) + nrm2(rv2[1]);
    }
    block_store2(rz, rr, 2, S, S, gridDim.x, partial);
}

template <typename R>
__global__ void cocg_pupdate_kernel(long long n, int S, const int* __restrict__ pg, const SysState* __restrict__ st,
                                    const typename V2<R>::T* __restrict__ z, typename V2<R>::T* __restrict__ p) {
    long long g = (long long)blockIdx.x * VB + threadIdx.x;
    if (g >= n * S) return;
    const int sy = sys_of_row(pg, n / 2, g / S, S, (int)(g % S));
    if (!st[sy].active) return;
    double2 b = st[sy].beta;
    R br = (R)b.x, bi = (R)b.y;
    typename V2<R>::T zv = z[g], pv = p[g];
    p[g] = mk2<R>(zv.x + br * pv.x - bi * pv.y, zv.y + br * pv.y + bi * pv.x);
}

// ---- BiCGStab vector kernels ----
// r_hat = r, p = v = 0, partial (r_hat, r) = ||r||^2
template <typename R>
__global__ void __launch_bounds__(VB) bicg_init_kernel(long long h, int S, const typename V2<R>::T* __restrict__ r,
                                                       typename V2<R>::T* __restrict__ rh, typename V2<R>::T* __restrict__ p,
                                                       typename V2<R>::T* __restrict__ v, double2* __restrict__ partial) {
    const int s = threadIdx.x % S;
    double2 c = make_double2(0, 0);
    for (int q = threadIdx.x / S; q < vec_pairs(S); q += VB / S) {
        const long long i = (long long)blockIdx.x * vec_pairs(S) + q;
        if (i >= h) break;
#pragma unroll
        for (int half = 0; half < 2; half++) {
            const long long g = (i + half * h) * S + s;
            typename V2<R>::T rv = r[g];
            rh[g] = rv;
            p[g] = mk2<R>(0, 0);
            v[g] = mk2<R>(0, 0);
            c.x += nrm2(rv);
        }
    }
    block_store2(c, c, 1, S, S, gridDim.x, partial);
}

// p = r + beta (p - omega v); p_hat = M^-1 p   (thread per DOF pair)
template <typename R>
__global__ void __launch_bounds__(VB) bicg_p_kernel(long long h, int S, int precond, const int* __restrict__ pg,
                                                    const SysState* __restrict__ st,
                                                    const typename V2<R>::T* __restrict__ r, typename V2<R>::T* __restrict__ p,
                                                    const typename V2<R>::T* __restrict__ v, typename V2<R>::T* __restrict__ ph,
                                                    const typename V2<R>::T* __restrict__ minv, typename V2<R>::T* __restrict__ rh) {
    typedef typename V2<R>::T T;
    long long g = (long long)blockIdx.x * VB + threadIdx.x;
    long long i = g / S;
    int s = (int)(g % S);
    if (i >= h) return;
    const int sy = sys_of_row(pg, h, i, S, s);
    if (!st[sy].active) return;
    double2 b = st[sy].beta, w = st[sy].omega;
    R br = (R)b.x, bi = (R)b.y, wr = (R)w.x, wi = (R)w.y;
    if (st[sy].restart) {
        rh[i * S + s] = r[i * S + s];
        rh[(i + h) * S + s] = r[(i + h) * S + s];
    }
    T pn[2];
#pragma unroll
    for (int half = 0; half < 2; half++) {
        long long k = (i + half * h) * S + s;
        T rv = r[k], pv = p[k], vv = v[k];
        R tr = pv.x - (wr * vv.x - wi * vv.y), ti = pv.y - (wr * vv.y + wi * vv.x);
        pn[half] = mk2<R>(rv.x + br * tr - bi * ti, rv.y + br * ti + bi * tr);
        p[k] = pn[half];
    }
    T zl, zh;
    apply_pair<R>(precond, minv, S, i, s, pn[0], pn[1], zl, zh);
    ph[i * S + s] = zl;
    ph[(i + h) * S + s] = zh;
}

// s = r - alpha v (stored in r); s_hat = M^-1 s
template <typename R>
__global__ void __launch_bounds__(VB) bicg_s_kernel(long long h, int S, int precond, const int* __restrict__ pg,
                                                    const SysState* __restrict__ st,
                                                    typename V2<R>::T* __restrict__ r, const typename V2<R>::T* __restrict__ v,
                                                    typename V2<R>::T* __restrict__ sh, const typename V2<R>::T* __restrict__ minv) {
    typedef typename V2<R>::T T;
    long long g = (long long)blockIdx.x * VB + threadIdx.x;
    long long i = g / S;
    int s = (int)(g % S);
    if (i >= h) return;
    if (!st[sys_of_row(pg, h, i, S, s)].active) return;
    double2 a = st[sys_of_row(pg, h, i, S, s)].alpha;
    R ar = (R)a.x, ai = (R)a.y;
    T sn[2];
#pragma unroll
    for (int half = 0; half < 2; half++) {
        long long k = (i + half * h) * S + s;
        T rv = r[k], vv = v[k];
        sn[half] = mk2<R>(rv.x - (ar * vv.x - ai * vv.y), rv.y - (ar * vv.y + ai * vv.x));
        r[k] = sn[half];
    }
    T zl, zh;
    apply_pair<R>(precond, minv, S, i, s, sn[0], sn[1], zl, zh);
    sh[i * S + s] = zl;
    sh[(i + h) * S + s] = zh;
}

// x += alpha p_hat + omega s_hat; r = s - omega t; partial (r_hat, r) and ||r||^2
template <typename R>
__global__ void __launch_bounds__(VB) bicg_x_kernel(long long h, int S, int cut, long long nb, const int* __restrict__ pg,
                                                    const SysState* __restrict__ st,
                                                    typename V2<R>::T* __restrict__ x, typename V2<R>::T* __restrict__ r,
                                                    const typename V2<R>::T* __restrict__ ph, const typename V2<R>::T* __restrict__ sh,
                                                    const typename V2<R>::T* __restrict__ t, const typename V2<R>::T* __restrict__ rh,
                                                    double2* __restrict__ partial) {
    typedef typename V2<R>::T T;
    const int s = threadIdx.x % S, slot = threadIdx.x / S, W = VB / cut;
    const long long p = (long long)blockIdx.x * (cut / S) + slot / W;
    double2 c0 = make_double2(0, 0), c1 = c0;
    for (int q = slot % W; q < vec_pairs(cut); q += W) {
        const long long i = p * vec_pairs(cut) + q;
        if (i >= h) break;
        const int sy = sys_of_row(pg, h, i, S, s);
        if (!st[sy].active) continue;
        double2 a = st[sy].alpha, w = st[sy].omega;
        R ar = (R)a.x, ai = (R)a.y, wr = (R)w.x, wi = (R)w.y;
#pragma unroll
        for (int half = 0; half < 2; half++) {
            const long long g = (i + half * h) * S + s;
            T xv = x[g], pv = ph[g], sv = sh[g], rv = r[g], tv = t[g];
            xv.x += ar * pv.x - ai * pv.y + wr * sv.x - wi * sv.y;
            xv.y += ar * pv.y + ai * pv.x + wr * sv.y + wi * sv.x;
            rv.x -= wr * tv.x - wi * tv.y;
            rv.y -= wr * tv.y + wi * tv.x;
            x[g] = xv;
            r[g] = rv;
            double2 d = dotc(rh[g], rv);
            c0.x += d.x; c0.y += d.y;
            c1.x += nrm2(rv);
        }
    }
    block_store2(c0, c1, 2, S, cut, nb, partial);
}

// ---- setup kernels -------------------------------------------------------------------
__global__ void mask_vec_kernel(long long n, int S, const uint8_t* mask, double2* v) {
    long long g = (long long)blockIdx.x * VB + threadIdx.x;
    if (g >= n * S) return;
    if (!mask[g / S]) v[g] = make_double2(0, 0);
}

// r = b - Ax on free DOFs; partials ||b||^2 and ||r||^2
__global__ void __launch_bounds__(VB) residual_kernel(long long h, int S, const uint8_t* __restrict__ mask,
                                                       const double2* __restrict__ b, const double2* __restrict__ Ax,
                                                       double2* __restrict__ r, double2* __restrict__ partial) {
    const int s = threadIdx.x % S;
    double2 cb = make_double2(0, 0), cr = cb;
    for (int q = threadIdx.x / S; q < vec_pairs(S); q += VB / S) {
        const long long i = (long long)blockIdx.x * vec_pairs(S) + q;
        if (i >= h) break;
#pragma unroll
        for (int half = 0; half < 2; half++) {
            const long long row = i + half * h, g = row * S + s;
            double2 res = make_double2(0, 0);
            if (mask[row]) {
                double2 bv = b[g], av = Ax[g];
                res = make_double2(bv.x - av.x, bv.y - av.y);
                cb.x += bv.x * bv.x + bv.y * bv.y;
                cr.x += res.x * res.x + res.y * res.y;
            }
            r[g] = res;
        }
    }
    block_store2(cb, cr, 2, S, S, gridDim.x, partial);
}

// Operator entry (row, col) of system s (E - k0^2 B + patch), used by the preconditioner setup.
__device__ __forceinline__ double2 row_value(const OpArgs& a, long long row, long long col, int sy) {
    const double2* Ev = (const double2*)a.E;
    const double2* Bv = (const double2*)a.B;
    int lo = a.indptr[row], hi = a.indptr[row + 1] - 1;
    double2 v = make_double2(0, 0);
    if (hi >= lo) {
        while (lo < hi) { int mid = (lo + hi) >> 1; if (a.indices[mid] < col) lo = mid + 1; else hi = mid; }
        if (a.indices[lo] == col) {
            double2 e = Ev[lo];
            double k2 = a.k0sq[sy];
            v = e;
            if (Bv) { double2 b = Bv[lo]; v.x -= k2 * b.x; v.y -= k2 * b.y; }
        }
    }
    int pr = a.patch_of_row ? a.patch_of_row[row] : -1;
    if (pr >= 0) {
        const double2* Pv = (const double2*)a.patch_vals;
        for (int j = a.patch_rowptr[pr]; j < a.patch_rowptr[pr + 1]; j++) {
            if (a.patch_cols[j] != col) continue;
            int q = a.patch_port[j];
            if ((unsigned)q >= (unsigned)a.n_ports) continue;                // as in spmv_kernel
            double gr = a.gamma[2 * (sy * a.n_ports + q)], gi = a.gamma[2 * (sy * a.n_ports + q) + 1];
            double2 pv = Pv[j];
            v.x += gr * pv.x - gi * pv.y;
            v.y += gr * pv.y + gi * pv.x;
        }
    }
    return v;
}

// Inverse 2x2 pair blocks (precond 2) or inverse diagonals (precond 1); op is the FP64 operator.
template <typename R>
__global__ void precond_setup_kernel(OpArgs a, int precond, typename V2<R>::T* __restrict__ minv) {
    long long h = a.n / 2;
    long long g = (long long)blockIdx.x * VB + threadIdx.x;
    int S = a.S;
    if (g >= h * S) return;
    long long i = g / S;
    int s = (int)(g % S);
    long long j = i + h;
    const int sy = sys_of_row(a.pg, h, i, S, s);
    double2 m00 = make_double2(0, 0), m01 = m00, m10 = m00, m11 = m00;
    bool fi = a.mask[i] != 0, fj = a.mask[j] != 0;
    double2 a00 = fi ? row_value(a, i, i, sy) : make_double2(1, 0);
    double2 a11 = fj ? row_value(a, j, j, sy) : make_double2(1, 0);
    double2 a01 = (fi && fj) ? row_value(a, i, j, sy) : make_double2(0, 0);
    double2 a10 = (fi && fj) ? row_value(a, j, i, sy) : make_double2(0, 0);
    auto inv1 = [](double2 v) { return cabs1(v) > 0 ? cdiv2(make_double2(1, 0), v) : make_double2(1, 0); };
    bool done = false;
    if (precond == 2) {
        double2 det = make_double2(a00.x * a11.x - a00.y * a11.y - (a01.x * a10.x - a01.y * a10.y),
                                   a00.x * a11.y + a00.y * a11.x - (a01.x * a10.y + a01.y * a10.x));
        double sc = cabs1(a00) * cabs1(a11);
        if (cabs1(det) > 1e-12 * sc && isfinite(cabs1(det))) {
            double2 id = cdiv2(make_double2(1, 0), det);
            m00 = cmul2(a11, id);
            m11 = cmul2(a00, id);
            m01 = cmul2(make_double2(-a01.x, -a01.y), id);
            m10 = cmul2(make_double2(-a10.x, -a10.y), id);
            done = true;
        }
    }
    if (!done) { m00 = inv1(a00); m11 = inv1(a11); }
    typename V2<R>::T* m = minv + (i * S + s) * 4;
    m[0] = mk2<R>((R)m00.x, (R)m00.y); m[1] = mk2<R>((R)m01.x, (R)m01.y);
    m[2] = mk2<R>((R)m10.x, (R)m10.y); m[3] = mk2<R>((R)m11.x, (R)m11.y);
}

// conversions / scaled copies for the mixed-precision refinement
// scale[q] = ||r_q|| of every system (grouped: G S of them)
__global__ void state_scale_kernel(int GS, const SysState* __restrict__ st64, double* __restrict__ scale) {
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < GS) scale[q] = sqrt(st64[q].rn2);
}

__global__ void to_f32_scaled_kernel(long long n, int S, const int* __restrict__ pg, const double2* __restrict__ src,
                                     const double* __restrict__ scale, float2* __restrict__ dst) {
    long long g = (long long)blockIdx.x * VB + threadIdx.x;
    if (g >= n * S) return;
    double rn = scale[sys_of_row(pg, n / 2, g / S, S, (int)(g % S))];
    double sc = rn > 0 ? 1.0 / rn : 0.0;
    double2 v = src[g];
    dst[g] = make_float2((float)(v.x * sc), (float)(v.y * sc));
}

__global__ void add_scaled_f32_kernel(long long n, int S, const int* __restrict__ pg, const float2* __restrict__ d,
                                      const double* __restrict__ scale, const SysState* __restrict__ outer,
                                      double2* __restrict__ x) {
    long long g = (long long)blockIdx.x * VB + threadIdx.x;
    if (g >= n * S) return;
    const int sy = sys_of_row(pg, n / 2, g / S, S, (int)(g % S));
    if (!outer[sy].active) return;
    double sc = scale[sy];
    float2 v = d[g];
    x[g].x += sc * (double)v.x;
    x[g].y += sc * (double)v.y;
}

// inner state for one refinement step: unit-norm rhs, relative tolerance `itol`, active = outer active
__global__ void inner_init_kernel(SysState* inner, const SysState* outer, int GS, double itol) {
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= GS) return;
    SysState z;
    z.rho = z.alpha = z.beta = z.omega = make_double2(0, 0);
    z.alpha.x = 1.0; z.omega.x = 1.0;
    z.active = outer[s].active;
    z.bn2 = z.active ? 1.0 : 0.0;
    z.rn2 = z.bn2;
    z.tol2 = itol * itol;
    z.iters = 0; z.status = 0; z.restart = 0; z.rh2 = 0;
    inner[s] = z;
}

__global__ void patch_map_kernel(long long np, const int* rows, int* patch_of_row) {
    long long g = (long long)blockIdx.x * VB + threadIdx.x;
    if (g < np) patch_of_row[rows[g]] = (int)g;
}

void launch_patch_map(long long np, const int* rows, int* pmap, cudaStream_t s) {
    patch_map_kernel<<<grid_for(np, VB), VB, 0, s>>>(np, rows, pmap);
}

__global__ void pad_copy_kernel(long long n, int nsys, int S, const double2* __restrict__ src, double2* __restrict__ dst) {
    long long g = (long long)blockIdx.x * VB + threadIdx.x;
    if (g >= n * S) return;
    long long i = g / S;
    int s = (int)(g % S);
    dst[g] = s < nsys ? src[i * nsys + s] : make_double2(0, 0);
}

__global__ void unpad_copy_kernel(long long n, int nsys, int S, const double2* __restrict__ src, double2* __restrict__ dst) {
    long long g = (long long)blockIdx.x * VB + threadIdx.x;
    if (g >= n * nsys) return;
    long long i = g / nsys;
    int s = (int)(g % nsys);
    dst[g] = src[i * S + s];
}

__global__ void combine_kernel(long long nnz, const double2* __restrict__ E, const double2* __restrict__ B, double k0sq,
                               double2* __restrict__ K) {
    long long g = (long long)blockIdx.x * VB + threadIdx.x;
    if (g >= nnz) return;
    double2 e = E[g], b = B[g];
    // (E - (B k0^2)) with the product rounded first, as the reference's E - B*k0**2
    double bx = __dmul_rn(b.x, k0sq), by = __dmul_rn(b.y, k0sq);
    K[g] = make_double2(__dsub_rn(e.x, bx), __dsub_rn(e.y, by));
}

__global__ void patch_add_kernel(long long np, const int* __restrict__ slot, const double2* __restrict__ vals,
                                 double gr, double gi, double2* __restrict__ K) {
    long long g = (long long)blockIdx.x * VB + threadIdx.x;
    if (g >= np) return;
    double2 v = vals[g];
    int s = slot[g];
    K[s].x += gr * v.x - gi * v.y;
    K[s].y += gr * v.y + gi * v.x;
}

// Columns of a batched vector moved to a batch of another width (column c of the narrower one holds column
// m[c] of the wider one, -1: zero).
struct ColMap { signed char m[64]; };
template <typename T>
__global__ void pack_columns_kernel(long long rows, int from, int to, ColMap map, const T* __restrict__ src, T* __restrict__ dst) {
    long long g = (long long)blockIdx.x * VB + threadIdx.x;
    if (g >= rows * to) return;
    const int c = map.m[g % to];
    T v;
    v.x = v.y = 0;
    if (c >= 0) v = src[g / to * from + c];
    dst[g] = v;
}
template <typename T>
__global__ void unpack_columns_kernel(long long rows, int from, int to, ColMap map, const T* __restrict__ src, T* __restrict__ dst) {
    long long g = (long long)blockIdx.x * VB + threadIdx.x;
    if (g >= rows * from) return;
    const int c = map.m[g % from];
    if (c >= 0) dst[g / from * to + c] = src[g];
}
// the same for the inverse 2 x 2 pair blocks, four values per pair and system
template <typename T>
__global__ void pack_blocks_kernel(long long h, int from, int to, ColMap map, const T* __restrict__ src, T* __restrict__ dst) {
    long long g = (long long)blockIdx.x * VB + threadIdx.x;
    if (g >= h * to) return;
    const int c = map.m[g % to];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        T v;
        v.x = v.y = 0;
        if (c >= 0) v = src[(g / to * from + c) * 4 + k];
        dst[g * 4 + k] = v;
    }
}

static int pow2_at_least(int v) {
    int p = 1;
    while (p < v) p <<= 1;
    return p;
}

// ---- workspace layout ----------------------------------------------------------------------
struct Layout {
    size_t off_state, off_snap, off_gamma, off_k0, off_partial, off_patchmap, off_scale, off_gpair, off_k0c, off_gammac;
    size_t off_x, off_b, off_r64, off_Ax;                  // FP64 vectors (n, S)
    size_t off_v[8];                                       // Krylov vectors of the inner precision
    size_t off_minv;
    size_t total;
};

static size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

static Layout make_layout(long long n, long long nnz, long long npatch, int S, int nports, int precision, int G = 1) {
    Layout L;
    size_t o = 0;
    long long nb = n / 16 + 2;          // spmv_pairs >= 8 and vec_pairs >= 8 pairs per block
    size_t vec64 = (size_t)n * S * sizeof(double2);
    size_t vecw = (size_t)n * S * (precision ? sizeof(float2) : sizeof(double2));
    L.off_state = o; o = align256(o + sizeof(SysState) * 2 * S * G);
    L.off_snap = o; o = align256(o + sizeof(SysState) * 2 * S * G);
    L.off_gamma = o; o = align256(o + sizeof(double) * 2 * S * G * (nports > 0 ? nports : 1));
    L.off_k0 = o; o = align256(o + sizeof(double) * S * G);
    L.off_partial = o; o = align256(o + sizeof(double2) * 3 * nb * S);
    L.off_patchmap = o; o = align256(o + sizeof(int) * n);
    L.off_scale = o; o = align256(o + sizeof(double) * S * G);
    L.off_gpair = o; o = align256(o + sizeof(int) * (G + 1));
    L.off_k0c = o; o = align256(o + sizeof(double) * S);
    L.off_gammac = o; o = align256(o + sizeof(double) * 2 * S * (nports > 0 ? nports : 1));
    L.off_x = o; o = align256(o + vec64);
    L.off_b = o; o = align256(o + vec64);
    L.off_r64 = o; o = align256(o + vec64);
    L.off_Ax = o; o = align256(o + vec64);
    for (int k = 0; k < 8; k++) { L.off_v[k] = o; o = align256(o + vecw); }
    L.off_minv = o; o = align256(o + vecw * 2);  // (n/2) * S * 4 entries
    (void)nnz; (void)npatch;
    L.total = o;
    return L;
}

// Batched Krylov solve in precision R from x = 0 with the initial residual already in r and the
// per-system state (bn2, tol2, active) in st.
template <typename R>
struct Krylov {
    typedef typename V2<R>::T T;
    int method = 1;            // 0 COCG, 1 BiCGStab
    OpArgs op;
    long long n = 0, h = 0;
    int S = 1, precond = 2, maxit = 1000, nsys = 1;
    T *x = nullptr, *r = nullptr, *minv = nullptr;
    T* v[7] = {nullptr};       // work vectors
    double2* partial = nullptr;
    SysState* st = nullptr;
    SysState* snap = nullptr;       // two copies of st, read by the host while the next replay runs
    cudaStream_t s = nullptr;
    // grouped systems: G groups of S systems, group of every DOF pair, group pair ranges
    int G = 1;
    const int* pg = nullptr;
    const int* gpair = nullptr;
    // auxiliary-space correction (precond 3: aux Jacobi, 4: learned network); BiCGStab only
    const emfem_aux_s* aux = nullptr;
    T* adinv = nullptr;
    // multifrontal LU of one system's operator (precond 5): M^-1 for every system of the batch
    emfem_mf_s* mf = nullptr;
    MfCols lucols = {};             // the columns that it is applied to
    int bj() const { return precond == 5 ? 0 : (precond >= 3 ? 2 : precond); }

    unsigned nb_all() const { return grid_for(n * (long long)S, VB); }
    unsigned nb_pair() const { return grid_for(h * (long long)S, VB); }

    int cut = 1;                    // width that the batch began with: every sum is cut by it

    // restart BiCGStab's shadow residual only when (r_hat, r) is at the rounding level of the
    // vectors' precision (the dots accumulate in FP64); a looser FP32 threshold restarts so often
    // that the Krylov memory is lost
    double restart_eps = sizeof(R) == 8 ? 1e-9 : 1e-6;
    void reduce(int ncomp, unsigned nblocks, int ppb, int mode) {
        reduce_update_kernel<<<G * S, VB, 0, s>>>(partial, (int)nblocks, S, ncomp, st, mode, maxit, restart_eps, nsys, G,
                                                  ppb, gpair);
    }
    void reduce_spmv(int ncomp, int mode) { reduce(ncomp, spmv_blocks(n, cut), spmv_pairs(cut), mode); }
    void reduce_vec(int ncomp, int mode) { reduce(ncomp, vec_blocks(h, cut), vec_pairs(cut), mode); }
    void spmv(const T* in, T* out, int dotmode, const T* w) { launch_spmv<R>(op, in, out, partial, dotmode, w, cut, s); }

    int start() {
        cut = S;
        lucols.ld = lucols.count = S;
        if (method == 0) {
            T *z = v[0], *p = v[1];
            cocg_init_kernel<R><<<vec_blocks(h, S), VB, 0, s>>>(h, S, precond, r, z, p, minv, partial);
            reduce_vec(1, UPD_SET_RHO);
        } else {
            T *rh = v[0], *p = v[1], *vv = v[2];
            bicg_init_kernel<R><<<vec_blocks(h, S), VB, 0, s>>>(h, S, r, rh, p, vv, partial);
            reduce_vec(1, UPD_SET_RHO);
        }
        return check_cuda(cudaGetLastError(), "krylov start");
    }

    int iteration() {
        if (method == 0) {
            T *z = v[0], *p = v[1], *q = v[2];
            spmv(p, q, DOT_XY, nullptr);
            reduce_spmv(1, UPD_COCG_ALPHA);
            cocg_update_kernel<R><<<vec_blocks(h, S), VB, 0, s>>>(h, S, precond, pg, st, x, r, z, p, q, minv, partial);
            reduce_vec(2, UPD_COCG_BETA);
            cocg_pupdate_kernel<R><<<nb_all(), VB, 0, s>>>(n, S, pg, st, z, p);
        } else {
            T *rh = v[0], *p = v[1], *vv = v[2], *ph = v[3], *sh = v[4], *t = v[5];
            bicg_p_kernel<R><<<nb_pair(), VB, 0, s>>>(h, S, bj(), pg, st, r, p, vv, ph, minv, rh);
            if (aux) EMFEM_TRY(aux_correct<T>(aux, S, precond == 4, adinv, p, op.mask, ph, s));
            if constexpr (sizeof(R) == 8) {
                if (mf) EMFEM_TRY(mf_apply(mf, lucols, (const double2*)p, (double2*)ph, s));
            }
            spmv(ph, vv, DOT_CONJW_Y, rh);
            reduce_spmv(1, UPD_BICG_ALPHA);
            bicg_s_kernel<R><<<nb_pair(), VB, 0, s>>>(h, S, bj(), pg, st, r, vv, sh, minv);
            if (aux) EMFEM_TRY(aux_correct<T>(aux, S, precond == 4, adinv, r, op.mask, sh, s));
            if constexpr (sizeof(R) == 8) {
                if (mf) EMFEM_TRY(mf_apply(mf, lucols, (const double2*)r, (double2*)sh, s));
            }
            spmv(sh, t, DOT_CONJY_W_YY, r);
            reduce_spmv(3, UPD_BICG_OMEGA);
            const unsigned nb = vec_blocks(h, cut), per = cut / S;
            bicg_x_kernel<R><<<(nb + per - 1) / per, VB, 0, s>>>(h, S, cut, nb, pg, st, x, r, ph, sh, t, rh, partial);
            reduce_vec(2, UPD_BICG_RHO);
        }
        return check_cuda(cudaGetLastError(), "krylov iteration");
    }

    // ---- narrowing the batch (FP64 BiCGStab on one group) ----
    // Systems converge at different iterations, and a column that has stopped still takes its lanes and its
    // share of every gather.  When the active systems fit half the columns, their vectors, preconditioner
    // and scalars move to a batch of that width; a stopped system's solution goes back to its own column of
    // xfull.  No width from 8 columns on changes the order of a sum (dot products keep their cut; the SpMV and the
    // aux restriction deal a row's entries out to four lane groups; the network and the LU treat a column by
    // itself), so a system's bits do not depend on when it is moved, nor on whether it is: narrower than 8 a
    // batch does not become, and one of 8 or fewer is left as it is.  (An LU application, nearly all of its
    // iteration, takes the active columns out of the batch: a window of 9 frequencies at 24 576 tets 207 ms, 269
    // with all 8 columns to the end.)  Vectors of a narrower batch live in the two halves of the workspace by turns: `wide` holds what an
    // iteration recomputes (five vectors of the full batch), `held` the carried ones (three), each with a
    // separate place for the block inverses.
    T* xfull = nullptr;                       // (n, S0): non-null enables narrowing
    T *wide = nullptr, *held = nullptr, *minv_wide = nullptr, *minv_held = nullptr;
    double *k0c = nullptr, *gammac = nullptr; // narrowed batch's per-system scalars (device)
    std::vector<double> hk0, hgamma;          // per-system scalars of the full batch (host)
    int S0 = 0;                               // width of the full batch
    std::vector<int> col;                     // column of the full batch that each column holds, -1: none
    std::vector<SysState> done;               // states by column of the full batch
    bool in_wide = false;
    // Below this many vector entries an iteration is bound by its launches, not by its width.
    static constexpr long long NARROW_MIN = 1 << 18;
    static int width_for(int active) { return std::max(8, pow2_at_least(active)); }

    int pack(const T* src, T* dst, long long rows, int from, int to, const ColMap& m) {
        pack_columns_kernel<T><<<grid_for(rows * to, VB), VB, 0, s>>>(rows, from, to, m, src, dst);
        return check_cuda(cudaGetLastError(), "pack_columns_kernel");
    }
    // the solutions of the current columns into their columns of xfull
    int flush() {
        if (x == xfull) return EMFEM_OK;
        ColMap m;
        for (int c = 0; c < S; c++) m.m[c] = (signed char)col[c];
        unpack_columns_kernel<T><<<grid_for(n * (long long)S, VB), VB, 0, s>>>(n, S, S0, m, x, xfull);
        return check_cuda(cudaGetLastError(), "unpack_columns_kernel");
    }
    int narrow(const std::vector<SysState>& host, int to) {
        EMFEM_TRY(flush());
        ColMap m;
        std::vector<int> ncol(to, -1);
        std::vector<SysState> nst(to, SysState{});
        int c = 0;
        for (int k = 0; k < S; k++)
            if (host[k].active) { m.m[c] = (signed char)k; ncol[c] = col[k]; nst[c] = host[k]; c++; }
        for (int k = c; k < to; k++) m.m[k] = -1;
        T* o = in_wide ? held : wide;
        const size_t step = ((size_t)n * to + 15) & ~(size_t)15;
        T* nx = o;
        EMFEM_TRY(pack(x, nx, n, S, to, m));
        T* nr = o + step;
        EMFEM_TRY(pack(r, nr, n, S, to, m));
        T* nv[6];
        for (int q = 0; q < 6; q++) {
            nv[q] = o + (2 + q) * step;
            if (q < 3) EMFEM_TRY(pack(v[q], nv[q], n, S, to, m));      // r_hat, p, v; the others are recomputed
        }
        T* nm = in_wide ? minv_held : minv_wide;
        if (bj()) {
            pack_blocks_kernel<T><<<grid_for(h * (long long)to, VB), VB, 0, s>>>(h, S, to, m, minv, nm);
            EMFEM_TRY(check_cuda(cudaGetLastError(), "pack_blocks_kernel"));
        }
        if (aux) {
            T* na = (T*)aux_dinv_buffer(aux, to);      // ends before the wider batch's begins (to <= S / 2)
            EMFEM_TRY(pack(adinv, na, aux->na, S, to, m));
            adinv = na;
        }
        std::vector<double> pk(to, 0.0), pg_(2 * (size_t)to * (op.n_ports > 0 ? op.n_ports : 1), 0.0);
        for (int k = 0; k < c; k++) {
            pk[k] = hk0[ncol[k]];
            for (int q = 0; q < 2 * op.n_ports; q++) pg_[2 * (size_t)k * op.n_ports + q] = hgamma[2 * (size_t)ncol[k] * op.n_ports + q];
        }
        EMFEM_CUDA(cudaMemcpyAsync(k0c, pk.data(), sizeof(double) * pk.size(), cudaMemcpyHostToDevice, s));
        EMFEM_CUDA(cudaMemcpyAsync(gammac, pg_.data(), sizeof(double) * pg_.size(), cudaMemcpyHostToDevice, s));
        EMFEM_CUDA(cudaMemcpyAsync(st, nst.data(), sizeof(SysState) * to, cudaMemcpyHostToDevice, s));
        EMFEM_CUDA(cudaStreamSynchronize(s));
        x = nx; r = nr; minv = nm; col = ncol; S = to; nsys = c;
        for (int q = 0; q < 6; q++) v[q] = nv[q];
        op.S = to; op.k0sq = k0c; op.gamma = gammac;
        in_wide = !in_wide;
        return EMFEM_OK;
    }

    // the columns of the active systems, for the LU
    void lu_columns(const std::vector<SysState>& host) {
        lucols.ld = S;
        lucols.count = 0;
        for (int k = 0; k < S; k++)
            if (host[k].active) lucols.m[lucols.count++] = (signed char)k;
    }

    int read_states(std::vector<SysState>& host, const SysState* from, cudaStream_t on) {
        EMFEM_CUDA(cudaMemcpyAsync(host.data(), from, sizeof(SysState) * host.size(), cudaMemcpyDeviceToHost, on));
        EMFEM_CUDA(cudaStreamSynchronize(on));
        return EMFEM_OK;
    }
    static int count_active(const std::vector<SysState>& host) {
        int n_act = 0;
        for (const SysState& q : host) n_act += q.active != 0;
        return n_act;
    }

    // One eager iteration (loads every kernel before capture), then `chunk` iterations captured once and
    // replayed until no system is active, the iteration cap is reached or the batch is narrowed.  With `ahead`
    // the next replay is queued before the flags of the one before are read, so the GPU does not wait for the
    // host; the replay queued last finds every system stopped.  The host reads (on a second stream) a copy of the
    // states taken between two replays, two copies by turns, so what it decides depends on iteration counts
    // alone and not on how far the replay in flight has come.
    int run(int chunk) {
        const bool narrowing = xfull && method == 1 && G == 1;
        // With block Jacobi every kernel skips stopped systems and iterations are short: the replay for nothing at the
        // end costs less than the waits (200 iterations, 810 tets: 7.9 ms at one system, 8.3 with the waits).  The aux
        // correction, the network and the LU do not skip: 30 iterations of 32 systems at 6 000 tets with the aux space
        // took 12.9 ms ahead and 11.1 with the waits, and 142 iterations and more gain nothing from it.
        const bool ahead = !mf && !aux;
        if (narrowing) {
            S0 = S;
            col.resize(S);
            for (int k = 0; k < S; k++) col[k] = k;
            done.assign(S, SysState{});
        }
        cudaStream_t side = nullptr;
        cudaEvent_t ev[2] = {nullptr, nullptr};
        int rc = EMFEM_OK;
        if (ahead) {
            rc = check_cuda(cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking), "cudaStreamCreate");
            for (int q = 0; q < 2 && rc == EMFEM_OK; q++)
                rc = check_cuda(cudaEventCreateWithFlags(&ev[q], cudaEventDisableTiming), "cudaEventCreate");
        }
        int left = (maxit + chunk - 1) / chunk + 1;
        while (rc == EMFEM_OK && left > 0) {
            std::vector<SysState> host((size_t)G * S);
            cudaGraph_t graph = nullptr;
            cudaGraphExec_t exec = nullptr;
            if ((rc = iteration()) != EMFEM_OK) break;
            if ((rc = check_cuda(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal), "cudaStreamBeginCapture")) != EMFEM_OK) break;
            for (int k = 0; k < chunk && rc == EMFEM_OK; k++) rc = iteration();
            const cudaError_t e = cudaStreamEndCapture(s, &graph);
            if (rc == EMFEM_OK) rc = check_cuda(e, "cudaStreamEndCapture");
            if (rc == EMFEM_OK) rc = check_cuda(cudaGraphInstantiate(&exec, graph, 0), "cudaGraphInstantiate");
            int to = 0, active = 1, cur = 0;
            bool fewer = false;
            // one replay, then its states into copy q
            auto replay = [&](int q) -> int {
                EMFEM_CUDA(cudaGraphLaunch(exec, s));
                left--;
                if (!ahead) return EMFEM_OK;
                EMFEM_CUDA(cudaMemcpyAsync(snap + q * host.size(), st, sizeof(SysState) * host.size(), cudaMemcpyDeviceToDevice, s));
                EMFEM_CUDA(cudaEventRecord(ev[q], s));
                return EMFEM_OK;
            };
            if (ahead && rc == EMFEM_OK) rc = replay(0);
            while (rc == EMFEM_OK) {
                if (ahead) {
                    if (left > 0) { if ((rc = replay(1 - cur)) != EMFEM_OK) break; }
                    if ((rc = check_cuda(cudaStreamWaitEvent(side, ev[cur], 0), "cudaStreamWaitEvent")) != EMFEM_OK) break;
                    if ((rc = read_states(host, snap + cur * host.size(), side)) != EMFEM_OK) break;
                    cur = 1 - cur;
                } else {
                    if ((rc = replay(0)) != EMFEM_OK) break;
                    if ((rc = read_states(host, st, s)) != EMFEM_OK) break;
                }
                active = count_active(host);
                if (active == 0 || left <= 0) break;
                if (!narrowing || n * (long long)S < NARROW_MIN) continue;
                if (2 * width_for(active) <= S) {
                    to = width_for(active);
                    break;
                }
                if (mf && 2 * pow2_at_least(active) <= pow2_at_least(lucols.count)) {
                    fewer = true;
                    break;
                }
            }
            // the replay queued ahead may have stopped more systems: read the states again when all is done
            if (rc == EMFEM_OK) rc = read_states(host, st, s);
            if (exec) cudaGraphExecDestroy(exec);
            if (graph) cudaGraphDestroy(graph);
            if (rc != EMFEM_OK) break;
            if (narrowing)
                for (int k = 0; k < S; k++) if (col[k] >= 0) done[col[k]] = host[k];
            active = count_active(host);
            if (active == 0 || !(to || fewer)) break;
            if (to) {
                rc = narrow(host, width_for(active));
                for (int k = 0; k < S; k++) host[k].active = k < active;
            }
            if (mf) lu_columns(host);
        }
        if (rc == EMFEM_OK && narrowing && S != S0) {
            rc = flush();
            if (rc == EMFEM_OK)
                rc = check_cuda(cudaMemcpyAsync(st, done.data(), sizeof(SysState) * S0, cudaMemcpyHostToDevice, s), "copy state");
        }
        const int rs = check_cuda(cudaStreamSynchronize(s), "sync");
        for (cudaEvent_t q : ev) if (q) cudaEventDestroy(q);
        if (side) cudaStreamDestroy(side);
        return rc != EMFEM_OK ? rc : rs;
    }
};

}  // namespace emfem

using namespace emfem;

static void build_op(OpArgs& a, int64_t n, int S, const int32_t* indptr, const int32_t* indices, const void* E,
                     const void* B, const double* k0dev, const int* pmap, const int32_t* prowptr, const int32_t* pcols,
                     const void* pvals, const int32_t* pport, int nports, const double* gdev, const uint8_t* mask) {
    a.n = n; a.S = S; a.indptr = indptr; a.indices = indices; a.E = E; a.B = B; a.k0sq = k0dev;
    a.patch_of_row = pmap; a.patch_rowptr = prowptr; a.patch_cols = pcols; a.patch_vals = pvals; a.patch_port = pport;
    a.n_ports = nports; a.gamma = gdev; a.mask = mask;
    a.pg = nullptr; a.hh = n / 2; a.skip = nullptr;
}

extern "C" {

int emfem_krylov_workspace_size(int64_t n, int64_t nnz, int nsys, int precision, size_t* bytes) {
    EMFEM_REQUIRE(bytes && n > 0 && nsys > 0 && nsys <= 64 && nnz >= 0, "emfem_krylov_workspace_size: bad argument");
    EMFEM_REQUIRE(precision == 0 || precision == 1, "emfem_krylov_workspace_size: precision must be 0 or 1");
    int S = pow2_at_least(nsys);
    Layout L = make_layout(n, nnz, nnz, S, 8, precision);
    *bytes = L.total;
    return EMFEM_OK;
}

int emfem_sweep_combine(emfem_handle h, int64_t nnz, const void* E_vals, const void* B_vals, double k0sq,
                        int64_t n_patch, const int32_t* patch_slot, const void* patch_vals,
                        double gamma_re, double gamma_im, void* K_vals) {
    EMFEM_REQUIRE(h && E_vals && B_vals && K_vals && nnz >= 0, "emfem_sweep_combine: bad argument");
    EMFEM_REQUIRE(n_patch == 0 || (patch_slot && patch_vals), "emfem_sweep_combine: patch arrays missing");
    if (nnz > 0) {
        combine_kernel<<<grid_for(nnz, VB), VB, 0, h->h.stream>>>(nnz, (const double2*)E_vals, (const double2*)B_vals,
                                                                  k0sq, (double2*)K_vals);
        EMFEM_LAUNCH("combine_kernel");
    }
    if (n_patch > 0) {
        patch_add_kernel<<<grid_for(n_patch, VB), VB, 0, h->h.stream>>>(n_patch, patch_slot, (const double2*)patch_vals,
                                                                        gamma_re, gamma_im, (double2*)K_vals);
        EMFEM_LAUNCH("patch_add_kernel");
    }
    return EMFEM_OK;
}

int emfem_sweep_spmv(emfem_handle h, int64_t n, const int32_t* indptr, const int32_t* indices,
                     const void* E_vals, const void* B_vals, int nsys, const double* k0sq_dev,
                     int64_t n_patch_rows, const int32_t* patch_rows, const int32_t* patch_rowptr,
                     const int32_t* patch_cols, const void* patch_vals, const int32_t* patch_port,
                     int n_ports, const double* gamma_dev, const uint8_t* free_mask, const void* x, void* y) {
    EMFEM_REQUIRE(h && indptr && indices && E_vals && k0sq_dev && free_mask && x && y && n > 0,
                  "emfem_sweep_spmv: bad argument");
    EMFEM_REQUIRE(nsys >= 1 && nsys <= 256 && (nsys & (nsys - 1)) == 0,
                  "emfem_sweep_spmv: nsys must be a power of two <= 256");
    EMFEM_REQUIRE(n_patch_rows == 0 || (patch_rows && patch_rowptr && patch_cols && patch_vals && patch_port && gamma_dev),
                  "emfem_sweep_spmv: patch arrays missing");
    OpArgs a;
    build_op(a, n, nsys, indptr, indices, E_vals, B_vals, k0sq_dev, nullptr, patch_rowptr, patch_cols, patch_vals,
             patch_port, n_ports, gamma_dev, free_mask);
    launch_spmv<double>(a, (const double2*)x, (double2*)y, nullptr, DOT_NONE, nullptr, nsys, h->h.stream);
    EMFEM_LAUNCH("spmv_kernel");
    if (n_patch_rows > 0) {
        patch_rows_kernel<<<grid_for(n_patch_rows * 32, VB), VB, 0, h->h.stream>>>(n_patch_rows, patch_rows, a,
                                                                                    (const double2*)x, (double2*)y);
        EMFEM_LAUNCH("patch_rows_kernel");
    }
    return EMFEM_OK;
}

}  // extern "C"

// The batched solve behind emfem_krylov_solve (G = 1) and emfem_krylov_solve_grouped (G groups of
// nsys systems; row i of the (n, S) vectors belongs to group pair_group[i mod n/2]).
static int krylov_impl(emfem_handle hd, int method, int64_t n, int64_t nnz, const int32_t* indptr, const int32_t* indices,
                       const void* E_vals, const void* B_vals, int nsys, const double* k0sq,
                       int64_t n_patch_rows, const int32_t* patch_rows, const int32_t* patch_rowptr,
                       const int32_t* patch_cols, const void* patch_vals, const int32_t* patch_port,
                       int n_ports, const double* gamma, const uint8_t* free_mask, const void* rhs, void* x,
                       double tol, int maxit, int precond, int precision, void* workspace, size_t workspace_bytes,
                       int* status, int* iters, double* relres, emfem_aux aux, int G, const int32_t* pair_group,
                       emfem_mf_s* mf = nullptr) {
    EMFEM_REQUIRE(hd && indptr && indices && E_vals && k0sq && free_mask && rhs && x && workspace,
                  "emfem_krylov_solve: null argument");
    EMFEM_REQUIRE((precond == 5) == (mf != nullptr), "emfem_krylov_solve: the LU preconditioner goes with precond 5");
    EMFEM_REQUIRE(precond != 5 || (method == 1 && precision == 0 && G == 1),
                  "emfem_krylov_solve_lu: FP64 BiCGStab on one group only");
    EMFEM_REQUIRE(method == 0 || method == 1, "emfem_krylov_solve: method must be 0 (COCG) or 1 (BiCGStab)");
    EMFEM_REQUIRE(n > 0 && (n % 2) == 0, "emfem_krylov_solve: n must be even (DOF pairs i, i + n/2)");
    EMFEM_REQUIRE(nsys >= 1 && nsys <= 64, "emfem_krylov_solve: 1 <= nsys <= 64");
    EMFEM_REQUIRE(precond >= 0 && precond <= 5 && (precision == 0 || precision == 1), "emfem_krylov_solve: bad option");
    EMFEM_REQUIRE(precond < 3 || precond == 5 || (aux && method == 1 && aux->n == n && aux->have_operator && aux->nports == n_ports),
                  "emfem_krylov_solve: precond 3/4 need BiCGStab and an aux space of this field with its operator "
                  "set (emfem_aux_set_operator, same ports)");
    EMFEM_REQUIRE(precond != 4 || aux->params, "emfem_krylov_solve: precond 4 needs network parameters (emfem_aux_set_network)");
    EMFEM_REQUIRE(precond < 3 || precond == 5 || aux->ngroups == G,
                  "emfem_krylov_solve: the aux space's groups (emfem_aux_set_rows) must match the solve's groups");
    EMFEM_REQUIRE(n_ports >= 0 && n_ports <= 8, "emfem_krylov_solve: at most 8 ports");
    EMFEM_REQUIRE(n_patch_rows == 0 || (patch_rows && patch_rowptr && patch_cols && patch_vals && patch_port && gamma),
                  "emfem_krylov_solve: patch arrays missing");
    EMFEM_REQUIRE(tol > 0 && maxit > 0, "emfem_krylov_solve: tol and maxit must be positive");
    Handle* h = &hd->h;
    int S = pow2_at_least(nsys);
    int64_t npatch = 0;
    if (n_patch_rows > 0) {
        int32_t last = 0;
        EMFEM_CUDA(cudaMemcpy(&last, patch_rowptr + n_patch_rows, sizeof(int32_t), cudaMemcpyDeviceToHost));
        npatch = last;
    }
    EMFEM_REQUIRE(npatch <= nnz, "emfem_krylov_solve: more patch entries than nnz");
    EMFEM_REQUIRE(precond != 5 || mf_reserved(mf) >= S,
                  "emfem_krylov_solve_lu: call emfem_mf_reserve with at least the padded batch size first");
    EMFEM_REQUIRE(precond < 3 || precond == 5 || aux->kbuf_bytes >= aux_solve_bytes(aux, S),
                  "emfem_krylov_solve: call emfem_aux_reserve with at least nsys systems first");
    std::vector<int> hgpair(G + 1, 0);
    if (G > 1) {
        EMFEM_REQUIRE(pair_group, "emfem_krylov_solve_grouped: pair_group required");
        EMFEM_REQUIRE((n / 2) % VB == 0, "emfem_krylov_solve_grouped: n/2 must be a multiple of 256");
        std::vector<int> hp(n / 2);
        EMFEM_CUDA(cudaMemcpy(hp.data(), pair_group, sizeof(int) * (n / 2), cudaMemcpyDeviceToHost));
        // groups 0..G-1 in ascending order, none empty, each starting at a multiple of 256 pairs
        int prev = -1;
        for (long long i = 0; i < n / 2; i++) {
            int v = hp[i];
            if (v == prev) continue;
            EMFEM_REQUIRE(v == prev + 1 && v < G && i % VB == 0,
                          "emfem_krylov_solve_grouped: pair_group must run through 0..G-1 in order, each group "
                          "starting at a multiple of 256 pairs");
            hgpair[v] = (int)i;
            prev = v;
        }
        EMFEM_REQUIRE(prev == G - 1, "emfem_krylov_solve_grouped: every group needs at least one DOF pair");
        hgpair[G] = (int)(n / 2);
    }
    Layout L = make_layout(n, nnz, npatch, S, n_ports, precision, G);
    size_t need = make_layout(n, nnz, nnz, S, 8, precision, G).total;
    if (workspace_bytes < need) {
        set_error("emfem_krylov_solve: workspace of %zu bytes, %zu needed (emfem_krylov_workspace_size)", workspace_bytes, need);
        return EMFEM_ERR_WORKSPACE;
    }
    char* ws = (char*)workspace;
    cudaStream_t s = nullptr;
    EMFEM_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    cudaEvent_t ev;
    if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) {
        cudaStreamDestroy(s);
        set_error("emfem_krylov_solve: cudaEventCreate failed");
        return EMFEM_ERR_CUDA;
    }
    SysState* st = (SysState*)(ws + L.off_state);
    SysState* st_outer = st + (size_t)G * S;
    int* gpair = (int*)(ws + L.off_gpair);
    const unsigned nbv = vec_blocks(n / 2, S);
    double* gdev = (double*)(ws + L.off_gamma);
    double* k0dev = (double*)(ws + L.off_k0);
    double2* partial = (double2*)(ws + L.off_partial);
    int* pmap = (int*)(ws + L.off_patchmap);
    double* scale = (double*)(ws + L.off_scale);
    double2* x64 = (double2*)(ws + L.off_x);
    double2* b64 = (double2*)(ws + L.off_b);
    double2* r64 = (double2*)(ws + L.off_r64);
    double2* Ax = (double2*)(ws + L.off_Ax);
    long long nS = n * (long long)S;
    unsigned gv = grid_for(nS, VB);
    std::vector<double> hk0((size_t)G * S, 0.0), hg(2 * (size_t)G * S * (n_ports > 0 ? n_ports : 1), 0.0);
    for (int g = 0; g < G; g++)
        for (int k = 0; k < nsys; k++) {
            hk0[g * S + k] = k0sq[g * nsys + k];
            for (int q = 0; q < n_ports; q++) {
                hg[2 * ((g * S + k) * n_ports + q)] = gamma[2 * ((g * nsys + k) * n_ports + q)];
                hg[2 * ((g * S + k) * n_ports + q) + 1] = gamma[2 * ((g * nsys + k) * n_ports + q) + 1];
            }
        }
    OpArgs op64;
    int rc = EMFEM_OK;
#define STRY(x) do { rc = (x); if (rc != EMFEM_OK) goto done; } while (0)
    STRY(check_cuda(cudaEventRecord(ev, h->stream), "event"));
    STRY(check_cuda(cudaStreamWaitEvent(s, ev, 0), "wait"));
    STRY(check_cuda(cudaMemcpyAsync(k0dev, hk0.data(), sizeof(double) * hk0.size(), cudaMemcpyHostToDevice, s), "copy k0"));
    STRY(check_cuda(cudaMemcpyAsync(gpair, hgpair.data(), sizeof(int) * (G + 1), cudaMemcpyHostToDevice, s), "copy gpair"));
    STRY(check_cuda(cudaMemcpyAsync(gdev, hg.data(), sizeof(double) * hg.size(), cudaMemcpyHostToDevice, s), "copy gamma"));
    STRY(check_cuda(cudaMemsetAsync(pmap, 0xff, sizeof(int) * n, s), "memset"));
    if (n_patch_rows > 0) {
        patch_map_kernel<<<grid_for(n_patch_rows, VB), VB, 0, s>>>(n_patch_rows, patch_rows, pmap);
        STRY(check_cuda(cudaGetLastError(), "patch_map_kernel"));
    }
    pad_copy_kernel<<<gv, VB, 0, s>>>(n, nsys, S, (const double2*)rhs, b64);
    pad_copy_kernel<<<gv, VB, 0, s>>>(n, nsys, S, (const double2*)x, x64);
    mask_vec_kernel<<<gv, VB, 0, s>>>(n, S, free_mask, b64);
    mask_vec_kernel<<<gv, VB, 0, s>>>(n, S, free_mask, x64);
    STRY(check_cuda(cudaGetLastError(), "setup copies"));
    build_op(op64, n, S, indptr, indices, E_vals, B_vals, k0dev, n_patch_rows ? pmap : nullptr, patch_rowptr,
             patch_cols, patch_vals, patch_port, n_ports, gdev, free_mask);
    if (G > 1) op64.pg = pair_group;
    // initial residual r64 = b - A x0 and the outer state (||b||, tolerance, active)
    launch_spmv<double>(op64, x64, Ax, nullptr, DOT_NONE, nullptr, S, s);
    residual_kernel<<<nbv, VB, 0, s>>>(n / 2, S, free_mask, b64, Ax, r64, partial);
    reduce_update_kernel<<<G * S, VB, 0, s>>>(partial, (int)nbv, S, 2, st_outer, UPD_INIT, maxit, tol, nsys, G,
                                              vec_pairs(S), gpair);
    STRY(check_cuda(cudaGetLastError(), "initial residual"));

    if (precision == 0) {
        Krylov<double> k;
        k.method = method; k.op = op64; k.n = n; k.h = n / 2; k.S = S; k.precond = precond; k.maxit = maxit; k.nsys = nsys;
        k.x = x64; k.r = (double2*)(ws + L.off_r64); k.minv = (double2*)(ws + L.off_minv);
        for (int q = 0; q < 7; q++) k.v[q] = (double2*)(ws + L.off_v[q]);
        k.partial = partial; k.st = st; k.snap = (SysState*)(ws + L.off_snap); k.s = s;
        k.op.skip = st;
        k.G = G; k.pg = G > 1 ? pair_group : nullptr; k.gpair = gpair;
        if (k.bj()) {
            precond_setup_kernel<double><<<grid_for((n / 2) * (long long)S, VB), VB, 0, s>>>(op64, k.bj(), k.minv);
            STRY(check_cuda(cudaGetLastError(), "precond_setup"));
        }
        if (precond == 3 || precond == 4) {
            k.aux = aux;
            k.adinv = (double2*)aux_dinv_buffer(aux, S);
            STRY(aux_setup_dinv<double2>(aux, S, nsys, k0dev, gdev, k.adinv, s));
        }
        k.mf = mf;
        if (method == 1 && G == 1) {
            k.xfull = x64; k.k0c = (double*)(ws + L.off_k0c); k.gammac = (double*)(ws + L.off_gammac);
            k.hk0 = hk0; k.hgamma = hg;
            k.wide = k.v[3]; k.held = k.v[0];
            k.minv_wide = Ax; k.minv_held = (double2*)(ws + L.off_minv);
        }
        // the recurrence tolerance is half the requested one so the FP64 true residual meets it
        reduce_update_kernel<<<G * S, VB, 0, s>>>(partial, (int)nbv, S, 2, st, UPD_INIT, maxit, 0.5 * tol, nsys, G,
                                              vec_pairs(S), gpair);
        STRY(check_cuda(cudaGetLastError(), "init state"));
        STRY(k.start());
        STRY(k.run(mf ? 2 : 16));     // an LU solve takes a few iterations of two applications, some 250 launches each
    } else {
        OpArgs op32 = op64;  // FP64 values, FP32 vectors (see spmv_kernel)
        Krylov<float> k;
        k.method = method; k.op = op32; k.n = n; k.h = n / 2; k.S = S; k.precond = precond; k.nsys = nsys;
        float2* r32 = (float2*)(ws + L.off_v[6]);
        float2* d32 = (float2*)(ws + L.off_v[7]);
        k.x = d32; k.r = r32; k.minv = (float2*)(ws + L.off_minv);
        for (int q = 0; q < 6; q++) k.v[q] = (float2*)(ws + L.off_v[q]);
        k.partial = partial; k.st = st; k.snap = (SysState*)(ws + L.off_snap); k.s = s;
        k.op.skip = st;
        k.G = G; k.pg = G > 1 ? pair_group : nullptr; k.gpair = gpair;
        const int* pgk = k.pg;
        const size_t GSm = (size_t)G * S;
        if (precond) {
            precond_setup_kernel<float><<<grid_for((n / 2) * (long long)S, VB), VB, 0, s>>>(op64, k.bj(), k.minv);
            STRY(check_cuda(cudaGetLastError(), "precond_setup"));
        }
        if (precond >= 3) {
            k.aux = aux;
            k.adinv = (float2*)aux_dinv_buffer(aux, S);
            STRY(aux_setup_dinv<float2>(aux, S, nsys, k0dev, gdev, k.adinv, s));
        }
        std::vector<SysState> ho(GSm);
        int used = 0;
        for (int outer = 0; outer < 60; outer++) {
            STRY(check_cuda(cudaMemcpyAsync(ho.data(), st_outer, sizeof(SysState) * GSm, cudaMemcpyDeviceToHost, s), "copy"));
            STRY(check_cuda(cudaStreamSynchronize(s), "sync"));
            bool any = false;
            for (size_t q = 0; q < GSm; q++) any |= ho[q].active != 0;
            if (!any || used >= maxit) break;
            state_scale_kernel<<<grid_for((long long)GSm, 64), 64, 0, s>>>((int)GSm, st_outer, scale);
            to_f32_scaled_kernel<<<gv, VB, 0, s>>>(n, S, pgk, r64, scale, r32);
            STRY(check_cuda(cudaMemsetAsync(d32, 0, sizeof(float2) * nS, s), "memset d"));
            inner_init_kernel<<<grid_for((long long)GSm, 64), 64, 0, s>>>(st, st_outer, (int)GSm, EMFEM_INNER_TOL);
            k.maxit = std::max(1, maxit - used);
            STRY(k.start());
            STRY(k.run(16));
            std::vector<SysState> hin(GSm);
            STRY(check_cuda(cudaMemcpyAsync(hin.data(), st, sizeof(SysState) * GSm, cudaMemcpyDeviceToHost, s), "copy"));
            STRY(check_cuda(cudaStreamSynchronize(s), "sync"));
            int mx = 1;
            for (size_t q = 0; q < GSm; q++) if (ho[q].active) mx = std::max(mx, hin[q].iters);
            used += mx;
            add_scaled_f32_kernel<<<gv, VB, 0, s>>>(n, S, pgk, d32, scale, st_outer, x64);
            launch_spmv<double>(op64, x64, Ax, nullptr, DOT_NONE, nullptr, S, s);
            residual_kernel<<<nbv, VB, 0, s>>>(n / 2, S, free_mask, b64, Ax, r64, partial);
            // the inner state array is free now: reuse it to reduce ||b||^2, ||r||^2 of the new residual
            reduce_update_kernel<<<G * S, VB, 0, s>>>(partial, (int)nbv, S, 2, st, UPD_INIT, maxit, 1.0, S, G,
                                              vec_pairs(S), gpair);
            STRY(check_cuda(cudaGetLastError(), "refinement"));
            std::vector<SysState> hr(GSm);
            STRY(check_cuda(cudaMemcpyAsync(hr.data(), st, sizeof(SysState) * GSm, cudaMemcpyDeviceToHost, s), "copy"));
            STRY(check_cuda(cudaStreamSynchronize(s), "sync"));
            // a correction that did not lower the FP64 residual is reverted and the system stops
            std::vector<double> rev(GSm, 0.0);
            bool any_rev = false;
            for (size_t q = 0; q < GSm; q++) {
                if (!ho[q].active) continue;
                ho[q].iters += hin[q].iters;
                double prev = ho[q].rn2;
                if (!std::isfinite(hr[q].rn2) || hr[q].rn2 >= prev) {
                    rev[q] = -std::sqrt(prev);
                    any_rev = true;
                    ho[q].active = 0; ho[q].status = 2;
                    continue;
                }
                ho[q].rn2 = hr[q].rn2;
                if (ho[q].rn2 <= ho[q].tol2) { ho[q].active = 0; ho[q].status = 0; }
                else if (ho[q].rn2 >= 0.98 * prev) { ho[q].active = 0; ho[q].status = 2; }
            }
            if (any_rev) {
                STRY(check_cuda(cudaMemcpyAsync(scale, rev.data(), sizeof(double) * GSm, cudaMemcpyHostToDevice, s), "copy"));
                add_scaled_f32_kernel<<<gv, VB, 0, s>>>(n, S, pgk, d32, scale, st_outer, x64);
                STRY(check_cuda(cudaGetLastError(), "revert"));
            }
            STRY(check_cuda(cudaMemcpyAsync(st_outer, ho.data(), sizeof(SysState) * GSm, cudaMemcpyHostToDevice, s), "copy"));
        }
        STRY(check_cuda(cudaMemcpyAsync(ho.data(), st_outer, sizeof(SysState) * GSm, cudaMemcpyDeviceToHost, s), "copy"));
        STRY(check_cuda(cudaStreamSynchronize(s), "sync"));
        for (size_t q = 0; q < GSm; q++) if (ho[q].active) { ho[q].active = 0; ho[q].status = 1; }
        STRY(check_cuda(cudaMemcpyAsync(st, ho.data(), sizeof(SysState) * GSm, cudaMemcpyHostToDevice, s), "copy"));
    }
    {
        // final FP64 true residual and solution copy-out
        const size_t GS = (size_t)G * S;
        std::vector<SysState> hs(GS);
        STRY(check_cuda(cudaMemcpyAsync(hs.data(), st, sizeof(SysState) * GS, cudaMemcpyDeviceToHost, s), "copy"));
        launch_spmv<double>(op64, x64, Ax, nullptr, DOT_NONE, nullptr, S, s);
        residual_kernel<<<nbv, VB, 0, s>>>(n / 2, S, free_mask, b64, Ax, r64, partial);
        reduce_update_kernel<<<G * S, VB, 0, s>>>(partial, (int)nbv, S, 2, st_outer, UPD_INIT, maxit, tol, S, G,
                                              vec_pairs(S), gpair);
        unpad_copy_kernel<<<grid_for(n * (long long)nsys, VB), VB, 0, s>>>(n, nsys, S, x64, (double2*)x);
        STRY(check_cuda(cudaGetLastError(), "final residual"));
        std::vector<SysState> hf(GS);
        STRY(check_cuda(cudaMemcpyAsync(hf.data(), st_outer, sizeof(SysState) * GS, cudaMemcpyDeviceToHost, s), "copy"));
        STRY(check_cuda(cudaStreamSynchronize(s), "sync"));
        bool all_ok = true;
        for (int g = 0; g < G; g++)
            for (int q = 0; q < nsys; q++) {
                const SysState &e = hs[g * S + q], &f = hf[g * S + q];
                double rel = f.bn2 > 0 ? std::sqrt(f.rn2 / f.bn2) : 0.0;
                int stat = e.active ? 1 : e.status;
                if (stat == 0 && rel > tol) stat = 1;  // the recurrence drifted from the true residual
                if (status) status[g * nsys + q] = stat;
                if (iters) iters[g * nsys + q] = e.iters;
                if (relres) relres[g * nsys + q] = rel;
                all_ok &= stat == 0;
            }
        if (!all_ok) {
            set_error("emfem_krylov_solve: not every system reached the tolerance");
            rc = EMFEM_ERR_NOT_CONVERGED;
        }
    }
done:
    cudaEventRecord(ev, s);
    cudaStreamWaitEvent(h->stream, ev, 0);
    cudaStreamSynchronize(s);
    cudaEventDestroy(ev);
    cudaStreamDestroy(s);
    return rc;
#undef STRY
}

extern "C" {

int emfem_krylov_solve(emfem_handle hd, int method, int64_t n, int64_t nnz, const int32_t* indptr, const int32_t* indices,
                       const void* E_vals, const void* B_vals, int nsys, const double* k0sq,
                       int64_t n_patch_rows, const int32_t* patch_rows, const int32_t* patch_rowptr,
                       const int32_t* patch_cols, const void* patch_vals, const int32_t* patch_port,
                       int n_ports, const double* gamma, const uint8_t* free_mask, const void* rhs, void* x,
                       double tol, int maxit, int precond, int precision, void* workspace, size_t workspace_bytes,
                       int* status, int* iters, double* relres, emfem_aux aux) {
    return krylov_impl(hd, method, n, nnz, indptr, indices, E_vals, B_vals, nsys, k0sq, n_patch_rows, patch_rows,
                       patch_rowptr, patch_cols, patch_vals, patch_port, n_ports, gamma, free_mask, rhs, x, tol, maxit,
                       precond, precision, workspace, workspace_bytes, status, iters, relres, aux, 1, nullptr);
}

int emfem_krylov_solve_lu(emfem_handle hd, int64_t n, int64_t nnz, const int32_t* indptr, const int32_t* indices,
                          const void* E_vals, const void* B_vals, int nsys, const double* k0sq, int64_t n_patch_rows,
                          const int32_t* patch_rows, const int32_t* patch_rowptr, const int32_t* patch_cols,
                          const void* patch_vals, const int32_t* patch_port, int n_ports, const double* gamma,
                          const uint8_t* free_mask, const void* rhs, void* x, double tol, int maxit, emfem_mf lu,
                          void* workspace, size_t workspace_bytes, int* status, int* iters, double* relres) {
    EMFEM_REQUIRE(lu, "emfem_krylov_solve_lu: no factorization");
    return krylov_impl(hd, 1, n, nnz, indptr, indices, E_vals, B_vals, nsys, k0sq, n_patch_rows, patch_rows,
                       patch_rowptr, patch_cols, patch_vals, patch_port, n_ports, gamma, free_mask, rhs, x, tol, maxit,
                       5, 0, workspace, workspace_bytes, status, iters, relres, nullptr, 1, nullptr, lu);
}

int emfem_krylov_workspace_size_grouped(int64_t n, int64_t nnz, int nsys, int ngroups, int precision, size_t* bytes) {
    EMFEM_REQUIRE(bytes && n > 0 && nsys > 0 && nsys <= 64 && nnz >= 0 && ngroups >= 1 && (precision == 0 || precision == 1),
                  "emfem_krylov_workspace_size_grouped: bad argument");
    *bytes = make_layout(n, nnz, nnz, pow2_at_least(nsys), 8, precision, ngroups).total;
    return EMFEM_OK;
}

int emfem_krylov_solve_grouped(emfem_handle hd, int method, int64_t n, int64_t nnz, const int32_t* indptr,
                               const int32_t* indices, const void* E_vals, const void* B_vals, int ngroups,
                               const int32_t* pair_group, int nsys, const double* k0sq, int64_t n_patch_rows,
                               const int32_t* patch_rows, const int32_t* patch_rowptr, const int32_t* patch_cols,
                               const void* patch_vals, const int32_t* patch_port, int n_ports, const double* gamma,
                               const uint8_t* free_mask, const void* rhs, void* x, double tol, int maxit, int precond,
                               int precision, void* workspace, size_t workspace_bytes, int* status, int* iters,
                               double* relres, emfem_aux aux) {
    EMFEM_REQUIRE(ngroups >= 1 && ngroups <= 4096, "emfem_krylov_solve_grouped: 1 <= ngroups <= 4096");
    return krylov_impl(hd, method, n, nnz, indptr, indices, E_vals, B_vals, nsys, k0sq, n_patch_rows, patch_rows,
                       patch_rowptr, patch_cols, patch_vals, patch_port, n_ports, gamma, free_mask, rhs, x, tol, maxit,
                       precond, precision, workspace, workspace_bytes, status, iters, relres, aux, ngroups, pair_group);
}

}  // extern "C"

// ---- allocation-free variant of emfem_sweep_spmv ------------------------------------------------
// Some callers cannot call cudaMalloc: applications that hand all device memory to their own pool
// allocator up front (a raw cudaMalloc fails or fragments it), and latency-critical loops in which an
// allocation's implicit device synchronisation is not acceptable.  This entry point computes exactly
// what emfem_sweep_spmv computes, but keeps its only scratch — the row -> Robin-patch-row map, one int
// per row — in the fixed array below instead of a stream-ordered allocation.  The array is part of
// this library's device image: every GPU that loads the library holds its 16 MiB until the process
// exits.  All calls share it and it keeps the last call's contents, so every call resets the rows it
// uses before filling them, and calls that overlap on the GPU (different streams or threads) race.
#include <mutex>

namespace emfem {
static __device__ __align__(256) int g_noalloc_patch_map[EMFEM_NOALLOC_MAX_ROWS];

constexpr int NOALLOC_MAX_DEVICES = 64;
struct NoallocSlot {
    int* addr = nullptr;
    unsigned long long ctx_id = 0;     // the context the address was resolved in (0 = unknown)
};
static NoallocSlot g_noalloc[NOALLOC_MAX_DEVICES];
static std::mutex g_noalloc_mutex;

// The current context's unique id through the driver's cuCtxGetCurrent / cuCtxGetId, looked up at run
// time (the library links only the CUDA runtime).  0 when no context is current or the lookup failed.
static unsigned long long current_ctx_id() {
    typedef int (*GetCurrentFn)(void** ctx);
    typedef int (*GetIdFn)(void* ctx, unsigned long long* id);
    static GetCurrentFn get_current = nullptr;
    static GetIdFn get_id = nullptr;
    static bool looked_up = false;
    if (!looked_up) {
        looked_up = true;
        cudaDriverEntryPointQueryResult q1, q2;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", (void**)&get_current, 12000, cudaEnableDefault, &q1) !=
                cudaSuccess || q1 != cudaDriverEntryPointSuccess)
            get_current = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", (void**)&get_id, 12000, cudaEnableDefault, &q2) !=
                cudaSuccess || q2 != cudaDriverEntryPointSuccess)
            get_id = nullptr;
    }
    if (!get_current || !get_id) return 0;
    void* ctx = nullptr;
    unsigned long long id = 0;
    if (get_current(&ctx) != 0 || ctx == nullptr) return 0;
    if (get_id(ctx, &id) != 0) return 0;
    return id;
}

// Device address of the static map on `device` (which must be current).  Resolved with
// cudaGetSymbolAddress once per device and context: host code only holds a host-side stand-in for the
// symbol, which must never be passed to a kernel.  A new context on the device (after cudaDeviceReset,
// the module is loaded again and the array may move) is seen by its id and resolves the address anew.
static int noalloc_scratch(int device, int** out) {
    if (device < 0 || device >= NOALLOC_MAX_DEVICES) {
        set_error("emfem_sweep_spmv_noalloc: device %d beyond the supported %d", device, NOALLOC_MAX_DEVICES);
        return EMFEM_ERR_INVALID_ARG;
    }
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    NoallocSlot& slot = g_noalloc[device];
    unsigned long long ctx = current_ctx_id();
    if (slot.addr == nullptr || ctx == 0 || ctx != slot.ctx_id) {
        int* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress((void**)&p, g_noalloc_patch_map);
        if (e != cudaSuccess) {
            set_error("emfem_sweep_spmv_noalloc: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
            return EMFEM_ERR_CUDA;
        }
        slot.addr = p;
        slot.ctx_id = current_ctx_id();     // the lookup above made the device's context current
    }
    *out = slot.addr;
    return EMFEM_OK;
}
}  // namespace emfem

extern "C" int emfem_sweep_spmv_noalloc(emfem_handle h, int64_t n, const int32_t* indptr, const int32_t* indices,
                                        const void* E_vals, const void* B_vals, int nsys, const double* k0sq_dev,
                                        int64_t n_patch_rows, const int32_t* patch_rows, const int32_t* patch_rowptr,
                                        const int32_t* patch_cols, const void* patch_vals, const int32_t* patch_port,
                                        int n_ports, const double* gamma_dev, const uint8_t* free_mask,
                                        const void* x, void* y) {
    EMFEM_REQUIRE(h && indptr && indices && E_vals && k0sq_dev && free_mask && x && y && n > 0,
                  "emfem_sweep_spmv_noalloc: bad argument");
    EMFEM_REQUIRE(n <= EMFEM_NOALLOC_MAX_ROWS,
                  "emfem_sweep_spmv_noalloc: %lld rows exceed the fixed scratch of %d rows; use emfem_sweep_spmv",
                  (long long)n, EMFEM_NOALLOC_MAX_ROWS);
    EMFEM_REQUIRE(nsys >= 1 && nsys <= 256 && (nsys & (nsys - 1)) == 0,
                  "emfem_sweep_spmv_noalloc: nsys must be a power of two <= 256");
    EMFEM_REQUIRE(n_patch_rows == 0 || (patch_rows && patch_rowptr && patch_cols && patch_vals && patch_port && gamma_dev),
                  "emfem_sweep_spmv_noalloc: patch arrays missing");
    int prev = 0;
    EMFEM_CUDA(cudaGetDevice(&prev));
    if (prev != h->h.device) EMFEM_CUDA(cudaSetDevice(h->h.device));
    int* pmap = nullptr;
    int rc = EMFEM_OK;
    if (n_patch_rows > 0) {
        rc = noalloc_scratch(h->h.device, &pmap);
        if (rc == EMFEM_OK) rc = check_cuda(cudaMemsetAsync(pmap, 0xff, sizeof(int) * n, h->h.stream), "cudaMemsetAsync");
        if (rc == EMFEM_OK) {
            patch_map_kernel<<<grid_for(n_patch_rows, VB), VB, 0, h->h.stream>>>(n_patch_rows, patch_rows, pmap);
            rc = check_cuda(cudaGetLastError(), "patch_map_kernel");
        }
    }
    if (rc == EMFEM_OK) {
        OpArgs a;
        build_op(a, n, nsys, indptr, indices, E_vals, B_vals, k0sq_dev, pmap, patch_rowptr, patch_cols, patch_vals,
                 patch_port, n_ports, gamma_dev, free_mask);
        launch_spmv<double>(a, (const double2*)x, (double2*)y, nullptr, DOT_NONE, nullptr, nsys, h->h.stream);
        rc = check_cuda(cudaGetLastError(), "spmv_kernel");
    }
    if (prev != h->h.device) cudaSetDevice(prev);
    return rc;
}
