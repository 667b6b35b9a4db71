// FP64 Cholesky solve of one symmetric positive definite system A x = g per block of CH_THREADS
// threads (solver.h:70-105, cuSOLVER DPOTRF/DPOTRS in the reference), shared by the shape solve
// and the landmark initializer.
//
// Arithmetic (shared with the oracle): pivots l_jj = sqrt(s_j); L(i,j) = t_ij r_j with
// r_j = 1 / l_jj (DIV = false) or t_ij / l_jj (DIV = true), where t_ij is a_ij minus L(i,k) L(j,k)
// for k = 0, 1, ... in increasing k (each product and difference rounded); forward y_i and back
// x_i alike, terms in increasing and in decreasing k. The right-hand side is carried as row n of
// the matrix: its entries become y, by the very operations of the forward substitution.
//
// What bounds it is the chain of pivots. Dependent FP64 operations take 9 cycles, a square root
// 95, a reciprocal 76, a division 127 (measured): with one product and one difference a column
// costs at least 200 cycles, 17 k for 85 columns. So the chain has a warp to itself: in step j it
// forms the pivot of column j + 1 from that column's two entries in row j + 1 and its diagonal,
// while the CH_WORKERS others update the triangle, which they hold in registers (thread (tr, tc) =
// (tid % 16, tid / 16) owns the entries (tr + 16 a, tc + 16 b)): they scale column j, subtract its
// products from their entries, and publish column j + 1 and the diagonal entry of column
// j + 2. One barrier per column (with DIV another among the workers, whose column is divided once
// into shared memory). A pivot that is not positive is noticed at the end of the group in which the chain
// formed it, by every thread: the chain is a step ahead of what the workers have read, so group J's
// mark has a slot by J's parity, read after the group's last barrier and written again 16 barriers later
// at the earliest. Each entry receives its updates in increasing k, the sequence of the oracle's
// left-looking dot products. Entries left of the current column or above the diagonal are
// updated too, without tests: nothing reads them again. Columns run in groups of 16, one
// instantiation each, so that every register block has a compile-time index.
// Back substitution in one warp, three to five rows per lane, the coefficients of CH_BU steps loaded
// ahead of the chain, each unknown broadcast by shuffle.
//
// One 85 x 85 system with the shape solve's trial point: the pivot formed by its owner among the
// workers and both substitutions by shuffles took 58 us; panels of 16 columns factored by one
// warp (shuffles or shifts) 60 to 146 us, their 30 products and differences per column issue at
// one per 3.5 cycles from a single warp and delay the chain; this form 33 us
// (1,024 frames in one launch 253 -> 143 us).
#pragma once
#include <cuda_runtime.h>

namespace tdi {

constexpr int CH_WORKERS = 256;
constexpr int CH_THREADS = CH_WORKERS + 32;
constexpr int CH_BU = 8;                    // back substitution: steps whose coefficients are in flight

// Column pitch of the factor: n rows and the right-hand side, odd so that a row's reads fall on
// distinct banks.
__host__ __device__ __forceinline__ int chol_ld(int n) { return (n + 1) | 1; }
__host__ __device__ __forceinline__ size_t chol_smem(int n, int RB)
{
    return ((size_t)n * chol_ld(n) + 5 * 16 * RB + 3) * sizeof(double);
}

struct CholMem {
    double *Lf;      // [n][LD] the factor, column-major, row n the right-hand side
    double *raw;     // [2][16 RB] column j before its scaling, by step parity
    double *rv;      // [16 RB] reciprocal pivots
    double *lv;      // [16 RB] pivots
    double *xs;      // [16 RB] the solution
    double *dd;      // [2] diagonal entry of the column after next, by parity
    int *fail;       // [2] a pivot formed in a group was not positive, by group parity
};

// t / l, correctly rounded, from r = 1 / l correctly rounded: two residual corrections with fused
// multiply-adds (Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", 1990): the first brings the quotient within one unit in the last place, the second
// rounds it correctly. Five dependent operations (45 cycles) instead of a division's 127. Operands
// far from the middle of the exponent range take the division.
__device__ __noinline__ double chol_div_any(double t, double l) { return t / l; }

__device__ __forceinline__ double chol_div(double t, double l, double r)
{
    const double at = fabs(t);
    const double q0 = t * r;
    const double q1 = fma(fma(-q0, l, t), r, q0);
    const double q = fma(fma(-q1, l, t), r, q1);
    if (at == 0.0) return t;                             // (l > 0)
    if (!(at > 1e-150 && at < 1e150 && l > 1e-100 && l < 1e100)) return chol_div_any(t, l);
    return q;
}

__device__ __forceinline__ void chol_worker_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(CH_WORKERS) : "memory"); }

// Steps of column group J (columns 16 J ... 16 J + 15), then the next group; false when a pivot was not
// positive (its reciprocal is then NaN or infinite, what follows it is not used).
template <int RB, bool DIV, int J>
__device__ __forceinline__ bool chol_group(double (&v)[RB][RB], const CholMem &cm, int n, int LD, int tid, int tr,
                                           int tc)
{
    if (16 * J >= n) return true;
    const int jend = min(n, 16 * J + 16);
    for (int j = 16 * J; j < jend; ++j) {
        const double *rj = cm.raw + (j & 1) * 16 * RB;
        const double p = cm.rv[j];
        if (tid >= CH_WORKERS) {
            if (j + 1 < n) {
                const double t = rj[j + 1], d = cm.dd[(j + 1) & 1];
                const double c = DIV ? chol_div(t, cm.lv[j], p) : t * p;
                const double s = d - c * c;
                const double l = sqrt(s);
                const double r = __drcp_rn(l);
                if (tid == CH_WORKERS) {
                    cm.rv[j + 1] = r;
                    if (DIV) cm.lv[j + 1] = l;
                    if (!(s > 0.0)) cm.fail[J & 1] = 1;
                }
            }
        } else {
            double *col = cm.Lf + (size_t)j * LD;
            double ci[RB], cl[RB];
            if constexpr (DIV) {
                if (tid > j && tid <= n) col[tid] = chol_div(rj[tid], cm.lv[j], p);
                chol_worker_barrier();
#pragma unroll
                for (int a = J; a < RB; ++a) { ci[a] = col[tr + 16 * a]; cl[a] = col[tc + 16 * a]; }
            } else {
#pragma unroll
                for (int a = J; a < RB; ++a) { ci[a] = rj[tr + 16 * a] * p; cl[a] = rj[tc + 16 * a] * p; }
            }
            double *rn = cm.raw + ((j + 1) & 1) * 16 * RB;
            const int jn = j + 1, j2 = j + 2;
            if (j < 16 * J + 15) {
                // block column J first: it holds column j + 1
#pragma unroll
                for (int a = J; a < RB; ++a) v[a][J] -= ci[a] * cl[J];
                if (tc == (jn & 15)) {
#pragma unroll
                    for (int a = J; a < RB; ++a) rn[tr + 16 * a] = v[a][J];
                }
            }
#pragma unroll
            for (int b = J + 1; b < RB; ++b)
#pragma unroll
                for (int a = b; a < RB; ++a) v[a][b] -= ci[a] * cl[b];
            if constexpr (J + 1 < RB) {
                if (j == 16 * J + 15 && tc == 0) {
#pragma unroll
                    for (int a = J + 1; a < RB; ++a) rn[tr + 16 * a] = v[a][J + 1];
                }
            }
            if (tr == tc && tr == (j2 & 15)) cm.dd[j2 & 1] = (j < 16 * J + 14 || J + 1 >= RB) ? v[J][J] : v[J + 1 < RB ? J + 1 : J][J + 1 < RB ? J + 1 : J];
            if constexpr (!DIV) {
                // the scaled column, for the back substitution
                if (tc == (j & 15)) {
#pragma unroll
                    for (int a = J; a < RB; ++a)
                        if (tr + 16 * a <= n) col[tr + 16 * a] = ci[a];
                }
            }
        }
        __syncthreads();
    }
    if (cm.fail[J & 1]) return false;
    if constexpr (J + 1 < RB) return chol_group<RB, DIV, J + 1>(v, cm, n, LD, tid, tr, tc);
    else return true;
}

// Solves A x = g: A(i, l) for n > i >= l through a(i, l), g_l through rhs(l); needs n < 16 RB.
// All CH_THREADS threads call it. sm: chol_smem(n, RB) bytes, not in use when called. Returns
// false (in every thread) when a pivot is not positive; else xs[i] = x_i (in sm), readable by all.
template <int RB, bool DIV, class A, class G>
__device__ __forceinline__ bool chol_solve(int n, double *sm, A a_of, G rhs, double *&xs)
{
    const int LD = chol_ld(n), tid = threadIdx.x, tr = tid & 15, tc = tid >> 4;
    CholMem cm;
    cm.Lf = sm;
    cm.raw = cm.Lf + (size_t)n * LD;
    cm.rv = cm.raw + 2 * 16 * RB;
    cm.lv = cm.rv + 16 * RB;
    cm.xs = cm.lv + 16 * RB;
    cm.dd = cm.xs + 16 * RB;
    cm.fail = reinterpret_cast<int *>(cm.dd + 2);
    xs = cm.xs;
    double v[RB][RB];
#pragma unroll
    for (int a = 0; a < RB; ++a)
#pragma unroll
        for (int b = 0; b <= a; ++b) {
            const int i = tr + 16 * a, l = tc + 16 * b;
            // (clamped, so that all of a thread's loads can be in flight together)
            const int lc = min(l, n - 1), ic = max(min(i, n - 1), lc);
            const double e = a_of(ic, lc), g = a == n / 16 ? rhs(lc) : 0.0;
            v[a][b] = l < n ? (i < n ? e : i == n ? g : 0.0) : 0.0;
        }
    // column 0, and the diagonal of column 1
    if (tid < CH_WORKERS) {
        if (tc == 0) {
#pragma unroll
            for (int a = 0; a < RB; ++a) cm.raw[tr + 16 * a] = v[a][0];
        }
        if (tr == 1 && tc == 1) cm.dd[1] = v[0][0];
        if (tid == 0) {
            const double l = sqrt(v[0][0]);
            cm.lv[0] = l;
            cm.rv[0] = __drcp_rn(l);
            cm.fail[0] = !(v[0][0] > 0.0);
            cm.fail[1] = 0;
        }
    }
    __syncthreads();
    if (!chol_group<RB, DIV, 0>(v, cm, n, LD, tid, tr, tc)) return false;
    // back substitution: rows lane + 32 q in t[q]
    if (tid < 32) {
        constexpr int TQ = (RB + 1) / 2;
        const double *Lf = cm.Lf;
        double t[TQ], po[TQ], lo[TQ];
#pragma unroll
        for (int q = 0; q < TQ; ++q) {
            const int i = tid + 32 * q;
            t[q] = i < n ? Lf[(size_t)i * LD + n] : 0.0;
            po[q] = i < n ? cm.rv[i] : 1.0;
            lo[q] = DIV && i < n ? cm.lv[i] : 1.0;
        }
#pragma unroll
        for (int q = TQ - 1; q >= 0; --q) {              // unknowns 32 q + 31 ... 32 q
            if (32 * q >= n) continue;
#pragma unroll 1
            for (int u0 = 32 - CH_BU; u0 >= 0; u0 -= CH_BU) {
                const int k0 = 32 * q + u0;
                if (k0 >= n) continue;
                double co[CH_BU][TQ];                    // L(k, i) of the lane's rows i for the next steps k
#pragma unroll
                for (int u = CH_BU - 1; u >= 0; --u)
#pragma unroll
                    for (int qq = 0; qq <= q; ++qq) {
                        const int i = tid + 32 * qq, k = k0 + u;
                        co[u][qq] = k < n && i < k ? Lf[(size_t)i * LD + k] : 0.0;
                    }
#pragma unroll
                for (int u = CH_BU - 1; u >= 0; --u) {
                    if (k0 + u >= n) continue;
                    const double xo = DIV ? chol_div(t[q], lo[q], po[q]) : t[q] * po[q];     // meaningful in the owner's lane
                    const double xk = __shfl_sync(0xffffffffu, xo, u0 + u);
                    if (tid == u0 + u) cm.xs[k0 + u] = xo;
#pragma unroll
                    for (int qq = 0; qq <= q; ++qq)
                        if (tid + 32 * qq < k0 + u) t[qq] -= co[u][qq] * xk;
                }
            }
        }
    }
    __syncthreads();
    return true;
}

}  // namespace tdi
