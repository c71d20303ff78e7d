// log det M and its gradient d log det M / d phi in FP64 on the device (HubbardExp::logDetM / gradLogDetM,
// hubbardExp.tpp:129-211; HubbardDiag::logDetM / gradLogDetM, hubbardDiag.tpp:169-250, with the time-slice matrix
// 1 - sgn delta K in place of exp(+-sgn delta K), the product taken in increasing t and i sgn sum(phi) added).
//
// logDetM (one matrix; batches go through logdet_many below): the time-slice matrices
// B_t = exp(sgn delta K) diag(phiExp[(t+1) % Nt]) (hubbardExp.tpp:142) are built by one kernel, multiplied as a balanced
// product tree of batched complex GEMMs (log2(Nt) levels instead of Nt sequential products; the product is the same
// B_{Nt-1} ... B_0), then 1 + prod is LU-factorised with partial pivoting (right-looking, panels of 32 columns: one panel
// kernel, the row swaps, a triangular solve for the block row of U and one GEMM update of the trailing matrix per panel)
// and log det = sum log(u_kk) + i pi (#row swaps), folded onto the principal branch like log(det(.))
// (src/NSL/LinAlg/det.tpp:15-20). Summing logs instead of forming det() avoids the overflow that makes the
// reference's value NaN at low temperature.
//
// gradLogDetM: Fk(t) = diag(phiExpInv[(t-1) % Nt]) exp(-sgn delta K); suffix products S(t) = Fk(t) ... Fk(Nt-1)
// and prefix products P(t) = (1 + S(0))^{-1} Fk(0) ... Fk(t) (hubbardExp.tpp:165-208). By size: scans of log2(Nt) levels
// (up to 32 sites and 8 matrices), a whole chain per launch (k_chain, a real exp(delta K) up to 144 sites), else Nt-1
// batched products. The inverse is a Gauss-Jordan elimination in shared memory (up to 64 sites; on clusters while few
// matrices leave SMs free) or the blocked LU. The diagonal of S(t+1) P(t) needs only O(Nx^2) per slice (a row-column dot
// per site) instead of the reference's full GEMM per slice.

#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <set>
#include <string>
#include <vector>

#include "fm_internal.cuh"

namespace nslg {

namespace {

// B[t, i, j] = E[i, j] * ph[(t + shift) mod Nt, j]          (column scaling: E diag(ph))
// or, with rowscale, B[t, i, j] = ph[(t + shift) mod Nt, i] * E[i, j]   (row scaling: diag(ph) E)
// With reverse, slice t is stored at position Nt - 1 - t (the product tree then forms M_0 M_1 ... M_{Nt-1}).
__global__ void k_slices(const double2 *__restrict__ E, const double2 *__restrict__ ph, double2 *__restrict__ B,
                         int Nt, int Nx, int shift, bool rowscale, bool reverse = false) {
    const int64_t nn = (int64_t)Nx * Nx;
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= nn * Nt) return;
    const int t = (int)(idx / nn);
    const int64_t ij = idx - (int64_t)t * nn;
    const int i = (int)(ij / Nx), j = (int)(ij - (int64_t)i * Nx);
    const int ts = ((t + shift) % Nt + Nt) % Nt;
    const double2 s = ph[(int64_t)ts * Nx + (rowscale ? i : j)];
    B[(reverse ? (int64_t)(Nt - 1 - t) * nn : (int64_t)t * nn) + ij] = cmul(E[ij], s);
}

// Sum of n complex values in a fixed order (one block).
__global__ void k_sum_c128(const double2 *__restrict__ v, int64_t n, double2 *__restrict__ out) {
    __shared__ double2 red[256];
    double2 acc = make_double2(0, 0);
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        acc.x += v[i].x;
        acc.y += v[i].y;
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            red[threadIdx.x].x += red[threadIdx.x + w].x;
            red[threadIdx.x].y += red[threadIdx.x + w].y;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = red[0];
}

__global__ void k_add_identity(double2 *A, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) A[(int64_t)i * n + i].x += 1.0;
}

// ---- LU with partial pivoting -------------------------------------------------------------------------------------
// Pivot of column k: p = argmax_{i>=k} |A[i,k]| (first index on ties, k itself where every entry is NaN, so that a row index
// never leaves the matrix); the multipliers l_ik = A[i,k] / A[k,k] are stored in place, the running log of the pivots and the
// number of row swaps give log det.
constexpr int LT = 1024;

// ---- blocked LU: panels of NB columns ------------------------------------------------------------------------------
// Right-looking: factor the panel (one block, column by column, pivots as above), apply its row swaps
// to the other columns, solve for the panel's block row of U, update the trailing matrix with one GEMM. Every step
// of the column-at-a-time version becomes one of four launches per panel.
//
// Panel width: FP64 arithmetic is slow per SM on this part (a panel runs on one SM per matrix), so large matrices use
// narrow panels (NB = 8: a quarter of the in-panel work of NB = 32, the rest moves into the trailing GEMM, which
// spreads over the GPU); matrices of at most 64 rows keep NB = 32 (one panel, fewest launches).
inline int panel_width(int n) { return n <= 64 ? 32 : 8; }

__global__ void __launch_bounds__(LT) k_lu_panel(double2 *A, int n, int k0, int nb, int *piv, double2 *pivots,
                                                 int *swaps, int *singular, int64_t mstride) {
    // matrix blockIdx.x of a batch
    A += blockIdx.x * mstride;
    piv += (int64_t)blockIdx.x * n;
    pivots += (int64_t)blockIdx.x * n;
    swaps += blockIdx.x;
    __shared__ double best[LT];
    __shared__ int bidx[LT];
    for (int k = k0; k < k0 + nb; ++k) {
        double bv = -1.0;
        int bi = k;
        for (int i = k + threadIdx.x; i < n; i += LT) {
            const double2 v = A[(int64_t)i * n + k];
            const double m = hypot(v.x, v.y);
            if (m > bv || (m == bv && i < bi)) {
                bv = m;
                bi = i;
            }
        }
        best[threadIdx.x] = bv;
        bidx[threadIdx.x] = bi;
        __syncthreads();
        for (int w = LT / 2; w > 0; w >>= 1) {
            if (threadIdx.x < w) {
                const double o = best[threadIdx.x + w];
                const int oi = bidx[threadIdx.x + w];
                if (o > best[threadIdx.x] || (o == best[threadIdx.x] && oi < bidx[threadIdx.x])) {
                    best[threadIdx.x] = o;
                    bidx[threadIdx.x] = oi;
                }
            }
            __syncthreads();
        }
        const int p = bidx[0];
        if (p != k)  // the panel's columns; the others are swapped by k_lu_laswp
            for (int j = k0 + threadIdx.x; j < k0 + nb; j += LT) {
                const double2 a = A[(int64_t)k * n + j];
                A[(int64_t)k * n + j] = A[(int64_t)p * n + j];
                A[(int64_t)p * n + j] = a;
            }
        __syncthreads();
        const double2 d = A[(int64_t)k * n + k];
        const double dd = d.x * d.x + d.y * d.y;
        const double2 inv = dd == 0.0 ? make_double2(0.0, 0.0) : make_double2(d.x / dd, -d.y / dd);
        for (int i = k + 1 + threadIdx.x; i < n; i += LT) A[(int64_t)i * n + k] = cmul(A[(int64_t)i * n + k], inv);
        if (threadIdx.x == 0) {
            piv[k] = p;
            pivots[k] = d;
            if (p != k) *swaps += 1;
            if (dd == 0.0) *singular = 1;
        }
        __syncthreads();
        // rank-1 update of the rest of the panel: A[i, j] -= l_ik u_kj, i > k, k < j < k0 + nb
        const int w = k0 + nb - k - 1;
        const int64_t cnt = (int64_t)(n - k - 1) * w;
        for (int64_t e = threadIdx.x; e < cnt; e += LT) {
            const int i = k + 1 + (int)(e / w), j = k + 1 + (int)(e % w);
            const double2 l = A[(int64_t)i * n + k], u = A[(int64_t)k * n + j];
            double2 a = A[(int64_t)i * n + j];
            a.x -= l.x * u.x - l.y * u.y;
            a.y -= l.x * u.y + l.y * u.x;
            A[(int64_t)i * n + j] = a;
        }
        __syncthreads();
    }
}

// The same panel factorisation with the panel (rows [k0, n), columns [k0, k0 + nb)) held in shared memory, row
// stride NB + 1 so that a column read spreads over the banks. Used while the panel fits (PANEL_SMEM bytes):
// one load and one store of the panel instead of global traffic and a block-wide reduction tree per column.
constexpr int PANEL_SMEM = 219648;  // dynamic shared memory of the panel kernel: 416 rows at NB = 32, 1525 at NB = 8

__device__ __forceinline__ bool piv_better(double m, int i, double bm, int bi) {
    return m > bm || (m == bm && i < bi);
}

template <int LPT, int NB>
__global__ void __launch_bounds__(LPT) k_lu_panel_smem(double2 *A, int n, int k0, int nb, int *piv, double2 *pivots,
                                                       int *swaps, int *singular, int64_t mstride) {
    constexpr int PS = NB + 1;
    extern __shared__ double2 Ps[];  // (n - k0) x PS
    // matrix blockIdx.x of a batch (LPT threads: 512 for large panels, 128 for small matrices)
    A += blockIdx.x * mstride;
    piv += (int64_t)blockIdx.x * n;
    pivots += (int64_t)blockIdx.x * n;
    swaps += blockIdx.x;
    __shared__ double wbest[LPT / 32];
    __shared__ int widx[LPT / 32];
    __shared__ int pivot;
    const int rows = n - k0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int e = threadIdx.x; e < rows * nb; e += LPT) {
        const int i = e / nb, j = e % nb;
        Ps[i * PS + j] = A[(int64_t)(k0 + i) * n + k0 + j];
    }
    __syncthreads();
    int nswap = 0, sing = 0;
    for (int kk = 0; kk < nb; ++kk) {
        // pivot: largest |a_ik|^2 over rows i >= kk, first index on ties
        double bm = -1.0;
        int bi = kk;
        for (int i = kk + threadIdx.x; i < rows; i += LPT) {
            const double2 v = Ps[i * PS + kk];
            const double m = v.x * v.x + v.y * v.y;
            if (piv_better(m, i, bm, bi)) {
                bm = m;
                bi = i;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double om = __shfl_down_sync(0xffffffffu, bm, o);
            const int oi = __shfl_down_sync(0xffffffffu, bi, o);
            if (piv_better(om, oi, bm, bi)) {
                bm = om;
                bi = oi;
            }
        }
        if (lane == 0) {
            wbest[warp] = bm;
            widx[warp] = bi;
        }
        __syncthreads();
        if (warp == 0) {
            bm = lane < LPT / 32 ? wbest[lane] : -1.0;
            bi = lane < LPT / 32 ? widx[lane] : kk;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double om = __shfl_down_sync(0xffffffffu, bm, o);
                const int oi = __shfl_down_sync(0xffffffffu, bi, o);
                if (piv_better(om, oi, bm, bi)) {
                    bm = om;
                    bi = oi;
                }
            }
            if (lane == 0) pivot = bi;
        }
        __syncthreads();
        const int p = pivot;
        if (p != kk && threadIdx.x < nb) {
            const double2 a = Ps[kk * PS + threadIdx.x];
            Ps[kk * PS + threadIdx.x] = Ps[p * PS + threadIdx.x];
            Ps[p * PS + threadIdx.x] = a;
        }
        __syncthreads();
        const double2 d = Ps[kk * PS + kk];
        const double dd = d.x * d.x + d.y * d.y;
        const double rdd = dd == 0.0 ? 0.0 : 1.0 / dd;
        const double2 inv = make_double2(d.x * rdd, -d.y * rdd);
        for (int i = kk + 1 + threadIdx.x; i < rows; i += LPT) Ps[i * PS + kk] = cmul(Ps[i * PS + kk], inv);
        if (threadIdx.x == 0) {
            piv[k0 + kk] = k0 + p;
            pivots[k0 + kk] = d;  // log det's terms are summed afterwards, off this column-by-column path
            if (p != kk) ++nswap;
            if (dd == 0.0) sing = 1;
        }
        __syncthreads();
        // rank-1 update of the rest of the panel: A[i, j] -= l_ik u_kj, i > kk, kk < j < nb
        const int w = nb - kk - 1;
        if (w > 0) {
            const int cnt = (rows - kk - 1) * w;
            for (int e = threadIdx.x; e < cnt; e += LPT) {
                const int i = kk + 1 + e / w, j = kk + 1 + e % w;
                const double2 l = Ps[i * PS + kk], u = Ps[kk * PS + j];
                double2 a = Ps[i * PS + j];
                a.x -= l.x * u.x - l.y * u.y;
                a.y -= l.x * u.y + l.y * u.x;
                Ps[i * PS + j] = a;
            }
        }
        __syncthreads();
    }
    for (int e = threadIdx.x; e < rows * nb; e += LPT) {
        const int i = e / nb, j = e % nb;
        A[(int64_t)(k0 + i) * n + k0 + j] = Ps[i * PS + j];
    }
    // panel rows swapped above are whole rows of the panel only; k_lu_laswp swaps the other columns
    if (threadIdx.x == 0) {
        *swaps += nswap;
        if (sing) *singular = 1;
    }
}

// Row swaps of the panel [k0, k0 + nb) applied to every column outside it, in order; one thread per column.
__global__ void k_lu_laswp(double2 *A, int n, int k0, int nb, const int *piv, int64_t mstride) {
    A += blockIdx.y * mstride;  // matrix blockIdx.y of a batch
    piv += (int64_t)blockIdx.y * n;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n || (c >= k0 && c < k0 + nb)) return;
    for (int k = k0; k < k0 + nb; ++k) {
        const int p = piv[k];
        if (p != k) {
            const double2 a = A[(int64_t)k * n + c];
            A[(int64_t)k * n + c] = A[(int64_t)p * n + c];
            A[(int64_t)p * n + c] = a;
        }
    }
}

// Unit-lower triangular solve with the diagonal block L[k0:k0+nb, k0:k0+nb] on columns [c0, n) of rows
// k0..k0+nb of X (X = A for the U block row, X = B for a forward substitution); one thread per column, the
// column's nb unknowns in registers (loops fully unrolled over the LB-row block), four independent partial sums per
// row so that the dependent FP64 chain is a quarter as long, TRSM_T threads per block so that the few columns of a
// small matrix still spread over many SMs. Matrix blockIdx.y of a batch (strides sL, sX).
constexpr int TRSM_T = 32;

__device__ __forceinline__ void csub_mul(double2 &a, double2 l, double2 x) {
    a.x -= l.x * x.x - l.y * x.y;
    a.y -= l.x * x.y + l.y * x.x;
}

template <int LB>
__global__ void __launch_bounds__(TRSM_T) k_trsm_lower_block(const double2 *__restrict__ L, double2 *X, int n, int k0,
                                                             int nb, int c0, int64_t sL, int64_t sX) {
    L += blockIdx.y * sL;
    X += blockIdx.y * sX;
    __shared__ double2 Ls[LB][LB];
    for (int e = threadIdx.x; e < nb * nb; e += blockDim.x)
        Ls[e / nb][e % nb] = L[(int64_t)(k0 + e / nb) * n + k0 + e % nb];
    __syncthreads();
    const int c = c0 + blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    double2 x[LB];
#pragma unroll
    for (int r = 0; r < LB; ++r)  // all loads first: one memory latency instead of one per row
        if (r < nb) x[r] = X[(int64_t)(k0 + r) * n + c];
#pragma unroll
    for (int r = 0; r < LB; ++r) {
        if (r < nb) {
            double2 a[4] = {x[r], make_double2(0, 0), make_double2(0, 0), make_double2(0, 0)};
#pragma unroll
            for (int q = 0; q < r; ++q) csub_mul(a[q & 3], Ls[r][q], x[q]);
            x[r] = make_double2((a[0].x + a[1].x) + (a[2].x + a[3].x), (a[0].y + a[1].y) + (a[2].y + a[3].y));
        }
    }
#pragma unroll
    for (int r = 0; r < LB; ++r)
        if (r < nb) X[(int64_t)(k0 + r) * n + c] = x[r];
}

// Upper triangular solve with the diagonal block U[k0:k0+nb, k0:k0+nb] on all columns of rows k0..k0+nb of B
// (registers, partial sums and block size as above; the reciprocals of the diagonal are formed once per block).
template <int LB>
__global__ void __launch_bounds__(TRSM_T) k_trsm_upper_block(const double2 *__restrict__ U, double2 *B, int n, int k0,
                                                             int nb, int64_t sU, int64_t sB) {
    U += blockIdx.y * sU;
    B += blockIdx.y * sB;
    __shared__ double2 Us[LB][LB];
    __shared__ double2 Ui[LB];
    for (int e = threadIdx.x; e < nb * nb; e += blockDim.x)
        Us[e / nb][e % nb] = U[(int64_t)(k0 + e / nb) * n + k0 + e % nb];
    __syncthreads();
    for (int r = threadIdx.x; r < nb; r += blockDim.x) {
        const double2 d = Us[r][r];
        const double dd = d.x * d.x + d.y * d.y;
        const double rdd = dd == 0.0 ? 0.0 : 1.0 / dd;
        Ui[r] = make_double2(d.x * rdd, -d.y * rdd);
    }
    __syncthreads();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    double2 x[LB];
#pragma unroll
    for (int r = 0; r < LB; ++r)
        if (r < nb) x[r] = B[(int64_t)(k0 + r) * n + c];
#pragma unroll
    for (int r = LB - 1; r >= 0; --r) {
        if (r < nb) {
            double2 a[4] = {x[r], make_double2(0, 0), make_double2(0, 0), make_double2(0, 0)};
#pragma unroll
            for (int q = r + 1; q < LB; ++q)
                if (q < nb) csub_mul(a[q & 3], Us[r][q], x[q]);
            const double2 v = make_double2((a[0].x + a[1].x) + (a[2].x + a[3].x), (a[0].y + a[1].y) + (a[2].y + a[3].y));
            x[r] = cmul(v, Ui[r]);
        }
    }
#pragma unroll
    for (int r = 0; r < LB; ++r)
        if (r < nb) B[(int64_t)(k0 + r) * n + c] = x[r];
}

// out[t, x] = i * sum_k A_t[k, x] B_t[k, x] (the diagonal of A_t^T B_t) for every slice in one launch, with
// A_t = T[(t + 1) mod Nt] and B_t = P[t] for t < Nt - 1, B_{Nt-1} = G. A block covers 32 columns (one per lane,
// coalesced rows) of one slice; its CD_W warps split k and are summed in shared memory.
constexpr int CD_W = 8;

__global__ void __launch_bounds__(32 * CD_W) k_coldot_slices(const double2 *__restrict__ T, const double2 *__restrict__ P,
                                                             const double2 *__restrict__ G, double2 *__restrict__ out,
                                                             int n, int Nt) {
    const int t = blockIdx.y;
    const int64_t nn = (int64_t)n * n;
    const double2 *A = T + (int64_t)((t + 1) % Nt) * nn;
    const double2 *B = t == Nt - 1 ? G : P + (int64_t)t * nn;
    const int x = blockIdx.x * 32 + threadIdx.x;
    double2 acc = make_double2(0, 0);
    if (x < n)
        for (int k = threadIdx.y; k < n; k += CD_W) {
            const double2 a = A[(int64_t)k * n + x], b = B[(int64_t)k * n + x];
            acc.x += a.x * b.x - a.y * b.y;
            acc.y += a.x * b.y + a.y * b.x;
        }
    __shared__ double2 red[CD_W][32];
    red[threadIdx.y][threadIdx.x] = acc;
    __syncthreads();
    if (threadIdx.y == 0 && x < n) {
        double2 sum = red[0][threadIdx.x];
#pragma unroll
        for (int w = 1; w < CD_W; ++w) {
            sum.x += red[w][threadIdx.x].x;
            sum.y += red[w][threadIdx.x].y;
        }
        out[(int64_t)t * n + x] = make_double2(-sum.y, sum.x);  // i * sum
    }
}

// out[j, i] = E[j, i] * d[i]
__global__ void k_colscale(const double2 *__restrict__ E, const double2 *__restrict__ d, double2 *__restrict__ out,
                           int n) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (int64_t)n * n) return;
    out[idx] = cmul(E[idx], d[idx % n]);
}

// out = T^T + 1
__global__ void k_transpose_plus_identity(const double2 *__restrict__ T, double2 *__restrict__ out, int n) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (int64_t)n * n) return;
    const int i = (int)(idx / n), j = (int)(idx % n);
    double2 v = T[(int64_t)j * n + i];
    if (i == j) v.x += 1.0;
    out[idx] = v;
}

}  // namespace

// Factors nmat matrices at once (matrix g at A + g * mstride, mstride 0 = n * n): each panel step is one launch
// over the whole batch, so independent matrices (the two species, many configurations) factor side by side on
// different SMs. Pivots, log sums and swap counts are per matrix; the singular flag is shared.
// logsum[g] = sum_k (log|u_kk| + i arg u_kk) over matrix g's pivots (zero pivots, flagged singular, are skipped),
// one block per matrix, fixed-order tree sum.
__global__ void k_pivot_logsum(const double2 *__restrict__ pivots, int n, double2 *__restrict__ logsum) {
    __shared__ double2 red[256];
    const double2 *pv = pivots + (int64_t)blockIdx.x * n;
    double2 acc = make_double2(0, 0);
    for (int k = threadIdx.x; k < n; k += 256) {
        const double2 d = pv[k];
        if (d.x != 0.0 || d.y != 0.0) {
            acc.x += log(hypot(d.x, d.y));
            acc.y += atan2(d.y, d.x);
        }
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            red[threadIdx.x].x += red[threadIdx.x + w].x;
            red[threadIdx.x].y += red[threadIdx.x + w].y;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) logsum[blockIdx.x] = red[0];
}

namespace {
template <int NB>
int lu_factor_nb(nslg_fm *fm, double2 *A, int n, LuScratch &s, int nmat, int64_t mstride) {
    cudaStream_t st = fm->ctx->stream;
    const double2 minus_one = make_double2(-1, 0);
    for (int k0 = 0; k0 < n; k0 += NB) {
        const int nb = std::min(NB, n - k0);
        const size_t smem = (size_t)(n - k0) * (NB + 1) * sizeof(double2);
        if (n - k0 <= 64)
            k_lu_panel_smem<128, NB><<<nmat, 128, smem, st>>>(A, n, k0, nb, s.piv, s.pivots, s.swaps, s.singular,
                                                              mstride);
        else if (smem <= (size_t)PANEL_SMEM)
            k_lu_panel_smem<512, NB><<<nmat, 512, smem, st>>>(A, n, k0, nb, s.piv, s.pivots, s.swaps, s.singular,
                                                              mstride);
        else
            k_lu_panel<<<nmat, LT, 0, st>>>(A, n, k0, nb, s.piv, s.pivots, s.swaps, s.singular, mstride);
        note_launch(st);
        if (n > nb) {
            k_lu_laswp<<<dim3((unsigned)ceil_div(n, 128), (unsigned)nmat), 128, 0, st>>>(A, n, k0, nb, s.piv, mstride);
            note_launch(st);
        }
        const int rest = n - k0 - nb;
        if (rest > 0) {
            // U12 = L11^{-1} A12, then A22 -= L21 U12
            k_trsm_lower_block<NB><<<dim3((unsigned)ceil_div(rest, TRSM_T), (unsigned)nmat), TRSM_T, 0, st>>>(
                A, A, n, k0, nb, k0 + nb, mstride, mstride);
            note_launch(st);
            const double2 *L21 = A + (int64_t)(k0 + nb) * n + k0, *U12 = A + (int64_t)k0 * n + k0 + nb;
            double2 *A22 = A + (int64_t)(k0 + nb) * n + k0 + nb;
            NSLG_TRY(zgemm(st, rest, rest, nb, minus_one, L21, n, mstride, U12, n, mstride, A22, n, mstride, nmat,
                           false, true));
        }
    }
    return NSLG_OK;
}

}  // namespace

// Factors nmat matrices at once (matrix g at A + g * mstride, mstride 0 = n * n): each panel step is one launch
// over the whole batch, so independent matrices (the two species, many configurations) factor side by side on
// different SMs. Pivots, log sums and swap counts are per matrix; the singular flag is shared.
int lu_factor(nslg_fm *fm, double2 *A, int n, LuScratch &s, int nmat, int64_t mstride, bool want_logsum) {
    cudaStream_t st = fm->ctx->stream;
    if (mstride == 0) mstride = (int64_t)n * n;
    {
        // the panel kernels' shared-memory limit, raised once per device (first call is never inside a capture:
        // the captured trajectory runs eagerly first)
        static std::mutex mu;
        static std::set<int> done;
        std::lock_guard<std::mutex> lock(mu);
        if (!done.count(fm->ctx->device)) {
            NSLG_CUDA(cudaFuncSetAttribute(k_lu_panel_smem<512, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           PANEL_SMEM));
            NSLG_CUDA(cudaFuncSetAttribute(k_lu_panel_smem<128, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           PANEL_SMEM));
            NSLG_CUDA(cudaFuncSetAttribute(k_lu_panel_smem<512, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           PANEL_SMEM));
            NSLG_CUDA(cudaFuncSetAttribute(k_lu_panel_smem<128, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           PANEL_SMEM));
            done.insert(fm->ctx->device);
        }
    }
    NSLG_CUDA(cudaMemsetAsync(s.swaps, 0, (size_t)nmat * sizeof(int), st));
    if (!fm->defer_checks) NSLG_CUDA(cudaMemsetAsync(s.singular, 0, sizeof(int), st));
    if (panel_width(n) == 32) NSLG_TRY(lu_factor_nb<32>(fm, A, n, s, nmat, mstride));
    else NSLG_TRY(lu_factor_nb<8>(fm, A, n, s, nmat, mstride));
    if (want_logsum) {
        k_pivot_logsum<<<(unsigned)nmat, 256, 0, st>>>(s.pivots, n, s.logsum);
        note_launch(st);
    }
    NSLG_CUDA(cudaGetLastError());
    return NSLG_OK;
}

namespace {
template <int NB>
int lu_solve_nb(nslg_fm *fm, const double2 *LU, double2 *B, int n, int nmat, int64_t lu_stride, int64_t b_stride) {
    cudaStream_t st = fm->ctx->stream;
    const double2 minus_one = make_double2(-1, 0);
    const dim3 gc((unsigned)ceil_div(n, TRSM_T), (unsigned)nmat);
    for (int k0 = 0; k0 < n; k0 += NB) {  // forward: L y = P b
        const int nb = std::min(NB, n - k0);
        k_trsm_lower_block<NB><<<gc, TRSM_T, 0, st>>>(LU, B, n, k0, nb, 0, lu_stride, b_stride);
        note_launch(st);
        const int rest = n - k0 - nb;
        if (rest > 0)
            NSLG_TRY(zgemm(st, rest, n, nb, minus_one, LU + (int64_t)(k0 + nb) * n + k0, n, lu_stride,
                           B + (int64_t)k0 * n, n, b_stride, B + (int64_t)(k0 + nb) * n, n, b_stride, nmat, false,
                           true));
    }
    for (int k0 = ((n - 1) / NB) * NB; k0 >= 0; k0 -= NB) {  // backward: U x = y
        const int nb = std::min(NB, n - k0);
        k_trsm_upper_block<NB><<<gc, TRSM_T, 0, st>>>(LU, B, n, k0, nb, lu_stride, b_stride);
        note_launch(st);
        if (k0 > 0)
            NSLG_TRY(zgemm(st, k0, n, nb, minus_one, LU + k0, n, lu_stride, B + (int64_t)k0 * n, n, b_stride, B, n,
                           b_stride, nmat, false, true));
    }
    return NSLG_OK;
}

// B[g] = P_g W[g] (the identity for a null W): the factorisation's row swaps applied in order (row k of the result is row
// perm[k], perm the composition of the swaps). Each block rebuilds perm in shared memory with one thread, then
// its threads write rows [row0, row0 + rows_per_block) of matrix blockIdx.x.
__global__ void k_perm_rows(double2 *B, const double2 *W, int n, const int *piv, int64_t bstride, int rows_per_block) {
    extern __shared__ int perm[];
    const int g = blockIdx.x;
    piv += (int64_t)g * n;
    B += g * bstride;
    if (threadIdx.x == 0) {
        for (int k = 0; k < n; ++k) perm[k] = k;
        for (int k = 0; k < n; ++k) {
            const int p = piv[k];
            const int a = perm[k];
            perm[k] = perm[p];
            perm[p] = a;
        }
    }
    __syncthreads();
    const int r0 = blockIdx.y * rows_per_block, r1 = min(n, r0 + rows_per_block);
    for (int64_t e = (int64_t)r0 * n + threadIdx.x; e < (int64_t)r1 * n; e += blockDim.x) {
        const int k = (int)(e / n), j = (int)(e % n);
        B[e] = W ? W[g * bstride + (int64_t)perm[k] * n + j] : make_double2(j == perm[k] ? 1.0 : 0.0, 0.0);
    }
}

// G[g] = (A_g + 1)^{-1} for small matrices (n <= GJ_MAX) in one launch: in-place Gauss-Jordan elimination with partial
// pivoting in shared memory, one CTA per matrix. Rows are never swapped: column k's pivot is the largest entry among the
// rows that have not been pivots yet (first row on ties, the same choice as an LU with row swaps makes up to the row
// order), and the permutation is applied on the way out, inv[k, p_j] = W[p_k, j]. A step is the scaled pivot row and one
// update of all n^2 elements, which the FP64 pipe of one SM bounds for large n (n^3 complex FMAs, 2 FP64 FMAs per clock);
// beside it one warp looks ahead: it forms the next column, finds its pivot (integer comparisons of the FP64 bit patterns:
// an FP64 comparison costs a warp 64 cycles) and the reciprocal, ~20 dependent FP64 operations that bound small n.
// Measured: 52 us -> 32 us at n = 18 (38 without the look-ahead); panel factorisation, triangular solves and permutation of
// 32 matrices of n = 50 690 us -> 254 us (293 without).
constexpr int GJ_MAX = 64;
constexpr int GJ_T = 512;
constexpr int SCAN_MAX = 32;           // the small-lattice gradient uses scans up to this size
constexpr int SCAN_MAX_MATRICES = 8;   // and up to this many matrices per call

constexpr size_t gj_smem(int n) { return (size_t)n * (n + 1) * sizeof(double2); }

// a b and a - l u with their roundings spelled out: both kernels below give the same bits
__device__ __forceinline__ double2 gj_mul(double2 a, double2 b) {
    return make_double2(fma(a.x, b.x, -__dmul_rn(a.y, b.y)), fma(a.x, b.y, __dmul_rn(a.y, b.x)));
}
__device__ __forceinline__ double2 gj_update(double2 a, double2 l, double2 u) {
    const double2 t = gj_mul(l, u);
    return make_double2(__dsub_rn(a.x, t.x), __dsub_rn(a.y, t.y));
}

struct GjPivot {
    int row;
    bool mine, zero;  // this lane holds it; it is zero
    double2 inv;      // its reciprocal, in that lane
};

// One warp: the pivot among the rows not in `used`, from the column's values c[0], c[1] at rows lane, lane + 32.
__device__ __forceinline__ GjPivot gj_choose(int n, unsigned long long used, const double2 (&c)[2]) {
    unsigned long long bm = 0;
    int bi = GJ_MAX;
    double2 bv = make_double2(0, 0);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int i = (int)(threadIdx.x % 32) + 32 * h;
        if (i >= n || (used >> i & 1)) continue;
        const unsigned long long m = (unsigned long long)__double_as_longlong(fma(c[h].x, c[h].x, c[h].y * c[h].y));
        if (bi == GJ_MAX || m > bm) {
            bm = m;
            bi = i;
            bv = c[h];
        }
    }
    const int mine = bi;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long om = __shfl_xor_sync(0xffffffffu, bm, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (oi < GJ_MAX && (bi == GJ_MAX || om > bm || (om == bm && oi < bi))) {
            bm = om;
            bi = oi;
        }
    }
    GjPivot q{bi, mine == bi, false, make_double2(0, 0)};
    if (q.mine) {
        const double dd = __longlong_as_double((long long)bm);  // |bv|^2
        const double rdd = dd == 0.0 ? 0.0 : 1.0 / dd;
        q.inv = make_double2(bv.x * rdd, -bv.y * rdd);
        q.zero = dd == 0.0;
    }
    return q;
}

__global__ void __launch_bounds__(GJ_T) k_gj_inverse(const double2 *__restrict__ A, int64_t astride,
                                                     double2 *__restrict__ G, int n, int *singular) {
    extern __shared__ double2 W[];  // n x (n + 1)
    __shared__ double2 f[GJ_MAX], u[GJ_MAX], next[GJ_MAX];
    __shared__ double2 inv_sh;
    __shared__ int pivot, piv[GJ_MAX];
    const int ld = n + 1, T = blockDim.x, tid = threadIdx.x;
    const int g = blockIdx.x;
    A += g * astride;
    G += (int64_t)g * n * n;
    for (int e = tid; e < n * n; e += T) {
        const int i = e / n, j = e - i * n;
        double2 v = A[e];
        if (i == j) v.x += 1.0;
        W[i * ld + j] = v;
    }
    __syncthreads();
    // warps 1 .. update all elements; warp 0 only looks ahead: it forms the next column, finds its pivot and the pivot's
    // reciprocal (a chain of ~10 dependent FP64 steps) while they do
    const int TB = T - 32, tb = tid - 32;
    const int di = TB / n, dj = TB - di * n;  // (i, j) steps of this thread's elements
    const int i0 = tb / n, j0 = tb - i0 * n;
    unsigned long long used = 0;  // rows that have been pivots (warp 0)
    int sing = 0;
    auto choose = [&](int k, const double2 (&c)[2]) {
        const GjPivot q = gj_choose(n, used, c);
        used |= 1ull << q.row;
        if (q.mine) {  // the lane that holds the pivot
            inv_sh = q.inv;
            pivot = q.row;
            piv[k] = q.row;
            if (q.zero) sing = 1;
        }
    };
    if (tid < 32) {
        const double2 c[2] = {tid < n ? W[tid * ld] : make_double2(0, 0),
                              tid + 32 < n ? W[(tid + 32) * ld] : make_double2(0, 0)};
        choose(0, c);
    }
    __syncthreads();
    int last = -1;  // the previous pivot row
    for (int k = 0; k < n; ++k) {
        const int p = pivot;
        const double2 inv = inv_sh;
        for (int j = tid; j < n; j += T) {
            u[j] = j == k ? inv : gj_mul(W[p * ld + j], inv);
            f[j] = (k == 0 || j == last) ? W[j * ld + k] : next[j];
        }
        __syncthreads();
        if (tid < 32) {
            if (k + 1 < n) {
                const double2 uj = u[k + 1];
                double2 c[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int i = tid + 32 * h;
                    c[h] = make_double2(0, 0);
                    if (i < n && i != p) {
                        const double2 l = f[i];
                        const double2 a = gj_update(W[i * ld + k + 1], l, uj);
                        c[h] = a;
                        next[i] = a;  // column k + 1 as the next step's multipliers (W keeps its old values, unread)
                    } else if (i == p) {
                        c[h] = uj;
                    }
                }
                choose(k + 1, c);
            }
        } else {
            for (int e = tb, i = i0, j = j0; e < n * n; e += TB) {
                if (j != k + 1 || i == p) {  // (the rest of column k + 1 is warp 0's)
                    const double2 uj = u[j];
                    double2 a = uj;
                    if (i != p) {
                        const double2 l = f[i];
                        a = gj_update(j == k ? make_double2(0, 0) : W[i * ld + j], l, uj);
                    }
                    W[i * ld + j] = a;
                }
                i += di;
                j += dj;
                if (j >= n) {
                    j -= n;
                    ++i;
                }
            }
        }
        __syncthreads();
        last = p;
    }
    for (int e = tid; e < n * n; e += T) {
        const int k = e / n, j = e - k * n;
        G[k * n + piv[j]] = W[piv[k] * ld + j];
    }
    if (sing) *singular = 1;
}

// The same elimination on a cluster of GC CTAs per matrix, columns dealt out in turn: the update of n^2 elements, which one
// SM's FP64 pipe takes 2 n^2 cycles for, is shared, and what is left of a step is the look-ahead. The owner of column k + 1
// writes it, its pivot and the reciprocal into every CTA's shared memory (two buffers); one cluster barrier per step.
// Every element sees the operations of k_gj_inverse. Measured, 32 matrices of n = 50: 253 us -> 128 us.
constexpr int GC = 4;
constexpr int GC_T = 384;
constexpr int GC_MIN = 24;  // sites from which clusters are used

__global__ void __launch_bounds__(GC_T) k_gj_cluster(const double2 *__restrict__ A, int64_t astride,
                                                     double2 *__restrict__ G, int n, int *singular) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    constexpr int NC = (GJ_MAX + GC - 1) / GC, LD = NC + 1;
    __shared__ double2 W[GJ_MAX * LD];  // row i, local column jl (column jl GC + rank)
    __shared__ double2 f[2][GJ_MAX], u[NC], inv_sh[2];
    __shared__ int pivot[2], piv[GJ_MAX];
    const int tid = threadIdx.x, T = blockDim.x, rank = (int)cl.block_rank();
    const int g = blockIdx.x / GC;
    const int nc = (n - rank + GC - 1) / GC;  // (n > GC)
    A += g * astride;
    G += (int64_t)g * n * n;
    for (int e = tid; e < n * nc; e += T) {
        const int i = e / nc, jl = e - i * nc, j = jl * GC + rank;
        double2 v = A[(int64_t)i * n + j];
        if (i == j) v.x += 1.0;
        W[i * LD + jl] = v;
    }
    unsigned long long used = 0;
    int sing = 0;
    // warp 0 of column k's owner: the column, its pivot and reciprocal to every CTA
    auto publish = [&](int k, const double2 (&c)[2]) {
        const GjPivot q = gj_choose(n, used, c);
        const int b = k & 1;
#pragma unroll
        for (int r = 0; r < GC; ++r) {
            double2 *fr = cl.map_shared_rank(&f[b][0], r);
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (tid + 32 * h < n) fr[tid + 32 * h] = c[h];
            if (q.mine) {
                *cl.map_shared_rank(&inv_sh[b], r) = q.inv;
                *cl.map_shared_rank(&pivot[b], r) = q.row;
            }
        }
        if (q.mine && q.zero) sing = 1;
    };
    cl.sync();  // every CTA has started (and loaded)
    if (rank == 0 && tid < 32) {
        const double2 c[2] = {tid < n ? W[tid * LD] : make_double2(0, 0),
                              tid + 32 < n ? W[(tid + 32) * LD] : make_double2(0, 0)};
        publish(0, c);
    }
    cl.sync();
    const int TB = T - 32, tb = tid - 32;
    const int di = TB / nc, dj = TB - di * nc, i0 = tb / nc, j0 = tb - i0 * nc;
    for (int k = 0; k < n; ++k) {
        const int b = k & 1, p = pivot[b];
        used |= 1ull << p;
        const int kl = k % GC == rank ? k / GC : -1;                // this CTA's column k
        const int nl = (k + 1) % GC == rank && k + 1 < n ? (k + 1) / GC : -1;  // and column k + 1
        if (tid == 0) piv[k] = p;
        if (tid < nc) u[tid] = tid == kl ? inv_sh[b] : gj_mul(W[p * LD + tid], inv_sh[b]);
        __syncthreads();
        if (tid < 32) {
            if (nl >= 0) {
                const double2 uj = u[nl];
                double2 c[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int i = tid + 32 * h;
                    c[h] = make_double2(0, 0);
                    if (i < n) c[h] = i == p ? uj : gj_update(W[i * LD + nl], f[b][i], uj);
                }
                publish(k + 1, c);
            }
        } else {
            for (int e = tb, i = i0, jl = j0; e < n * nc; e += TB) {
                if (jl != nl || i == p) {  // (the rest of column k + 1 lives on in f)
                    const double2 uj = u[jl];
                    W[i * LD + jl] = i == p ? uj : gj_update(jl == kl ? make_double2(0, 0) : W[i * LD + jl], f[b][i], uj);
                }
                i += di;
                jl += dj;
                if (jl >= nc) {
                    jl -= nc;
                    ++i;
                }
            }
        }
        cl.sync();
    }
    for (int e = tid; e < n * nc; e += T) {
        const int k = e / nc, jl = e - k * nc;
        G[(int64_t)k * n + piv[jl * GC + rank]] = W[piv[k] * LD + jl];
    }
    if (sing) *singular = 1;
}

// G[g] = (A_g + 1)^{-1} (astride elements apart, G dense), n <= GJ_MAX.
int gj_inverse_plus_one(nslg_fm *fm, const double2 *A, int64_t astride, double2 *G, int n, int nmat, int *singular) {
    {
        static std::mutex mu;
        static std::set<int> done;
        std::lock_guard<std::mutex> lock(mu);
        if (!done.count(fm->ctx->device)) {
            NSLG_CUDA(cudaFuncSetAttribute(k_gj_inverse, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)gj_smem(GJ_MAX)));
            done.insert(fm->ctx->device);
        }
    }
    // clusters from 24 sites on while two CTAs per SM hold all matrices. One gradient (ring, Nt = 8), one CTA and clusters:
    // 14 sites 90 and 92 us, 16 97 and 97, 18 108 and 102, 22 118 and 111, 24 122 and 115, 28 136 and 126, 32 160 and 139.
    // Trajectories of 5 forces, one CTA per matrix against clusters: n = 32, 2 matrices 904 and 803 us; n = 50 2.15 and
    // 1.51 ms, 48 matrices 5.33 and 4.90 ms, 76 6.64 and 6.50 ms; n = 64, 2 matrices 3.05 and 1.54 ms, 48 5.94 and 4.94 ms.
    if (n >= GC_MIN && (int64_t)nmat * GC <= 2 * std::max(1, num_sms())) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)nmat * GC);
        cfg.blockDim = dim3(GC_T);
        cfg.stream = fm->ctx->stream;
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = GC;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        NSLG_CUDA(cudaLaunchKernelEx(&cfg, k_gj_cluster, A, astride, G, n, singular));
        note_launch(fm->ctx->stream);
        return NSLG_OK;
    }
    k_gj_inverse<<<(unsigned)nmat, GJ_T, gj_smem(n), fm->ctx->stream>>>(A, astride, G, n, singular);
    note_launch(fm->ctx->stream);
    NSLG_CUDA(cudaGetLastError());
    return NSLG_OK;
}

// One level of the Hillis-Steele scans over the slices of nmat matrices (n <= SCAN_MAX), prefix and suffix in one launch:
//   Qn(t) = Q(t - o) Q(t) (t >= o, Q(t) below),  Sn(t) = S(t) S(t + o) (t < Nt - o, S(t) above).
// A CTA computes 32 outputs of one product, its four warps a quarter of the k sum each (one per scheduler).
__global__ void __launch_bounds__(128) k_scan_level(const double2 *__restrict__ Q, const double2 *__restrict__ S,
                                                    double2 *__restrict__ Qn, double2 *__restrict__ Sn, int n, int Nt,
                                                    int o) {
    __shared__ double2 red[3][32];
    const int lane = threadIdx.x % 32, w = threadIdx.x / 32;
    const int t = blockIdx.y;
    const bool suffix = blockIdx.z & 1;
    const int64_t nn = (int64_t)n * n, base = (int64_t)(blockIdx.z >> 1) * Nt * nn;
    const int e = blockIdx.x * 32 + lane;
    const double2 *X = (suffix ? S : Q) + base;
    double2 *Y = (suffix ? Sn : Qn) + base;
    const int ta = suffix ? t : t - o, tb = suffix ? t + o : t;
    if (ta < 0 || tb >= Nt) {  // no partner at this distance
        if (w == 0 && e < nn) Y[t * nn + e] = X[t * nn + e];
        return;
    }
    double2 acc = make_double2(0, 0);
    if (e < nn) {
        const int i = e / n, j = e - i * n;
        const double2 *a = X + ta * nn + i * n, *b = X + tb * nn + j;
#pragma unroll 8
        for (int k = w; k < n; k += 4) {
            const double2 av = a[k], bv = b[k * n];
            acc.x = fma(av.x, bv.x, acc.x);
            acc.x = fma(-av.y, bv.y, acc.x);
            acc.y = fma(av.x, bv.y, acc.y);
            acc.y = fma(av.y, bv.x, acc.y);
        }
    }
    if (w > 0) red[w - 1][lane] = acc;
    __syncthreads();
    if (w == 0 && e < nn) {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            acc.x += red[q][lane].x;
            acc.y += red[q][lane].y;
        }
        Y[t * nn + e] = acc;
    }
}

// out[g, t, x] = i sum_k S(t + 1)[x, k] (G Q(t))[k, x], and i sum_k S(0)[x, k] G[k, x] at t = Nt - 1: the diagonal of the
// gradient from the scans without storing G Q(t). A CTA owns XB sites of one slice, a thread one (site, k).
__global__ void __launch_bounds__(128) k_scan_grad(const double2 *__restrict__ S, const double2 *__restrict__ Q,
                                                   const double2 *__restrict__ G, double2 *__restrict__ out, int n,
                                                   int Nt, int XB) {
    __shared__ double2 term[128];
    const int t = blockIdx.y, g = blockIdx.z;
    const int64_t nn = (int64_t)n * n;
    const int xl = threadIdx.x / n, k = threadIdx.x - xl * n, x = blockIdx.x * XB + xl;
    const double2 *Gg = G + g * nn;
    if (xl < XB && x < n) {
        const double2 s = S[((int64_t)g * Nt + (t + 1) % Nt) * nn + x * n + k];
        double2 p;
        if (t == Nt - 1) {
            p = Gg[k * n + x];
        } else {
            const double2 *q = Q + ((int64_t)g * Nt + t) * nn + x;
            double2 r[4] = {make_double2(0, 0), make_double2(0, 0), make_double2(0, 0), make_double2(0, 0)};
            for (int l0 = 0; l0 < n; l0 += 4)
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (l0 + c < n) {
                        const double2 a = Gg[k * n + l0 + c], b = q[(l0 + c) * n];
                        r[c].x = fma(a.x, b.x, r[c].x);
                        r[c].x = fma(-a.y, b.y, r[c].x);
                        r[c].y = fma(a.x, b.y, r[c].y);
                        r[c].y = fma(a.y, b.x, r[c].y);
                    }
            p = make_double2(((r[0].x + r[1].x) + r[2].x) + r[3].x, ((r[0].y + r[1].y) + r[2].y) + r[3].y);
        }
        term[threadIdx.x] = cmul(s, p);
    }
    for (int o = 16; o > 0; o >>= 1) {  // tree sum over k (n <= 32)
        __syncthreads();
        if (k < o && k + o < n && xl < XB && x < n) {
            double2 v = term[threadIdx.x];
            v.x += term[threadIdx.x + o].x;
            v.y += term[threadIdx.x + o].y;
            term[threadIdx.x] = v;
        }
    }
    if (k == 0 && xl < XB && x < n) {
        const double2 v = term[threadIdx.x];
        out[((int64_t)g * Nt + t) * n + x] = make_double2(-v.y, v.x);  // i * sum
    }
}

}  // namespace

// G[g] = A_g^{-1} for nmat factored matrices (LU of matrix g at LU + g * lu_stride, G dense (nmat, n, n)).
int lu_inverse(nslg_fm *fm, const double2 *LU, double2 *G, int n, const LuScratch &s, int nmat, int64_t lu_stride) {
    cudaStream_t st = fm->ctx->stream;
    const int64_t nn = (int64_t)n * n;
    if (lu_stride == 0) lu_stride = nn;
    const int rpb = 32;
    k_perm_rows<<<dim3((unsigned)nmat, (unsigned)ceil_div(n, rpb)), 256, (size_t)n * sizeof(int), st>>>(
        G, nullptr, n, s.piv, nn, rpb);
    note_launch(st);
    if (panel_width(n) == 32) NSLG_TRY(lu_solve_nb<32>(fm, LU, G, n, nmat, lu_stride, nn));
    else NSLG_TRY(lu_solve_nb<8>(fm, LU, G, n, nmat, lu_stride, nn));
    NSLG_CUDA(cudaGetLastError());
    return NSLG_OK;
}

// Y[g] = A_g^{-1} W[g]: the right-hand sides' rows in pivot order, then both substitutions.
int lu_solve(nslg_fm *fm, const double2 *LU, const double2 *W, double2 *Y, int n, const LuScratch &s, int nmat,
             int64_t lu_stride) {
    cudaStream_t st = fm->ctx->stream;
    const int64_t nn = (int64_t)n * n;
    const int rpb = 32;
    k_perm_rows<<<dim3((unsigned)nmat, (unsigned)ceil_div(n, rpb)), 256, (size_t)n * sizeof(int), st>>>(Y, W, n, s.piv, nn,
                                                                                                    rpb);
    note_launch(st);
    if (panel_width(n) == 32) NSLG_TRY(lu_solve_nb<32>(fm, LU, Y, n, nmat, lu_stride, nn));
    else NSLG_TRY(lu_solve_nb<8>(fm, LU, Y, n, nmat, lu_stride, nn));
    NSLG_CUDA(cudaGetLastError());
    return NSLG_OK;
}

int get_lu_scratch(nslg_fm *fm, int n, LuScratch &s, int nmat, const char *tag) {
    const std::string t = tag ? tag : "lu";
    NSLG_TRY(ws_get(fm, (t + "_piv").c_str(), (size_t)n * nmat, &s.piv));
    NSLG_TRY(ws_get(fm, (t + "_logsum").c_str(), (size_t)nmat, &s.logsum));
    NSLG_TRY(ws_get(fm, (t + "_pivots").c_str(), (size_t)n * nmat, &s.pivots));
    NSLG_TRY(ws_get(fm, (t + "_swaps").c_str(), (size_t)nmat, &s.swaps));
    NSLG_TRY(ws_get(fm, "lu_singular", 1, &s.singular));
    return NSLG_OK;
}

namespace {

// In-place product tree over T matrices in buf (T, n, n): after the call buf[0] = M_{T-1} ... M_0.
int product_tree(nslg_fm *fm, double2 *buf, double2 *tmp, int T, int n) {
    cudaStream_t st = fm->ctx->stream;
    const int64_t nn = (int64_t)n * n;
    const double2 one = make_double2(1, 0);
    while (T > 1) {
        const int pairs = T / 2;
        // tmp[k] = buf[2k+1] @ buf[2k]
        NSLG_TRY(zgemm(st, n, n, n, one, buf + nn, n, 2 * nn, buf, n, 2 * nn, tmp, n, nn, pairs, false));
        NSLG_CUDA(cudaMemcpyAsync(buf, tmp, pairs * nn * sizeof(double2), cudaMemcpyDeviceToDevice, st));
        if (T & 1)
            NSLG_CUDA(cudaMemcpyAsync(buf + pairs * nn, buf + (T - 1) * nn, nn * sizeof(double2),
                                      cudaMemcpyDeviceToDevice, st));
        T = pairs + (T & 1);
    }
    return NSLG_OK;
}

}  // namespace

// log det M for the populated configuration and current species; result on the host.
int fm_logdet(nslg_fm *fm, double2 *out) {
    cudaStream_t st = fm->ctx->stream;
    const int Nt = (int)fm->Nt, n = (int)fm->Nx;
    const int64_t nn = (int64_t)n * n;
    const bool diag = fm->kind == NSLG_FM_DIAG;
    const double2 d = make_double2(fm->sgn * fm->delta.x, fm->sgn * fm->delta.y);
    if (use_stratified(fm)) {
        const ExpEntry *Ep, *Ed;
        NSLG_TRY(get_exp(fm, make_double2(-d.x, -d.y), &Ep));
        NSLG_TRY(get_exp(fm, d, &Ed));
        const int sg = fm->sgn;
        return logdet_strat(fm, 1, &Ep, &Ed, &sg, fm->phase, fm->phase_inv, out);
    }
    const ExpEntry *E;
    if (diag) NSLG_TRY(get_lin(fm, d, 1, &E));  // 1 - sgn delta K
    else NSLG_TRY(get_exp(fm, d, &E));
    double2 *B, *tmp, *phisum;
    NSLG_TRY(ws_get(fm, "ld_slices", (size_t)Nt * nn, &B));
    NSLG_TRY(ws_get(fm, "ld_tmp", (size_t)((Nt + 1) / 2) * nn, &tmp));
    NSLG_TRY(ws_get(fm, "ld_phisum", 1, &phisum));
    LuScratch s;
    NSLG_TRY(get_lu_scratch(fm, n, s));
    // Exp: B_t = exp(sgn delta K) diag(phiExp[t+1]), product B_{Nt-1} ... B_0 (hubbardExp.tpp:140-147).
    // Diag: fk_t = (1 - sgn delta K) diag(phiExpInv[t+1]), product fk_0 ... fk_{Nt-1} (hubbardDiag.tpp:176-187).
    k_slices<<<(unsigned)ceil_div(nn * Nt, 256), 256, 0, st>>>(E->full, diag ? fm->phase_inv : fm->phase, B, Nt, n,
                                                                1, false, diag);
    note_launch(st);
    NSLG_CUDA(cudaGetLastError());
    NSLG_TRY(product_tree(fm, B, tmp, Nt, n));
    k_add_identity<<<(unsigned)ceil_div(n, 256), 256, 0, st>>>(B, n);
    note_launch(st);
    NSLG_TRY(lu_factor(fm, B, n, s));
    double2 ls;
    int sw = 0, sing = 0;
    NSLG_CUDA(cudaMemcpyAsync(&ls, s.logsum, sizeof(double2), cudaMemcpyDeviceToHost, st));
    NSLG_CUDA(cudaMemcpyAsync(&sw, s.swaps, sizeof(int), cudaMemcpyDeviceToHost, st));
    NSLG_CUDA(cudaMemcpyAsync(&sing, s.singular, sizeof(int), cudaMemcpyDeviceToHost, st));
    NSLG_CUDA(cudaStreamSynchronize(st));
    if (sing) {
        *out = make_double2(-INFINITY, 0.0);
        return NSLG_OK;
    }
    double im = ls.y + (sw & 1 ? M_PI : 0.0);
    im = std::remainder(im, 2.0 * M_PI);  // principal branch, like log(det(.))
    if (im <= -M_PI) im += 2.0 * M_PI;
    *out = make_double2(ls.x, im);
    if (diag) {  // + i sgn sum(phi), not folded (hubbardDiag.tpp:189-191)
        k_sum_c128<<<1, 256, 0, st>>>(fm->phi, (int64_t)Nt * n, phisum);
        note_launch(st);
        double2 ps;
        NSLG_CUDA(cudaMemcpyAsync(&ps, phisum, sizeof(double2), cudaMemcpyDeviceToHost, st));
        NSLG_CUDA(cudaStreamSynchronize(st));
        out->x += -fm->sgn * ps.y;
        out->y += fm->sgn * ps.x;
    }
    return NSLG_OK;
}

namespace {

// Batched k_slices: B[g, t, i, j] = E_g[i, j] * ph[g, (t + shift) mod Nt, rowscale ? i : j] with
// E_g = (g & emask) ? E1 : E0.
__global__ void k_slices_many(const double2 *__restrict__ E0, const double2 *__restrict__ E1, int emask,
                              const double2 *__restrict__ ph, double2 *__restrict__ B, int nmat, int Nt, int n,
                              int shift, bool rowscale) {
    const int64_t nn = (int64_t)n * n;
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= nn * Nt * nmat) return;
    const int64_t gt = idx / nn;
    const int g = (int)(gt / Nt), t = (int)(gt % Nt);
    const int64_t ij = idx - gt * nn;
    const int i = (int)(ij / n), j = (int)(ij - (int64_t)i * n);
    const double2 *E = (g & emask) ? E1 : E0;
    const int ts = ((t + shift) % Nt + Nt) % Nt;
    B[idx] = cmul(E[ij], ph[((int64_t)g * Nt + ts) * n + (rowscale ? i : j)]);
}

// A[g] += 1 for nmat matrices at stride mstride
__global__ void k_add_identity_many(double2 *A, int n, int nmat, int64_t mstride) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (int64_t)n * nmat) return;
    const int g = (int)(idx / n), i = (int)(idx % n);
    A[g * mstride + (int64_t)i * n + i].x += 1.0;
}

// out[g, t, x] = i * sum_k S[g, (t + 1) mod Nt][x, k] B[k, x] with B = P[g, t] (t < Nt - 1) or G[g] (t = Nt - 1): a CTA
// owns 32 sites x of one slice and turns 32 x 32 blocks of S through shared memory, so that both matrices are read
// along their rows; its eight warps split k.
__global__ void __launch_bounds__(256) k_diagprod_many(const double2 *__restrict__ S, const double2 *__restrict__ P,
                                                       const double2 *__restrict__ G, double2 *__restrict__ out, int n,
                                                       int Nt) {
    __shared__ double2 tile[32][33];
    __shared__ double2 red[8][32];
    const int64_t gt = blockIdx.x;
    const int g = (int)(gt / Nt), t = (int)(gt % Nt);
    const int lane = threadIdx.x % 32, w = threadIdx.x / 32;
    const int x0 = blockIdx.y * 32, x = x0 + lane;
    const int64_t nn = (int64_t)n * n;
    const double2 *Sm = S + ((int64_t)g * Nt + (t + 1) % Nt) * nn;
    const double2 *B = t == Nt - 1 ? G + (int64_t)g * nn : P + gt * nn;
    double2 acc = make_double2(0, 0);
    for (int k0 = 0; k0 < n; k0 += 32) {
        if (k0) __syncthreads();
        for (int r = w; r < 32; r += 8)
            if (x0 + r < n && k0 + lane < n) tile[r][lane] = Sm[(int64_t)(x0 + r) * n + k0 + lane];
        __syncthreads();
        if (x < n)
            for (int kk = w; kk < min(32, n - k0); kk += 8) {
                const double2 a = tile[lane][kk], bv = B[(int64_t)(k0 + kk) * n + x];
                acc.x += a.x * bv.x - a.y * bv.y;
                acc.y += a.x * bv.y + a.y * bv.x;
            }
    }
    red[w][lane] = acc;
    __syncthreads();
    if (w == 0 && x < n) {
#pragma unroll
        for (int q = 1; q < 8; ++q) {
            acc.x += red[q][lane].x;
            acc.y += red[q][lane].y;
        }
        out[gt * n + x] = make_double2(-acc.y, acc.x);  // i * acc
    }
}

int diagprod_many(cudaStream_t st, const double2 *S, const double2 *P, const double2 *G, double2 *out, int n, int Nt,
                  int nmat) {
    // (slices on grid.x: Nt alone may exceed grid.y's 65535)
    k_diagprod_many<<<dim3((unsigned)((int64_t)nmat * Nt), (unsigned)ceil_div(n, 32)), 256, 0, st>>>(S, P, G, out, n, Nt);
    note_launch(st);
    NSLG_CUDA(cudaGetLastError());
    return NSLG_OK;
}

// dst[g] = diag(ph[g, row]) E_g for nmat matrices (E_g = (g & emask) ? E1 : E0), dst dstride elements apart.
__global__ void k_first_slice(const double2 *__restrict__ E0, const double2 *__restrict__ E1, int emask,
                              const double2 *__restrict__ ph, int row, double2 *__restrict__ dst, int64_t dstride,
                              int nmat, int Nt, int n) {
    const int64_t nn = (int64_t)n * n, idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= nn * nmat) return;
    const int g = (int)(idx / nn);
    const int64_t e = idx - g * nn;
    dst[g * dstride + e] = cmul(((g & emask) ? E1 : E0)[e], ph[((int64_t)g * Nt + row) * n + e / n]);
}

// X[g] = diag(ph[g, 2 mod Nt]) E_g diag(ph[g, 1 mod Nt]), without the row scale for one slice.
__global__ void k_logdet_first(const double2 *__restrict__ E0, const double2 *__restrict__ E1, int emask,
                               const double2 *__restrict__ ph, double2 *__restrict__ X, int nmat, int Nt, int n) {
    const int64_t nn = (int64_t)n * n, idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= nn * nmat) return;
    const int g = (int)(idx / nn);
    const int64_t e = idx - g * nn;
    const double2 *p = ph + (int64_t)g * Nt * n;
    double2 v = cmul(((g & emask) ? E1 : E0)[e], p[(int64_t)(1 % Nt) * n + e % n]);
    if (Nt > 1) v = cmul(p[(int64_t)(2 % Nt) * n + e / n], v);
    X[idx] = v;
}

// A product of every matrix of a batch with its real factor E_g: the factor as A (left) or B, as a two-level batch.
ZProd factor_product(int n, const double2 *E0, const double2 *E1, int emask, bool left, const double2 *X, int64_t sX,
                     double2 *Y, int64_t sY) {
    const int64_t dE = emask ? (int64_t)((reinterpret_cast<intptr_t>(E1) - reinterpret_cast<intptr_t>(E0)) /
                                         (intptr_t)sizeof(double2))
                             : 0;
    const int b2 = emask ? 2 : 1;
    ZProd p(n, n, n, left ? E0 : X, n, left ? 0 : b2 * sX, left ? X : E0, n, left ? b2 * sX : 0, Y, n, b2 * sY);
    (left ? p.sA2 : p.sB2) = dE;
    (left ? p.sB2 : p.sA2) = sX;
    p.sC2 = sY;
    p.batch2 = b2;
    p.real = left ? 1 : 2;
    return p;
}

// ---- whole chains in one launch --------------------------------------------------------------------------------------
// The rows of P(t) = (P(t-1) D_t) E' and the columns of S(t) = D_t (E' S(t+1)) (and of the log det's product) are
// independent through the whole chain, so a CTA takes V of them through all Nt steps: the vectors stay in shared memory
// beside the real factor, one barrier per step, no launch per time slice. A thread owns one output of one vector and sums it in
// ascending order whatever the split, so that a batch follows its single configurations bit by bit (and the products of
// one launch per step). With 2 FP64 FMAs per clock per SM a step is bound by its FMAs once every SM
// has some ten vectors, by the chain of one output's FMAs below.
// Measured, 31 steps on 32 matrices of 50 sites: 777 us as one launch per step -> 515 us.
//
// FORM 0: rows of P, out[t] stored for t = 0 .. steps - 1, the scale of step t applied to the vector before the product.
// FORM 1: columns of S, out[Nt - 2 - t] stored, the scale applied to the result. FORM 2: as 1 in increasing t, only the
// last result stored, unscaled (the log det's product).
constexpr int CH_T = 512;             // threads per CTA at most
constexpr size_t CH_SMEM = 200 * 1024;

struct ChainArgs {
    const double2 *E0, *E1;  // the real factor of matrix g is (g & emask) ? E1 : E0
    int emask;
    const double2 *first;    // the starting matrices, sfirst elements apart
    int64_t sfirst;
    const double2 *ph;       // scale rows (Nt, n) per matrix
    double2 *out;            // matrix g, step t at out + g * sout + t * n * n
    int64_t sout;
    int Nt, n, steps, V;
};

inline size_t chain_smem(int n, int V) { return (size_t)n * n * sizeof(double) + (size_t)2 * V * (n | 1) * sizeof(double2); }

template <int FORM> __global__ void __launch_bounds__(CH_T) k_chain(ChainArgs A) {
    extern __shared__ double2 sm[];
    const int n = A.n, V = A.V, Nt = A.Nt;
    const int L = n | 1;  // distance of the vectors: neighbouring ones in different banks
    const int64_t nn = (int64_t)n * n;
    double2 *Y = sm;                                              // two buffers of V vectors
    double *E = reinterpret_cast<double *>(sm + 2 * V * L);       // E[k n + o]: factor from input k to output o
    const int g = blockIdx.y, v0 = blockIdx.x * V, nv = min(V, n - v0);
    const double2 *Eg = (g & A.emask) ? A.E1 : A.E0;
    const double2 *first = A.first + g * A.sfirst, *ph = A.ph + (int64_t)g * Nt * n;
    double2 *out = A.out + g * A.sout;
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int i = e / n, j = e - i * n;
        E[FORM == 0 ? e : j * n + i] = Eg[e].x;  // rows: sum_k y_k E'[k, o]; columns: sum_k E'[o, k] y_k
    }
    // phase row of step t
    auto row = [&](int t) -> const double2 * {
        const int r = FORM == 0 ? t - 1 : FORM == 1 ? Nt - 3 - t : t + 3;
        return ph + (int64_t)((r + Nt) % Nt) * n;
    };
    // element (vector v, index k) of a matrix: row v0 + v, column k, or column v0 + v, row k
    auto at = [&](int v, int k) -> int64_t { return FORM == 0 ? (int64_t)(v0 + v) * n + k : (int64_t)k * n + v0 + v; };
    for (int e = threadIdx.x; e < nv * n; e += blockDim.x) {
        const int v = e / n, k = e - v * n;
        double2 y = first[at(v, k)];
        if (FORM == 0) y = cmul(y, row(0)[k]);
        Y[v * L + k] = y;
    }
    __syncthreads();
    for (int t = 0; t < A.steps; ++t) {
        const double2 *cur = Y + (t & 1) * V * L;
        double2 *nxt = Y + ((t + 1) & 1) * V * L;
        const bool last = t + 1 == A.steps, scaled = !(FORM == 2 && last);
        const double2 *sc = FORM == 0 ? row(last ? t : t + 1) : row(t);
        double2 *dst = FORM == 0 ? out + t * nn : FORM == 1 ? out + (int64_t)(Nt - 2 - t) * nn : out;
        for (int e = threadIdx.x; e < nv * n; e += blockDim.x) {
            // rows: consecutive threads, consecutive columns; columns: consecutive threads, neighbouring vectors
            const int v = FORM == 0 ? e / n : e % nv, o = FORM == 0 ? e - v * n : e / nv;
            const double2 scale = scaled ? sc[o] : make_double2(1, 0);
            const double2 *y = cur + v * L;
            const double *w = E + o;
            double2 acc = make_double2(0, 0);
#pragma unroll 8
            for (int k = 0; k < n; ++k) {
                acc.x = fma(y[k].x, w[k * n], acc.x);
                acc.y = fma(y[k].y, w[k * n], acc.y);
            }
            if (FORM != 0 && scaled) acc = cmul(scale, acc);
            if (FORM != 2 || last) dst[at(v, o)] = acc;
            nxt[v * L + o] = FORM == 0 ? cmul(acc, scale) : acc;
        }
        __syncthreads();
    }
}

// Vectors per CTA: the least estimated time, from the FP64 issue of the busiest SM and the chain of one output. Taken while
// eight vectors fit beside the factor (n <= 144): a trajectory (2 to 128 matrices, Nt = 16 and 32) against one launch per
// step was 0.42 to 0.95 of its time at n = 40 to 98, 0.73 to 0.99 at n = 112 and 128, 0.75 to 0.97 at n = 144, but up to
// 1.04 at n = 150 and 1.08 at n = 156, where one CTA per SM and few vectors leave the pipe waiting at each step.
bool plan_chain(int n, int nmat, ChainArgs &A, int *threads) {
    if (n < 2 || chain_smem(n, std::min(n, 8)) > CH_SMEM || nmat > 65535) return false;
    const int sms = std::max(1, num_sms());
    double best = 1e300;
    for (int V = 1; V <= std::min(n, 16) && chain_smem(n, V) <= CH_SMEM; ++V) {
        const int thr = std::min(CH_T, 32 * (int)ceil_div((int64_t)V * n, 32));
        const int64_t ctas = ceil_div(n, V) * nmat;
        const int64_t fit = std::max<int64_t>(1, std::min<int64_t>(1536 / thr, (int64_t)(220 * 1024 / chain_smem(n, V))));
        const double warps = (double)ceil_div((int64_t)V * n, 32);  // warp-sized pieces of a CTA's step, 2 n FMAs each
        const double res = (double)std::min<int64_t>(fit, ceil_div(ctas, sms));
        const double waves = (double)ceil_div(ctas, (int64_t)(sms * res));
        const double step = std::max(res * warps * 2.0 * n * 16.0, (double)ceil_div((int64_t)V * n, thr) * 2.0 * n * 64.0);
        if (waves * (step + 1500.0) < best) {  // (barrier, scale and store of a step: some 1500 clocks)
            best = waves * (step + 1500.0);
            A.V = V;
            *threads = thr;
        }
    }
    return true;
}

template <int FORM> int launch_chain(nslg_fm *fm, const ChainArgs &A, int threads, int nmat) {
    {
        static std::mutex mu;
        static std::set<int> done;
        std::lock_guard<std::mutex> lock(mu);
        if (!done.count(fm->ctx->device)) {
            NSLG_CUDA(cudaFuncSetAttribute(k_chain<FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CH_SMEM));
            done.insert(fm->ctx->device);
        }
    }
    k_chain<FORM><<<dim3((unsigned)ceil_div(A.n, A.V), (unsigned)nmat), threads, chain_smem(A.n, A.V), fm->ctx->stream>>>(A);
    note_launch(fm->ctx->stream);
    NSLG_CUDA(cudaGetLastError());
    return NSLG_OK;
}

}  // namespace

namespace {

// Tensor-core form of the gradient (force precision NSLG_PREC_BF16_SPLIT; exponential discretisation with a real
// exp(-sgn delta K), symmetric because K is real and Hermitian). Both chains become split-BF16 products Y E'^T with
// a diagonal scale, E' = exp(-sgn delta K), D_t = phiExpInv[(t - 1) mod Nt]:
//   T(t) = S(t)^T = T(t+1) E'^T D_t         (column scale of the product),  T(Nt-1) = E' D_{Nt-1}
//   P(t) = P(t-1) Fk(t) = (P(t-1) D_t) E'    (column scale of the operand),  P(-1) = G = (1 + S(0))^{-1} (FP64 LU)
//   pi_dot(t) = i diag(S(t+1) P(t)) = i sum_k T(t+1)[k, x] P(t)[k, x]
int grad_logdet_tc(nslg_fm *fm, const ExpEntry *E, double2 *out) {
    const ExpEntry *Es[1] = {E};
    return grad_logdet_tc_many(fm, 1, Es, fm->phase_inv, out);
}

}  // namespace

// The split-BF16 gradient for nmat matrices (matrix g: factor E[g], phase rows ph_inv + g * Nt * Nx, output
// out + g * Nt * Nx): the FP64 LU of the nmat matrices 1 + S(0) and the solves against the identity run as one
// batch, so the two species of a force share the single-SM LU launches; with two matrices the second one's
// tensor-core chains run on the handle's side stream, beside the first one's (each chain product fills only a
// few dozen SMs).
int grad_logdet_tc_many(nslg_fm *fm, int nmat, const ExpEntry *const *E, const double2 *ph_inv, double2 *out) {
    cudaStream_t st = fm->ctx->stream;
    const int Nt = (int)fm->Nt, n = (int)fm->Nx;
    const int64_t nn = (int64_t)n * n, ms = (int64_t)Nt * nn;
    NSLG_REQUIRE(nmat == 1 || nmat == 2, NSLG_ERR_ARG, "split-BF16 gradient: one or two matrices");
    std::vector<OzPlanes *> Pz(nmat);
    for (int g = 0; g < nmat; ++g) NSLG_TRY(oz_planes(fm, E[g], &Pz[g]));
    double2 *T, *P, *G;
    NSLG_TRY(ws_get(fm, "gr_S", (size_t)nmat * ms, &T));
    NSLG_TRY(ws_get(fm, "gr_P", (size_t)nmat * ms, &P));
    NSLG_TRY(ws_get(fm, "gr_G", (size_t)nmat * nn, &G));
    const size_t dg_elems = oz_digit_bytes(n, n);  // digits of one product's operand
    char *dg;
    int *rexp;
    NSLG_TRY(ws_get(fm, "fz_digits", dg_elems * nmat, &dg));
    NSLG_TRY(ws_get(fm, "fz_rexp", (size_t)2 * n * nmat, &rexp));
    cudaStream_t sg[2] = {st, st};
    if (nmat == 2) {
        if (!fm->side) NSLG_CUDA(cudaStreamCreateWithFlags(&fm->side, cudaStreamNonBlocking));
        if (!fm->ev_fork) NSLG_CUDA(cudaEventCreateWithFlags(&fm->ev_fork, cudaEventDisableTiming));
        if (!fm->ev_join) NSLG_CUDA(cudaEventCreateWithFlags(&fm->ev_join, cudaEventDisableTiming));
        sg[1] = fm->side;
    }
    auto fork = [&]() -> int {
        if (nmat == 2) {
            NSLG_CUDA(cudaEventRecord(fm->ev_fork, st));
            NSLG_CUDA(cudaStreamWaitEvent(fm->side, fm->ev_fork, 0));
        }
        return NSLG_OK;
    };
    auto join = [&]() -> int {
        if (nmat == 2) {
            NSLG_CUDA(cudaEventRecord(fm->ev_join, fm->side));
            NSLG_CUDA(cudaStreamWaitEvent(st, fm->ev_join, 0));
        }
        return NSLG_OK;
    };
    LuScratch s;
    NSLG_TRY(get_lu_scratch(fm, n, s, nmat));
    auto D = [&](int g, int t) { return ph_inv + ((int64_t)g * Nt + ((t - 1) % Nt + Nt) % Nt) * n; };
    auto Tg = [&](int g, int t) { return T + g * ms + (int64_t)t * nn; };
    auto Pg = [&](int g, int t) { return P + g * ms + (int64_t)t * nn; };
    auto dgg = [&](int g) { return (void *)(dg + g * dg_elems); };
    const unsigned g2 = (unsigned)ceil_div(nn, 256);
    NSLG_TRY(fork());
    for (int g = 0; g < nmat; ++g) {
        k_colscale<<<g2, 256, 0, sg[g]>>>(E[g]->full, D(g, Nt - 1), Tg(g, Nt - 1), n);
        note_launch(sg[g]);
        for (int t = Nt - 2; t >= 0; --t)
            NSLG_TRY(oz_gemm(Tg(g, t + 1), Tg(g, t), nullptr, D(g, t), *Pz[g], dgg(g), rexp + 2 * n * g, n, n,
                             fm->tc_err, sg[g]));
        k_transpose_plus_identity<<<g2, 256, 0, sg[g]>>>(Tg(g, 0), Pg(g, 0), n);  // 1 + S(0) in P[g, 0] as scratch
        note_launch(sg[g]);
    }
    NSLG_TRY(join());
    NSLG_TRY(lu_factor(fm, P, n, s, nmat, ms, false));
    NSLG_TRY(lu_inverse(fm, P, G, n, s, nmat, ms));
    NSLG_TRY(fork());
    for (int g = 0; g < nmat; ++g)
        for (int t = 0; t < Nt - 1; ++t) {
            const double2 *prev = t == 0 ? G + g * nn : Pg(g, t - 1);
            NSLG_TRY(oz_gemm(prev, Pg(g, t), D(g, t), nullptr, *Pz[g], dgg(g), rexp + 2 * n * g, n, n, fm->tc_err,
                             sg[g]));
        }
    NSLG_TRY(join());
    for (int g = 0; g < nmat; ++g) {
        k_coldot_slices<<<dim3((unsigned)ceil_div(n, 32), (unsigned)Nt), dim3(32, CD_W), 0, st>>>(
            T + g * ms, P + g * ms, G + g * nn, out + (int64_t)g * Nt * n, n, Nt);
        note_launch(st);
    }
    NSLG_CUDA(cudaGetLastError());
    return NSLG_OK;
}

// d log det M / d phi (Nt, Nx) into a device buffer.
int fm_grad_logdet(nslg_fm *fm, double2 *out) {
    cudaStream_t st = fm->ctx->stream;
    const int n = (int)fm->Nx;
    // Fk(t) = diag(phiExpInv[t-1]) exp(-sgn delta K) (Exp) or diag(phiExpInv[t-1]) (1 - sgn delta K) (Diag,
    // hubbardDiag.tpp:203-205)
    const ExpEntry *E;
    if (fm->kind == NSLG_FM_DIAG) NSLG_TRY(get_lin(fm, make_double2(fm->sgn * fm->delta.x, fm->sgn * fm->delta.y), 1, &E));
    else NSLG_TRY(get_exp(fm, make_double2(-fm->sgn * fm->delta.x, -fm->sgn * fm->delta.y), &E));
    if (use_stratified_grad(fm)) {
        const ExpEntry *Ed;
        NSLG_TRY(get_exp(fm, make_double2(fm->sgn * fm->delta.x, fm->sgn * fm->delta.y), &Ed));
        return grad_logdet_strat(fm, 1, &E, &Ed, fm->phase, fm->phase_inv, out);
    } else if (fm->force_precision == NSLG_PREC_BF16_SPLIT && fm->kind == NSLG_FM_EXP && E->is_real && n <= 2048) {
        NSLG_TRY(grad_logdet_tc(fm, E, out));
    } else {
        NSLG_TRY(grad_logdet_many(fm, 1, E, E, 0, fm->phase_inv, out));
    }
    if (fm->defer_checks) return NSLG_OK;  // the captured trajectory checks the sticky flag after its replay
    LuScratch s;
    NSLG_TRY(get_lu_scratch(fm, n, s));
    int sing = 0;
    NSLG_CUDA(cudaMemcpyAsync(&sing, s.singular, sizeof(int), cudaMemcpyDeviceToHost, st));
    NSLG_CUDA(cudaStreamSynchronize(st));
    NSLG_REQUIRE(!sing, NSLG_ERR_ARG, "gradLogDetM: 1 + A^{-1} is singular");
    return NSLG_OK;
}


// d log det M / d phi for nmat matrices at once (hubbardExp.tpp:153-211), FP64: matrix g has the time-slice factor
// E_g = (g & emask) ? E1 : E0 and the phase rows ph_inv[g] = phiExpInv (Nt, Nx); out is (nmat, Nt, Nx).
//   Fk(t) = diag(phiExpInv[(t - 1) mod Nt]) E,  S(t) = Fk(t) S(t+1), S(Nt-1) = Fk(Nt-1),
//   G = (1 + S(0))^{-1},  P(t) = P(t-1) Fk(t), P(-1) = G,  pi_dot(t) = i diag(S(t+1) P(t)), pi_dot(Nt-1) = i diag(S(0) G).
// Every chain step is one batched GEMM over the nmat matrices and the LU/solve factor them side by side, so the
// species of one configuration, or many configurations, share each launch.
int grad_logdet_many(nslg_fm *fm, int nmat, const ExpEntry *e0, const ExpEntry *e1, int emask, const double2 *ph_inv,
                     double2 *out) {
    cudaStream_t st = fm->ctx->stream;
    const int Nt = (int)fm->Nt, n = (int)fm->Nx;
    const int64_t nn = (int64_t)n * n, ms = (int64_t)Nt * nn;
    const double2 *E0 = e0->full, *E1 = e1->full;
    const bool real = e0->is_real && e1->is_real && (emask == 0 || (emask == 1 && nmat % 2 == 0));
    const bool scan = n <= SCAN_MAX && Nt > 1 && Nt <= 65535 && nmat <= SCAN_MAX_MATRICES;
    double2 *Fk = nullptr, *S, *P, *G;
    NSLG_TRY(ws_get(fm, "gr_S", (size_t)nmat * ms, &S));
    NSLG_TRY(ws_get(fm, "gr_P", (size_t)nmat * ms, &P));
    NSLG_TRY(ws_get(fm, "gr_G", (size_t)nmat * nn, &G));
    LuScratch s;
    NSLG_TRY(get_lu_scratch(fm, n, s, nmat));
    const double2 one = make_double2(1, 0);
    if (scan || !real) {
        NSLG_TRY(ws_get(fm, "gr_Fk", (size_t)nmat * ms, &Fk));
        k_slices_many<<<(unsigned)ceil_div(ms * nmat, 256), 256, 0, st>>>(E0, E1, emask, ph_inv, Fk, nmat, Nt, n, -1,
                                                                           true);
        note_launch(st);
    }
    if (scan) {
        // Small matrices, few of them: the chains are latency-bound (each product is a few microseconds of dependent
        // FP64 steps on a handful of SMs), so they become scans with log2(Nt) levels of batched products
        // (Hillis-Steele: ~Nt log2 Nt products instead of 2 (Nt - 1), all of a level in one launch; with many
        // matrices the chains already fill the GPU and the scans' extra products would cost more than they save):
        //   Q(t) = Fk(0) ... Fk(t) (prefix), S(t) = Fk(t) ... Fk(Nt-1) (suffix),
        // G = (1 + S(0))^{-1} from one Gauss-Jordan launch, and P(t) = G Q(t) only as the terms of the diagonal.
        double2 *Q0, *Q1, *S1;
        NSLG_TRY(ws_get(fm, "gr_Q0", (size_t)nmat * ms, &Q0));
        NSLG_TRY(ws_get(fm, "gr_Q1", (size_t)nmat * ms, &Q1));
        NSLG_TRY(ws_get(fm, "gr_S1", (size_t)nmat * ms, &S1));
        const double2 *Qc = Fk, *Sc = Fk;
        double2 *Qbuf[2] = {Q0, Q1}, *Sbuf[2] = {S, S1};
        int lvl = 0;
        for (int o = 1; o < Nt; o <<= 1, ++lvl) {
            double2 *Qn = Qbuf[lvl & 1], *Sn = Sbuf[lvl & 1];
            k_scan_level<<<dim3((unsigned)ceil_div(nn, 32), (unsigned)Nt, 2u * nmat), 128, 0, st>>>(Qc, Sc, Qn, Sn, n,
                                                                                                  Nt, o);
            note_launch(st);
            Qc = Qn;
            Sc = Sn;
        }
        if (!fm->defer_checks) NSLG_CUDA(cudaMemsetAsync(s.singular, 0, sizeof(int), st));
        NSLG_TRY(gj_inverse_plus_one(fm, Sc, ms, G, n, nmat, s.singular));
        const int XB = std::min(n, 128 / n);
        k_scan_grad<<<dim3((unsigned)ceil_div(n, XB), (unsigned)Nt, (unsigned)nmat), 128, 0, st>>>(Sc, Qc, G, out, n, Nt,
                                                                                                 XB);
        note_launch(st);
        NSLG_CUDA(cudaGetLastError());
        return NSLG_OK;
    }
    // S(Nt-1) = Fk(Nt-1), then the suffix chain; a real E' keeps its products real-by-complex, with the phases as a
    // scale of the result's rows: S(t) = D_t (E' S(t+1)), D_t = diag(phiExpInv[t-1])
    auto row = [&](int t) { return ((t - 1) % Nt + Nt) % Nt; };
    k_first_slice<<<(unsigned)ceil_div(nn * nmat, 256), 256, 0, st>>>(E0, E1, emask, ph_inv, row(Nt - 1),
                                                                       S + (int64_t)(Nt - 1) * nn, ms, nmat, Nt, n);
    note_launch(st);
    const int64_t sph = (int64_t)Nt * n;
    ChainArgs ca{E0, E1, emask, S + (int64_t)(Nt - 1) * nn, ms, ph_inv, S, ms, Nt, n, Nt - 1, 1};
    int cthreads = 0;
    const bool chain = real && Nt > 1 && plan_chain(n, nmat, ca, &cthreads);
    if (chain) NSLG_TRY(launch_chain<1>(fm, ca, cthreads, nmat));
    for (int t = Nt - 2; t >= 0 && !chain; --t) {
        if (!real) {
            NSLG_TRY(zgemm(st, n, n, n, one, Fk + t * nn, n, ms, S + (t + 1) * nn, n, ms, S + t * nn, n, ms, nmat, false));
            continue;
        }
        ZProd p = factor_product(n, E0, E1, emask, true, S + (t + 1) * nn, ms, S + t * nn, ms);
        p.rscale = ph_inv + (int64_t)row(t) * n;
        p.srs = p.batch2 * sph;
        p.srs2 = sph;
        NSLG_TRY(zprod(st, p, nmat / p.batch2));
    }
    // G = (1 + S(0))^{-1}
    if (n <= GJ_MAX) {
        if (!fm->defer_checks) NSLG_CUDA(cudaMemsetAsync(s.singular, 0, sizeof(int), st));
        NSLG_TRY(gj_inverse_plus_one(fm, S, ms, G, n, nmat, s.singular));
    } else {  // 1 + S(0) in P[g, 0] as scratch
        NSLG_CUDA(cudaMemcpy2DAsync(P, ms * sizeof(double2), S, ms * sizeof(double2), nn * sizeof(double2), nmat,
                                    cudaMemcpyDeviceToDevice, st));
        k_add_identity_many<<<(unsigned)ceil_div((int64_t)n * nmat, 256), 256, 0, st>>>(P, n, nmat, ms);
        note_launch(st);
        NSLG_TRY(lu_factor(fm, P, n, s, nmat, ms, false));
        NSLG_TRY(lu_inverse(fm, P, G, n, s, nmat, ms));
    }
    // prefix chain P(t) = P(t-1) Fk(t) = (P(t-1) D_t) E', P(-1) = G
    if (chain) {
        ca.first = G;
        ca.sfirst = nn;
        ca.out = P;
        NSLG_TRY(launch_chain<0>(fm, ca, cthreads, nmat));
    }
    for (int t = 0; t < Nt - 1 && !chain; ++t) {
        const double2 *prev = t == 0 ? G : P + (t - 1) * nn;
        const int64_t sp = t == 0 ? nn : ms;
        if (!real) {
            NSLG_TRY(zgemm(st, n, n, n, one, prev, n, sp, Fk + t * nn, n, ms, P + t * nn, n, ms, nmat, false));
            continue;
        }
        ZProd p = factor_product(n, E0, E1, emask, false, prev, sp, P + t * nn, ms);
        p.kscale = ph_inv + (int64_t)row(t) * n;
        p.sks = p.batch2 * sph;
        p.sks2 = sph;
        NSLG_TRY(zprod(st, p, nmat / p.batch2));
    }
    return diagprod_many(st, S, P, G, out, n, Nt, nmat);
}

// log det M for nmat matrices of the exponential discretisation at once (hubbardExp.tpp:129-150): matrix g has
// B_t = E_g diag(phiExp_g[(t + 1) mod Nt]) with E_g = (g & emask) ? E1 : E0 and phase rows ph[g] (Nt, Nx). The
// product B_{Nt-1} ... B_0 is a chain of batched GEMMs (one launch per t for all g), 1 + product is factored by the
// batched LU and log det = sum log u_kk + i pi (#swaps) on the principal branch; out[g] on the host (-inf for a
// singular matrix).
int logdet_many(nslg_fm *fm, int nmat, const ExpEntry *e0, const ExpEntry *e1, int emask, const double2 *ph,
                double2 *out) {
    cudaStream_t st = fm->ctx->stream;
    const int Nt = (int)fm->Nt, n = (int)fm->Nx;
    const int64_t nn = (int64_t)n * n, ms = (int64_t)Nt * nn, sph = (int64_t)Nt * n;
    const double2 *E0 = e0->full, *E1 = e1->full;
    const bool real = e0->is_real && e1->is_real && (emask == 0 || (emask == 1 && nmat % 2 == 0));
    double2 *R;
    NSLG_TRY(ws_get(fm, "ldm_prod", (size_t)2 * nmat * nn, &R));
    LuScratch s;
    NSLG_TRY(get_lu_scratch(fm, n, s, nmat));
    const double2 one = make_double2(1, 0);
    double2 *cur = R, *nxt = R + (int64_t)nmat * nn;
    if (real) {
        // X_t = D_{t+2} B_t ... B_0 with D_t = diag(phiExp[t]): X_t = D_{t+2} (E X_{t-1}), a real-by-complex product with
        // a row scale (none on the last)
        k_logdet_first<<<(unsigned)ceil_div(nn * nmat, 256), 256, 0, st>>>(E0, E1, emask, ph, cur, nmat, Nt, n);
        note_launch(st);
        ChainArgs ca{E0, E1, emask, cur, nn, ph, nxt, nn, Nt, n, Nt - 1, 1};
        int cthreads = 0;
        const bool chain = Nt > 1 && plan_chain(n, nmat, ca, &cthreads);
        if (chain) {
            NSLG_TRY(launch_chain<2>(fm, ca, cthreads, nmat));
            std::swap(cur, nxt);
        }
        for (int t = 1; t < Nt && !chain; ++t) {
            ZProd p = factor_product(n, E0, E1, emask, true, cur, nn, nxt, nn);
            if (t + 1 < Nt) {
                p.rscale = ph + (int64_t)((t + 2) % Nt) * n;
                p.srs = p.batch2 * sph;
                p.srs2 = sph;
            }
            NSLG_TRY(zprod(st, p, nmat / p.batch2));
            std::swap(cur, nxt);
        }
    } else {
        double2 *B;
        NSLG_TRY(ws_get(fm, "ldm_slices", (size_t)nmat * ms, &B));
        k_slices_many<<<(unsigned)ceil_div(ms * nmat, 256), 256, 0, st>>>(E0, E1, emask, ph, B, nmat, Nt, n, 1, false);
        note_launch(st);
        NSLG_CUDA(cudaMemcpy2DAsync(cur, nn * sizeof(double2), B, ms * sizeof(double2), nn * sizeof(double2), nmat,
                                    cudaMemcpyDeviceToDevice, st));
        for (int t = 1; t < Nt; ++t) {
            NSLG_TRY(zgemm(st, n, n, n, one, B + t * nn, n, ms, cur, n, nn, nxt, n, nn, nmat, false));
            std::swap(cur, nxt);
        }
    }
    k_add_identity_many<<<(unsigned)ceil_div((int64_t)n * nmat, 256), 256, 0, st>>>(cur, n, nmat, nn);
    note_launch(st);
    NSLG_TRY(lu_factor(fm, cur, n, s, nmat, nn));
    std::vector<double2> ls(nmat);
    std::vector<int> sw(nmat);
    int sing = 0;
    NSLG_CUDA(cudaMemcpyAsync(ls.data(), s.logsum, nmat * sizeof(double2), cudaMemcpyDeviceToHost, st));
    NSLG_CUDA(cudaMemcpyAsync(sw.data(), s.swaps, nmat * sizeof(int), cudaMemcpyDeviceToHost, st));
    NSLG_CUDA(cudaMemcpyAsync(&sing, s.singular, sizeof(int), cudaMemcpyDeviceToHost, st));
    NSLG_CUDA(cudaStreamSynchronize(st));
    NSLG_REQUIRE(!sing, NSLG_ERR_ARG, "logDetM: 1 + prod B_t is singular for a configuration of the batch");
    for (int g = 0; g < nmat; ++g) {
        double im = ls[g].y + (sw[g] & 1 ? M_PI : 0.0);
        im = std::remainder(im, 2.0 * M_PI);
        if (im <= -M_PI) im += 2.0 * M_PI;
        out[g] = make_double2(ls[g].x, im);
    }
    return NSLG_OK;
}

}  // namespace nslg
