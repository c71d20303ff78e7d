// Dense FP64 complex linear algebra used off the per-iteration path: a batched complex GEMM, the matrix exponential
// exp(d K) of the hopping matrix (SpatialLattice::exp_hopping_matrix, lattice.tpp:52-58) and the phase factors of
// HubbardExp::populate (hubbardExp.hpp:116-128).

#include <algorithm>
#include <tuple>

#include "fm_internal.cuh"

namespace nslg {

namespace {

// C = alpha * (A o kscale) @ B (o rscale) (+ I) (+ C with accumulate), batched over blockIdx.z.
//
// GB300 runs FP64 at ~2 FMAs per clock per SM: a warp's DFMA occupies its scheduler for 64 cycles, so operand reads from
// shared memory and L1 fit in its shadow and what matters is that no lane computes padding and that all 608 schedulers
// have equal work. A thread owns one column of TM consecutive rows; a CTA's threads are the flattened (row group,
// column) pairs of whole rows (N <= 256) or a run of columns of one row group; A is staged in shared memory, B is read
// in place (consecutive lanes, consecutive columns). zsplit() picks the split. Every output sums over k in ascending
// order whatever the split. Measured: 32 products of 50 x 50 matrices, one factor real, 58 -> 25 us (of it a factor of two
// from the real factor), 26 real-by-complex products at n = 288 2.82 -> 2.07 ms (the rate of the FP64 pipe).
// REAL: 1 = A holds real numbers (imaginary parts zero), 2 = B does, 3 = both; the product then skips the FMAs with the
// zero imaginary parts (2 or 1 instead of 4 per term). TA: A is given as its adjoint (A[i, k] = conj(At[k lda + i])).
constexpr int ZKC = 32;    // reduction depth per staged chunk
constexpr int ZMAXT = 256;  // threads per CTA at most

template <int REAL, bool TA, int TM>
__global__ void __launch_bounds__(ZMAXT) k_zgemm(ZProd p, int G, int CW) {
    extern __shared__ double2 As[];  // (G TM) x LS
    const int LS = min(ZKC, p.K) + 1;
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32, nwarps = blockDim.x / 32;
    const int R = G * TM;
    const int m0 = blockIdx.x * R;
    const int z1 = blockIdx.z / p.batch2, z2 = blockIdx.z % p.batch2;
    const double2 *A = p.A + p.sA * z1 + p.sA2 * z2;
    const double2 *B = p.B + p.sB * z1 + p.sB2 * z2;
    double2 *C = p.C + p.sC * z1 + p.sC2 * z2;
    const double2 *ks = p.kscale ? p.kscale + p.sks * z1 + p.sks2 * z2 : nullptr;
    const int g = tid / CW, c = tid - g * CW;
    const int col = blockIdx.y * CW + c;
    if (p.upper && min(p.N, (int)(blockIdx.y + 1) * CW) <= m0) return;  // every column of this CTA is left of its rows
    const bool act = g < G && col < p.N && m0 + g * TM < p.M;
    double2 acc[TM];
#pragma unroll
    for (int i = 0; i < TM; ++i) acc[i] = make_double2(0, 0);
    const int kbeg = p.a_upper ? m0 : 0;  // A upper triangular: nothing left of its diagonal
    for (int k0 = kbeg; k0 < p.K; k0 += ZKC) {
        const int kc = min(ZKC, p.K - k0);
        if (k0 != kbeg) __syncthreads();
        if constexpr (TA) {
            for (int e = tid; e < R * kc; e += blockDim.x) {
                const int kk = e / R, row = e - kk * R;
                double2 v = make_double2(0, 0);
                if (m0 + row < p.M) v = A[(int64_t)(k0 + kk) * p.lda + m0 + row];
                As[row * LS + kk] = make_double2(v.x, -v.y);
            }
        } else {
            for (int row = warp; row < R; row += nwarps)
                for (int kk = lane; kk < kc; kk += 32) {
                    double2 v = make_double2(0, 0);
                    if (m0 + row < p.M) {
                        v = A[(int64_t)(m0 + row) * p.lda + k0 + kk];
                        if (ks) v = cmul(v, ks[k0 + kk]);
                    }
                    As[row * LS + kk] = v;
                }
        }
        __syncthreads();
        if (act) {
            const double2 *as = As + g * TM * LS;
            const double2 *b = B + (int64_t)k0 * p.ldb + col;
#pragma unroll 8
            for (int kk = 0; kk < kc; ++kk) {
                const double2 bv = b[(int64_t)kk * p.ldb];
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const double2 a = as[i * LS + kk];
                    if constexpr (REAL == 3) {  // both real
                        acc[i].x = fma(a.x, bv.x, acc[i].x);
                    } else if constexpr (REAL == 2) {  // B real
                        acc[i].x = fma(a.x, bv.x, acc[i].x);
                        acc[i].y = fma(a.y, bv.x, acc[i].y);
                    } else if constexpr (REAL == 1) {  // A real
                        acc[i].x = fma(a.x, bv.x, acc[i].x);
                        acc[i].y = fma(a.x, bv.y, acc[i].y);
                    } else {
                        acc[i].x = fma(a.x, bv.x, acc[i].x);
                        acc[i].x = fma(-a.y, bv.y, acc[i].x);
                        acc[i].y = fma(a.x, bv.y, acc[i].y);
                        acc[i].y = fma(a.y, bv.x, acc[i].y);
                    }
                }
            }
        }
    }
    if (!act) return;
    const double2 *rs = p.rscale ? p.rscale + p.srs * z1 + p.srs2 * z2 : nullptr;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int r = m0 + g * TM + i;
        if (r >= p.M || (p.upper && col < r)) continue;
        double2 v = acc[i];
        if (p.alpha.y != 0.0) v = cmul(p.alpha, v);
        else if (p.alpha.x != 1.0) v = make_double2(p.alpha.x * v.x, p.alpha.x * v.y);
        if (rs) v = cmul(rs[r], v);
        if (p.add_identity && r == col) v.x += 1.0;
        if (p.accumulate) {
            const double2 o = C[(int64_t)r * p.ldc + col];
            v.x += o.x;
            v.y += o.y;
        }
        C[(int64_t)r * p.ldc + col] = v;
    }
}

// Small products (M, N, K <= ZSMALL): what bounds them is the dependent chain of FP64 steps of one output, so a CTA takes
// 32 outputs (flattened, no padded tile) and its four warps, one per scheduler, a quarter of the k sum each.
constexpr int ZSMALL = 32;

template <int REAL, bool TA> __global__ void __launch_bounds__(128) k_zgemm_small(ZProd p) {
    __shared__ double2 red[3][32];
    const int lane = threadIdx.x % 32, w = threadIdx.x / 32;
    const int z1 = blockIdx.z / p.batch2, z2 = blockIdx.z % p.batch2;
    const double2 *A = p.A + p.sA * z1 + p.sA2 * z2;
    const double2 *B = p.B + p.sB * z1 + p.sB2 * z2;
    double2 *C = p.C + p.sC * z1 + p.sC2 * z2;
    const double2 *ks = p.kscale ? p.kscale + p.sks * z1 + p.sks2 * z2 : nullptr;
    const int e = blockIdx.x * 32 + lane;
    const int r = e / p.N, c = e - r * p.N;
    const bool act = r < p.M && !(p.upper && c < r);
    double2 acc = make_double2(0, 0);
    if (act) {
#pragma unroll 8
        for (int k = w; k < p.K; k += 4) {
            double2 a = TA ? A[(int64_t)k * p.lda + r] : A[(int64_t)r * p.lda + k];
            if (TA) a.y = -a.y;
            if (ks) a = cmul(a, ks[k]);
            const double2 b = B[(int64_t)k * p.ldb + c];
            if constexpr (REAL == 3) {
                acc.x = fma(a.x, b.x, acc.x);
            } else if constexpr (REAL == 2) {
                acc.x = fma(a.x, b.x, acc.x);
                acc.y = fma(a.y, b.x, acc.y);
            } else if constexpr (REAL == 1) {
                acc.x = fma(a.x, b.x, acc.x);
                acc.y = fma(a.x, b.y, acc.y);
            } else {
                acc.x = fma(a.x, b.x, acc.x);
                acc.x = fma(-a.y, b.y, acc.x);
                acc.y = fma(a.x, b.y, acc.y);
                acc.y = fma(a.y, b.x, acc.y);
            }
        }
    }
    if (w > 0) red[w - 1][lane] = acc;
    __syncthreads();
    if (w > 0 || !act) return;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        acc.x += red[q][lane].x;
        acc.y += red[q][lane].y;
    }
    double2 v = cmul(p.alpha, acc);
    if (p.rscale) v = cmul(p.rscale[p.srs * z1 + p.srs2 * z2 + r], v);
    if (p.add_identity && r == c) v.x += 1.0;
    if (p.accumulate) {
        const double2 o = C[(int64_t)r * p.ldc + c];
        v.x += o.x;
        v.y += o.y;
    }
    C[(int64_t)r * p.ldc + c] = v;
}

__global__ void k_set_identity(double2 *A, int n) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)n * n) return;
    const int r = (int)(i / n), c = (int)(i % n);
    A[i] = make_double2(r == c ? 1.0 : 0.0, 0.0);
}

__global__ void k_scale(double2 *out, const double2 *in, double2 s, int64_t n) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = cmul(s, in[i]);
}

// Planes of exp(d K): re/im FP64 row-major, re transposed in FP64 and FP32, plus a flag set when any imaginary part is
// nonzero.
__global__ void k_split_planes(const double2 *E, double *re, double *im, double *reT, float *re32T, int n,
                               int *nonreal) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)n * n) return;
    const double2 v = E[i];
    const int64_t j = (i % n) * n + i / n;
    re[i] = v.x;
    im[i] = v.y;
    reT[j] = v.x;
    re32T[j] = (float)v.x;
    if (v.y != 0.0) atomicOr(nonreal, 1);
}
// the transposed imaginary planes of a complex entry
__global__ void k_split_imag(const double2 *E, double *imT, float *im32T, int n) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)n * n) return;
    const int64_t j = (i % n) * n + i / n;
    imT[j] = E[i].y;
    im32T[j] = (float)E[i].y;
}

// 1-norm (max column sum of |K|) of a complex (n, n) matrix, one block.
__global__ void k_norm1(const double2 *A, int n, double *out) {
    __shared__ double red[256];
    double best = 0;
    int other = 0;  // entries that are not finite real numbers
    for (int c = threadIdx.x; c < n; c += blockDim.x) {
        double s = 0;
        for (int r = 0; r < n; ++r) {
            const double2 v = A[(int64_t)r * n + c];
            other |= !(v.y == 0.0 && isfinite(v.x));
            s += hypot(v.x, v.y);
        }
        best = fmax(best, s);
    }
    red[threadIdx.x] = best;
    other = __syncthreads_or(other);
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + w]);
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        out[0] = red[0];
        double2 tr = make_double2(0, 0);
        for (int i = 0; i < n; ++i) {
            tr.x += A[(int64_t)i * n + i].x;
            tr.y += A[(int64_t)i * n + i].y;
        }
        out[1] = tr.x;
        out[2] = tr.y;
        out[3] = other ? 1.0 : 0.0;
    }
}

// phase = exp(i sgn phi + sgn mu), phase_inv = exp(-i sgn phi - sgn mu)  (hubbardExp.hpp:121-127)
__global__ void k_phases(const double2 *phi, double2 *phase, double2 *phase_inv, float2 *phase32, int sgn,
                         double2 mu, int64_t n) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double2 f = phi[i];
    // i*sgn*phi + sgn*mu = (-sgn*f.y + sgn*mu.x) + i (sgn*f.x + sgn*mu.y)
    const double a = sgn * (mu.x - f.y);
    const double b = sgn * (f.x + mu.y);
    double sb, cb;
    sincos(b, &sb, &cb);
    const double ea = exp(a), eia = exp(-a);
    phase[i] = make_double2(ea * cb, ea * sb);
    phase_inv[i] = make_double2(eia * cb, -eia * sb);
    phase32[i] = make_float2((float)(ea * cb), (float)(ea * sb));
}

}  // namespace

namespace {

// How an (M, N) product of nz matrices is cut into CTAs: columns per CTA, row groups, rows per thread (as the
// CUDA-core operator's split).
struct ZSplit {
    int CW, G, TM, threads, gx, gy;
};

size_t zsmem(int G, int TM, int K) { return (size_t)G * TM * (std::min(ZKC, K) + 1) * sizeof(double2); }

ZSplit zsplit(int M, int N, int K, int64_t nz) {
    ZSplit S;
    if (N > ZMAXT) {  // a run of columns of one row group, all runs alike and a whole number of warps
        const int runs = (int)ceil_div(N, 128);
        S.CW = (int)ceil_div(ceil_div(N, runs), 32) * 32;
        S.gy = (int)ceil_div(N, S.CW);
        S.G = 1;
    } else {  // whole rows: as many row groups as leave the fewest idle lanes in the last warp
        S.CW = N;
        S.gy = 1;
        S.G = 1;
        double best = 0;
        for (int G = 1; G * N <= ZMAXT && G <= M; ++G) {
            const double eff = (double)(G * N) / (32.0 * (double)ceil_div(G * N, 32));
            if (eff > best + 0.03) {
                best = eff;
                S.G = G;
            }
        }
    }
    S.threads = 32 * (int)ceil_div(S.G * S.CW, 32);
    // rows per thread: the most that still keep the schedulers (4 per SM) evenly busy to 90 %, else the best balance
    const int64_t sched = 4 * (int64_t)std::max(1, num_sms());
    double best = 0;
    S.TM = 1;
    for (int TM = 8; TM >= 1; TM /= 2) {
        if (TM > 1 && zsmem(S.G, TM, K) > 48 * 1024) continue;  // (one or two columns: many rows of A staged at once)
        const int64_t rb = ceil_div(M, (int64_t)S.G * TM);
        const int64_t warps = rb * S.gy * (S.threads / 32) * nz;
        const double eff = (double)warps / (double)(sched * ceil_div(warps, sched)) * (double)M / (double)(rb * S.G * TM);
        if (eff > 1.02 * best) {
            best = eff;
            S.TM = TM;
        }
        if (eff >= 0.9) break;
    }
    S.gx = (int)ceil_div(M, (int64_t)S.G * S.TM);
    return S;
}

template <int REAL, bool TA> void launch_zgemm(const ZSplit &S, unsigned nz, const ZProd &p, cudaStream_t st) {
    const dim3 grid((unsigned)S.gx, (unsigned)S.gy, nz);
    const size_t smem = zsmem(S.G, S.TM, p.K);  // <= 48 KB
    if (S.TM == 8) k_zgemm<REAL, TA, 8><<<grid, S.threads, smem, st>>>(p, S.G, S.CW);
    else if (S.TM == 4) k_zgemm<REAL, TA, 4><<<grid, S.threads, smem, st>>>(p, S.G, S.CW);
    else if (S.TM == 2) k_zgemm<REAL, TA, 2><<<grid, S.threads, smem, st>>>(p, S.G, S.CW);
    else k_zgemm<REAL, TA, 1><<<grid, S.threads, smem, st>>>(p, S.G, S.CW);
}

}  // namespace

int zprod(cudaStream_t st, const ZProd &p, int batch) {
    if (p.M <= 0 || p.N <= 0 || batch == 0 || p.batch2 == 0) return NSLG_OK;
    const int64_t nz = (int64_t)batch * p.batch2;
    NSLG_REQUIRE(nz <= 65535, NSLG_ERR_SHAPE, "zgemm: at most 65535 products per launch");
    if (p.M <= ZSMALL && p.N <= ZSMALL && p.K <= ZSMALL) {
        const dim3 grid((unsigned)ceil_div((int64_t)p.M * p.N, 32), 1, (unsigned)nz);
        if (p.a_adjoint) k_zgemm_small<0, true><<<grid, 128, 0, st>>>(p);
        else if (p.real == 1) k_zgemm_small<1, false><<<grid, 128, 0, st>>>(p);
        else if (p.real == 2) k_zgemm_small<2, false><<<grid, 128, 0, st>>>(p);
        else if (p.real == 3) k_zgemm_small<3, false><<<grid, 128, 0, st>>>(p);
        else k_zgemm_small<0, false><<<grid, 128, 0, st>>>(p);
        note_launch(st);
        NSLG_CUDA(cudaGetLastError());
        return NSLG_OK;
    }
    const ZSplit S = zsplit(p.M, p.N, p.K, nz);
    if (p.a_adjoint) launch_zgemm<0, true>(S, (unsigned)nz, p, st);
    else if (p.real == 1) launch_zgemm<1, false>(S, (unsigned)nz, p, st);
    else if (p.real == 2) launch_zgemm<2, false>(S, (unsigned)nz, p, st);
    else if (p.real == 3) launch_zgemm<3, false>(S, (unsigned)nz, p, st);
    else launch_zgemm<0, false>(S, (unsigned)nz, p, st);
    note_launch(st);
    NSLG_CUDA(cudaGetLastError());
    return NSLG_OK;
}

int zgemm(cudaStream_t st, int M, int N, int K, double2 alpha, const double2 *A, int64_t lda, int64_t sA,
          const double2 *B, int64_t ldb, int64_t sB, double2 *C, int64_t ldc, int64_t sC, int batch,
          bool add_identity, bool accumulate) {
    ZProd p(M, N, K, A, lda, sA, B, ldb, sB, C, ldc, sC);
    p.alpha = alpha;
    p.add_identity = add_identity;
    p.accumulate = accumulate;
    return zprod(st, p, batch);
}

// Two-level batched product: C[z1, z2] = alpha A[z1, z2] B[z1, z2] with element offsets z1 * s + z2 * s2, for
// batch x batch2 products in one launch.
int zgemm2(cudaStream_t st, int M, int N, int K, double2 alpha, const double2 *A, int64_t lda, int64_t sA,
           int64_t sA2, const double2 *B, int64_t ldb, int64_t sB, int64_t sB2, double2 *C, int64_t ldc, int64_t sC,
           int64_t sC2, int batch, int batch2, int real) {
    ZProd p(M, N, K, A, lda, sA, B, ldb, sB, C, ldc, sC);
    p.alpha = alpha;
    p.sA2 = sA2;
    p.sB2 = sB2;
    p.sC2 = sC2;
    p.batch2 = batch2;
    p.real = real;
    return zprod(st, p, batch);
}

int compute_phases(nslg_fm *fm) {
    const int64_t n = fm->Nt * fm->Nx;
    const double2 mu = fm->mu_tilde;
    k_phases<<<(unsigned)ceil_div(n, 256), 256, 0, fm->ctx->stream>>>(fm->phi, fm->phase, fm->phase_inv,
                                                                     fm->phase32, fm->sgn, mu, n);
    note_launch(fm->ctx->stream);
    NSLG_CUDA(cudaGetLastError());
    return NSLG_OK;
}

void free_planes(ExpEntry &e) {
    cudaFree(e.re);
    cudaFree(e.im);
    cudaFree(e.reT);
    cudaFree(e.imT);
    cudaFree(e.re32T);
    cudaFree(e.im32T);
    e.re = e.im = e.reT = e.imT = nullptr;
    e.re32T = e.im32T = nullptr;
    if (e.tc) {
        cudaFree(e.tc->hi);
        cudaFree(e.tc->lo);
        delete e.tc;
    }
    if (e.oz) {
        cudaFree(e.oz->planes);
        cudaFree(e.oz->col_exp);
        cudaFree(e.oz->klist);
        delete e.oz;
    }
    if (e.dd) {
        cudaFree(e.dd->planes);
        cudaFree(e.dd->col_exp);
        cudaFree(e.dd->klist);
        delete e.dd;
    }
    e.tc = nullptr;
    e.oz = nullptr;
    e.dd = nullptr;
}

static int make_entry(nslg_fm *fm, double2 *full, nslg::ExpEntry *e) {
    const int64_t n = fm->Nx * fm->Nx;
    cudaStream_t st = fm->ctx->stream;
    e->full = full;
    NSLG_CUDA(cudaMalloc(&e->re, n * sizeof(double)));
    NSLG_CUDA(cudaMalloc(&e->im, n * sizeof(double)));
    NSLG_CUDA(cudaMalloc(&e->reT, n * sizeof(double)));
    NSLG_CUDA(cudaMalloc(&e->re32T, n * sizeof(float)));
    int *flag;
    NSLG_TRY(ws_get(fm, "exp_flag", 1, &flag));
    NSLG_CUDA(cudaMemsetAsync(flag, 0, sizeof(int), st));
    k_split_planes<<<(unsigned)ceil_div(n, 256), 256, 0, st>>>(full, e->re, e->im, e->reT, e->re32T, (int)fm->Nx, flag);
    note_launch(st);
    NSLG_CUDA(cudaGetLastError());
    int h = 0;
    NSLG_CUDA(cudaMemcpyAsync(&h, flag, sizeof(int), cudaMemcpyDeviceToHost, st));
    NSLG_CUDA(cudaStreamSynchronize(st));
    e->is_real = (h == 0);
    if (!e->is_real) {
        NSLG_CUDA(cudaMalloc(&e->imT, n * sizeof(double)));
        NSLG_CUDA(cudaMalloc(&e->im32T, n * sizeof(float)));
        k_split_imag<<<(unsigned)ceil_div(n, 256), 256, 0, st>>>(full, e->imT, e->im32T, (int)fm->Nx);
        note_launch(st);
        NSLG_CUDA(cudaGetLastError());
    }
    return NSLG_OK;
}

int install_exp(nslg_fm *fm, double2 d, const double2 *E_dev) {
    const auto key = std::make_pair(d.x, d.y);
    const int64_t n = fm->Nx * fm->Nx;
    auto it = fm->memo.find(key);
    if (it != fm->memo.end()) {
        NSLG_CUDA(cudaMemcpyAsync(it->second.full, E_dev, n * sizeof(double2), cudaMemcpyDeviceToDevice,
                                  fm->ctx->stream));
        // everything derived from the old matrix goes with it: planes and digits (built again on their next use), and the
        // captured graphs, which hold their addresses (a group's graphs are keyed by ws_generation)
        NSLG_CUDA(cudaStreamSynchronize(fm->ctx->stream));
        drop_graphs(fm);
        fm->lf_seen.clear();
        ++fm->ws_generation;
        free_planes(it->second);
        return make_entry(fm, it->second.full, &it->second);
    }
    double2 *full;
    NSLG_CUDA(cudaMalloc(&full, n * sizeof(double2)));
    NSLG_CUDA(cudaMemcpyAsync(full, E_dev, n * sizeof(double2), cudaMemcpyDeviceToDevice, fm->ctx->stream));
    ExpEntry e;
    NSLG_TRY(make_entry(fm, full, &e));
    fm->memo[key] = e;
    return NSLG_OK;
}

__global__ void k_lin(const double2 *__restrict__ K, double2 d, int one_minus, double2 *__restrict__ out, int n) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)n * n) return;
    double2 v = cmul(d, K[i]);
    if (one_minus) {
        v.x = -v.x;
        v.y = -v.y;
        if (i / n == i % n) v.x += 1.0;
    }
    out[i] = v;
}

int get_lin(nslg_fm *fm, double2 d, int one_minus, const ExpEntry **out) {
    const auto key = std::make_tuple(d.x, d.y, one_minus);
    auto it = fm->lin.find(key);
    if (it == fm->lin.end()) {
        const int n = (int)fm->Nx;
        double2 *full;
        NSLG_CUDA(cudaMalloc(&full, (size_t)n * n * sizeof(double2)));
        k_lin<<<(unsigned)ceil_div((int64_t)n * n, 256), 256, 0, fm->ctx->stream>>>(fm->hops, d, one_minus, full, n);
        note_launch(fm->ctx->stream);
        NSLG_CUDA(cudaGetLastError());
        ExpEntry e;
        NSLG_TRY(make_entry(fm, full, &e));
        it = fm->lin.emplace(key, e).first;
    }
    *out = &it->second;
    return NSLG_OK;
}

int get_factor(nslg_fm *fm, double2 d, const ExpEntry **out) {
    return fm->kind == NSLG_FM_DIAG ? get_lin(fm, d, 0, out) : get_exp(fm, d, out);
}

// exp(d K) by scaling and squaring of the Taylor series: A = d K / 2^s with |A|_1 <= 1/2, T = sum_{k<=14} A^k/k!
// (Horner form, truncation below 3e-17 relative), then T <- T^2 s times.
int get_exp(nslg_fm *fm, double2 d, const ExpEntry **out) {
    const auto key = std::make_pair(d.x, d.y);
    auto it = fm->memo.find(key);
    if (it != fm->memo.end()) {
        *out = &it->second;
        return NSLG_OK;
    }
    const int n = (int)fm->Nx;
    const int64_t nn = (int64_t)n * n;
    cudaStream_t st = fm->ctx->stream;
    const double anorm = hypot(d.x, d.y) * fm->hops_norm1;
    int s = 0;
    while (anorm / std::ldexp(1.0, s) > 0.5) ++s;
    const double scale = std::ldexp(1.0, -s);
    double2 *A, *T0, *T1;
    NSLG_TRY(ws_get(fm, "expm_A", nn, &A));
    NSLG_TRY(ws_get(fm, "expm_T0", nn, &T0));
    NSLG_TRY(ws_get(fm, "expm_T1", nn, &T1));
    k_scale<<<(unsigned)ceil_div(nn, 256), 256, 0, st>>>(A, fm->hops, make_double2(d.x * scale, d.y * scale), nn);
    note_launch(st);
    NSLG_CUDA(cudaGetLastError());
    k_set_identity<<<(unsigned)ceil_div(nn, 256), 256, 0, st>>>(T0, n);
    note_launch(st);
    NSLG_CUDA(cudaGetLastError());
    // Real K and d: every product is real by real, a quarter of the FMAs, which is what bounds it (the terms left out are
    // exact zeros; beyond |d K| = 600 an entry could overflow and its infinity times zero would be lost). Measured, the
    // first operator call of a new matrix against complex products in square tiles: 2.60 -> 1.14 ms at 240 sites, 145 -> 37 ms
    // at 1152.
    const int real = fm->hops_real && d.y == 0.0 && anorm < 600.0 ? 3 : 0;
    auto product = [&](double alpha, const double2 *X, bool identity) {  // T1 = alpha X T0 (+ I)
        ZProd p(n, n, n, X, n, 0, T0, n, 0, T1, n, 0);
        p.alpha = make_double2(alpha, 0);
        p.add_identity = identity;
        p.real = real;
        return zprod(st, p, 1);
    };
    const int m = 14;
    for (int j = m; j >= 1; --j) {  // T <- I + (A / j) T
        NSLG_TRY(product(1.0 / j, A, true));
        std::swap(T0, T1);
    }
    for (int k = 0; k < s; ++k) {
        NSLG_TRY(product(1.0, T0, false));
        std::swap(T0, T1);
    }
    NSLG_TRY(install_exp(fm, d, T0));
    *out = &fm->memo[key];
    return NSLG_OK;
}

int compute_hops_norm(nslg_fm *fm) {
    double *dn;
    NSLG_TRY(ws_get(fm, "norm1", 4, &dn));
    k_norm1<<<1, 256, 0, fm->ctx->stream>>>(fm->hops, (int)fm->Nx, dn);
    note_launch(fm->ctx->stream);
    NSLG_CUDA(cudaGetLastError());
    double h[4];
    NSLG_CUDA(cudaMemcpyAsync(h, dn, sizeof h, cudaMemcpyDeviceToHost, fm->ctx->stream));
    NSLG_CUDA(cudaStreamSynchronize(fm->ctx->stream));
    fm->hops_norm1 = h[0];
    fm->hops_trace = make_double2(h[1], h[2]);
    fm->hops_real = h[3] == 0.0;
    return NSLG_OK;
}

}  // namespace nslg
