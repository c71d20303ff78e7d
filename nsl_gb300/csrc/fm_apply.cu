// Fused fermion-matrix applications M psi and M^dagger psi (exponential discretisation) on CUDA cores.
//
// One launch evaluates, for every right-hand side r and time slice t (hubbardExp.tpp:13-75),
//   M:    out[r, t+1] = psi[r, t+1] - B_{t+1} * expK (phase[t] o psi[r, t])           (B_0 = -1)
//   Mdag: out[r, t-1] = psi[r, t-1] - conj(phase[t-1]) o B'_{t-1} * expK* psi[r, t]    (B'_{Nt-1} = -1)
// as one GEMM over the spatial index with the phase multiply in the operand load (prologue) and the time shift,
// the anti-periodic boundary sign and the "psi -" in the epilogue, so psi is read once and out written once.
// The GEMM rows are the (r, t) pairs, the columns the output site x and the reduction runs over the input site y:
//   Z[(r,t), x] = sum_y Y[(r,t), y] E[x, y].
// expK is real whenever delta and the hopping matrix are real (honeycomb, ring with real kappa); the kernel then
// does a complex-by-real product (2 real FMAs per term instead of 4).
//
// The diagonal discretisation (HubbardDiag, hubbardDiag.tpp:10-71) uses the same GEMM with E = sgn delta K on the
// unshifted slice and adds its phase term element-wise in the epilogue:
//   M:    out[r, t] = psi[r, t] - (sgn delta K psi[r, t]) - B_t phase[t-1] psi[r, t-1]               (B_0 = -1)
//   Mdag: out[r, t] = psi[r, t] - (sgn delta* K psi[r, t]) - conj(phase[t]) B'_t psi[r, t+1]     (B'_{Nt-1} = -1)
//
// A system mask (sys_mask, sys_rows consecutive rows per system) lets whole tiles of unflagged systems return at once:
// the reliable updates of a batched CG evaluate b - A x only for the systems that asked for one.
//
// Vectors are FP64 (Tio = double) in both forms. Tc = double is the FP64 drop-in (DFMA); Tc = float is the FP32
// operator of the mixed-precision solver (FFMA): psi is rounded to FP32 in the operand load, the product runs in FP32
// and the epilogue forms psi - s * z in FP64.
//
// What bounds the FP64 form is the FP64 pipe, ~2 FMAs per clock per SM: a warp's DFMA occupies its scheduler for 64
// cycles, so shared-memory reads, L1 reads and synchronisation all fit in its shadow and the only losses are lanes
// that compute padding and schedulers that run dry. k_fm_apply therefore has no square tile: a thread owns one output
// site of TM consecutive rows, the threads of a CTA are the flattened (row group, site) pairs of whole rows (Nx <= 256)
// or a run of sites of one row group, and exp(delta K) is read transposed, straight from L1/L2 (consecutive lanes,
// consecutive sites). TM shrinks until every scheduler has work. Every output sums over y in ascending order
// whatever TM is. Measured, MM^dagger on 64 right-hand sides at honeycomb 12x12, Nt = 64: 3540 us -> 2486 us (a 2160 us
// floor at the FP64 pipe's rate); M on one right-hand side at honeycomb 3x3, Nt = 16: 67 us -> 4 us of kernel time (the
// figures before are 64 x 64 tiles through shared memory).

#include <algorithm>

#include "fm_internal.cuh"

namespace nslg {

namespace {

constexpr int MAXT = 256;  // threads per CTA at most
constexpr int KC = 64;     // reduction sites per staged operand chunk

// Row stride of the staged operand: 16-byte aligned rows that start in different banks.
template <typename T> __host__ __device__ __forceinline__ int row_stride(int Nx) {
    const int k = Nx < KC ? Nx : KC;
    return sizeof(T) == 8 ? k + 1 : (k + 1) / 2 * 2 + 2;
}

// psi row -> operand value of the GEMM (MODE_M: phase o psi, rounded to T first)
template <typename T, int MODE>
__device__ __forceinline__ cplx_t<T> load_operand(const double2 *__restrict__ psi, const cplx_t<T> *__restrict__ phase,
                                                  int64_t grow, int t, int Nx, int y) {
    const double2 w = psi[grow * Nx + y];
    cplx_t<T> v = cmake<cplx_t<T>>((T)w.x, (T)w.y);
    if (MODE == MODE_M) v = cmul(phase[(int64_t)t * Nx + y], v);  // the diagonal modes multiply psi by nothing
    return v;
}

// epilogue at (row, site): time shift, boundary sign, phase (Mdag) and psi - .
template <typename T, int MODE>
__device__ __forceinline__ void store_output(const double2 *__restrict__ psi, double2 *__restrict__ out,
                                             const cplx_t<T> *__restrict__ phase, int64_t grow, int x, int Nt, int Nx,
                                             cplx_t<T> z) {
    const int64_t r = grow / Nt;
    const int t = (int)(grow - r * Nt);
    int to;
    double s;
    if (MODE == MODE_M) {
        to = (t + 1 == Nt) ? 0 : t + 1;
        s = (to == 0) ? -1.0 : 1.0;
    } else if (MODE == MODE_MDAG) {
        to = (t == 0) ? Nt - 1 : t - 1;
        s = (t == 0) ? -1.0 : 1.0;
    } else {  // diagonal modes: the GEMM stays on its slice
        to = t;
        s = 1.0;
    }
    const int64_t orow = (r * Nt + to) * Nx;
    if (MODE == MODE_MDAG) z = cmulc(phase[(int64_t)to * Nx + x], z);
    const double2 p = psi[orow + x];
    double2 o;
    o.x = p.x - s * (double)z.x;
    o.y = p.y - s * (double)z.y;
    if (MODE == MODE_DIAG_M || MODE == MODE_DIAG_MDAG) {
        // the neighbouring slice of the element-wise phase term and its boundary sign
        const int tn = (MODE == MODE_DIAG_M) ? (t == 0 ? Nt - 1 : t - 1) : (t + 1 == Nt ? 0 : t + 1);
        const double sn = (MODE == MODE_DIAG_M) ? (t == 0 ? -1.0 : 1.0) : (t + 1 == Nt ? -1.0 : 1.0);
        const double2 q = psi[(r * Nt + tn) * Nx + x];
        const cplx_t<T> ph = phase[(int64_t)(MODE == MODE_DIAG_M ? tn : t) * Nx + x];
        const double phx = (double)ph.x, phy = (MODE == MODE_DIAG_M) ? (double)ph.y : -(double)ph.y;  // phase or conj
        o.x -= sn * (phx * q.x - phy * q.y);
        o.y -= sn * (phx * q.y + phy * q.x);
    }
    out[orow + x] = o;
}

__device__ __forceinline__ bool rows_flagged(const int *__restrict__ sys_mask, int64_t sys_rows, int64_t m0,
                                             int64_t end) {
    bool any = false;
    for (int64_t s = m0 / sys_rows; s <= (end - 1) / sys_rows; ++s) any |= sys_mask[s] != 0;
    return any;
}

// CTA: rows [m0, m0 + G TM), sites [blockIdx.y CW, + CW); thread (g, c) = (tid / CW, tid % CW), tid < G CW, owns rows
// m0 + g TM + i (i < TM) at site c of the run. EreT / EimT: exp(delta K) transposed, EreT[y Nx + x] = E[x, y].
template <typename T, bool CE, int MODE, int TM>
__global__ void __launch_bounds__(MAXT) k_fm_apply(const double2 *__restrict__ psi, double2 *__restrict__ out,
                                                   const cplx_t<T> *__restrict__ phase, const T *__restrict__ EreT,
                                                   const T *__restrict__ EimT, int Nt, int Nx, int64_t rows, int G,
                                                   int CW, const int *__restrict__ sys_mask, int64_t sys_rows) {
    using C = cplx_t<T>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *Ys = reinterpret_cast<C *>(smem_raw);  // (G TM) x LS
    const int LS = row_stride<T>(Nx);
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32, nwarps = blockDim.x / 32;
    const int R = G * TM;
    const int64_t m0 = (int64_t)blockIdx.x * R;
    if (sys_mask && !rows_flagged(sys_mask, sys_rows, m0, min(rows, m0 + R))) return;
    const int t0 = (int)(m0 % Nt);
    const int g = tid / CW, c = tid - g * CW;
    const int x = blockIdx.y * CW + c;
    const bool act = g < G && x < Nx;
    C acc[TM];
#pragma unroll
    for (int i = 0; i < TM; ++i) acc[i] = cmake<C>(0, 0);
    auto term = [&](C a, T b, T bi, C &s) {
        s.x = fma(a.x, b, s.x);
        s.y = fma(a.y, b, s.y);
        if (CE) {
            s.x = fma(-a.y, bi, s.x);
            s.y = fma(a.x, bi, s.y);
        }
    };
    for (int k0 = 0; k0 < Nx; k0 += KC) {
        const int kc = min(KC, Nx - k0);
        if (k0) __syncthreads();
        for (int row = warp; row < R; row += nwarps) {  // one warp per row
            const int64_t grow = m0 + row;
            const int t = MODE == MODE_M ? (t0 + row) % Nt : 0;
            for (int kk = lane; kk < kc; kk += 32)
                Ys[row * LS + kk] = grow < rows ? load_operand<T, MODE>(psi, phase, grow, t, Nx, k0 + kk)
                                                : cmake<C>(0, 0);
        }
        __syncthreads();
        if (act) {
            const C *ys = Ys + g * TM * LS;
            const T *er = EreT + (int64_t)k0 * Nx + x;
            const T *ei = CE ? EimT + (int64_t)k0 * Nx + x : nullptr;
            int kk = 0;
            if constexpr (sizeof(T) == 4) {  // FP32: the operand reads bound the loop, so two y per 16-byte read
#pragma unroll 4
                for (; kk + 1 < kc; kk += 2) {
                    const T b0 = er[(int64_t)kk * Nx], b1 = er[(int64_t)(kk + 1) * Nx];
                    const T i0 = CE ? ei[(int64_t)kk * Nx] : T(0), i1 = CE ? ei[(int64_t)(kk + 1) * Nx] : T(0);
#pragma unroll
                    for (int i = 0; i < TM; ++i) {
                        const float4 a = *reinterpret_cast<const float4 *>(ys + i * LS + kk);
                        term(cmake<C>(a.x, a.y), b0, i0, acc[i]);
                        term(cmake<C>(a.z, a.w), b1, i1, acc[i]);
                    }
                }
            }
#pragma unroll 8
            for (; kk < kc; ++kk) {
                const T b = er[(int64_t)kk * Nx];
                const T bi = CE ? ei[(int64_t)kk * Nx] : T(0);
#pragma unroll
                for (int i = 0; i < TM; ++i) term(ys[i * LS + kk], b, bi, acc[i]);
            }
        }
    }
    if (!act) return;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int64_t grow = m0 + g * TM + i;
        if (grow < rows) store_output<T, MODE>(psi, out, phase, grow, x, Nt, Nx, acc[i]);
    }
}

// The FP32 M^dagger (and diagonal) products of large batches: 64 x 64 tiles, 4 x 4 outputs per thread. FP32 FMAs are not
// what bounds that product (128 per clock per SM), operand reads are, and the square micro-tile needs the fewest.
constexpr int BM = 64, BN = 64, BK = 16;

template <bool CE, int MODE>
__global__ void __launch_bounds__(256) k_fm_apply32_tile(const double2 *__restrict__ psi, double2 *__restrict__ out,
                                                         const float2 *__restrict__ phase,
                                                         const float *__restrict__ EreT,
                                                         const float *__restrict__ EimT, int Nt, int Nx, int64_t rows,
                                                         const int *__restrict__ sys_mask, int64_t sys_rows) {
    __shared__ float2 As[BK][BM + 1];
    __shared__ float Bs[BK][BN + 1];
    __shared__ float Bsi[CE ? BK : 1][BN + 1];
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    const int64_t m0 = (int64_t)blockIdx.x * BM;
    const int n0 = blockIdx.y * BN;
    if (sys_mask && !rows_flagged(sys_mask, sys_rows, m0, min(rows, m0 + BM))) return;
    float2 acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0, 0);
    for (int k0 = 0; k0 < Nx; k0 += BK) {
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            const int idx = tid + l * 256;
            const int row = idx / BK, kk = idx % BK, y = k0 + kk;
            const int64_t grow = m0 + row;
            As[kk][row] = (grow < rows && y < Nx) ? load_operand<float, MODE>(psi, phase, grow, (int)(grow % Nt), Nx, y)
                                                  : make_float2(0, 0);
            const int n = idx % BN, bk = idx / BN, x = n0 + n, yb = k0 + bk;
            const bool ok = x < Nx && yb < Nx;
            Bs[bk][n] = ok ? EreT[(int64_t)yb * Nx + x] : 0.f;
            if (CE) Bsi[bk][n] = ok ? EimT[(int64_t)yb * Nx + x] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 a = As[kk][ty + 16 * i];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float b = Bs[kk][tx + 16 * j];
                    acc[i][j].x = fma(a.x, b, acc[i][j].x);
                    acc[i][j].y = fma(a.y, b, acc[i][j].y);
                    if (CE) {
                        const float bi = Bsi[kk][tx + 16 * j];
                        acc[i][j].x = fma(-a.y, bi, acc[i][j].x);
                        acc[i][j].y = fma(a.x, bi, acc[i][j].y);
                    }
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int64_t grow = m0 + ty + 16 * i;
        if (grow >= rows) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int x = n0 + tx + 16 * j;
            if (x < Nx) store_output<float, MODE>(psi, out, phase, grow, x, Nt, Nx, acc[i][j]);
        }
    }
}

// How a (rows, Nx) product is cut into CTAs: sites per CTA, row groups, rows per thread.
struct Split {
    int CW, G, TM, threads;
    unsigned gx, gy;
};

Split split_of(int64_t rows, int Nx) {
    Split S;
    const int64_t sched = 4 * (int64_t)std::max(1, num_sms());
    if (Nx > MAXT) {  // a run of sites of one row group, all runs alike and a whole number of warps
        const int runs = (int)ceil_div(Nx, 128);
        S.CW = (int)ceil_div(ceil_div(Nx, runs), 32) * 32;
        S.gy = (unsigned)ceil_div(Nx, S.CW);
        S.G = 1;
    } else {  // whole rows: as many row groups as leave the fewest idle lanes in the last warp, small CTAs first
        S.CW = Nx;
        S.gy = 1;
        S.G = 1;
        double best = 0;
        for (int G = 1; G * Nx <= MAXT && G <= rows; ++G) {
            const double eff = (double)(G * Nx) / (32.0 * (double)ceil_div(G * Nx, 32));
            if (eff > best + 0.03) {
                best = eff;
                S.G = G;
            }
        }
    }
    S.threads = 32 * (int)ceil_div(S.G * S.CW, 32);
    // rows per thread: the most that still keep the schedulers (4 per SM) evenly busy to 90 %, else the best balance
    double best = 0;
    S.TM = 1;
    for (int TM = 8; TM >= 1; TM /= 2) {
        const int64_t warps = ceil_div(rows, (int64_t)S.G * TM) * S.gy * (S.threads / 32);
        const double waves = (double)warps / (double)sched;
        const double eff = waves / (double)ceil_div(warps, sched) * (double)rows /
                           (double)(ceil_div(rows, (int64_t)S.G * TM) * S.G * TM);
        if (eff > 1.02 * best) {
            best = eff;
            S.TM = TM;
        }
        if (eff >= 0.9) break;
    }
    S.gx = (unsigned)ceil_div(rows, (int64_t)S.G * S.TM);
    return S;
}

template <typename T, bool CE, int TM>
void launch_tm(int mode, const Split &S, const double2 *psi, double2 *out, const cplx_t<T> *phase, const T *Ere,
               const T *Eim, int Nt, int Nx, int64_t rows, cudaStream_t st, const int *mask, int64_t sys_rows) {
    const dim3 grid(S.gx, S.gy);
    const size_t smem = (size_t)S.G * TM * row_stride<T>(Nx) * sizeof(cplx_t<T>);  // <= 37 KB (G Nx <= 256)
    if (mode == MODE_M)
        k_fm_apply<T, CE, MODE_M, TM><<<grid, S.threads, smem, st>>>(psi, out, phase, Ere, Eim, Nt, Nx, rows, S.G, S.CW,
                                                                     mask, sys_rows);
    else if (mode == MODE_MDAG)
        k_fm_apply<T, CE, MODE_MDAG, TM><<<grid, S.threads, smem, st>>>(psi, out, phase, Ere, Eim, Nt, Nx, rows, S.G,
                                                                        S.CW, mask, sys_rows);
    else if (mode == MODE_DIAG_M)
        k_fm_apply<T, CE, MODE_DIAG_M, TM><<<grid, S.threads, smem, st>>>(psi, out, phase, Ere, Eim, Nt, Nx, rows, S.G,
                                                                          S.CW, mask, sys_rows);
    else
        k_fm_apply<T, CE, MODE_DIAG_MDAG, TM><<<grid, S.threads, smem, st>>>(psi, out, phase, Ere, Eim, Nt, Nx, rows,
                                                                             S.G, S.CW, mask, sys_rows);
}

template <typename T, bool CE>
int launch_mode(int mode, const double2 *psi, double2 *out, const cplx_t<T> *phase, const T *Ere, const T *Eim,
                int Nt, int Nx, int64_t rows, cudaStream_t st, const int *mask, int64_t sys_rows) {
    if constexpr (sizeof(T) == 4) {
        // measured, M^dagger: 75 us here against 79 below (64 right-hand sides, honeycomb 12x12, Nt = 64), 198 against 251
        // (8, honeycomb 24x24, Nt = 128), but 147 against 93 with one; M, whose phase is formed once per site block,
        // is faster below (139 and 289 us here, 89 and 221 below)
        const int64_t tiles = ceil_div(rows, BM) * ceil_div(Nx, BN);
        if (mode != MODE_M && Nx > MAXT && tiles >= 2 * num_sms()) {
            const dim3 grid((unsigned)ceil_div(rows, BM), (unsigned)ceil_div(Nx, BN));
            if (mode == MODE_MDAG)
                k_fm_apply32_tile<CE, MODE_MDAG><<<grid, 256, 0, st>>>(psi, out, phase, Ere, Eim, Nt, Nx, rows, mask,
                                                                       sys_rows);
            else if (mode == MODE_DIAG_M)
                k_fm_apply32_tile<CE, MODE_DIAG_M><<<grid, 256, 0, st>>>(psi, out, phase, Ere, Eim, Nt, Nx, rows, mask,
                                                                         sys_rows);
            else
                k_fm_apply32_tile<CE, MODE_DIAG_MDAG><<<grid, 256, 0, st>>>(psi, out, phase, Ere, Eim, Nt, Nx, rows,
                                                                            mask, sys_rows);
            note_launch(st);
            NSLG_CUDA(cudaGetLastError());
            return NSLG_OK;
        }
    }
    const Split S = split_of(rows, Nx);
    if (S.TM == 8) launch_tm<T, CE, 8>(mode, S, psi, out, phase, Ere, Eim, Nt, Nx, rows, st, mask, sys_rows);
    else if (S.TM == 4) launch_tm<T, CE, 4>(mode, S, psi, out, phase, Ere, Eim, Nt, Nx, rows, st, mask, sys_rows);
    else if (S.TM == 2) launch_tm<T, CE, 2>(mode, S, psi, out, phase, Ere, Eim, Nt, Nx, rows, st, mask, sys_rows);
    else launch_tm<T, CE, 1>(mode, S, psi, out, phase, Ere, Eim, Nt, Nx, rows, st, mask, sys_rows);
    note_launch(st);
    NSLG_CUDA(cudaGetLastError());
    return NSLG_OK;
}

}  // namespace

template <typename T>
int fm_apply_simt(int mode, const double2 *psi, double2 *out, const cplx_t<T> *phase, const T *Ere, const T *Eim,
                  int Nt, int Nx, int64_t rows, cudaStream_t st, const int *sys_mask, int64_t sys_rows) {
    if (rows == 0) return NSLG_OK;
    NSLG_REQUIRE(!sys_mask || sys_rows >= 1, NSLG_ERR_ARG, "operator row mask: rows per system must be positive");
    if (Eim) return launch_mode<T, true>(mode, psi, out, phase, Ere, Eim, Nt, Nx, rows, st, sys_mask, sys_rows);
    return launch_mode<T, false>(mode, psi, out, phase, Ere, nullptr, Nt, Nx, rows, st, sys_mask, sys_rows);
}

template int fm_apply_simt<double>(int, const double2 *, double2 *, const double2 *, const double *, const double *,
                                   int, int, int64_t, cudaStream_t, const int *, int64_t);
template int fm_apply_simt<float>(int, const double2 *, double2 *, const float2 *, const float *, const float *,
                                  int, int, int64_t, cudaStream_t, const int *, int64_t);

}  // namespace nslg
