// M psi and M^dagger psi in double-double on the tensor cores: twelve digits of nine bits, every digit product and every
// accumulation exact.
//
// The CUDA-core form (fm_apply_dd.cu) spends 34 FP64 operations per term, and GB300 does ~2 of them per clock per SM. Here
// both factors are cut into balanced base-512 digits at per-row power-of-two scales, as in the FP64-class operator
// (fm_apply_oz.cu, oz_digits.cuh), but to D = 12 digits (107 bits): the pair x_hi + x_lo, and the FP64 entries of
// exp(delta K), whose small entries reach below the row maximum's last bit. Digit products of order d = a + b < D go into D
// FP32 accumulators in TMEM; what is dropped (orders >= D) and rounded is below 2^-105 of the row maxima.
//
// Exactness. An accumulator stays exact while its partial sums are integers below 2^24. For every operand
//   |G_d(x)| <= 256 sum_{l, y} |b_l(x, y)|  over the sites y accumulated, b_l the digits of row x of exp(delta K),
// so the reduction over y is cut into segments of k-blocks for which that sum stays below 2^24 for every x of the tile
// (k_ddtc_klist; a single 16-site k-block is at most 12 * 16 * 2^16 < 2^24, so every matrix has such a cut). After each
// segment the epilogue folds the accumulators into one 128-bit integer per output, sum_d G_d 2^{9(D-1-d)}; over all segments
// |G_d| <= (d + 1) 2^16 Nx, so for Nx <= 2048 the integer stays below 2^127. Only the finished integer is turned into a
// double-double.
//
// One persistent CTA per SM as in fm_apply_oz.cu: warp 0 streams k-blocks (one bulk copy per operand), warp 1 issues one
// MMA per operand digit (N = 16 sites x the digits that meet it; as there, MMAs of different N on overlapping accumulators,
// executed in issue order), four epilogue warps finish 128 x 16 tiles from one of two
// accumulator sets while the next segment runs in the other.
// Measured, M on 64 right-hand sides at honeycomb 12x12, Nt = 64: 23.8 ms on the CUDA cores, 0.49 ms here; on 2 at 24x24,
// Nt = 128: 23.8 and 0.32 ms.

#include <algorithm>

#include "dd_math.cuh"
#include "fm_internal.cuh"
#include "oz_digits.cuh"
#include "tc_common.cuh"

namespace nslg {

namespace {

constexpr int D = 12;                        // digits per operand
constexpr int DT_BM = OZ_TILE_A;             // real GEMM rows per tile
constexpr int DT_BN = 16;                    // output sites per tile
constexpr int DT_A_SLICE = DT_BM * 2 * OZ_KB;  // 4 KB
constexpr int DT_B_SLICE = DT_BN * 2 * OZ_KB;  // 512 B
constexpr int DT_STAGE = D * (DT_A_SLICE + DT_B_SLICE);  // 54 KB per k-block
constexpr int DT_STAGES = 4;
constexpr int DT_THREADS = 192;              // copy warp, MMA warp, four epilogue warps
constexpr int DT_TMEM_COLS = 512;            // two accumulator sets of D * DT_BN = 192 columns
constexpr int DT_SMEM = DT_STAGES * DT_STAGE + 1024 /*alignment*/ + 1024 /*barriers*/;
constexpr int DT_BITS = 9 * D - 1;           // operands are rounded to 2^{e - 107}
constexpr int64_t DT_BLOCK_ELEMS = 1 << 21;  // elements per block of rows (workspace of 160 MB)
constexpr int DT_NONFINITE = 1 << 28;        // row scale of a row with an infinity or a NaN
static_assert(DT_SMEM <= 227 * 1024, "shared memory per CTA");
static_assert(2 * D * DT_BN <= DT_TMEM_COLS, "TMEM columns");

using i128 = __int128;

// round(v 2^{DT_BITS - e}) of one FP64 number, |v| <= 2^e.
__device__ __forceinline__ i128 scaled_int128(double v, int e) {
    const unsigned long long bits = (unsigned long long)__double_as_longlong(v);
    const int ex = (int)((bits >> 52) & 0x7FF);
    if (ex == 0) return 0;  // zero (subnormals are far below every row scale)
    const unsigned long long mant = (bits & 0xFFFFFFFFFFFFFull) | (1ull << 52);
    const int sh = ex - 1075 + DT_BITS - e;  // v = mant 2^{ex - 1075}
    i128 u;
    if (sh >= 0) u = (i128)mant << min(sh, 70);
    else if (sh <= -64) u = 0;
    else u = (i128)((mant + (1ull << (-sh - 1))) >> -sh);
    return (bits >> 63) ? -u : u;
}

// Balanced base-512 digits of N, |N| <= 2^107: digit k has weight 2^{9(D-1-k)}, |a_0| <= 256, the others in [-256, 255].
__device__ __forceinline__ void digits12(i128 N, int (&a)[D]) {
#pragma unroll
    for (int k = D - 1; k > 0; --k) {
        const int d = (int)(((unsigned)(unsigned long long)N + 256u) & 511u) - 256;
        a[k] = d;
        N = (N - d) >> 9;
    }
    a[0] = (int)N;
}

// Byte offset of (row, digit l, site y) in D-digit planes of TILE-row tiles (the layout of digit_offset, oz_digits.cuh).
template <int TILE> __device__ __forceinline__ int64_t dt_offset(int64_t row, int l, int y, int nkb) {
    const int m = (int)(row % TILE);
    return (((row / TILE) * nkb + y / OZ_KB) * D + l) * (TILE * 32) + m * 32 + (((y >> 3 & 1) ^ (m >> 2 & 1)) << 4) +
           (y & 7) * 2;
}

__device__ __forceinline__ unsigned long long wmax(unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Digits of exp(d K) (one block of 256 threads per row x) and, per k-block, sum_l sum_y |b_l| and the digits present.
__global__ void __launch_bounds__(256) k_ddtc_planes(const double2 *__restrict__ E, char *planes, int *col_exp, int *sums,
                                                     int *masks, int Nx, int nkb) {
    const int x = blockIdx.x;
    __shared__ unsigned long long red[8];
    unsigned long long m = 0ull;
    for (int y = threadIdx.x; y < Nx; y += 256) m = max(m, abs_bits(E[(int64_t)x * Nx + y].x));
    m = wmax(m);
    if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = m;
    __syncthreads();
    for (int w = 0; w < 8; ++w) m = max(m, red[w]);
    const int e = scale_exponent(m);
    if (threadIdx.x == 0) col_exp[x] = e;
    for (int y = threadIdx.x; y < nkb * OZ_KB; y += 256) {
        int a[D], s = 0, mk = 0;
        digits12(scaled_int128(y < Nx ? E[(int64_t)x * Nx + y].x : 0.0, e), a);
#pragma unroll
        for (int l = 0; l < D; ++l) {
            *reinterpret_cast<__nv_bfloat16 *>(planes + dt_offset<DT_BN>(x, l, y, nkb)) = __float2bfloat16_rn((float)a[l]);
            s += abs(a[l]);
            mk |= (a[l] != 0) << l;
        }
        atomicAdd(&sums[(int64_t)x * nkb + y / OZ_KB], s);
        if (mk) atomicOr(&masks[(x / DT_BN) * nkb + y / OZ_KB], mk);
    }
}

// k-blocks of every tile of output sites: klist[tile (nkb + 1)] = count, then k-block | digits << 14 | end << 30. A segment's
// first k-block has every digit (it starts all accumulators); k-blocks without a digit are left out. One thread per tile.
__global__ void k_ddtc_klist(const int *__restrict__ sums, const int *__restrict__ masks, int *klist, int Nx, int ntn,
                             int nkb) {
    const int nt = blockIdx.x * blockDim.x + threadIdx.x;
    if (nt >= ntn) return;
    int *kl = klist + (int64_t)nt * (nkb + 1);
    long long acc[DT_BN];
    int n = 0;
    bool fresh = true;
    for (int kb = 0; kb < nkb; ++kb) {
        const int mask = masks[nt * nkb + kb];
        if (!mask && !(kb == nkb - 1 && n == 0)) continue;
        bool over = false;
        for (int i = 0; i < DT_BN; ++i) {
            const int x = nt * DT_BN + i;
            const long long s = x < Nx ? sums[(int64_t)x * nkb + kb] : 0;
            over |= !fresh && (acc[i] + s) * 256 >= (1ll << 24);
        }
        if (over) {
            kl[n] |= 1 << 30;
            fresh = true;
        }
        for (int i = 0; i < DT_BN; ++i) {
            const int x = nt * DT_BN + i;
            const long long s = x < Nx ? sums[(int64_t)x * nkb + kb] : 0;
            acc[i] = fresh ? s : acc[i] + s;
        }
        kl[1 + n++] = kb | (fresh ? (1 << D) - 1 : mask) << 14;
        fresh = false;
    }
    kl[n] |= 1 << 30;  // n >= 1: the last k-block stands in for a tile without a digit
    kl[0] = n;
}

// One warp per row (r, t) of rows [row0, row0 + rows) (digits, scales, vh and vl are indexed from row0): the operand (phase o x
// for M, stored to vh, vl; x itself for M^dagger), its scales (real and imaginary parts) and its digits.
template <int MODE>
__global__ void __launch_bounds__(256) k_ddtc_digits(const double2 *__restrict__ xh, const double2 *__restrict__ xl,
                                                     const double2 *__restrict__ phase, double2 *__restrict__ vh,
                                                     double2 *__restrict__ vl, int Nt, int Nx, int64_t row0, int64_t rows,
                                                     int nkb, char *__restrict__ planes, int *__restrict__ rexp,
                                                     const int *__restrict__ sys_mask, int64_t sys_rows) {
    const int64_t grow = (int64_t)blockIdx.x * 8 + threadIdx.x / 32;
    const int lane = threadIdx.x % 32;
    if (grow >= rows || (sys_mask && !sys_mask[(row0 + grow) / sys_rows])) return;
    const int t = (int)((row0 + grow) % Nt);
    xh += row0 * Nx;
    xl += row0 * Nx;
    unsigned long long mr = 0, mi = 0;
    for (int y = lane; y < Nx; y += 32) {
        const double2 h = xh[grow * Nx + y], l = xl[grow * Nx + y];
        ddc v = {fast_two_sum(h.x, l.x), fast_two_sum(h.y, l.y)};
        if (MODE == MODE_M) v = cmul_d(phase[(int64_t)t * Nx + y], v);
        if (MODE == MODE_M) {
            vh[grow * Nx + y] = make_double2(v.re.hi, v.im.hi);
            vl[grow * Nx + y] = make_double2(v.re.lo, v.im.lo);
        }
        mr = max(mr, abs_bits(v.re.hi));
        mi = max(mi, abs_bits(v.im.hi));
    }
    mr = wmax(mr);
    mi = wmax(mi);
    const int er = scale_exponent(mr), ei = scale_exponent(mi);
    if (lane == 0) {
        rexp[2 * grow] = (mr >> 52) >= 0x7FF ? DT_NONFINITE : er;  // (a NaN may keep its sign bit)
        rexp[2 * grow + 1] = (mi >> 52) >= 0x7FF ? DT_NONFINITE : ei;
    }
    const double2 *sh = MODE == MODE_M ? vh : xh, *sl = MODE == MODE_M ? vl : xl;  // (each lane reads what it wrote)
    for (int y = lane; y < nkb * OZ_KB; y += 32) {
        dd re = {0.0, 0.0}, im = {0.0, 0.0};
        if (y < Nx) {
            const double2 h = sh[grow * Nx + y], l = sl[grow * Nx + y];
            re = fast_two_sum(h.x, l.x);
            im = fast_two_sum(h.y, l.y);
        }
        int a[D], b[D];
        digits12(scaled_int128(re.hi, er) + scaled_int128(re.lo, er), a);
        digits12(scaled_int128(im.hi, ei) + scaled_int128(im.lo, ei), b);
        char *p = planes + dt_offset<DT_BM>(2 * grow, 0, y, nkb);
#pragma unroll
        for (int l = 0; l < D; ++l) {
            *reinterpret_cast<__nv_bfloat16 *>(p + l * DT_A_SLICE) = __float2bfloat16_rn((float)a[l]);
            *reinterpret_cast<__nv_bfloat16 *>(p + l * DT_A_SLICE + 32) = __float2bfloat16_rn((float)b[l]);
        }
    }
}

// T 2^e as a double-double: the leading 53 bits and the rest.
__device__ __forceinline__ dd int128_to_dd(i128 T, int e) {
    if (T == 0) return {0.0, 0.0};
    const bool neg = T < 0;
    unsigned __int128 u = neg ? (unsigned __int128)(-T) : (unsigned __int128)T;
    const unsigned long long top = (unsigned long long)(u >> 64);
    const int lz = top ? __clzll((long long)top) : 64 + __clzll((long long)(unsigned long long)u);
    u <<= lz;  // leading one at bit 127: |T| = u 2^-lz
    const long long m = (long long)(u >> 75);             // 53 bits
    unsigned long long rest = (unsigned long long)(u >> 12) & ((1ull << 63) - 1);  // the next 63 bits
    const double hi = scaled_to_double(neg ? -m : m, e + 75 - lz);
    const double lo = scaled_to_double(neg ? -(long long)rest : (long long)rest, e + 12 - lz);
    return fast_two_sum(hi, lo);
}

template <int MODE>
__global__ void __launch_bounds__(DT_THREADS, 1)
    k_fm_apply_ddtc(const double2 *__restrict__ xh, const double2 *__restrict__ xl, double2 *__restrict__ oh,
                    double2 *__restrict__ ol, const double2 *__restrict__ phase, const int *__restrict__ row_exp,
                    const int *__restrict__ col_exp, const int *__restrict__ klist, const uint8_t *__restrict__ dga,
                    const uint8_t *__restrict__ dgb, int Nt, int Nx, int64_t row0, int64_t rows, int nkb, int *err,
                    const int *__restrict__ sys_mask, int64_t sys_rows) {
    constexpr int STAGE = DT_STAGE, BN = DT_BN;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *bar_full = reinterpret_cast<uint64_t *>(smem + DT_STAGES * STAGE);
    uint64_t *bar_empty = bar_full + DT_STAGES;
    uint64_t *bar_tfull = bar_empty + DT_STAGES;  // [2]: an accumulator set holds a finished segment
    uint64_t *bar_tempty = bar_tfull + 2;         // [2]: the epilogue has read an accumulator set
    uint64_t *bar_done = bar_tempty + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bar_done + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(bar_done + 2);
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const int nmt = (int)((rows + DT_BM / 2 - 1) / (DT_BM / 2));
    const int ntn = (Nx + BN - 1) / BN;
    const int ntiles = nmt * ntn;
    auto live = [&](int t) -> bool {  // some row of the tile belongs to a flagged system
        if (!sys_mask) return true;
        const int64_t g0 = (int64_t)(t / ntn) * (DT_BM / 2);
        const int64_t last = min(rows, g0 + DT_BM / 2) - 1;
        for (int64_t s = (row0 + g0) / sys_rows; s <= (row0 + last) / sys_rows; ++s)
            if (sys_mask[s] != 0) return true;
        return false;
    };
    if (tid == 0) {
        for (int i = 0; i < DT_STAGES; ++i) {
            tc::mbar_init(&bar_full[i], 1);
            tc::mbar_init(&bar_empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            tc::mbar_init(&bar_tfull[i], 1);
            tc::mbar_init(&bar_tempty[i], 4);
        }
        tc::mbar_init(bar_done, 1);
        *abort_flag = 0;
        tc::fence_mbar_init();
    }
    if (warp == 1) tc::tmem_alloc(tmem_slot, DT_TMEM_COLS);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            int it = 0;
            for (int t = blockIdx.x; t < ntiles && !*abort_flag; t += gridDim.x) {
                if (!live(t)) continue;
                const uint8_t *at = dga + (int64_t)(t / ntn) * nkb * (D * DT_A_SLICE);
                const uint8_t *bt = dgb + (int64_t)(t % ntn) * nkb * (D * DT_B_SLICE);
                const int *kl = klist + (int64_t)(t % ntn) * (nkb + 1);
                const int nk = kl[0];
                for (int i = 1; i <= nk; ++i, ++it) {
                    const int kb = kl[i] & 0x3FFF, mask = kl[i] >> 14 & ((1 << D) - 1);
                    const int b0 = __ffs(mask) - 1, nb = 32 - __clz(mask) - b0, na = D - b0;
                    const int s = it % DT_STAGES;
                    if (it >= DT_STAGES &&
                        (*abort_flag || !tc::mbar_wait(&bar_empty[s], ((it / DT_STAGES) - 1) & 1, err, 41))) {
                        *abort_flag = 1;
                        break;
                    }
                    uint8_t *a_base = smem + s * STAGE;
                    uint8_t *b_base = a_base + D * DT_A_SLICE;
                    tc::mbar_arrive_expect_tx(&bar_full[s], na * DT_A_SLICE + nb * DT_B_SLICE);
                    tc::bulk_load(a_base, at + (int64_t)kb * (D * DT_A_SLICE), na * DT_A_SLICE, &bar_full[s]);
                    tc::bulk_load(b_base + b0 * DT_B_SLICE, bt + ((int64_t)kb * D + b0) * DT_B_SLICE, nb * DT_B_SLICE,
                                  &bar_full[s]);
                }
            }
            for (int u = it - 1; u >= 0 && u >= it - DT_STAGES; --u)
                if (!tc::mbar_wait(&bar_full[u % DT_STAGES], (u / DT_STAGES) & 1, err, 44)) *abort_flag = 1;
        }
    } else if (warp == 1) {
        if (lane == 0) {
            int it = 0, seg = 0;  // segments so far: accumulator set seg & 1
            bool ok = true;
            const uint64_t dsm0 = tc::sdesc_kmajor_sw32(tc::smem_addr(smem));
            for (int t = blockIdx.x; t < ntiles && ok && !*abort_flag; t += gridDim.x) {
                if (!live(t)) continue;
                const int *kl = klist + (int64_t)(t % ntn) * (nkb + 1);
                const int nk = kl[0];
                bool first = true;
                for (int i = 1; i <= nk; ++i, ++it) {
                    const int entry = kl[i], mask = entry >> 14 & ((1 << D) - 1);
                    const int buf = seg & 1, use = seg >> 1;
                    if (first && use >= 1 && !tc::mbar_wait(&bar_tempty[buf], (use - 1) & 1, err, 45)) ok = false;
                    if (first) tc::tc_fence_after();
                    const int s = it % DT_STAGES;
                    if (!ok || *abort_flag || !tc::mbar_wait(&bar_full[s], (it / DT_STAGES) & 1, err, 42)) {
                        ok = false;
                        break;
                    }
                    const uint32_t dbase = tmem + (uint32_t)(buf * D * BN);
                    const uint64_t dst = dsm0 + (uint64_t)((s * STAGE) >> 4);
                    const int b0 = __ffs(mask) - 1, b1 = 31 - __clz(mask);
                    const uint64_t db = dst + (uint64_t)((D * DT_A_SLICE + b0 * DT_B_SLICE) >> 4);
                    for (int a = 0; a < D - b0; ++a) {
                        const int n = min(b1, D - 1 - a) - b0 + 1;
                        tc::mma_bf16(dbase + (uint32_t)((a + b0) * BN), dst + (uint64_t)((a * DT_A_SLICE) >> 4), db,
                                     tc::idesc_bf16(DT_BM, n * BN), (first && a == 0) ? 0u : 1u);
                    }
                    tc::mma_commit(&bar_empty[s]);
                    first = false;
                    if (entry >> 30 & 1) {
                        tc::mma_commit(&bar_tfull[buf]);
                        ++seg;
                        first = true;
                    }
                }
            }
            if (!ok) *abort_flag = 1;
            tc::mma_commit(bar_done);
            if (!tc::mbar_wait(bar_done, 0, err, 43)) *abort_flag = 1;
        }
    } else {
        // TMEM lane = GEMM row m of the tile (real or imaginary part of complex row j); 16 sites per lane, of which the
        // two lanes of a complex row finish alternate ones (as in fm_apply_oz.cu)
        const int m = 32 * (warp % 4) + lane, j = m >> 1, comp = m & 1;
        const uint32_t lane_base = tmem + ((uint32_t)(32 * (warp % 4)) << 16);
        int seg = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
            if (!live(t)) continue;
            const int mt = t / ntn, nt = t % ntn;
            const int *kl = klist + (int64_t)nt * (nkb + 1);
            const int nk = kl[0];
            i128 T[BN];
#pragma unroll
            for (int i = 0; i < BN; ++i) T[i] = 0;
            for (int i = 1; i <= nk; ++i) {
                if (!(kl[i] >> 30 & 1)) continue;  // one pass per segment
                const int buf = seg & 1, use = seg >> 1;
                // (a vote: a warp leaves whole, or its shuffles and TMEM reads would wait for lanes that have gone)
                if (!__all_sync(0xffffffffu, *abort_flag == 0 && tc::mbar_wait(&bar_tfull[buf], use & 1, err, 46))) {
                    ok = false;
                    break;
                }
                tc::tc_fence_after();
#pragma unroll
                for (int q = 0; q < BN / 8; ++q) {
                    uint32_t v[D][8];
#pragma unroll
                    for (int d = 0; d < D; ++d)
                        tc::tmem_ld8_async(lane_base + (uint32_t)(buf * D * BN + d * BN + 8 * q), v[d]);
                    tc::tmem_wait_ld<D>(v);
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        i128 g = 0;
#pragma unroll
                        for (int d = 0; d < D; ++d)  // integer-valued
                            g = g * 512 + (i128)__float2int_rn(__uint_as_float(v[d][c]));
                        T[8 * q + c] += g;
                    }
                }
                tc::tc_fence_before();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&bar_tempty[buf]);
                ++seg;
            }
            if (!ok) {
                *abort_flag = 1;
                break;
            }
            const int64_t lrow = (int64_t)mt * (DT_BM / 2) + j, grow = row0 + lrow;
            const bool row_ok = lrow < rows && (!sys_mask || sys_mask[grow / sys_rows] != 0);
            const int64_t r = grow / Nt;
            const int tt = (int)(grow - r * Nt);
            int to;
            bool neg;  // boundary slice: psi + z
            if (MODE == MODE_M) {
                to = (tt + 1 == Nt) ? 0 : tt + 1;
                neg = to == 0;
            } else {
                to = (tt == 0) ? Nt - 1 : tt - 1;
                neg = tt == 0;
            }
            const int64_t orow = (r * Nt + to) * Nx;
            const int re = row_ok ? row_exp[(int64_t)mt * DT_BM + m] : 0;
#pragma unroll
            for (int s = 0; s < BN / 2; ++s) {
                const int x0 = nt * BN + 2 * s;
                dd z[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    // 2^{e_row + e_x - 16} sum_d 2^{-9d} G_d
                    z[h] = int128_to_dd(T[2 * s + h], re + (x0 + h < Nx ? col_exp[x0 + h] : 0) - 16 - 9 * (D - 1));
                    if (re == DT_NONFINITE) z[h] = {__longlong_as_double(0x7FF8000000000000ll), 0.0};
                }
                // lane pairs exchange: this lane finishes site x0 + comp
                const dd give = comp ? z[0] : z[1], keep = comp ? z[1] : z[0];
                const dd recv = {__shfl_xor_sync(0xffffffffu, give.hi, 1), __shfl_xor_sync(0xffffffffu, give.lo, 1)};
                ddc w = comp ? ddc{recv, keep} : ddc{keep, recv};
                const int x = x0 + comp;
                if (row_ok && x < Nx) {
                    if (MODE == MODE_MDAG) w = cmulc_d(phase[(int64_t)to * Nx + x], w);
                    const double2 h = xh[orow + x], l = xl[orow + x];
                    const dd pr = fast_two_sum(h.x, l.x), pi = fast_two_sum(h.y, l.y);
                    const dd ore = neg ? dd_add(pr, w.re) : dd_add(pr, dd_neg(w.re));
                    const dd oim = neg ? dd_add(pi, w.im) : dd_add(pi, dd_neg(w.im));
                    oh[orow + x] = make_double2(ore.hi, oim.hi);
                    ol[orow + x] = make_double2(ore.lo, oim.lo);
                }
            }
        }
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc::tc_fence_after();
        tc::tmem_dealloc(tmem, DT_TMEM_COLS);
    }
}

int planes_of(nslg_fm *fm, const ExpEntry *e, DdPlanes **out) {
    auto *E = const_cast<ExpEntry *>(e);
    if (!E->dd) {
        cudaStream_t st = fm->ctx->stream;
        const int Nx = (int)fm->Nx, ntn = (int)ceil_div(Nx, DT_BN), nkb = oz_ld(Nx) / OZ_KB;
        const size_t bytes = (size_t)ntn * nkb * D * DT_B_SLICE, nlist = (size_t)ntn * (nkb + 1);
        int *sums, *masks;
        NSLG_TRY(ws_get(fm, "ddtc_sums", (size_t)Nx * nkb, &sums));
        NSLG_TRY(ws_get(fm, "ddtc_masks", (size_t)ntn * nkb, &masks));
        auto *P = new DdPlanes;
        if (cudaMalloc(&P->planes, bytes) != cudaSuccess || cudaMalloc(&P->col_exp, Nx * sizeof(int)) != cudaSuccess ||
            cudaMalloc(&P->klist, nlist * sizeof(int)) != cudaSuccess) {
            cudaGetLastError();
            cudaFree(P->planes);
            cudaFree(P->col_exp);
            delete P;
            set_error("double-double digit planes: device allocation failed");
            return NSLG_ERR_OOM;
        }
        E->dd = P;  // freed with the entry
        NSLG_CUDA(cudaMemsetAsync(P->planes, 0, bytes, st));
        NSLG_CUDA(cudaMemsetAsync(sums, 0, (size_t)Nx * nkb * sizeof(int), st));
        NSLG_CUDA(cudaMemsetAsync(masks, 0, (size_t)ntn * nkb * sizeof(int), st));
        NSLG_CUDA(cudaMemsetAsync(P->klist, 0, nlist * sizeof(int), st));
        k_ddtc_planes<<<Nx, 256, 0, st>>>(E->full, static_cast<char *>(P->planes), P->col_exp, sums, masks, Nx, nkb);
        k_ddtc_klist<<<(unsigned)ceil_div(ntn, 32), 32, 0, st>>>(sums, masks, P->klist, Nx, ntn, nkb);
        note_launch(st, 2);
        NSLG_CUDA(cudaGetLastError());
        NSLG_CUDA(cudaFuncSetAttribute(k_fm_apply_ddtc<MODE_M>, cudaFuncAttributeMaxDynamicSharedMemorySize, DT_SMEM));
        NSLG_CUDA(cudaFuncSetAttribute(k_fm_apply_ddtc<MODE_MDAG>, cudaFuncAttributeMaxDynamicSharedMemorySize, DT_SMEM));
    }
    *out = E->dd;
    return NSLG_OK;
}

}  // namespace

// Measured, one M of a few vectors, CUDA cores and tensor cores: 4608 elements on 18 sites 349 and 44 us, 4096 on 64 sites 681
// and 51 us, 4608 on 72 sites 846 and 54 us. Below the line the tensor cores are ahead too (128 elements on 8 sites 172 and
// 35 us, 1024 on 64 sites 660 and 47 us): it is where they were first tried, not where the two forms meet.
bool ddtc_applies(const ExpEntry *e, int Nx, int64_t rows) {
    return e->is_real && Nx <= 2048 && rows * Nx >= 4096;
}

int fm_apply_ddtc(nslg_fm *fm, int mode, const ExpEntry *e, const double2 *xh, const double2 *xl, double2 *oh,
                  double2 *ol, int64_t rows, const int *sys_mask, int64_t sys_rows) {
    cudaStream_t st = fm->ctx->stream;
    const int Nt = (int)fm->Nt, Nx = (int)fm->Nx, nkb = oz_ld(Nx) / OZ_KB;
    DdPlanes *P;
    NSLG_TRY(planes_of(fm, e, &P));
    // The workspace (80 bytes per element) is bounded: longer vectors go through it in blocks of rows.
    const int64_t block = std::max<int64_t>(DT_BM / 2, DT_BLOCK_ELEMS / Nx / (DT_BM / 2) * (DT_BM / 2));
    const int64_t most = std::min(rows, block);
    char *dg;
    int *rexp;
    double2 *vh = nullptr, *vl = nullptr;
    NSLG_TRY(ws_get(fm, "ddtc_digits", (size_t)ceil_div(2 * most, DT_BM) * nkb * D * DT_A_SLICE, &dg));
    NSLG_TRY(ws_get(fm, "ddtc_rexp", (size_t)ceil_div(2 * most, DT_BM) * DT_BM, &rexp));
    if (mode == MODE_M) {
        NSLG_TRY(ws_get(fm, "ddtc_vh", (size_t)(most * Nx), &vh));
        NSLG_TRY(ws_get(fm, "ddtc_vl", (size_t)(most * Nx), &vl));
    }
    const auto *dga = reinterpret_cast<const uint8_t *>(dg), *dgb = static_cast<const uint8_t *>(P->planes);
    for (int64_t row0 = 0; row0 < rows; row0 += block) {
        const int64_t cnt = std::min(block, rows - row0);
        const unsigned blocks = (unsigned)ceil_div(cnt, 8);
        const int64_t tiles = ceil_div(cnt, DT_BM / 2) * ceil_div(Nx, DT_BN);
        const unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(tiles, std::max(1, num_sms())));
        if (mode == MODE_M) {
            k_ddtc_digits<MODE_M><<<blocks, 256, 0, st>>>(xh, xl, fm->phase, vh, vl, Nt, Nx, row0, cnt, nkb, dg, rexp,
                                                          sys_mask, sys_rows);
            k_fm_apply_ddtc<MODE_M><<<grid, DT_THREADS, DT_SMEM, st>>>(xh, xl, oh, ol, fm->phase, rexp, P->col_exp,
                                                                       P->klist, dga, dgb, Nt, Nx, row0, cnt, nkb,
                                                                       fm->tc_err, sys_mask, sys_rows);
        } else {
            k_ddtc_digits<MODE_MDAG><<<blocks, 256, 0, st>>>(xh, xl, nullptr, nullptr, nullptr, Nt, Nx, row0, cnt, nkb, dg,
                                                             rexp, sys_mask, sys_rows);
            k_fm_apply_ddtc<MODE_MDAG><<<grid, DT_THREADS, DT_SMEM, st>>>(xh, xl, oh, ol, fm->phase, rexp, P->col_exp,
                                                                          P->klist, dga, dgb, Nt, Nx, row0, cnt, nkb,
                                                                          fm->tc_err, sys_mask, sys_rows);
        }
        note_launch(st, 2);
        NSLG_CUDA(cudaGetLastError());
    }
    return NSLG_OK;
}

}  // namespace nslg
