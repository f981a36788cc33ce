// Large-front column block, first half of K3 + K4: factor the nb x nb
// diagonal block of one column block and invert it.
//
// One launch per column block of all large fronts of a level, one CTA per
// front. The CTA factors the block in shared memory, writes L back in place,
// stores the full inverse inv(L) (nb x nb, column-major, ld ldi) to scratch and
// the 64 x 64 diagonal blocks of inv(L) after the panels for the triangular
// solves. The rows below the block are then solved on the tensor cores as the
// GEMM  X := X inv(L)^T  (launched by the host right after this kernel), so
// the O(m nb^2) part of the TRSM runs at GEMM speed.
//
// The block (padded to a multiple of 32 with an identity tail) is processed in
// 32 x 32 tiles I = 0 .. nblk-1, right-looking, three barriers per tile column:
//   phase A  the tiles below, L_RI = A_RI inv(L_II)^T, and the inverse tiles
//            inv(L)_IJ = -inv(L_II) sum_K P_IJK (J < I), in halves of 16 columns, one
//            warp each;
//   phase B  tile (I+1, I+1) -= L_{I+1,I} L_{I+1,I}^T, four columns a warp;
//   phase C  warp 0 factors tile (I+1, I+1) (lane = row) and warp 1 inverts it (lane =
//            column) four pivots behind; warps 2-7 meanwhile run the other trailing
//            updates A_RC -= L_RI L_CI^T (R >= C > I) and the products
//            P_{I+1,J,K} = L_{I+1,K} inv(L)_KJ (J <= K <= I) that the next
//            off-diagonal inverse tiles need (they only read final tiles).
// What bounds it is the chain of pivots of one warp: everything else is split over the
// warps so that it does not lengthen the chain. Clocks at 128 columns in FP32: 84,800
// with whole-tile products on the chain, the inverse in the factoring warp and
// four-way bank conflicts in the load; 67,600 now (47 -> 35 us a launch). At 64 columns
// in FP64: 47,300 and 35,500 (32 -> 19 us).
// The code is kept compact (rolled loops): the work per CTA is small, and fully unrolled
// variants spent most of their time refetching instructions.
#include "device.h"

#include <type_traits>

namespace mfs {

namespace {

constexpr int kPanelThreads = 256;

template <typename T>
struct Vec16;
template <>
struct Vec16<float> {
    using type = float4;
};
template <>
struct Vec16<double> {
    using type = double2;
};

template <typename T>
__device__ __forceinline__ T recip_sqrt(T x);
template <>
__device__ __forceinline__ double recip_sqrt<double>(double x) { return rsqrt(x); }
template <>
__device__ __forceinline__ float recip_sqrt<float>(float x) { return rsqrtf(x); }

// inv(L) feeding a single-pass TF32 tensor-core row solve is stored rounded to
// TF32 (nearest); the tensor cores would truncate it.
template <typename T>
__device__ __forceinline__ T round_operand(T x) { return x; }
template <>
__device__ __forceinline__ float round_operand<float>(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
}

// Largest value of type T at or below x (x >= 0): p > x in FP64 exactly when p > down(x).
template <typename T>
__device__ __forceinline__ T round_down(double x);
template <>
__device__ __forceinline__ double round_down<double>(double x) { return x; }
template <>
__device__ __forceinline__ float round_down<float>(double x) { return __double2float_rd(x); }

// Warp-level tile product: c[r][q] += sum_{k < 32} A(4 rq + r, k) * B(NC cq + q, k) with
// rq = lane % 8, cq = lane / 8: 32 rows, 4 NC columns; A(i, k) = A0[k * lda + i],
// B(j, k) = B0[j * sj + k * sk].
template <typename T, int NC>
__device__ __forceinline__ void tile_mma(T (&c)[4][NC], const T *A0, int lda, const T *B0, int sj, int sk, int lane) {
    const int rq = lane & 7, cq = lane >> 3;
    const T *a = A0 + 4 * rq;
    const T *b = B0 + NC * cq * sj;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int q = 0; q < NC; ++q) c[r][q] = T(0);
#pragma unroll 4
    for (int k = 0; k < 32; ++k) {
        T av[4], bv[NC];
#pragma unroll
        for (int r = 0; r < 4; ++r) av[r] = a[k * lda + r];
#pragma unroll
        for (int q = 0; q < NC; ++q) bv[q] = b[q * sj + k * sk];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int q = 0; q < NC; ++q) c[r][q] += av[r] * bv[q];
    }
}

// Store a lane's 4 x NC patch into a column-major tile (element (i, j) at M[j * ldm + i]),
// scaled by s (and added to the old value when add is set).
template <typename T, int NC>
__device__ __forceinline__ void tile_store(T *M, int ldm, const T (&c)[4][NC], T s, bool add, int lane) {
    const int rq = lane & 7, cq = lane >> 3;
#pragma unroll
    for (int q = 0; q < NC; ++q)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            T *p = M + (NC * cq + q) * ldm + 4 * rq + r;
            *p = add ? *p + s * c[r][q] : s * c[r][q];
        }
}

// Pivot rule of a diagonal tile, one lane per column: a bad pivot (at or below `tiny`, or
// NaN) is replaced (by 1, or under refinement by the larger of its magnitude and `floor`)
// and remembered by the lane; what it means is settled after the tile.
template <typename T>
struct PivotRule {
    T tiny, floor;
    bool perturb, bad;
    __device__ __forceinline__ T operator()(T p, bool mine) {
        const bool b = !(p > tiny);
        const T m = fabs(p);
        const T sub = !perturb ? T(1) : m > floor ? m : floor > T(0) ? floor : T(1);
        bad |= b & mine;
        return b ? sub : p;
    }
};

// The four columns under way go from the factoring to the inverting warp (and back to its
// own lanes) through two buffers of Lq: [32 rows][4] of L, then the four reciprocal pivots.
constexpr int kLq = 32 * 4 + 4;
__device__ __forceinline__ void pair_sync() { asm volatile("bar.sync 2, 64;" ::: "memory"); }

template <typename T>
__device__ __forceinline__ void load4(T (&c)[4], const T *p) {
    using V = typename Vec16<T>::type;
    constexpr int E = 16 / int(sizeof(T));
#pragma unroll
    for (int v = 0; v < 4 / E; ++v) *reinterpret_cast<V *>(&c[v * E]) = reinterpret_cast<const V *>(p)[v];
}
template <typename T>
__device__ __forceinline__ void store4(T *p, const T (&c)[4]) {
    using V = typename Vec16<T>::type;
    constexpr int E = 16 / int(sizeof(T));
#pragma unroll
    for (int v = 0; v < 4 / E; ++v) reinterpret_cast<V *>(p)[v] = *reinterpret_cast<const V *>(&c[v * E]);
}

// Pivots k0 .. k0 + 3 of a diagonal tile, with LEN columns left. r[j] = A(lane, k0 + j). The
// four columns are updated among themselves through shuffles; the rank-4 update that the
// four before left pending on r[4 ..] (l4, Lq buffer `old`) fills the chain's latency; what
// the next four need of these is done at the end.
template <typename T, int LEN>
__device__ __forceinline__ void factor_steps(T (&r)[32], T (&l4)[4], T &piv, PivotRule<T> &rule, int k0, T *Dt, T *Lq,
                                             int LDD, int lane) {
    constexpr int P = (LEN - 4) / 4;                 // pending columns per pivot
    const T *old = Lq + (((k0 >> 2) & 1) ^ 1) * kLq;
    T *cur = Lq + ((k0 >> 2) & 1) * kLq;
    T l[4], rs[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        const int k = k0 + t;
        rs[t] = recip_sqrt(piv);
        l[t] = (lane == k) ? piv * rs[t] : r[t] * rs[t];
        if (t < 3) {
            // the next pivot, on its own lane: nothing else of this step is on the chain
            piv = __shfl_sync(0xffffffffu, rule(r[t + 1] - l[t] * l[t], lane == k + 1), k + 1);
        }
#pragma unroll
        for (int u = t + 1; u < 4; ++u) r[u] -= l[t] * __shfl_sync(0xffffffffu, l[t], k0 + u);
        if (lane >= k) Dt[k * LDD + lane] = l[t];
#pragma unroll
        for (int j = 4 + t * P; j < 4 + (t + 1) * P; ++j) {
            T c[4];                                  // (rows past the tile: not used later)
            load4(c, old + ((k0 + j) & 31) * 4);
#pragma unroll
            for (int e = 0; e < 4; ++e) r[j] -= l4[e] * c[e];
        }
    }
    store4(cur + lane * 4, l);
    if (lane == 0) store4(cur + 128, rs);
    pair_sync();
    // the next four columns, and their first pivot
#pragma unroll
    for (int j = 4; j < 8; ++j) {
        T c[4];
        load4(c, cur + ((k0 + j) & 31) * 4);
#pragma unroll
        for (int e = 0; e < 4; ++e) r[j] -= l[e] * c[e];
    }
    piv = __shfl_sync(0xffffffffu, rule(r[4], lane == k0 + 4), (k0 + 4) & 31);
#pragma unroll
    for (int j = 0; j < LEN - 4; ++j) r[j] = r[j + 4];
#pragma unroll
    for (int e = 0; e < 4; ++e) l4[e] = l[e];
}

// The inverting warp's part of the same pivots: lane = column, y[j] = Y(k0 + j, lane);
// Y_k = y[t] / L(k, k), then y[j] -= L(k0 + j, k) Y_k.
template <typename T, int LEN>
__device__ __forceinline__ void invert_steps(T (&y)[32], int k0, T *It, const T *Lq, int LDD, int lane) {
    const T *cur = Lq + ((k0 >> 2) & 1) * kLq;
    pair_sync();
    T rs[4], yk[4];
    load4(rs, cur + 128);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        T c[4];
        load4(c, cur + (k0 + t) * 4);
#pragma unroll
        for (int e = 0; e < t; ++e) y[t] -= c[e] * yk[e];
        yk[t] = y[t] * rs[t];
        if (k0 + t >= lane) It[lane * LDD + k0 + t] = yk[t];
    }
#pragma unroll
    for (int j = 4; j < LEN; ++j) {
        T c[4];
        load4(c, cur + ((k0 + j) & 31) * 4);
#pragma unroll
        for (int e = 0; e < 4; ++e) y[j] -= c[e] * yk[e];
    }
#pragma unroll
    for (int j = 0; j < LEN - 4; ++j) y[j] = y[j + 4];
}

// Cholesky of the 32 x 32 tile at (c0, c0) of D by warp 0 and its inverse by warp 1. The
// 32-entry register vectors are taken four entries at a time and then shifted by four, so
// that every register index is static in a rolled loop; the second half holds 16. Clocks of
// a tile: FP32 7,300, FP64 10,500 (9,829 and 12,214 with both in one warp and a
// shared-memory round trip a pivot).
template <typename T>
__device__ __noinline__ void factor_tile(T *D, T *Lq, int LDD, int c0, int nb, int lane, int col_base, int *fail_col,
                                         int *perturbed, const double *dorig, int *sflag) {
    T *Dt = D + c0 * LDD + c0;                       // tile element (i, j) at Dt[j * LDD + i]
    T r[32], l4[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll
    for (int j = 0; j < 32; ++j) r[j] = (j <= lane) ? Dt[j * LDD + lane] : T(0);
    store4(Lq + kLq + lane * 4, l4);                 // (nothing is pending at first)
    __syncwarp();
    const bool in = c0 + lane < nb;                  // (columns past nb are the identity's)
    const int col = col_base + c0 + lane;
    const double d = (dorig && in) ? fabs(dorig[col]) : 0.0;
    // with an FP64 re-factor pending (sflag) a tiny pivot is bad too; the identity's are not
    const T tiny = !in ? T(-1) : sflag ? round_down<T>(kRefactorTiny * d) : T(0);
    PivotRule<T> rule{tiny, T(1e-3 * d), dorig != nullptr, false};
    T piv = __shfl_sync(0xffffffffu, rule(r[0], lane == 0), 0);
#pragma unroll 1
    for (int k0 = 0; k0 < 16; k0 += 4) factor_steps<T, 32>(r, l4, piv, rule, k0, Dt, Lq, LDD, lane);
#pragma unroll 1
    for (int k0 = 16; k0 < 32; k0 += 4) factor_steps<T, 16>(r, l4, piv, rule, k0, Dt, Lq, LDD, lane);
    if (rule.bad) {
        // the same rule as the small-front kernel: report (plain) or perturb (refined FP32);
        // a block to be factored again in FP64 is only marked
        if (sflag) *sflag = 1;
        else if (dorig) atomicAdd(perturbed, 1);
        else atomicMin(fail_col, col);
    }
}
template <typename T>
__device__ __noinline__ void invert_tile(T *Iv, const T *Lq, int LDD, int c0, int lane) {
    T *It = Iv + c0 * LDD + c0;
    T y[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) y[j] = (j == lane) ? T(1) : T(0);
#pragma unroll 1
    for (int k0 = 0; k0 < 16; k0 += 4) invert_steps<T, 32>(y, k0, It, Lq, LDD, lane);
#pragma unroll 1
    for (int k0 = 16; k0 < 32; k0 += 4) invert_steps<T, 16>(y, k0, It, Lq, LDD, lane);
}

// FP64 re-factor of one FP32 diagonal block whose FP32 factorization met a
// non-positive or tiny pivot (pivot <= kRefactorTiny * injected diagonal): the
// block's stored (assembled and updated) values are factored by right-looking
// Cholesky in FP64 and inverted in place (lower-triangular inverse, columns from
// the last), then L, inv(L) (rounded for the tensor-core row solve when asked) and
// the 64 x 64 diagonal inverses are written as the FP32 pass would have. A pivot
// that stays non-positive in FP64 takes the refinement floor and is counted.
// Shared memory: the block as doubles (ld nb + 1) and one column of scratch.
template <typename T>
__device__ __noinline__ void refactor_block_fp64(const PanelTask &tk, T *blk, T *inv_scratch, T *factor,
                                                 const PivotCtl &pv, bool round_inv, unsigned char *smem) {
    const int nb = tk.nb, ld = tk.ld, LD = nb + 1;
    const int tid = threadIdx.x, nt = blockDim.x;
    double *F = reinterpret_cast<double *>(smem);          // (i, j) at F[j * LD + i]
    double *tmp = F + nb * LD;
    __shared__ double pivot;
    for (int q = tid; q < nb * nb; q += nt) {
        const int j = q / nb, i = q - j * nb;
        F[j * LD + i] = i >= j ? double(blk[int64_t(j) * ld + i]) : 0.0;
    }
    __syncthreads();
    for (int k = 0; k < nb; ++k) {
        if (tid == 0) {
            double p = F[k * LD + k];
            if (!(p > 0.0)) {
                const double fl = 1e-3 * fabs(pv.dorig[tk.col + k]);
                p = fabs(p) > fl ? fabs(p) : (fl > 0.0 ? fl : 1.0);
                atomicAdd(pv.perturbed, 1);
            }
            pivot = sqrt(p);
            F[k * LD + k] = pivot;
        }
        __syncthreads();
        const double rp = 1.0 / pivot;
        for (int i = k + 1 + tid; i < nb; i += nt) F[k * LD + i] *= rp;
        __syncthreads();
        const int m = nb - k - 1;
        for (int q = tid; q < m * m; q += nt) {
            const int j = k + 1 + q / m, i = k + 1 + q % m;
            if (i >= j) F[j * LD + i] -= F[k * LD + i] * F[k * LD + j];
        }
        __syncthreads();
    }
    for (int q = tid; q < nb * nb; q += nt) {
        const int j = q / nb, i = q - j * nb;
        if (i >= j) blk[int64_t(j) * ld + i] = T(F[j * LD + i]);
    }
    __syncthreads();
    // inv(L) in place: column j below the diagonal = -(1 / L_jj) inv(L_22) L(j+1:, j)
    for (int j = nb - 1; j >= 0; --j) {
        if (tid == 0) F[j * LD + j] = 1.0 / F[j * LD + j];
        __syncthreads();
        const double ajj = -F[j * LD + j];
        for (int i = j + 1 + tid; i < nb; i += nt) {
            double acc = 0.0;
            for (int k = j + 1; k <= i; ++k) acc += F[k * LD + i] * F[j * LD + k];
            tmp[i] = acc;
        }
        __syncthreads();
        for (int i = j + 1 + tid; i < nb; i += nt) F[j * LD + i] = tmp[i] * ajj;
        __syncthreads();
    }
    for (int q = tid; q < nb * nb; q += nt) {
        const int j = q / nb, i = q - j * nb;
        const T v = i >= j ? T(F[j * LD + i]) : T(0);
        inv_scratch[tk.inv_full + int64_t(j) * tk.ldi + i] = round_inv ? round_operand(v) : v;
    }
    if (tk.inv_out >= 0) {
        const int nb64 = (nb + 63) / 64;
        T *inv = factor + tk.inv_out;
        for (int q = tid; q < nb64 * 4096; q += nt) {
            const int b = q >> 12, e = q & 4095;
            const int j = e >> 6, i = e & 63;
            const int gi = b * 64 + i, gj = b * 64 + j;
            inv[q] = (gi < nb && gj < nb && gi >= gj) ? T(F[gj * LD + gi]) : T(0);
        }
    }
    if (tid == 0) atomicAdd(pv.refactored, 1);
}

template <typename T>
__global__ void __launch_bounds__(kPanelThreads, 1) panel_kernel(const PanelTask *__restrict__ tasks,
                                                                 T *__restrict__ factor, T *__restrict__ inv_scratch,
                                                                 PivotCtl pv, bool round_inv) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const PanelTask tk = tasks[blockIdx.x];
    const int nb = tk.nb, ld = tk.ld;
    const int nblk = (nb + 31) / 32, NBP = nblk * 32;
    const int LDD = NBP + 1;
    T *Lq = reinterpret_cast<T *>(smem_raw);         // 2 x kLq: columns of a diagonal tile in work (16-byte aligned)
    T *D = Lq + 2 * kLq;                             // L, column-major, ld LDD (identity-padded)
    T *Iv = D + NBP * LDD;                           // inv(L), column-major, ld LDD
    T *P = Iv + NBP * LDD;                           // 6 x [32][33] partial products
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5;
    T *blk = factor + tk.off;
    __shared__ int refactor_flag;
    int *sflag = (std::is_same<T, float>::value && pv.refactored && pv.dorig) ? &refactor_flag : nullptr;
    if (tid == 0) refactor_flag = 0;
    // Load: a warp takes every eighth column, lane = row, the rows' four segments of 32; eight
    // columns' loads are issued before the first shared-memory store (neither the loads nor
    // the stores collide). Nothing above the diagonal is read.
    for (int jb = warp; jb < NBP; jb += 64) {
        T v[8][4];
#pragma unroll
        for (int u = 0; u < 8; ++u)
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                const int j = jb + 8 * u, i = 32 * g + lane;
                v[u][g] = (i == j) ? T(1) : T(0);
                if (i >= j && i < nb && j < nb) v[u][g] = blk[int64_t(j) * ld + i];
            }
#pragma unroll
        for (int u = 0; u < 8; ++u)
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                const int j = jb + 8 * u, i = 32 * g + lane;
                if (j < NBP && i < NBP) {
                    D[j * LDD + i] = v[u][g];
                    Iv[j * LDD + i] = T(0);
                }
            }
    }
    __syncthreads();
    auto diag = [&](int I) {
        if (warp == 0)
            factor_tile(D, Lq, LDD, 32 * I, nb, lane, tk.col, pv.fail_col, pv.perturbed, pv.dorig, sflag);
        else if (warp == 1)
            invert_tile(Iv, Lq, LDD, 32 * I, lane);
    };
    diag(0);
    __syncthreads();
    for (int I = 0; I < nblk; ++I) {
        const int c0 = 32 * I;
        // ---- phase A: tiles below (L_RI) and off-diagonal inverse tiles (inv(L)_IJ), in
        //      halves of 16 columns; a tile below is replaced, so its halves wait for each other
        {
            const int nbelow = nblk - 1 - I, nhalf = 2 * (nbelow + I);
            // T_IJ = sum_{K=J}^{I-1} P_IJK, gathered into the K = J slot
            if (I > 1) {
                for (int J = 0; J + 1 < I; ++J) {
                    T *Pj = P + (J * (J + 1) / 2 + J) * 32 * 33;
                    for (int e = tid; e < 32 * 33; e += nt) {
                        T sum = Pj[e];
                        for (int K = J + 1; K < I; ++K) sum += P[(K * (K + 1) / 2 + J) * 32 * 33 + e];
                        Pj[e] = sum;
                    }
                }
                __syncthreads();
            }
            T c[4][4];
            const int u = warp >> 1, h = 16 * (warp & 1);
            if (warp < nhalf) {
                if (u < nbelow) {
                    // B(j, k) = inv(L_II)(j, k)
                    tile_mma(c, D + c0 * LDD + 32 * (I + 1 + u), LDD, Iv + c0 * LDD + c0 + h, 1, LDD, lane);
                } else {
                    // B(j, t) = T_IJ(t, j)
                    const int J = u - nbelow;
                    tile_mma(c, Iv + c0 * LDD + c0, LDD, P + (J * (J + 1) / 2 + J) * 32 * 33 + h * 33, 33, 1, lane);
                }
            }
            __syncthreads();
            if (warp < nhalf) {
                if (u < nbelow) tile_store(D + (c0 + h) * LDD + 32 * (I + 1 + u), LDD, c, T(1), false, lane);
                else tile_store(Iv + (32 * (u - nbelow) + h) * LDD + c0, LDD, c, T(-1), false, lane);
            }
        }
        __syncthreads();
        if (I + 1 == nblk) break;
        // ---- phase B: the next diagonal tile's update, lane = row, four columns a warp
        {
            const T *Lr = D + c0 * LDD + c0 + 32;
            T sum[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll 8
            for (int k = 0; k < 32; ++k) {
                const T a = Lr[k * LDD + lane];
#pragma unroll
                for (int q = 0; q < 4; ++q) sum[q] += a * Lr[k * LDD + 4 * warp + q];
            }
            T *Dn = D + (c0 + 32 + 4 * warp) * LDD + c0 + 32 + lane;
#pragma unroll
            for (int q = 0; q < 4; ++q) Dn[q * LDD] -= sum[q];
        }
        __syncthreads();
        // ---- phase C: that tile factored and inverted; the other trailing updates of tile
        //      column I; products for the next inverse tiles
        if (warp < 2) {
            diag(I + 1);
        } else {
            const int m = nblk - 1 - I;                          // trailing tile rows / columns
            const int ntrail = m * (m + 1) / 2;                  // u = 0 is tile (I+1, I+1)
            const int nterm = (I + 1) * (I + 2) / 2;             // P_{I+1,J,K}, J <= K <= I
            for (int u = warp - 1; u < ntrail + nterm; u += 6) {
                T c[4][8];
                if (u < ntrail) {
                    int a = 0;
                    while ((a + 1) * (a + 2) / 2 <= u) ++a;
                    const int R = I + 1 + a, C = I + 1 + (u - a * (a + 1) / 2);   // R >= C
                    // B(j, k) = L_CI(j, k)
                    tile_mma(c, D + c0 * LDD + 32 * R, LDD, D + c0 * LDD + 32 * C, 1, LDD, lane);
                    tile_store(D + (32 * C) * LDD + 32 * R, LDD, c, T(-1), true, lane);
                } else {
                    const int t = u - ntrail;                     // t = K (K + 1) / 2 + J
                    int K = 0;
                    while ((K + 1) * (K + 2) / 2 <= t) ++K;
                    const int J = t - K * (K + 1) / 2;
                    // B(j, k) = inv(L)_KJ(k, j)
                    tile_mma(c, D + (32 * K) * LDD + 32 * (I + 1), LDD, Iv + (32 * J) * LDD + 32 * K, LDD, 1, lane);
                    tile_store(P + t * 32 * 33, 33, c, T(1), false, lane);
                }
            }
        }
        __syncthreads();
    }
    if (sflag) {
        __syncthreads();
        if (refactor_flag) {
            // the block has not been written back: factor its stored values again in FP64
            refactor_block_fp64(tk, blk, inv_scratch, factor, pv, round_inv, smem_raw);
            return;
        }
    }
    // L (lower triangle only: the strict upper part keeps its stored values), inv(L) (zeros
    // above the diagonal) and the 64 x 64 diagonal blocks of inv(L) (the inverses of L's
    // 64 x 64 diagonal blocks, zero past nb), a column a warp, lane = row
    T *inv = tk.inv_out >= 0 ? factor + tk.inv_out : nullptr;
    const int nb64 = (nb + 63) & ~63;
    for (int j = warp; j < nb64; j += 8) {
        T *dl = blk + int64_t(j) * ld;
        T *di = inv_scratch + tk.inv_full + int64_t(j) * tk.ldi;
        T *d64 = inv ? inv + (j >> 6) * 4096 + (j & 63) * 64 - (j & ~63) : nullptr;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            const int i = 32 * g + lane;
            if (i >= nb64) continue;
            const bool live = i < nb && j < nb;
            const T y = live && i >= j ? Iv[j * LDD + i] : T(0);
            if (live) {
                di[i] = round_inv ? round_operand(y) : y;
                if (i >= j) dl[i] = D[j * LDD + i];
            }
            if (d64 && (i >> 6) == (j >> 6)) d64[i] = y;
        }
    }
}

}  // namespace

size_t panel_smem_bytes(int nb, bool fp64) {
    const size_t el = fp64 ? 8 : 4;
    const size_t nbp = size_t((nb + 31) / 32) * 32;
    return (2 * kLq + 2 * nbp * (nbp + 1) + 6 * 32 * 33) * el;
}

template <typename T>
void launch_panel(const PanelTask *tasks, int ntasks, int max_nb, T *factor, T *inv_scratch, PivotCtl pv,
                  bool round_inv, cudaStream_t st) {
    if (ntasks <= 0) return;
    const size_t smem = panel_smem_bytes(max_nb, sizeof(T) == 8);
    // the opt-in limit counts static shared memory too
    static PerDeviceOnce once;
    once([] {
        cudaFuncAttributes fa{};
        cudaFuncGetAttributes(&fa, panel_kernel<T>);
        cudaFuncSetAttribute(panel_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kMaxSmemOptin - int(fa.sharedSizeBytes));
    });
    ++g_kernel_launches;
    panel_kernel<T><<<ntasks, kPanelThreads, smem, st>>>(tasks, factor, inv_scratch, pv, round_inv);
}

template void launch_panel<float>(const PanelTask *, int, int, float *, float *, PivotCtl, bool, cudaStream_t);
template void launch_panel<double>(const PanelTask *, int, int, double *, double *, PivotCtl, bool, cudaStream_t);

}  // namespace mfs
