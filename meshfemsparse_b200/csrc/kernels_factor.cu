// Numeric factorization kernels (K2 value injection, K3 POTRF, K4 TRSM,
// K5 Schur update + extend-add) for the multifrontal, level-scheduled
// supernodal Cholesky factorization.
//
// The reference delegates this stage to BlockCatamari's
// SparseLDL::RefactorWithFixedSparsityPattern (called at
// Solvers/CatamariFactorizer.cc:660): inject A (+ sigma I or sigma B) through
// the conversion plan, then a right-looking supernodal Cholesky where every
// supernode's Schur complement is merged into its parent through
// child_rel_indices. The GPU restatement keeps that structure:
//   * one injection pass over the plan (CatamariConversionPlan.hh:524-525);
//   * per elimination-tree level, small fronts are factored by one CTA each in
//     shared memory; large fronts run as tiled POTRF / TRSM / update kernels
//     whose task lists cover every large front of the level at once;
//   * a parent pulls its children's update matrices in child order
//     (deterministic, no atomics), so results are bit-identical run to run.
// Pivot failures never trap: the smallest failing column is recorded and the
// pivot replaced by 1 so the launch completes; the host turns it into
// the reference's "pivots successful" error (CatamariFactorizer.cc:701-705).
#include "device.h"

#include <cstdio>

namespace mfs {

namespace {

template <typename T>
__device__ __forceinline__ T dev_sqrt(T x);
template <>
__device__ __forceinline__ double dev_sqrt<double>(double x) { return sqrt(x); }
template <>
__device__ __forceinline__ float dev_sqrt<float>(float x) { return sqrtf(x); }

template <typename T>
__global__ void zero_kernel(T *p, int64_t n) {
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
        p[i] = T(0);
}

// K2: one thread per (plan entry, block component).
template <typename T>
__global__ void inject_kernel(const PlanEntryDev *__restrict__ plan, int64_t nplan, int vb, int src_ld,
                              const double *__restrict__ Ax, const double *__restrict__ Bx, double sigma_b,
                              T *__restrict__ factor) {
    const int vb2 = vb * vb;
    const int64_t total = nplan * vb2;
    for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t < total;
         t += int64_t(gridDim.x) * blockDim.x) {
        const int64_t e = t / vb2;
        const int comp = int(t - e * vb2);
        const int r = comp % vb, c = comp / vb;
        const PlanEntryDev pe = plan[e];
        if ((pe.flags & 2) && r < c) continue;   // diagonal block: lower part only
        const int64_t so = (pe.flags & 1) ? pe.src + int64_t(r) * src_ld + c : pe.src + int64_t(c) * src_ld + r;
        double v = Ax[so];
        if (Bx) v += sigma_b * Bx[so];
        factor[pe.dst + int64_t(c) * pe.ld + r] = T(v);
    }
}

template <typename T>
__global__ void diag_shift_kernel(const int64_t *__restrict__ diag_off, int64_t n, double sigma, T *factor) {
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
        factor[diag_off[i]] = T(double(factor[diag_off[i]]) + sigma);
}

__device__ __forceinline__ int child_rel(const int32_t *rel, int i, int vb) { return rel[i / vb] + i % vb; }

// A non-positive (or NaN) pivot. Without perturbation (plain solves, the
// reference's semantics) the smallest failing column is recorded and 1 is used
// so the launch completes; the host then reports the failure. With
// perturbation (the FP32 factor used as a preconditioner under FP64
// refinement) the pivot becomes max(|a|, kPivotFloor * A(col,col)) of the
// injected matrix, which keeps the factor SPD, and the event is counted.
constexpr double kPivotFloor = 1e-3;
template <typename T>
__device__ __forceinline__ T bad_pivot(T a, int col, const PivotCtl &pv, bool record) {
    if (pv.dorig) {
        const T floor_v = T(kPivotFloor * fabs(pv.dorig[col]));
        const T m = fabs(a);
        if (record) atomicAdd(pv.perturbed, 1);
        return (m > floor_v) ? m : (floor_v > T(0) ? floor_v : T(1));
    }
    if (record) atomicMin(pv.fail_col, col);
    return T(1);
}

template <typename T>
__global__ void extract_diag_kernel(const int64_t *__restrict__ diag_off, int64_t n, const T *__restrict__ factor,
                                    double *__restrict__ out) {
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
        out[i] = double(factor[diag_off[i]]);
}

// Small fronts: the whole (w+d)^2 front lives in shared memory.
template <typename T>
__global__ void __launch_bounds__(256) small_factor_kernel(const int32_t *__restrict__ list, SnDev sd,
                                                           T *__restrict__ factor, T *__restrict__ upd,
                                                           PivotCtl pv) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *F = reinterpret_cast<T *>(smem_raw);
    const int s = list[blockIdx.x];
    const int w = sd.w[s], d = sd.d[s], f = w + d;
    const int tid = threadIdx.x, nt = blockDim.x;
    T *pan = factor + sd.pan_off[s];
    const int ld = sd.ld[s];
    const int fw = f * w;
    for (int k = tid; k < f * f; k += nt) F[k] = k < fw ? pan[(k / f) * ld + k % f] : T(0);
    __syncthreads();
    const int vb = sd.vb;
    for (int ci = sd.child_ptr[s]; ci < sd.child_ptr[s + 1]; ++ci) {
        const int c = sd.child_list[ci];
        const int dc = sd.d[c];
        const T *U = upd + sd.upd_off[c];
        const int32_t *rel = sd.rel + sd.struct_ptr[c];
        for (int k = tid; k < dc * dc; k += nt) {
            const int j = k / dc, i = k - j * dc;
            if (i < j) continue;
            F[child_rel(rel, j, vb) * f + child_rel(rel, i, vb)] += U[k];
        }
        __syncthreads();
    }
    for (int k = 0; k < w; ++k) {
        T *colk = F + k * f;
        if (tid == 0) {
            T a = colk[k];
            if (!(a > T(0))) a = bad_pivot(a, sd.col0[s] + k, pv, true);
            colk[k] = dev_sqrt(a);
        }
        __syncthreads();
        const T piv = colk[k];
        for (int i = k + 1 + tid; i < f; i += nt) colk[i] = colk[i] / piv;
        __syncthreads();
        const int m = f - k - 1;
        for (int t = tid; t < m * m; t += nt) {
            const int jj = t / m, ii = t - jj * m;
            if (ii < jj) continue;
            const int j = k + 1 + jj, i = k + 1 + ii;
            F[j * f + i] -= colk[i] * colk[j];
        }
        __syncthreads();
    }
    for (int k = tid; k < fw; k += nt) pan[(k / f) * ld + k % f] = F[k];
    if (d > 0 && sd.upd_off[s] >= 0) {
        T *U = upd + sd.upd_off[s];
        for (int k = tid; k < d * d; k += nt) {
            const int j = k / d, i = k - j * d;
            U[k] = F[(w + j) * f + (w + i)];
        }
    }
}

// Extend-add of a large front: every element of its lower triangle is the injected value
// (panel columns) or zero (U_s) plus the children's update matrices, in child order, pulled
// through the children's inverse row maps. HBM-bound for the large fronts: each child's
// triangle is read and U_s written once (with scatters from the children U_s was zeroed
// whole and then read and written once per child: 4 d^2 against 1.5 d^2 elements for two
// children of the same size), latency-bound for the small ones. A thread has two rows of
// the tile's columns, eight columns at a time: 16 independent loads per child in flight at
// 4 (FP64 2) CTAs per SM, the row maps loaded once. (32 columns at once left one CTA per SM,
// 50 ms; tiles of 8 columns spent their time on the maps, 23 ms; tiles found by a search
// over the tasks and 512 rows for every front, 18.7 ms.)
// k = 64 in FP32 (23 launches): 22.3 ms before, 16.5 ms now; k = 20 in FP64: 53 us a
// launch before, 32 us now.
template <typename T, int VB, int NT, int RW>
__global__ void __launch_bounds__(NT, (sizeof(T) == 4 ? 1024 : 512) / NT)
    assemble_large_kernel(const AssembleTile *__restrict__ tiles, const AssembleTask *__restrict__ tasks, SnDev sd,
                          const AsmChild *__restrict__ children, const int32_t *__restrict__ cmap,
                          T *__restrict__ factor, T *upd) {
    const AssembleTile tile = tiles[blockIdx.x];
    const AssembleTask tk = tasks[tile.task];
    const int s = tk.sn;
    const int w = sd.w[s], d = sd.d[s], f = w + d, ld = sd.ld[s];
    const int c0 = tile.c0, r0 = tile.r0 + threadIdx.x;
    const int vb = VB > 0 ? VB : sd.vb;
    constexpr int G = 8;
    T *pan = factor + sd.pan_off[s];
    T *Us = d > 0 && sd.upd_off[s] >= 0 ? upd + sd.upd_off[s] : nullptr;
    // this thread's rows in a child (-1: none); kept for the first two children
    auto row_maps = [&](const AsmChild &ch, int (&mi)[RW]) {
#pragma unroll
        for (int q = 0; q < RW; ++q) {
            const int i = r0 + NT * q;
            mi[q] = -1;
            if (i < f) {
                const int b = i / vb, m = cmap[ch.map + b];
                if (m >= 0) mi[q] = m * vb + i - b * vb;
            }
        }
    };
    AsmChild kept[2];
    int kmi[2][RW];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        if (k >= tk.nchild) break;
        kept[k] = children[tk.child0 + k];
        row_maps(kept[k], kmi[k]);
    }
#pragma unroll 1
    for (int cg = c0; cg < min(f, c0 + kAsmCols); cg += G) {
        T acc[RW][G];
        unsigned touched = 0;                            // columns with a child's contribution
        // the panel's columns hold the injected values
#pragma unroll
        for (int q = 0; q < RW; ++q)
#pragma unroll
            for (int j = 0; j < G; ++j) {
                const int i = r0 + NT * q;
                acc[q][j] = T(0);
                if (cg + j < w && i >= cg + j && i < f) acc[q][j] = pan[int64_t(cg + j) * ld + i];
            }
        auto add = [&](const AsmChild &ch, const int (&mi)[RW]) {
            int mj[G], most = -1;                        // the columns in the child
#pragma unroll
            for (int j = 0; j < G; ++j) {
                mj[j] = -1;
                if (cg + j < f) {
                    const int b = (cg + j) / vb, m = cmap[ch.map + b];
                    if (m >= 0) mj[j] = m * vb + (cg + j) - b * vb;
                }
                most = max(most, mj[j]);
            }
            if (most < 0) return;                        // (the same for every thread)
            const T *U = upd + ch.upd;
            T v[RW][G];
#pragma unroll
            for (int j = 0; j < G; ++j) {
                if (mj[j] >= 0) touched |= 1u << j;
                const T *col = U + int64_t(mj[j]) * ch.d;
#pragma unroll
                for (int q = 0; q < RW; ++q) {
                    v[q][j] = T(0);
                    if (mj[j] >= 0 && mi[q] >= mj[j]) v[q][j] = col[mi[q]];
                }
            }
#pragma unroll
            for (int q = 0; q < RW; ++q)
#pragma unroll
                for (int j = 0; j < G; ++j) acc[q][j] += v[q][j];
        };
#pragma unroll
        for (int k = 0; k < 2; ++k)
            if (k < tk.nchild) add(kept[k], kmi[k]);
        for (int ci = 2; ci < tk.nchild; ++ci) {
            const AsmChild ch = children[tk.child0 + ci];
            int mi[RW];
            row_maps(ch, mi);
            add(ch, mi);
        }
#pragma unroll
        for (int j = 0; j < G; ++j) {
            const int col = cg + j;
#pragma unroll
            for (int q = 0; q < RW; ++q) {
                const int i = r0 + NT * q;
                if (col >= f || i < col || i >= f) continue;
                if (col >= w) Us[int64_t(col - w) * d + (i - w)] = acc[q][j];
                else if (touched >> j & 1) pan[int64_t(col) * ld + i] = acc[q][j];
            }
        }
    }
}

inline int grid_for(int64_t n, int threads) {
    int64_t g = (n + threads - 1) / threads;
    if (g > 148 * 32) g = 148 * 32;
    if (g < 1) g = 1;
    return int(g);
}

}  // namespace

template <typename T>
void launch_zero(T *p, int64_t n, cudaStream_t st) {
    if (n <= 0) return;
    ++g_kernel_launches;
    zero_kernel<T><<<grid_for(n, 256), 256, 0, st>>>(p, n);
}

template <typename T>
void launch_inject(const PlanEntryDev *plan, int64_t nplan, int vb, int src_ld, const double *Ax, const double *Bx,
                   double sigma_b, T *factor, cudaStream_t st) {
    if (nplan <= 0) return;
    ++g_kernel_launches;
    inject_kernel<T><<<grid_for(nplan * vb * vb, 256), 256, 0, st>>>(plan, nplan, vb, src_ld, Ax, Bx, sigma_b,
                                                                      factor);
}

template <typename T>
void launch_diag_shift(const int64_t *diag_off, int64_t n, double sigma, T *factor, cudaStream_t st) {
    if (n <= 0) return;
    ++g_kernel_launches;
    diag_shift_kernel<T><<<grid_for(n, 256), 256, 0, st>>>(diag_off, n, sigma, factor);
}

template <typename T>
void launch_small_factor(const int32_t *list, int count, int max_front, SnDev sd, T *factor, T *upd, PivotCtl pv,
                         cudaStream_t st) {
    if (count <= 0) return;
    const size_t smem = size_t(max_front) * max_front * sizeof(T);
    static PerDeviceOnce once;
    once([] { cudaFuncSetAttribute(small_factor_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmemOptin); });
    ++g_kernel_launches;
    small_factor_kernel<T><<<count, 256, smem, st>>>(list, sd, factor, upd, pv);
}

template <typename T>
void launch_assemble_large(const AssembleTile *tiles, int ntiles, int tile_rows, const AssembleTask *tasks, SnDev sd,
                           const AsmChild *children, const int32_t *cmap, T *factor, T *upd, cudaStream_t st) {
    if (ntiles <= 0) return;
    ++g_kernel_launches;
    auto go = [&](auto narrow, auto wide) {
        if (tile_rows == kAsmRowsSmall) narrow<<<ntiles, 128, 0, st>>>(tiles, tasks, sd, children, cmap, factor, upd);
        else wide<<<ntiles, 256, 0, st>>>(tiles, tasks, sd, children, cmap, factor, upd);
    };
    static_assert(kAsmRowsSmall == 128 && kAsmRows == 512, "rows of a tile: threads x rows per thread");
    if (sd.vb == 3) go(assemble_large_kernel<T, 3, 128, 1>, assemble_large_kernel<T, 3, 256, 2>);
    else if (sd.vb == 1) go(assemble_large_kernel<T, 1, 128, 1>, assemble_large_kernel<T, 1, 256, 2>);
    else go(assemble_large_kernel<T, 0, 128, 1>, assemble_large_kernel<T, 0, 256, 2>);
}

template <typename T>
void launch_extract_diag(const int64_t *diag_off, int64_t n, const T *factor, double *out, cudaStream_t st) {
    if (n <= 0) return;
    ++g_kernel_launches;
    extract_diag_kernel<T><<<grid_for(n, 256), 256, 0, st>>>(diag_off, n, factor, out);
}

#define MFS_INSTANTIATE(T)                                                                                        \
    template void launch_zero<T>(T *, int64_t, cudaStream_t);                                                      \
    template void launch_inject<T>(const PlanEntryDev *, int64_t, int, int, const double *, const double *, double, \
                                   T *, cudaStream_t);                                                            \
    template void launch_diag_shift<T>(const int64_t *, int64_t, double, T *, cudaStream_t);                       \
    template void launch_small_factor<T>(const int32_t *, int, int, SnDev, T *, T *, PivotCtl, cudaStream_t);      \
    template void launch_assemble_large<T>(const AssembleTile *, int, int, const AssembleTask *, SnDev,            \
                                           const AsmChild *, const int32_t *, T *, T *, cudaStream_t);                                               \
    template void launch_extract_diag<T>(const int64_t *, int64_t, const T *, double *, cudaStream_t);

MFS_INSTANTIATE(double)
MFS_INSTANTIATE(float)


namespace {
// One CTA per front: the largest injected diagonal over the front's rows (its own
// columns and its structure rows), then the exponent that keeps its square root
// below 2^12.
__global__ void __launch_bounds__(256) front_scale_kernel(const int32_t *__restrict__ fronts, SnDev sd,
                                                          const double *__restrict__ diag, int32_t *__restrict__ sexp) {
    const int s = fronts[blockIdx.x];
    const int w = sd.w[s], d = sd.d[s], c0 = sd.col0[s], vb = sd.vb;
    const int32_t *rows = sd.struct_rows + sd.struct_ptr[s];
    double m = 0.0;
    for (int i = threadIdx.x; i < w + d; i += blockDim.x) {
        const int r = i < w ? c0 + i : rows[(i - w) / vb] * vb + (i - w) % vb;
        m = fmax(m, fabs(diag[r]));
    }
    __shared__ double red[256];
    red[threadIdx.x] = m;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + o]);
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const double mx = red[0];
        sexp[s] = (mx > 0.0 && isfinite(mx)) ? ilogb(sqrt(mx)) + 1 - 12 : 0;
    }
}
}  // namespace

void launch_front_scale(const int32_t *fronts, int nfronts, SnDev sd, const double *diag, int32_t *sexp,
                        cudaStream_t st) {
    if (nfronts <= 0) return;
    ++g_kernel_launches;
    front_scale_kernel<<<nfronts, 256, 0, st>>>(fronts, sd, diag, sexp);
}

}  // namespace mfs
