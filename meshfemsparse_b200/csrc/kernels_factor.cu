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
__device__ __forceinline__ T dev_rsqrt(T x);
template <>
__device__ __forceinline__ double dev_rsqrt<double>(double x) { return rsqrt(x); }
template <>
__device__ __forceinline__ float dev_rsqrt<float>(float x) { return rsqrtf(x); }

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

// Small fronts: the front's lower triangle lives in shared memory, packed by columns.
// Assembly pulls the children through their inverse row maps (a warp has four columns, a
// lane the rows lane + 32 g); the factorization takes four columns at a time: every thread
// factors the 4 x 4 diagonal block for itself, one thread per row solves the row against it
// (to the factor and to Lp), then the rank-4 update of the trailing triangle, a warp per
// column. Two barriers per four columns; bound by the chain of pivots (four reciprocal square
// roots in a row) for narrow fronts and by the triangle's read and write in shared memory
// for wide ones, hence rank 4 and not 1. With rank-1 steps, a division per element and three
// barriers a column over the whole square the 20-sided cube took 587 us in FP64 (5
// launches), 150 us now; the batch of 48 cubes in FP32 4,550 us (9 launches), 1,255 us now.
constexpr int kSmallCols = 4;

// Column c of block row b of a front of ManyDev (its list: entries e0 to e1 - 1): a warp calls
// add(front row, value) over each child's rows from the column's own on, in child order. 32
// list entries and their children are loaded at a time, a lane each, then the values of four
// children before the first is added: what is left between two adds is the add.
template <typename T, typename Add>
__device__ __forceinline__ void many_column(const ManyDev &many, const AsmChild *__restrict__ children, const T *upd,
                                            int64_t e0, int64_t e1, int c, int vb, int lane, Add add) {
    for (int64_t e = e0; e < e1; e += 32) {
        const int n = int(min(int64_t(32), e1 - e));
        int2 en = make_int2(0, 0);
        AsmChild ch{0, 0, 0, 0};
        if (lane < n) {
            en = many.ent[e + lane];
            ch = children[en.x];
        }
#pragma unroll 1
        for (int k0 = 0; k0 < n; k0 += 4) {
            T v[4];
            int ri[4], d[4], jc[4];
            int64_t map[4], up[4];
            auto value = [&](int u, int ic) {            // row ic of the child's column
                const int b = ic / vb;
                ri[u] = many.rel[map[u] + b] + ic - b * vb;
                v[u] = upd[up[u] + int64_t(jc[u]) * d[u] + ic];
            };
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int k = min(k0 + u, n - 1);
                d[u] = k0 + u < n ? __shfl_sync(0xffffffffu, ch.d, k) : 0;
                jc[u] = __shfl_sync(0xffffffffu, en.y, k) * vb + c;
                map[u] = __shfl_sync(0xffffffffu, ch.map, k);
                up[u] = __shfl_sync(0xffffffffu, ch.upd, k);
                if (jc[u] + lane < d[u]) value(u, jc[u] + lane);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (jc[u] + lane < d[u]) add(ri[u], v[u]);
#pragma unroll 4
                for (int ic = jc[u] + lane + 32; ic < d[u]; ic += 32) {
                    value(u, ic);
                    add(ri[u], v[u]);
                }
                __syncwarp();                            // (the next child may meet the same rows)
            }
        }
    }
}

// The children of a small front of ManyDev, added to its triangle F by the CTA. (A call: rare,
// and inlined it costs the kernel registers.)
template <typename T>
__device__ __noinline__ void small_many(const SmallTask *tk, int vb, const ManyDev &many, const AsmChild *children,
                                        const T *upd, T *F) {
    const int f = tk->f;
    const int64_t *ptr = many.ptr + many.fronts[tk->many].rows;
    for (int j = threadIdx.x >> 5; j < f; j += 8) {
        T *Fj = F + j * f - ((j * (j + 1)) >> 1);
        many_column(many, children, upd, ptr[j / vb], ptr[j / vb + 1], j % vb, vb, threadIdx.x & 31,
                    [&](int i, T x) { Fj[i] += x; });
    }
}

template <typename T, int VB, int NSEG, int MINB>
__global__ void __launch_bounds__(256, MINB)
    small_factor_kernel(const SmallTask *__restrict__ tasks, int vb_, int lp, const AsmChild *__restrict__ children,
                        const int32_t *__restrict__ cmap, ManyDev many, T *__restrict__ factor, T *upd, PivotCtl pv) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *Lp = reinterpret_cast<T *>(smem_raw);             // [4][lp]: the four columns under way
    T *F = Lp + kSmallCols * lp;
    const SmallTask tk = tasks[blockIdx.x];
    const int w = tk.w, f = tk.f, d = f - w, ld = tk.ld;
    const int vb = VB > 0 ? VB : vb_;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    T *pan = factor + tk.pan;
    // packed triangle: (i, j) at F[col(j) + i], i >= j
    auto col = [f](int j) { return j * f - ((j * (j + 1)) >> 1); };
    {
        auto row_maps = [&](const AsmChild &ch, int (&mi)[NSEG]) {
#pragma unroll
            for (int g = 0; g < NSEG; ++g) {
                const int i = lane + 32 * g;
                mi[g] = -1;
                if (i < f) {
                    const int b = i / vb, m = cmap[ch.map + b];
                    if (m >= 0) mi[g] = m * vb + i - b * vb;
                }
            }
        };
        AsmChild kept[2];
        int kmi[2][NSEG];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (k >= tk.nchild) break;
            kept[k] = children[tk.child0 + k];
            row_maps(kept[k], kmi[k]);
        }
        for (int j0 = 4 * warp; j0 < f; j0 += 32) {
            T v[4][NSEG];
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int g = 0; g < NSEG; ++g) {
                    const int j = j0 + u, i = lane + 32 * g;
                    v[u][g] = T(0);
                    if (j < w && i >= j && i < f) v[u][g] = pan[int64_t(j) * ld + i];
                }
            auto add = [&](const AsmChild &ch, const int (&mi)[NSEG]) {
                int mj[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    mj[u] = -1;
                    if (j0 + u < f) {
                        const int b = (j0 + u) / vb, m = cmap[ch.map + b];
                        if (m >= 0) mj[u] = m * vb + (j0 + u) - b * vb;
                    }
                }
                const T *U = upd + ch.upd;
                T x[4][NSEG];
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int g = 0; g < NSEG; ++g) {
                        x[u][g] = T(0);
                        if (mj[u] >= 0 && mi[g] >= mj[u]) x[u][g] = U[mj[u] * ch.d + mi[g]];
                    }
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int g = 0; g < NSEG; ++g) v[u][g] += x[u][g];
            };
#pragma unroll
            for (int k = 0; k < 2; ++k)
                if (k < tk.nchild) add(kept[k], kmi[k]);
            for (int ci = 2; ci < tk.nchild; ++ci) {
                const AsmChild ch = children[tk.child0 + ci];
                int mi[NSEG];
                row_maps(ch, mi);
                add(ch, mi);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int g = 0; g < NSEG; ++g) {
                    const int j = j0 + u, i = lane + 32 * g;
                    if (j < f && i >= j && i < f) F[col(j) + i] = v[u][g];
                }
        }
    }
    if (tk.many >= 0) {
        __syncthreads();
        small_many(tasks + blockIdx.x, vb, many, children, upd, F);
    }
    __syncthreads();
    for (int k = 0; k < w; k += kSmallCols) {
        const int nb = min(kSmallCols, w - k);
        T a[4][4], rs[4];                                // a: lower triangle of the block, then of its L
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int t = u; t < 4; ++t) a[t][u] = (t < nb) ? F[col(k + u) + k + t] : T(0);
        const int i = k + tid;                           // this thread's row
        T l[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) l[u] = (u < nb && i >= k + nb && i < f) ? F[col(k + u) + i] : T(0);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            rs[u] = T(0);
            if (u < nb) {
                T p = a[u][u];
                if (!(p > T(0))) p = bad_pivot(p, tk.col0 + k + u, pv, tid == 0);
                rs[u] = dev_rsqrt(p);
                a[u][u] = rs[u] > T(0) ? p * rs[u] : p;  // (an infinite pivot: L = inf, zeros below)
#pragma unroll
                for (int t = u + 1; t < 4; ++t) {
                    a[t][u] *= rs[u];
#pragma unroll
                    for (int v = u + 1; v <= t; ++v) a[t][v] -= a[t][u] * a[v][u];
                }
            }
        }
        if (i >= k + nb) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
#pragma unroll
                for (int v = 0; v < u; ++v) l[u] -= l[v] * a[u][v];
                l[u] *= rs[u];
            }
        } else {
#pragma unroll
            for (int t = 0; t < 4; ++t)
#pragma unroll
                for (int u = 0; u <= t; ++u)
                    if (tid == t) l[u] = a[t][u];
        }
        if (i < f) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                Lp[u * lp + i] = l[u];
                if (u < nb && i >= k + u) pan[int64_t(k + u) * ld + i] = l[u];
            }
        }
        __syncthreads();
        T li[4][NSEG];
#pragma unroll
        for (int g = 0; g < NSEG; ++g)
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int r = lane + 32 * g;
                li[u][g] = (r >= k + nb && r < f) ? Lp[u * lp + r] : T(0);
            }
        for (int j = k + nb + warp; j < f; j += 8) {
            T lj[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) lj[u] = Lp[u * lp + j];
            T *Fj = F + col(j);
#pragma unroll
            for (int g = 0; g < NSEG; ++g) {
                const int r = lane + 32 * g;
                if (r >= j && r < f) {
                    T x = Fj[r];
#pragma unroll
                    for (int u = 0; u < 4; ++u) x -= li[u][g] * lj[u];
                    Fj[r] = x;
                }
            }
        }
        __syncthreads();
    }
    if (d > 0 && tk.upd >= 0) {
        T *U = upd + tk.upd;
        for (int j = w + warp; j < f; j += 8)
            for (int i = j + lane; i < f; i += 32) U[(j - w) * d + (i - w)] = F[col(j) + i];
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

// The children of a large front of ManyDev, whose panel and (zeroed) U_s are in place: a warp
// per block column, added to in global memory.
template <typename T>
__global__ void __launch_bounds__(256) assemble_many_kernel(const ManyTask *__restrict__ tasks, SnDev sd, ManyDev many,
                                                            const AsmChild *__restrict__ children,
                                                            T *factor, T *upd) {
    const ManyTask tk = tasks[blockIdx.x];
    const int s = tk.sn, lane = threadIdx.x & 31, b = tk.b + (threadIdx.x >> 5);
    const int w = sd.w[s], d = sd.d[s], vb = sd.vb;
    if (b * vb >= w + d) return;
    const int64_t *ptr = many.ptr + many.fronts[tk.many].rows + b;
    T *pan = factor + sd.pan_off[s], *Us = upd + sd.upd_off[s];
    for (int c = 0; c < vb; ++c) {
        const int j = b * vb + c;
        T *dst = j < w ? pan + int64_t(j) * sd.ld[s] : Us + int64_t(j - w) * d - w;
        many_column(many, children, upd, ptr[0], ptr[1], c, vb, lane, [&](int i, T x) { dst[i] += x; });
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
void launch_small_factor(const SmallTask *tasks, int count, int max_front, int vb, const AsmChild *children,
                         const int32_t *cmap, ManyDev many, T *factor, T *upd, PivotCtl pv, cudaStream_t st) {
    if (count <= 0) return;
    const int lp = (max_front + 3) & ~3;
    const size_t smem = (size_t(kSmallCols) * lp + size_t(max_front) * (max_front + 1) / 2) * sizeof(T);
    auto go = [&](auto kern, PerDeviceOnce &once) {
        once([kern] { cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmemOptin); });
        kern<<<count, 256, smem, st>>>(tasks, vb, lp, children, cmap, many, factor, upd, pv);
    };
    // rows per lane from the level's largest front
    auto by_front = [&](auto k2, auto k3, auto k5, auto k8, PerDeviceOnce(&once)[4]) {
        if (max_front <= 64) go(k2, once[0]);
        else if (max_front <= 96) go(k3, once[1]);
        else if (max_front <= 160) go(k5, once[2]);
        else go(k8, once[3]);
    };
    ++g_kernel_launches;
    static PerDeviceOnce once3[4], once1[4], once0[4];
    constexpr int B2 = sizeof(T) == 4 ? 4 : 3, B5 = sizeof(T) == 4 ? 3 : 2;
    if (vb == 3)
        by_front(small_factor_kernel<T, 3, 2, B2>, small_factor_kernel<T, 3, 3, B2>, small_factor_kernel<T, 3, 5, B5>,
                 small_factor_kernel<T, 3, 8, 1>, once3);
    else if (vb == 1)
        by_front(small_factor_kernel<T, 1, 2, B2>, small_factor_kernel<T, 1, 3, B2>, small_factor_kernel<T, 1, 5, B5>,
                 small_factor_kernel<T, 1, 8, 1>, once1);
    else
        by_front(small_factor_kernel<T, 0, 2, B2>, small_factor_kernel<T, 0, 3, B2>, small_factor_kernel<T, 0, 5, B5>,
                 small_factor_kernel<T, 0, 8, 1>, once0);
}

template <typename T>
void launch_assemble_many(const ManyTask *tasks, int ntasks, SnDev sd, ManyDev many, const AsmChild *children, T *factor,
                          T *upd, cudaStream_t st) {
    if (ntasks <= 0) return;
    ++g_kernel_launches;
    assemble_many_kernel<T><<<ntasks, 256, 0, st>>>(tasks, sd, many, children, factor, upd);
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
    template void launch_small_factor<T>(const SmallTask *, int, int, int, const AsmChild *, const int32_t *,      \
                                         ManyDev, T *, T *, PivotCtl, cudaStream_t);                               \
    template void launch_assemble_many<T>(const ManyTask *, int, SnDev, ManyDev, const AsmChild *, T *, T *,       \
                                          cudaStream_t);                                                           \
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
