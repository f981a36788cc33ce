// Multi-RHS forward / backward solves (K6) over the lower part of the assembly
// tree, one independent subtree per CTA or per warp and right-hand side.
//
// Below the cut level the tree has many small fronts and few rows per front: what a front
// costs is its chain of dependent loads, not its bytes. A walk goes over a whole subtree (a
// contiguous postorder range of supernodes):
//   forward  (postorder)  v = [x(cols); 0] + children's u (child order, through their inverse
//            row maps); y = L11^{-1} v[0:w]; u = v[w:f] - L21 y; y -> x, u -> solve arena
//            (read by the parent, later in this walk or above the cut);
//   backward (reverse postorder) v = [x(cols); x(struct rows)] (ancestors are final);
//            v[0:w] -= L21^T x_struct; x = L11^{-T} v[0:w].
// Fronts factored in shared memory (no stored diagonal inverses) are one warp's, for up to
// four right-hand sides, v in its registers (lane = rows lane + 32 g): column substitution
// forward (a column's chain is a shuffle, a product with the reciprocal diagonal and a fused
// multiply-add), backward eight columns at a time (sums over the rows below, the triangle). Both
// read columns only; an entry is read and widened once for the four. The largest subtrees of
// such fronts alone are a launch of their own, spread over all warps: nothing there waits
// at a barrier. The fronts above them are a CTA's per subtree of the cut, four right-hand
// sides at a time, through the stored 64 x 64 inverses, v in shared memory. In one CTA walk for
// all, with barriers, a division a column and the children one after the other, a pass over
// the batch of 48 cubes (FP32, 8 right-hand sides) took 1,160 us forward and 1,170 us backward;
// now 209 us (small fronts) and 377 us (above them) forward, 406 and 498 us backward. The
// 64-sided cube with 4: 687 us forward and 694 us backward before, 140 + 366 and 271 + 464 us
// now (the fronts with stored inverses read L straight from global memory, which is what
// bounds the larger half). Subtrees are assigned round-robin in order of decreasing work.
#include "device.h"

#include <algorithm>
#include <type_traits>

namespace mfs {

namespace {

constexpr int kSubThreads = 256;
constexpr int kSubRhs = 4;                 // right-hand sides per pass or warp (more are looped)
constexpr int kSubRed = 4 * kSubRhs * 64;  // split-k partials of a 64-row block

// Division by the block size as a product: exact for rows of a front below the cut (at most
// 2048 of them, so at most 2048 a block).
struct BlockDiv {
    int vb;
    uint32_t m;                            // ceil(2^26 / vb)
    explicit BlockDiv(int v) : vb(v), m(((1u << 26) + uint32_t(v) - 1) / uint32_t(v)) {}
    __device__ __forceinline__ int operator()(int i) const { return int((uint64_t(uint32_t(i)) * m) >> 26); }
};

__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
    return x;
}

// ------------------------------------------------------------------ forward
// A front with stored inverses, the whole CTA.
template <typename T>
__device__ __forceinline__ void fwd_front(int s, const SnDev &sd, BlockDiv div, const T *__restrict__ factor,
                                          const T *pan, double *__restrict__ X, int64_t ldx, int nrhs, int rg, int nr,
                                          double *__restrict__ sol, double *v, double *red) {
    const int tid = threadIdx.x, nt = blockDim.x;
    const int w = sd.w[s], d = sd.d[s], f = w + d, c0 = sd.col0[s], ld = sd.ld[s];
    for (int q = tid; q < nr * f; q += nt) {
        const int r = q / f, i = q - r * f;
        v[q] = i < w ? X[c0 + i + int64_t(rg + r) * ldx] : 0.0;
    }
    __syncthreads();
    for (int ci = sd.child_ptr[s]; ci < sd.child_ptr[s + 1]; ++ci) {
        const int c = sd.child_list[ci];
        const int dc = sd.d[c];
        if (dc == 0) continue;
        const int32_t *rel = sd.rel + sd.struct_ptr[c];
        const double *uc = sol + sd.sol_off[c] * nrhs;
        for (int q = tid; q < nr * dc; q += nt) {
            const int r = q / dc, i = q - r * dc, b = div(i);
            v[r * f + rel[b] + i - b * div.vb] += uc[i + int64_t(rg + r) * dc];
        }
        __syncthreads();
    }
    const int64_t inv = sd.inv_off[s];
    const int nbw = (w + 63) / 64;
    const int i = tid & 63, g = tid >> 6;             // row of the block, k-split group (4)
    for (int rb = 0; rb < nbw; ++rb) {
        const int r0 = rb * 64, nrr = min(64, w - r0);
        if (rb > 0) {
            // v[r0 + i] -= sum_{j < r0} L(r0 + i, j) y_j, j split over the 4 groups
            double acc[kSubRhs] = {0.0, 0.0, 0.0, 0.0};
            if (i < nrr)
                for (int j = g; j < r0; j += 4) {
                    const double l = double(pan[int64_t(j) * ld + r0 + i]);
#pragma unroll
                    for (int r = 0; r < kSubRhs; ++r)
                        if (r < nr) acc[r] += l * v[r * f + j];
                }
#pragma unroll
            for (int r = 0; r < kSubRhs; ++r) red[(g * kSubRhs + r) * 64 + i] = acc[r];
            __syncthreads();
            if (g == 0 && i < nrr)
#pragma unroll
                for (int r = 0; r < kSubRhs; ++r)
                    if (r < nr)
                        v[r * f + r0 + i] -= red[r * 64 + i] + red[(kSubRhs + r) * 64 + i] +
                                             red[(2 * kSubRhs + r) * 64 + i] + red[(3 * kSubRhs + r) * 64 + i];
            __syncthreads();
        }
        // y = inv(L(rb, rb)) v_block, j split over the 4 groups
        {
            const T *ib = factor + inv + int64_t(rb) * 4096;   // column-major 64 x 64
            double acc[kSubRhs] = {0.0, 0.0, 0.0, 0.0};
            if (i < nrr)
                for (int j = g; j <= i; j += 4) {
                    const double l = double(ib[j * 64 + i]);
#pragma unroll
                    for (int r = 0; r < kSubRhs; ++r)
                        if (r < nr) acc[r] += l * v[r * f + r0 + j];
                }
#pragma unroll
            for (int r = 0; r < kSubRhs; ++r) red[(g * kSubRhs + r) * 64 + i] = acc[r];
            __syncthreads();
            if (g == 0 && i < nrr)
#pragma unroll
                for (int r = 0; r < kSubRhs; ++r)
                    if (r < nr)
                        v[r * f + r0 + i] = red[r * 64 + i] + red[(kSubRhs + r) * 64 + i] +
                                            red[(2 * kSubRhs + r) * 64 + i] + red[(3 * kSubRhs + r) * 64 + i];
            __syncthreads();
        }
    }
    // u = v[w:f] - L21 y
    for (int k = tid; k < d; k += nt) {
        double acc[kSubRhs] = {0.0, 0.0, 0.0, 0.0};
        for (int j = 0; j < w; ++j) {
            const double l = double(pan[int64_t(j) * ld + w + k]);
#pragma unroll
            for (int r = 0; r < kSubRhs; ++r)
                if (r < nr) acc[r] += l * v[r * f + j];
        }
#pragma unroll
        for (int r = 0; r < kSubRhs; ++r)
            if (r < nr) v[r * f + w + k] -= acc[r];
    }
    __syncthreads();
    const bool has_u = d > 0 && sd.sol_off[s] >= 0;
    for (int q = tid; q < nr * f; q += nt) {
        const int r = q / f, i = q - r * f;
        if (i < w) X[c0 + i + int64_t(rg + r) * ldx] = v[q];
        else if (has_u) sol[sd.sol_off[s] * nrhs + (i - w) + int64_t(rg + r) * d] = v[q];
    }
    __syncthreads();
}

// ------------------------------------------------------------------ backward
template <typename T>
__device__ __forceinline__ void bwd_front(int s, const SnDev &sd, BlockDiv div, const T *__restrict__ factor,
                                          const T *pan, double *__restrict__ X, int64_t ldx, int rg, int nr,
                                          double *v) {
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
    const int w = sd.w[s], d = sd.d[s], f = w + d, c0 = sd.col0[s], ld = sd.ld[s];
    const int32_t *rows = sd.struct_rows + sd.struct_ptr[s];
    for (int q = tid; q < nr * f; q += nt) {
        const int r = q / f, i = q - r * f;
        int64_t gi;
        if (i < w) gi = c0 + i;
        else {
            const int li = i - w, b = div(li);
            gi = int64_t(rows[b]) * div.vb + li - b * div.vb;
        }
        v[q] = X[gi + int64_t(rg + r) * ldx];
    }
    __syncthreads();
    const int64_t inv = sd.inv_off[s];
    // v[0:w] -= L21^T x_struct: one warp per column, lanes over rows
    if (d > 0) {
        for (int j = warp; j < w; j += nw) {
            double acc[kSubRhs] = {0.0, 0.0, 0.0, 0.0};
            for (int k = lane; k < d; k += 32) {
                const double l = double(pan[int64_t(j) * ld + w + k]);
#pragma unroll
                for (int r = 0; r < kSubRhs; ++r)
                    if (r < nr) acc[r] += l * v[r * f + w + k];
            }
#pragma unroll
            for (int r = 0; r < kSubRhs; ++r) {
                const double sum = warp_sum(acc[r]);
                if (lane == 0 && r < nr) v[r * f + j] -= sum;
            }
        }
        __syncthreads();
    }
    const int nbw = (w + 63) / 64;
    for (int rb = nbw - 1; rb >= 0; --rb) {
        const int r0 = rb * 64, nrr = min(64, w - r0);
        if (r0 + 64 < w) {
            // v[r0 + j] -= sum_{i >= r0 + 64} L(i, r0 + j) x_i
            for (int j = warp; j < nrr; j += nw) {
                double acc[kSubRhs] = {0.0, 0.0, 0.0, 0.0};
                for (int i = r0 + 64 + lane; i < w; i += 32) {
                    const double l = double(pan[int64_t(r0 + j) * ld + i]);
#pragma unroll
                    for (int r = 0; r < kSubRhs; ++r)
                        if (r < nr) acc[r] += l * v[r * f + i];
                }
#pragma unroll
                for (int r = 0; r < kSubRhs; ++r) {
                    const double sum = warp_sum(acc[r]);
                    if (lane == 0 && r < nr) v[r * f + r0 + j] -= sum;
                }
            }
            __syncthreads();
        }
        // x_block = inv(L(rb, rb))^T v_block, one warp per column of the inverse
        const T *ib = factor + inv + int64_t(rb) * 4096;
        for (int j0 = 0; j0 < nrr; j0 += 2 * nw) {          // 2 columns per warp and round
            double out[2][kSubRhs];
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const int j = j0 + warp + t * nw;
                double acc[kSubRhs] = {0.0, 0.0, 0.0, 0.0};
                if (j < nrr)
                    for (int i = j + lane; i < nrr; i += 32) {
                        const double l = double(ib[j * 64 + i]);
#pragma unroll
                        for (int r = 0; r < kSubRhs; ++r)
                            if (r < nr) acc[r] += l * v[r * f + r0 + i];
                    }
#pragma unroll
                for (int r = 0; r < kSubRhs; ++r) out[t][r] = warp_sum(acc[r]);
            }
            __syncthreads();                              // all reads of this round done
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const int j = j0 + warp + t * nw;
                if (lane == 0 && j < nrr)
#pragma unroll
                    for (int r = 0; r < kSubRhs; ++r)
                        if (r < nr) v[r * f + r0 + j] = out[t][r];
            }
            __syncthreads();
        }
    }
    __syncthreads();
    for (int q = tid; q < nr * w; q += nt) {
        const int r = q / w, j = q - r * w;
        X[c0 + j + int64_t(rg + r) * ldx] = v[r * f + j];
    }
    __syncthreads();
}

// ------------------------------------------------------------------ small fronts, one warp
// NSEG x 32 rows at least the front's; right-hand sides r0 to r0 + nr - 1, at most RB. A lane
// holds the rows from the 32 columns under way on (v[r][g]: row jb + lane + 32 g), moved by
// one entry from one such block of columns to the next, so that the loop over the blocks
// is rolled: unrolled, with the block sizes 1 and 3 as template parameters, this file took
// 674 s to compile and half of the object code was never run.
template <typename T, int NSEG, int RB, bool MANY>
__device__ __forceinline__ void fwd_small(const SubFront &sf, const T *__restrict__ factor,
                                          const SbChild *__restrict__ kids, const int32_t *__restrict__ cmap,
                                          const ManyDev &many, BlockDiv div, double *X, int64_t ldx, int nrhs, int r0, int nr, double *sol) {
    const int lane = threadIdx.x & 31;
    const int w = sf.w, f = sf.f;
    const T *pan = factor + sf.pan;
    double *x = X + sf.col0 + r0 * ldx;
    auto diagonal = [&](int i) { return i < w ? double(pan[int64_t(i) * sf.ld + i]) : 1.0; };
    double v[RB][NSEG];
    __syncwarp();                                        // the children's u (this warp's) are visible
    double d = diagonal(lane);
#pragma unroll
    for (int g = 0; g < NSEG; ++g) {
        const int i = lane + 32 * g;
#pragma unroll
        for (int r = 0; r < RB; ++r) v[r][g] = i < w && r < nr ? x[i + r * ldx] : 0.0;
    }
    for (int ci = 0; ci < sf.nchild; ++ci) {
        const SbChild ch = kids[sf.child0 + ci];
        const double *u = sol + ch.sol * nrhs + int64_t(r0) * ch.d;
        int m[NSEG];
#pragma unroll
        for (int g = 0; g < NSEG; ++g) {
            const int i = lane + 32 * g, b = div(i);
            m[g] = -1;
            if (i < f) {
                const int k = cmap[ch.map + b];
                if (k >= 0) m[g] = (k - b) * div.vb + i;
            }
        }
        double a[RB][NSEG];
#pragma unroll
        for (int r = 0; r < RB; ++r)
#pragma unroll
            for (int g = 0; g < NSEG; ++g) a[r][g] = m[g] >= 0 && r < nr ? u[m[g] + r * ch.d] : 0.0;
#pragma unroll
        for (int r = 0; r < RB; ++r)
#pragma unroll
            for (int g = 0; g < NSEG; ++g) v[r][g] += a[r][g];
    }
    if constexpr (MANY)
        if (sf.many >= 0) {                              // each row's own list, in child order
            const int64_t *ptr = many.ptr + many.fronts[sf.many].rows;
#pragma unroll
            for (int g = 0; g < NSEG; ++g) {
                const int i = lane + 32 * g, b = div(i);
                if (i >= f) continue;
#pragma unroll 1
                for (int64_t q = ptr[b]; q < ptr[b + 1]; ++q) {
                    const int2 en = many.ent[q];
                    const SbChild ch = kids[en.x];
                    const double *u = sol + ch.sol * nrhs + int64_t(r0) * ch.d + en.y * div.vb + i - b * div.vb;
#pragma unroll
                    for (int r = 0; r < RB; ++r) v[r][g] += r < nr ? u[r * ch.d] : 0.0;
                }
            }
        }
    int jb = 0;
#pragma unroll 1
    for (;; jb += 32) {
        const double rd = 1.0 / d;
        d = diagonal(jb + 32 + lane);
        const int je = min(32, w - jb);
#pragma unroll 1
        for (int j0 = 0; j0 < je; j0 += 4) {
            // four columns of L ahead of their use
            T l[4][NSEG];
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int g = 0; g < NSEG; ++g) {
                    const int i = jb + lane + 32 * g, j = jb + j0 + u;
                    l[u][g] = (j0 + u < je && i > j && i < f) ? pan[int64_t(j) * sf.ld + i] : T(0);
                }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (j0 + u >= je) break;
                double y[RB];
#pragma unroll
                for (int r = 0; r < RB; ++r) y[r] = __shfl_sync(0xffffffffu, v[r][0] * rd, j0 + u);
                if (lane == j0 + u)
#pragma unroll
                    for (int r = 0; r < RB; ++r) v[r][0] = y[r];
#pragma unroll
                for (int g = 0; g < NSEG; ++g) {
                    const double lv = double(l[u][g]);
#pragma unroll
                    for (int r = 0; r < RB; ++r) v[r][g] -= lv * y[r];
                }
            }
        }
        if (jb + 32 >= w) break;
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            if (r < nr) x[jb + lane + r * ldx] = v[r][0];
#pragma unroll
            for (int g = 0; g + 1 < NSEG; ++g) v[r][g] = v[r][g + 1];
            v[r][NSEG - 1] = 0.0;
        }
    }
    double *us = sf.sol >= 0 ? sol + sf.sol * nrhs + int64_t(r0) * (f - w) : nullptr;
#pragma unroll
    for (int r = 0; r < RB; ++r) {
        if (r >= nr) break;
#pragma unroll
        for (int g = 0; g < NSEG; ++g) {
            const int i = jb + lane + 32 * g;
            if (i < w) x[i + r * ldx] = v[r][g];
            else if (i < f && us) us[i - w + r * int64_t(f - w)] = v[r][g];
        }
    }
}

template <typename T, int NSEG, int RB>
__device__ __forceinline__ void bwd_small(const SubFront &sf, const T *__restrict__ factor,
                                          const int32_t *__restrict__ struct_rows, BlockDiv div, double *X, int64_t ldx,
                                          int r0, int nr) {
    const int lane = threadIdx.x & 31;
    const int w = sf.w, f = sf.f, wb = div(w);
    const T *pan = factor + sf.pan;
    const int32_t *rows = struct_rows + sf.rows - wb;
    double *x = X + r0 * ldx;
    auto diagonal = [&](int i) { return i < w ? double(pan[int64_t(i) * sf.ld + i]) : 1.0; };
    double v[RB][NSEG];                                  // x of the rows (own columns: not yet)
    __syncwarp();                                        // the parent's x (this warp's) is visible
    int jb = (w - 1) & ~31;
    double d = diagonal(jb + lane);
#pragma unroll
    for (int g = 0; g < NSEG; ++g) {
        const int i = jb + lane + 32 * g;
        int64_t gi = sf.col0 + i;
        if (i >= w && i < f) {
            const int b = div(i);
            gi = int64_t(rows[b]) * div.vb + i - b * div.vb;
        }
#pragma unroll
        for (int r = 0; r < RB; ++r) v[r][g] = i < f && r < nr ? x[gi + r * ldx] : 0.0;
    }
    // the blocks of 32 columns, last first; in each, eight columns at a time, last first: the
    // sums of L(i, j) x_i over the rows below them, spread over the lanes as they are
    // reduced (each step halves what a lane holds), then the 8 x 8 triangle, lane k of the
    // eight with column k
#pragma unroll 1
    for (;; jb -= 32) {
        const double rd = 1.0 / d;
        double vn[RB];                                   // the rows of the next block of columns
#pragma unroll
        for (int r = 0; r < RB; ++r) vn[r] = jb > 0 && r < nr ? x[sf.col0 + jb - 32 + lane + r * ldx] : 0.0;
        if (jb > 0) d = diagonal(jb - 32 + lane);
#pragma unroll 1
        for (int c0 = (min(32, w - jb) - 1) & ~7; c0 >= 0; c0 -= 8) {
            const int j0 = jb + c0, nb = min(8, w - j0), below = j0 + nb;
            const int k = lane - c0;                     // this lane's column of the eight
            T tri[8];
#pragma unroll
            for (int u = 1; u < 8; ++u)
                tri[u] = k >= 0 && k < u && u < nb ? pan[int64_t(j0 + k) * sf.ld + j0 + u] : T(0);
            double a[RB][8];
#pragma unroll
            for (int r = 0; r < RB; ++r)
#pragma unroll
                for (int u = 0; u < 8; ++u) a[r][u] = 0.0;
#pragma unroll
            for (int g = 0; g < NSEG; ++g) {
                const int i = jb + lane + 32 * g;
                T l[8];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    l[u] = (u < nb && i >= below && i < f) ? pan[int64_t(j0 + u) * sf.ld + i] : T(0);
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const double lv = double(l[u]);
#pragma unroll
                    for (int r = 0; r < RB; ++r) a[r][u] += lv * v[r][g];
                }
            }
#pragma unroll
            for (int r = 0; r < RB; ++r) {
#pragma unroll
                for (int h = 4; h > 0; h >>= 1) {        // lanes' bits 4, 3, 2 choose the column
                    const bool up = lane & (4 * h);
#pragma unroll
                    for (int u = 0; u < h; ++u) {
                        const double give = up ? a[r][u] : a[r][u + h], keep = up ? a[r][u + h] : a[r][u];
                        a[r][u] = keep + __shfl_xor_sync(0xffffffffu, give, 4 * h);
                    }
                }
                a[r][0] += __shfl_xor_sync(0xffffffffu, a[r][0], 2);
                a[r][0] += __shfl_xor_sync(0xffffffffu, a[r][0], 1);
                const double sum = __shfl_sync(0xffffffffu, a[r][0], (k & 7) * 4);
                if (k >= 0 && k < nb) v[r][0] -= sum;
            }
#pragma unroll
            for (int u = 7; u >= 0; --u) {
                if (u >= nb) continue;
                const double lv = u > 0 ? double(tri[u]) : 0.0;
#pragma unroll
                for (int r = 0; r < RB; ++r) {
                    const double xj = __shfl_sync(0xffffffffu, v[r][0] * rd, c0 + u);
                    if (k == u) v[r][0] = xj;
                    else v[r][0] -= lv * xj;             // lv: 0 outside the columns before u
                }
            }
        }
        if (jb + lane < w)
#pragma unroll
            for (int r = 0; r < RB; ++r)
                if (r < nr) x[sf.col0 + jb + lane + r * ldx] = v[r][0];
        if (jb == 0) break;
#pragma unroll
        for (int r = 0; r < RB; ++r) {
#pragma unroll
            for (int g = NSEG - 1; g > 0; --g) v[r][g] = v[r][g - 1];
            v[r][0] = vn[r];
        }
    }
}

// The same, for a small front in a CTA's walk: a call, so that the walk keeps its registers.
template <typename T>
__device__ __noinline__ void fwd_small_call(const SubFront *sf, const T *factor, const SbChild *kids,
                                            const int32_t *cmap, const ManyDev &many, BlockDiv div, double *X,
                                            int64_t ldx, int nrhs, int r, double *sol) {
    fwd_small<T, 8, 1, true>(*sf, factor, kids, cmap, many, div, X, ldx, nrhs, r, 1, sol);
}

template <typename T>
__device__ __noinline__ void bwd_small_call(const SubFront *sf, const T *factor, const int32_t *struct_rows,
                                            BlockDiv div, double *X, int64_t ldx, int r) {
    bwd_small<T, 8, 1>(*sf, factor, struct_rows, div, X, ldx, r, 1);
}

// The front's panel into L2, a line a lane.
template <typename T>
__device__ __forceinline__ void prefetch_panel(const SubFront &sf, const T *factor) {
    const char *p = reinterpret_cast<const char *>(factor + sf.pan);
    const int bytes = sf.ld * sf.w * int(sizeof(T));
    for (int o = (threadIdx.x & 31) * 128; o < bytes; o += 32 * 128)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p + o));
}

// Subtrees of small fronts only: a warp per subtree and RB right-hand sides.
template <typename T, int NSEG, int RB>
__global__ void __launch_bounds__(kSubThreads) subtree_small_fwd_kernel(
    const int2 *__restrict__ subs, int nsub, BlockDiv div, const SubFront *__restrict__ fronts,
    const SbChild *__restrict__ kids, const int32_t *__restrict__ cmap, const T *__restrict__ factor, double *X,
    int64_t ldx, int nrhs, double *sol) {
    const int nwarps = gridDim.x * (kSubThreads / 32), ngr = (nrhs + RB - 1) / RB;
    for (int q = blockIdx.x * (kSubThreads / 32) + (threadIdx.x >> 5); q < nsub * ngr; q += nwarps) {
        const int2 sr = subs[q / ngr];
        const int r0 = q % ngr * RB, nr = min(RB, nrhs - r0);
        SubFront next = fronts[sr.x];
        for (int s = sr.x; s <= sr.y; ++s) {
            const SubFront sf = next;
            if (s < sr.y) {
                next = fronts[s + 1];
                prefetch_panel(next, factor);
            }
            if (sf.f <= 64) fwd_small<T, 2, RB, false>(sf, factor, kids, cmap, ManyDev{}, div, X, ldx, nrhs, r0, nr, sol);
            else fwd_small<T, NSEG, RB, false>(sf, factor, kids, cmap, ManyDev{}, div, X, ldx, nrhs, r0, nr, sol);
        }
    }
}

// The fronts above those: a CTA per subtree of the cut, children first (tops: its fronts,
// top_ptr[k] to top_ptr[k + 1] in postorder).
template <typename T>
__global__ void __launch_bounds__(kSubThreads, 3) subtree_fwd_kernel(
    const int32_t *__restrict__ top_ptr, const int32_t *__restrict__ tops, int nsub, SnDev sd, BlockDiv div,
    const SubFront *__restrict__ fronts, const SbChild *__restrict__ kids, const int32_t *__restrict__ cmap,
    ManyDev many, const T *__restrict__ factor, double *X, int64_t ldx, int nrhs, double *sol) {
    extern __shared__ __align__(16) double sub_smem[];
    double *red = sub_smem, *v = red + kSubRed;
    const int warp = threadIdx.x >> 5;
    for (int k = blockIdx.x; k < nsub; k += gridDim.x) {
        const int t0 = top_ptr[k], t1 = top_ptr[k + 1];
        for (int t = t0; t < t1; ++t) {
            const int s = tops[t];
            __syncthreads();                             // the children's u are there
            if (fronts[s].inv < 0) {
                for (int r = warp; r < nrhs; r += kSubThreads / 32)
                    fwd_small_call<T>(fronts + s, factor, kids, cmap, many, div, X, ldx, nrhs, r, sol);
                continue;
            }
            for (int rg = 0; rg < nrhs; rg += kSubRhs)
                fwd_front<T>(s, sd, div, factor, factor + fronts[s].pan, X, ldx, nrhs, rg, min(kSubRhs, nrhs - rg), sol,
                             v, red);
        }
    }
}

template <typename T, int NSEG, int RB>
__global__ void __launch_bounds__(kSubThreads) subtree_small_bwd_kernel(
    const int2 *__restrict__ subs, int nsub, BlockDiv div, const int32_t *__restrict__ struct_rows,
    const SubFront *__restrict__ fronts, const T *__restrict__ factor, double *X, int64_t ldx, int nrhs) {
    const int nwarps = gridDim.x * (kSubThreads / 32), ngr = (nrhs + RB - 1) / RB;
    for (int q = blockIdx.x * (kSubThreads / 32) + (threadIdx.x >> 5); q < nsub * ngr; q += nwarps) {
        const int2 sr = subs[q / ngr];
        const int r0 = q % ngr * RB, nr = min(RB, nrhs - r0);
        SubFront next = fronts[sr.y];
        for (int s = sr.y; s >= sr.x; --s) {
            const SubFront sf = next;
            if (s > sr.x) {
                next = fronts[s - 1];
                prefetch_panel(next, factor);
            }
            if (sf.f <= 64) bwd_small<T, 2, RB>(sf, factor, struct_rows, div, X, ldx, r0, nr);
            else bwd_small<T, NSEG, RB>(sf, factor, struct_rows, div, X, ldx, r0, nr);
        }
    }
}

// The fronts above those: a CTA per subtree of the cut, parents first (tops: its fronts,
// top_ptr[k] to top_ptr[k + 1] in postorder).
template <typename T>
__global__ void __launch_bounds__(kSubThreads, 3) subtree_bwd_kernel(
    const int32_t *__restrict__ top_ptr, const int32_t *__restrict__ tops, int nsub, SnDev sd, BlockDiv div,
    const SubFront *__restrict__ fronts, const T *__restrict__ factor, double *X, int64_t ldx, int nrhs) {
    extern __shared__ __align__(16) double sub_smem[];
    double *v = sub_smem + kSubRed;
    const int warp = threadIdx.x >> 5;
    for (int k = blockIdx.x; k < nsub; k += gridDim.x) {
        const int t0 = top_ptr[k], t1 = top_ptr[k + 1];
        for (int t = t1 - 1; t >= t0; --t) {
            const int s = tops[t];
            __syncthreads();                             // the parent's x is there
            if (fronts[s].inv < 0) {
                for (int r = warp; r < nrhs; r += kSubThreads / 32)
                    bwd_small_call<T>(fronts + s, factor, sd.struct_rows, div, X, ldx, r);
                continue;
            }
            for (int rg = 0; rg < nrhs; rg += kSubRhs)
                bwd_front<T>(s, sd, div, factor, factor + fronts[s].pan, X, ldx, rg, min(kSubRhs, nrhs - rg), v);
        }
    }
}

}  // namespace

template <typename T>
void launch_subtree_small(bool forward, const int2 *subs, int nsub, int fmax, SnDev sd, const SubFront *fronts,
                          const SbChild *kids, const int32_t *cmap, const T *factor, double *X, int64_t ldx, int nrhs,
                          double *sol, cudaStream_t st) {
    if (nsub <= 0) return;
    const int rb = nrhs > 1 ? kSubRhs : 1;
    const int64_t warps = int64_t(nsub) * ((nrhs + rb - 1) / rb), ctas = (warps + kSubThreads / 32 - 1) / (kSubThreads / 32);
    const int grid = int(std::min<int64_t>(ctas, 1 << 20));
    const BlockDiv div(sd.vb);
    ++g_kernel_launches;
    auto launch = [&](auto seg, auto rbc) {
        constexpr int NSEG = decltype(seg)::value, RB = decltype(rbc)::value;
        if (forward)
            subtree_small_fwd_kernel<T, NSEG, RB>
                <<<grid, kSubThreads, 0, st>>>(subs, nsub, div, fronts, kids, cmap, factor, X, ldx, nrhs, sol);
        else
            subtree_small_bwd_kernel<T, NSEG, RB>
                <<<grid, kSubThreads, 0, st>>>(subs, nsub, div, sd.struct_rows, fronts, factor, X, ldx, nrhs);
    };
    auto run = [&](auto seg) {                           // rows per lane of the largest front
        if (nrhs > 1) launch(seg, std::integral_constant<int, kSubRhs>{});
        else launch(seg, std::integral_constant<int, 1>{});
    };
    if (fmax <= 96) run(std::integral_constant<int, 3>{});
    else if (fmax <= 160) run(std::integral_constant<int, 5>{});
    else run(std::integral_constant<int, 8>{});
}

template <typename T>
void launch_subtree_solve(bool forward, const int32_t *top_ptr, const int32_t *tops, int nsub, int fmax, SnDev sd,
                          const SubFront *fronts, const SbChild *kids, const int32_t *cmap, ManyDev many,
                          const T *factor, double *X, int64_t ldx, int nrhs, double *sol, cudaStream_t st) {
    if (nsub <= 0) return;
    const size_t smem = (size_t(kSubRed) + size_t(kSubRhs) * fmax) * sizeof(double);
    const int grid = std::min(nsub, 8 * device_sm_count());
    const BlockDiv div(sd.vb);
    static PerDeviceOnce once;
    once([] {
        cudaFuncSetAttribute(subtree_fwd_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmemOptin);
        cudaFuncSetAttribute(subtree_bwd_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmemOptin);
    });
    ++g_kernel_launches;
    if (forward)
        subtree_fwd_kernel<T><<<grid, kSubThreads, smem, st>>>(top_ptr, tops, nsub, sd, div, fronts, kids, cmap, many,
                                                               factor, X, ldx, nrhs, sol);
    else
        subtree_bwd_kernel<T><<<grid, kSubThreads, smem, st>>>(top_ptr, tops, nsub, sd, div, fronts, factor, X, ldx,
                                                               nrhs);
}

#define MFS_SUBTREE(T)                                                                                               \
    template void launch_subtree_small<T>(bool, const int2 *, int, int, SnDev, const SubFront *, const SbChild *,    \
                                          const int32_t *, const T *, double *, int64_t, int, double *,              \
                                          cudaStream_t);                                                             \
    template void launch_subtree_solve<T>(bool, const int32_t *, const int32_t *, int, int, SnDev, const SubFront *, \
                                          const SbChild *, const int32_t *, ManyDev, const T *, double *, int64_t,   \
                                          int, double *, cudaStream_t);
MFS_SUBTREE(float)
MFS_SUBTREE(double)
#undef MFS_SUBTREE

}  // namespace mfs
