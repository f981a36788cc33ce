// Symmetric block SpMV (K7), the fused
// pin-removal/permutation gathers, element assembly (K1) and the FP64
// vector kernels of the refinement loop.
//
// Reference counterparts:
//   SparseLDL::Solve (forward L y = b, backward L^T x = y, multi-RHS column-major,
//   ld = n) ............................ Solvers/CatamariFactorizer.cc:54,70,838-907
//   removeFixedEntries / extractFullSolution with the permutation fused
//   ..................................... Solvers/CholeskyFactorizerBase.hh:299-363
//   BlockCSCHessianBase::applyRawColumnRangeAccum (upper blocks + transposes)
//   ..................................... BlockCSCHessian.hh:1080-1120
//   ElementHessianContribAssembler<true>::run + ColumnScanner::addBlockAtLoc
//   ..................................... SystemAssembler.hh:60-98, BlockCSCHessian.hh:371-381
// The triangular solves themselves live in kernels_trisolve.cu.
#include "device.h"

#include <algorithm>

namespace mfs {

namespace {

constexpr int kReduceBlocks = 592;   // 4 x SM count; fixed so reductions are deterministic

__global__ void spmv_kernel(const int64_t *__restrict__ ptr, const int64_t *__restrict__ src,
                            const int32_t *__restrict__ col, const int32_t *__restrict__ flag, int64_t nrows, int vb,
                            int ld, const double *__restrict__ Ax, const double *__restrict__ X,
                            double *__restrict__ Y, int64_t ldx, int nrhs) {
    const int64_t total = nrows * vb * nrhs;
    for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t < total;
         t += int64_t(gridDim.x) * blockDim.x) {
        const int64_t rr = t / (nrows * vb);
        const int64_t q = t - rr * nrows * vb;
        const int64_t i = q / vb;
        const int r = int(q - i * vb);
        double acc = 0.0;
        for (int64_t e = ptr[i]; e < ptr[i + 1]; ++e) {
            const int64_t so = src[e];
            const int64_t xb = int64_t(col[e]) * vb + rr * ldx;
            const int fl = flag[e];
            for (int c = 0; c < vb; ++c) {
                double a;
                if (fl & 2) a = (r <= c) ? Ax[so + int64_t(c) * ld + r] : Ax[so + int64_t(r) * ld + c];
                else if (fl & 1) a = Ax[so + int64_t(r) * ld + c];
                else a = Ax[so + int64_t(c) * ld + r];
                acc += a * X[xb + c];
            }
        }
        Y[i * vb + r + rr * ldx] = acc;
    }
}

// Sum over the block's 256 threads, the same on every thread and in every block.
__device__ __forceinline__ double block_sum(double v, double *sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += sh[k];
    return s;
}
// Sum of the kReduceBlocks partial sums of one column (in every block that needs it: that
// costs less than a launch of its own).
__device__ __forceinline__ double partial_sum(const double *__restrict__ partials, double *sh) {
    double v = 0.0;
    for (int k = threadIdx.x; k < kReduceBlocks; k += 256) v += partials[k];
    return block_sum(v, sh);
}

// The 3 x 3 block form: eight lanes per block row, a lane per stored block (its 72 bytes read
// by one lane, the row's indices coalesced), NR right-hand sides a pass over the matrix.
// HBM- or L2-bound: every stored block is read for its row and for its column. One thread
// per scalar row took three passes over the indices, one pass over the matrix per
// right-hand side and one load at a time: k = 64, four right-hand sides 383 us before, 205 us
// now; one of them about 200 us before, 89 us now.
// dotp: kReduceBlocks partial sums of X . Y per column.
template <int NR>
__global__ void __launch_bounds__(256) spmv3_kernel(const int64_t *__restrict__ ptr, const int64_t *__restrict__ src,
                                                    const int32_t *__restrict__ col, const int32_t *__restrict__ flag,
                                                    int64_t nrows, int ld, const double *__restrict__ Ax,
                                                    const double *__restrict__ X, double *__restrict__ Y, int64_t ldx,
                                                    int nr, double *__restrict__ dotp, const int *__restrict__ stop) {
    if (stop && *stop) return;
    __shared__ double sh[8];
    const int lane = threadIdx.x & 7;
    double dot[NR];
#pragma unroll
    for (int k = 0; k < NR; ++k) dot[k] = 0.0;
    // (whole warps stay in the loop: the sums are exchanged among eight lanes)
    const int64_t stride = int64_t(gridDim.x) * 32;
    for (int64_t i0 = blockIdx.x * int64_t(32); i0 < nrows; i0 += stride) {
        const int64_t i = i0 + (threadIdx.x >> 3);
        double y[NR][3];
#pragma unroll
        for (int k = 0; k < NR; ++k) y[k][0] = y[k][1] = y[k][2] = 0.0;
        const int64_t e1 = i < nrows ? ptr[i + 1] : 0;
        for (int64_t e = (i < nrows ? ptr[i] : 0) + lane; e < e1; e += 8) {
            const double *b = Ax + src[e];
            const int fl = flag[e];
            const double *x = X + int64_t(col[e]) * 3;
            double m[3][3];                              // m[c][r]: stored column c
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int q = 0; q < 3; ++q) m[c][q] = b[int64_t(c) * ld + q];
            if (fl & 2) {                                // diagonal block: its upper triangle counts
                m[0][1] = m[1][0];
                m[0][2] = m[2][0];
                m[1][2] = m[2][1];
            } else if (fl & 1) {                         // transposed
                double t;
                t = m[0][1]; m[0][1] = m[1][0]; m[1][0] = t;
                t = m[0][2]; m[0][2] = m[2][0]; m[2][0] = t;
                t = m[1][2]; m[1][2] = m[2][1]; m[2][1] = t;
            }
#pragma unroll
            for (int k = 0; k < NR; ++k) {
                if (k >= nr) break;
                const double *xk = x + k * ldx;
                const double x0 = xk[0], x1 = xk[1], x2 = xk[2];
#pragma unroll
                for (int q = 0; q < 3; ++q) y[k][q] += m[0][q] * x0 + m[1][q] * x1 + m[2][q] * x2;
            }
        }
#pragma unroll
        for (int k = 0; k < NR; ++k)
#pragma unroll
            for (int q = 0; q < 3; ++q)
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) y[k][q] += __shfl_xor_sync(0xffffffffu, y[k][q], o);
        if (i < nrows && lane < 3) {
#pragma unroll
            for (int k = 0; k < NR; ++k) {
                if (k >= nr) break;
                const double v = lane == 0 ? y[k][0] : lane == 1 ? y[k][1] : y[k][2];
                const int64_t at = i * 3 + lane + k * ldx;
                Y[at] = v;
                if (dotp) dot[k] += X[at] * v;
            }
        }
    }
    if (!dotp) return;
#pragma unroll
    for (int k = 0; k < NR; ++k) {
        const double s = block_sum(dot[k], sh);
        if (threadIdx.x == 0 && k < nr) dotp[k * kReduceBlocks + blockIdx.x] = s;
    }
}

__global__ void gather_rows_kernel(const int64_t *__restrict__ map, int64_t n_in, const double *__restrict__ in,
                                   int64_t ld_in, double *__restrict__ out, int64_t ld_out, int nrhs) {
    const int64_t total = n_in * nrhs;
    for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t < total;
         t += int64_t(gridDim.x) * blockDim.x) {
        const int64_t r = t / n_in, i = t - r * n_in;
        const int64_t q = map ? map[i] : i;
        if (q >= 0) out[q + r * ld_out] = in[i + r * ld_in];
    }
}

__global__ void scatter_rows_kernel(const int64_t *__restrict__ map, int64_t n_out, const double *__restrict__ in,
                                    int64_t ld_in, double *__restrict__ out, int64_t ld_out, int nrhs) {
    const int64_t total = n_out * nrhs;
    for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t < total;
         t += int64_t(gridDim.x) * blockDim.x) {
        const int64_t r = t / n_out, i = t - r * n_out;
        const int64_t q = map ? map[i] : i;
        out[i + r * ld_out] = q >= 0 ? in[q + r * ld_in] : 0.0;
    }
}

// K1: one thread per (slot, component); contributions are summed in element order.
// contrib = (offset into Ke of the 3x3 block's upper-left) << 2 | kind,
// kind 0: O(r,c) = Ke[o + 12 r + c]; 1: O(r,c) = Ke[o + 12 c + r]; 2: diagonal, r <= c only.
// HBM-bound once kAsmBatch contributions are in flight per thread: k = 64 (1.81 GB of element
// matrices) 815 us with one after the other, 482 us now.
constexpr int kAsmBatch = 6;
__global__ void assemble_elements_kernel(const int64_t *__restrict__ slot_ptr, const int64_t *__restrict__ contrib,
                                         int64_t nslots, const double *__restrict__ Ke, double *__restrict__ Ax) {
    const int64_t total = nslots * 9;
    for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t < total;
         t += int64_t(gridDim.x) * blockDim.x) {
        const int64_t slot = t / 9;
        const int comp = int(t - slot * 9);
        const int c = comp / 3, r = comp - 3 * c;
        double acc = 0.0;
        const int64_t k1 = slot_ptr[slot + 1];
        for (int64_t k = slot_ptr[slot]; k < k1; k += kAsmBatch) {
            // the batch's codes, then its values, then the sum in element order
            int64_t code[kAsmBatch];
            double v[kAsmBatch];
#pragma unroll
            for (int u = 0; u < kAsmBatch; ++u) code[u] = k + u < k1 ? contrib[k + u] : -1;
#pragma unroll
            for (int u = 0; u < kAsmBatch; ++u) {
                v[u] = 0.0;
                const int kind = int(code[u] & 3);
                const int64_t o = code[u] >> 2;
                if (code[u] >= 0 && (kind != 2 || r <= c)) v[u] = Ke[o + (kind == 1 ? 12 * c + r : 12 * r + c)];
            }
#pragma unroll
            for (int u = 0; u < kAsmBatch; ++u) acc += v[u];
        }
        Ax[t] = acc;
    }
}

// Deterministic column dot products: fixed grid (x: blocks, y: columns), per-block partial
// sums, ordered final sum.
__global__ void __launch_bounds__(256) coldot_partial_kernel(const double *__restrict__ X,
                                                             const double *__restrict__ Y, int64_t n,
                                                             double *__restrict__ partials) {
    __shared__ double sh[8];
    const double *x = X + int64_t(blockIdx.y) * n, *y = Y + int64_t(blockIdx.y) * n;
    double acc = 0.0;
    for (int64_t i = blockIdx.x * int64_t(256) + threadIdx.x; i < n; i += int64_t(kReduceBlocks) * 256) acc += x[i] * y[i];
    acc = block_sum(acc, sh);
    if (threadIdx.x == 0) partials[blockIdx.y * kReduceBlocks + blockIdx.x] = acc;
}

__global__ void __launch_bounds__(256) coldot_final_kernel(const double *__restrict__ partials,
                                                           double *__restrict__ out) {
    __shared__ double sh[8];
    const double s = partial_sum(partials + blockIdx.x * kReduceBlocks, sh);
    if (threadIdx.x == 0) out[blockIdx.x] = s;
}

// x += alpha p, r -= alpha Ap with alpha = rz / pAp per column (columns with active == 0
// untouched); pAp from its partial sums. Z (optional): a copy of r. The squared norms of r
// go to hr by the block that finishes last; with a state it also settles convergence: active
// columns whose relative residual is at the tolerance end, and when none is left the
// kernels of the iterations already launched return at once.
__global__ void __launch_bounds__(256)
    pcg_xr_kernel(double *__restrict__ X, double *__restrict__ R, const double *__restrict__ P,
                  const double *__restrict__ AP, const double *__restrict__ rz, const double *__restrict__ pap_part,
                  int *active, int64_t n, double *__restrict__ Z, double *norm_part, double *__restrict__ hr,
                  unsigned *count, const double *__restrict__ hb, PcgState *st) {
    if (st && st->stop) return;
    __shared__ double sh[8];
    __shared__ bool last;
    const int c = blockIdx.y;
    const double pap = partial_sum(pap_part + c * kReduceBlocks, sh);
    const double alpha = pap != 0.0 ? rz[c] / pap : 0.0;
    const bool act = active[c] != 0;
    const int64_t o = int64_t(c) * n;
    double acc = 0.0;
    for (int64_t i = blockIdx.x * int64_t(256) + threadIdx.x; i < n; i += int64_t(kReduceBlocks) * 256) {
        double v = R[o + i];
        if (act) {
            X[o + i] += alpha * P[o + i];
            v -= alpha * AP[o + i];
            R[o + i] = v;
        }
        if (Z) Z[o + i] = v;
        acc += v * v;
    }
    acc = block_sum(acc, sh);
    if (threadIdx.x == 0) {
        norm_part[c * kReduceBlocks + blockIdx.x] = acc;
        __threadfence();
        last = atomicInc(count, gridDim.x * gridDim.y - 1) == gridDim.x * gridDim.y - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double worst = 0.0;
    bool left = false;
    for (int k = 0; k < gridDim.y; ++k) {
        double v = 0.0;
        for (int q = threadIdx.x; q < kReduceBlocks; q += 256) v += __ldcg(norm_part + k * kReduceBlocks + q);
        v = block_sum(v, sh);
        if (threadIdx.x != 0) continue;
        hr[k] = v;
        if (!st) continue;
        const double rel = hb[k] > 0.0 ? sqrt(v / hb[k]) : 0.0;
        if (active[k] && rel <= st->tol) active[k] = 0;
        left |= active[k] != 0;
        worst = fmax(worst, rel);
    }
    if (st && threadIdx.x == 0) {
        ++st->it;
        st->worst = worst;
        if (!left) st->stop = 1;
    }
}

// p = z + beta p with beta = rz_new / rz_old; rz_new from its partial sums, also stored.
__global__ void __launch_bounds__(256)
    pcg_p_kernel(double *__restrict__ P, const double *__restrict__ Z, const double *__restrict__ rz_part,
                 const double *__restrict__ rz_old, double *__restrict__ rz_new, const int *__restrict__ active,
                 int64_t n, const PcgState *st) {
    if (st && st->stop) return;
    __shared__ double sh[8];
    const int c = blockIdx.y;
    const double num = partial_sum(rz_part + c * kReduceBlocks, sh);
    if (blockIdx.x == 0 && threadIdx.x == 0) rz_new[c] = num;
    if (!active[c]) return;
    const double beta = rz_old[c] != 0.0 ? num / rz_old[c] : 0.0;
    const int64_t o = int64_t(c) * n;
    for (int64_t i = blockIdx.x * int64_t(256) + threadIdx.x; i < n; i += int64_t(gridDim.x) * 256)
        P[o + i] = Z[o + i] + beta * P[o + i];
}

// z = s s r (the Jacobi preconditioner, s = D^{-1/2}) and partial sums of r . z.
__global__ void __launch_bounds__(256)
    pcg_jacobi_kernel(const double *__restrict__ R, const double *__restrict__ s, double *__restrict__ Z, int64_t n,
                      double *__restrict__ rz_part, const int *__restrict__ stop) {
    if (stop && *stop) return;
    __shared__ double sh[8];
    const int64_t o = int64_t(blockIdx.y) * n;
    double acc = 0.0;
    for (int64_t i = blockIdx.x * int64_t(256) + threadIdx.x; i < n; i += int64_t(kReduceBlocks) * 256) {
        const double v = R[o + i], z = (v * s[i]) * s[i];
        Z[o + i] = z;
        acc += v * z;
    }
    acc = block_sum(acc, sh);
    if (threadIdx.x == 0) rz_part[blockIdx.y * kReduceBlocks + blockIdx.x] = acc;
}

__global__ void copy_kernel(double *__restrict__ dst, const double *__restrict__ src, int64_t count) {
    for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t < count;
         t += int64_t(gridDim.x) * blockDim.x)
        dst[t] = src[t];
}

__global__ void axpy_kernel(double *__restrict__ y, const double *__restrict__ x, double alpha, int64_t count) {
    for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t < count;
         t += int64_t(gridDim.x) * blockDim.x)
        y[t] += alpha * x[t];
}

inline int grid_for(int64_t n, int threads) {
    int64_t g = (n + threads - 1) / threads;
    if (g > 148 * 32) g = 148 * 32;
    if (g < 1) g = 1;
    return int(g);
}

}  // namespace

int reduce_partials_count() { return kReduceBlocks; }

void launch_spmv(const int64_t *ptr, const int64_t *src, const int32_t *col, const int32_t *flag, int64_t nrows,
                 int vb, int src_ld, const double *Ax, const double *X, double *Y, int64_t ld, int nrhs,
                 cudaStream_t st, double *dotp, const int *stop) {
    if (nrows <= 0) {
        if (dotp) cudaMemsetAsync(dotp, 0, size_t(kReduceBlocks) * nrhs * sizeof(double), st);
        return;
    }
    if (vb != 3) {
        ++g_kernel_launches;
        spmv_kernel<<<grid_for(nrows * vb * nrhs, 256), 256, 0, st>>>(ptr, src, col, flag, nrows, vb, src_ld, Ax, X, Y,
                                                                       ld, nrhs);
        if (dotp) launch_coldot_partial(X, Y, nrows * vb, nrhs, dotp, st);
        return;
    }
    const int grid = dotp ? kReduceBlocks : int(std::min<int64_t>((nrows + 31) / 32, 148 * 8));
    for (int r = 0; r < nrhs; r += 4) {
        const int nr = std::min(4, nrhs - r);
        auto kern = nr == 1 ? spmv3_kernel<1> : nr == 2 ? spmv3_kernel<2> : spmv3_kernel<4>;
        ++g_kernel_launches;
        kern<<<grid, 256, 0, st>>>(ptr, src, col, flag, nrows, src_ld, Ax, X + r * ld, Y + r * ld, ld, nr,
                                   dotp ? dotp + r * kReduceBlocks : nullptr, stop);
    }
}

void launch_gather_rows(const int64_t *map, int64_t n_in, const double *in, int64_t ld_in, double *out,
                        int64_t ld_out, int nrhs, cudaStream_t st) {
    if (n_in <= 0) return;
    ++g_kernel_launches;
    gather_rows_kernel<<<grid_for(n_in * nrhs, 256), 256, 0, st>>>(map, n_in, in, ld_in, out, ld_out, nrhs);
}

void launch_scatter_rows(const int64_t *map, int64_t n_out, const double *in, int64_t ld_in, double *out,
                         int64_t ld_out, int nrhs, cudaStream_t st) {
    if (n_out <= 0) return;
    ++g_kernel_launches;
    scatter_rows_kernel<<<grid_for(n_out * nrhs, 256), 256, 0, st>>>(map, n_out, in, ld_in, out, ld_out, nrhs);
}

void launch_assemble_elements(const int64_t *slot_ptr, const int64_t *contrib, int64_t nslots, const double *Ke,
                              double *Ax, cudaStream_t st) {
    if (nslots <= 0) return;
    ++g_kernel_launches;
    assemble_elements_kernel<<<grid_for(nslots * 9, 256), 256, 0, st>>>(slot_ptr, contrib, nslots, Ke, Ax);
}

void launch_coldot_partial(const double *X, const double *Y, int64_t n, int nrhs, double *partials, cudaStream_t st) {
    ++g_kernel_launches;
    coldot_partial_kernel<<<dim3(kReduceBlocks, nrhs), 256, 0, st>>>(X, Y, n, partials);
}

void launch_coldot(const double *X, const double *Y, int64_t n, int nrhs, double *partials, double *out,
                   cudaStream_t st) {
    launch_coldot_partial(X, Y, n, nrhs, partials, st);
    ++g_kernel_launches;
    coldot_final_kernel<<<nrhs, 256, 0, st>>>(partials, out);
}

void launch_colnorm2(const double *X, int64_t n, int nrhs, double *partials, double *out, cudaStream_t st) {
    launch_coldot(X, X, n, nrhs, partials, out, st);
}

void launch_pcg_update_x_r(double *X, double *R, const double *P, const double *AP, const double *rz,
                           const double *pap_part, int *active, int64_t n, int nrhs, double *Z, double *norm_part,
                           double *hr, unsigned *count, const double *hb, PcgState *state, cudaStream_t st) {
    ++g_kernel_launches;
    pcg_xr_kernel<<<dim3(kReduceBlocks, nrhs), 256, 0, st>>>(X, R, P, AP, rz, pap_part, active, n, Z, norm_part, hr,
                                                             count, hb, state);
}

void launch_pcg_update_p(double *P, const double *Z, const double *rz_part, const double *rz_old, double *rz_new,
                         const int *active, int64_t n, int nrhs, const PcgState *state, cudaStream_t st) {
    ++g_kernel_launches;
    pcg_p_kernel<<<dim3(kReduceBlocks, nrhs), 256, 0, st>>>(P, Z, rz_part, rz_old, rz_new, active, n, state);
}

void launch_pcg_jacobi(const double *R, const double *s, double *Z, int64_t n, int nrhs, double *rz_part,
                       const int *stop, cudaStream_t st) {
    ++g_kernel_launches;
    pcg_jacobi_kernel<<<dim3(kReduceBlocks, nrhs), 256, 0, st>>>(R, s, Z, n, rz_part, stop);
}

void launch_copy(double *dst, const double *src, int64_t count, cudaStream_t st) {
    if (count <= 0) return;
    ++g_kernel_launches;
    copy_kernel<<<grid_for(count, 256), 256, 0, st>>>(dst, src, count);
}

void launch_axpy(double *y, const double *x, double alpha, int64_t count, cudaStream_t st) {
    if (count <= 0) return;
    ++g_kernel_launches;
    axpy_kernel<<<grid_for(count, 256), 256, 0, st>>>(y, x, alpha, count);
}

}  // namespace mfs
