// Tensor-core tile GEMMs for the supernodal Schur updates (K5) and the
// inverse-based panel solves (K4):
//     mode 0:  C(i,j) -= sum_k A(i,k) B(j,k)      (SYRK / trailing update, "NT")
//     mode 1:  C(i,j)  = sum_k A(i,k) B(j,k)      (panel rows times inv(L_kk)^T)
// A, B and C are column-major sub-blocks addressed by per-task offsets; a task
// covers an m x n block with tiles_m x tiles_n CTA tiles and an optional lower
// mask (only i >= j is touched, tiles strictly above the diagonal exit early).
// One launch carries the tasks of every large front of a level.
//
// FP32 factors: single-pass TF32 runs on the 5th-generation tensor cores
// (tcgen05, kernels_gemm_tc.cu); the split 3xTF32 form (a = a_hi + a_lo, three
// products, FP32-level accuracy) and a legacy single-pass form run here on
// mma.sync m16n8k8. FP64 factors run on the FP64 tensor-core path (mma.sync
// m8n8k4 DMMA). Tiles are staged through shared memory with cp.async (FP32 4 bytes,
// double buffered; FP64 16 bytes, four stages). An FP32 task tile is 128 x 256 (the tcgen05 tile); the
// mma.sync kernel covers it as two 128 x 128 halves and ignores the tcgen05
// alignment shift (its extra tiles find no rows or columns).
#include "device.h"

#include <cstdint>

namespace mfs {

namespace {

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void cp_async4(void *dst, const void *src, bool valid) {
    const uint32_t d = smem_u32(dst);
    const int sz = valid ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(sz) : "memory");
}
// 16-byte copy of `bytes` (0, 8 or 16) source bytes, zero-filling the rest.
__device__ __forceinline__ void cp_async16(void *dst, const void *src, int bytes) {
    const uint32_t d = smem_u32(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ uint32_t to_tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

__device__ __forceinline__ int find_task(const GemmTask *tasks, int ntasks, int t) {
    int lo = 0, hi = ntasks - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (tasks[mid].tile_base <= t) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// ---------------------------------------------------------------- TF32 ----
constexpr int TBM = 128, TBN = 128, TBK = 32, TLD = TBM + 8;   // TLD % 32 == 8: conflict-free fragments
constexpr int kTF32Smem = 2 * 2 * TBK * TLD * 4;
constexpr int kTaskTileN32 = 256;                                // FP32 task tile width

template <int SPLIT>
__device__ __forceinline__ void tf32_tile(const GemmTask &tk, int i0, int j0, const float *Abase,
                                          const float *__restrict__ Bbase, float *Cbase, float *As, float *Bs) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp & 1, wn = warp >> 1;        // 2 x 4 warps, warp tile 64 x 32
    const int gid = lane >> 2, tig = lane & 3;
    const float *A = Abase + tk.a_off;
    const float *B = Bbase + tk.b_off;
    const int K = tk.k;

    auto load = [&](int stage, int k0) {
        float *as = As + stage * TBK * TLD;
        float *bs = Bs + stage * TBK * TLD;
#pragma unroll
        for (int r = 0; r < (TBK * TBM) / 256; ++r) {
            const int l = tid + 256 * r;
            const int kk = l / TBM, ii = l % TBM;
            const int gk = k0 + kk;
            const bool va = (i0 + ii < tk.m) && gk < K;
            const bool vb = (j0 + ii < tk.n) && gk < K;
            cp_async4(as + kk * TLD + ii, va ? A + int64_t(gk) * tk.lda + i0 + ii : A, va);
            cp_async4(bs + kk * TLD + ii, vb ? B + int64_t(gk) * tk.ldb + j0 + ii : B, vb);
        }
        cp_commit();
    };

    float acc[4][4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[a][b][c] = 0.f;

    const int nk = (K + TBK - 1) / TBK;
    load(0, 0);
    for (int kc = 0; kc < nk; ++kc) {
        if (kc + 1 < nk) {
            load((kc + 1) & 1, (kc + 1) * TBK);
            cp_wait<1>();
        } else {
            cp_wait<0>();
        }
        __syncthreads();
        const float *as = As + (kc & 1) * TBK * TLD;
        const float *bs = Bs + (kc & 1) * TBK * TLD;
#pragma unroll
        for (int k8 = 0; k8 < TBK; k8 += 8) {
            uint32_t ah[4][4], bh[4][2];
            uint32_t al[4][4], bl[4][2];
#pragma unroll
            for (int mt = 0; mt < 4; ++mt) {
                const int m = wm * 64 + mt * 16 + gid;
                const float v0 = as[(k8 + tig) * TLD + m], v1 = as[(k8 + tig) * TLD + m + 8];
                const float v2 = as[(k8 + tig + 4) * TLD + m], v3 = as[(k8 + tig + 4) * TLD + m + 8];
                ah[mt][0] = to_tf32(v0); ah[mt][1] = to_tf32(v1); ah[mt][2] = to_tf32(v2); ah[mt][3] = to_tf32(v3);
                if (SPLIT == 3) {
                    al[mt][0] = to_tf32(v0 - __uint_as_float(ah[mt][0]));
                    al[mt][1] = to_tf32(v1 - __uint_as_float(ah[mt][1]));
                    al[mt][2] = to_tf32(v2 - __uint_as_float(ah[mt][2]));
                    al[mt][3] = to_tf32(v3 - __uint_as_float(ah[mt][3]));
                }
            }
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                const int n = wn * 32 + nt * 8 + gid;
                const float v0 = bs[(k8 + tig) * TLD + n], v1 = bs[(k8 + tig + 4) * TLD + n];
                bh[nt][0] = to_tf32(v0); bh[nt][1] = to_tf32(v1);
                if (SPLIT == 3) {
                    bl[nt][0] = to_tf32(v0 - __uint_as_float(bh[nt][0]));
                    bl[nt][1] = to_tf32(v1 - __uint_as_float(bh[nt][1]));
                }
            }
#pragma unroll
            for (int mt = 0; mt < 4; ++mt)
#pragma unroll
                for (int nt = 0; nt < 4; ++nt) {
                    if (SPLIT == 3) {
                        mma_tf32(acc[mt][nt], al[mt], bh[nt]);
                        mma_tf32(acc[mt][nt], ah[mt], bl[nt]);
                    }
                    mma_tf32(acc[mt][nt], ah[mt], bh[nt]);
                }
        }
        __syncthreads();
    }
    float *C = Cbase + tk.c_off;
#pragma unroll
    for (int mt = 0; mt < 4; ++mt)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = i0 + wm * 64 + mt * 16 + gid + (e >> 1) * 8;
                const int j = j0 + wn * 32 + nt * 8 + tig * 2 + (e & 1);
                if (i >= tk.m || j >= tk.n || (tk.lower && i < j)) continue;
                float *p = C + int64_t(j) * tk.ldc + i;
                if (tk.mode == 0) *p -= acc[mt][nt][e];
                else *p = acc[mt][nt][e];
            }
}

template <int SPLIT>
__global__ void __launch_bounds__(256) gemm_tf32_kernel(const GemmTask *__restrict__ tasks, int ntasks,
                                                        const float *Abase, const float *__restrict__ Bbase,
                                                        float *Cbase) {
    extern __shared__ __align__(16) float sm[];
    float *As = sm;                           // [2][TBK][TLD]
    float *Bs = sm + 2 * TBK * TLD;           // [2][TBK][TLD]
    const int t = blockIdx.x;
    const GemmTask tk = tasks[find_task(tasks, ntasks, t)];
    const int local = t - tk.tile_base;
    const int ti = local % tk.tiles_m, tj = local / tk.tiles_m;
    const int i0 = ti * TBM;
    // The halves run in order; an in-place task (C == A, n <= 128) is finished
    // by the first half before the second one (which has no columns) starts.
    for (int h = 0; h < kTaskTileN32 / TBN; ++h) {
        const int j0 = tj * kTaskTileN32 + h * TBN;
        if (j0 >= tk.n || (tk.lower && i0 + TBM - 1 < j0)) break;
        if (h) __syncthreads();
        tf32_tile<SPLIT>(tk, i0, j0, Abase, Bbase, Cbase, As, Bs);
    }
}

// ---------------------------------------------------------------- FP64 ----
// DMMA m8n8k4; a CTA tile is 128 x 64, warps 4 x 2 of 32 x 32, two CTAs per SM. What
// bounds it: the tensor pipe for the large updates (37 TFLOP/s measured for DMMA alone),
// latency for the column-block chain, whose launches have a few tiles and k of 64 to 192.
// The operands come by 16-byte cp.async through a ring of DST stages of 16 k (a tile starts
// at the 2-element aligned row at or before its operand, the extra row and column are
// not stored), and C is loaded in two batches: written as C -= acc element by element, each
// load waited for the store before it, most of a 25 us launch at k = 64. (Accumulators that
// start as -C, so that its loads overlap the ring's first fill, were slower: the level SYRKs
// at 24 instead of 26 TFLOP/s.) All GEMM launches of a factorization of the 48-sided cube:
// 123 ms with 8-byte copies, two stages and the element-by-element epilogue, 105 ms now
// (level SYRKs 26, the largest 30 TFLOP/s).
// Launches of at most kF64FewTiles tiles (the column-block chain of the large fronts) split
// every tile into four of 32 rows (all of its columns: a row solve is in place), since a
// tile alone takes 1.1 us of its SM per 16 k: left-looking updates of the 20-sided cube
// 19 us a launch on whole tiles, 12 us split; with more tiles than SMs the split only
// costs reads of B.
constexpr int DBM = 128, DBN = 64, DBK = 16, DST = 4;
constexpr int kF64FewTiles = 148;
template <int BM>
struct F64Tile {
    static constexpr int LDA = BM + 4, LDB = DBN + 4;         // 8 bytes x (4 k + row): conflict-free fragments
    static constexpr int STAGE = DBK * (LDA + LDB);          // doubles
    static constexpr int SMEM = DST * STAGE * 8;
    static constexpr int WM = BM == 128 ? 4 : 2, WN = 8 / WM; // warps along m, n
    static constexpr int MT = BM / WM / 8, NT = DBN / WN / 8; // 8 x 8 products per warp
};

template <int BM>
__global__ void __launch_bounds__(256, 2) gemm_f64_kernel(const GemmTask *__restrict__ tasks, int ntasks,
                                                          const double *Abase, const double *__restrict__ Bbase,
                                                          double *Cbase) {
    using S = F64Tile<BM>;
    constexpr int LDA = S::LDA, LDB = S::LDB, MT = S::MT, NT = S::NT, PARTS = DBM / BM;
    extern __shared__ __align__(16) double smd[];
    const int t = blockIdx.x / PARTS;
    const GemmTask tk = tasks[find_task(tasks, ntasks, t)];
    const int local = t - tk.tile_base;
    const int ti = local % tk.tiles_m, tj = local / tk.tiles_m;
    const int da = tk.shift & 255, db = tk.shift >> 8;       // shifted row x is operand row x - d
    const int i0 = ti * DBM + int(blockIdx.x % PARTS) * BM, j0 = tj * DBN;   // tile origin in shifted coordinates
    if (i0 >= tk.m + da || (tk.lower && i0 + BM - 1 - da < j0 - db)) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp % S::WM, wn = warp / S::WM;
    const int gid = lane >> 2, tig = lane & 3;
    const double *A = Abase + (tk.a_off - da) + i0;
    const double *B = Bbase + (tk.b_off - db) + j0;
    const int am = tk.m + da - i0, bn = tk.n + db - j0;      // rows / columns left in shifted coordinates
    const int K = tk.k, nk = (K + DBK - 1) / DBK;
    // copies: BM / 2 (A) and 32 (B) 16-byte chunks a k row; a thread has one chunk and every
    // KA-th (eighth) k row
    constexpr int CA = BM / 2, KA = 256 / CA;
    const int ca = (tid % CA) * 2, ka = tid / CA, cb = (tid & 31) * 2, kb0 = tid >> 5;
    const int na = min(2, max(0, am - ca)) * 8, nb = min(2, max(0, bn - cb)) * 8;
    auto load = [&](int kc) {
        double *as = smd + (kc % DST) * S::STAGE;
        double *bs = as + DBK * LDA;
        const int k0 = kc * DBK;
#pragma unroll
        for (int r = 0; r < DBK / KA; ++r) {
            const int k = ka + KA * r, n = k0 + k < K ? na : 0;
            cp_async16(as + k * LDA + ca, n ? A + int64_t(k0 + k) * tk.lda + ca : Abase, n);
        }
#pragma unroll
        for (int r = 0; r < DBK / 8; ++r) {
            const int k = kb0 + 8 * r, n = k0 + k < K ? nb : 0;
            cp_async16(bs + k * LDB + cb, n ? B + int64_t(k0 + k) * tk.ldb + cb : Bbase, n);
        }
    };
    double acc[MT][NT][2];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) acc[mt][nt][0] = acc[mt][nt][1] = 0.0;
#pragma unroll
    for (int kc = 0; kc < DST - 1; ++kc) {
        if (kc < nk) load(kc);
        cp_commit();
    }
    for (int kc = 0; kc < nk; ++kc) {
        cp_wait<DST - 2>();
        __syncthreads();                                     // (also: stage kc - 1 is read)
        if (kc + DST - 1 < nk) load(kc + DST - 1);
        cp_commit();
        const double *as = smd + (kc % DST) * S::STAGE + wm * (8 * MT) + gid;
        const double *bs = smd + (kc % DST) * S::STAGE + DBK * LDA + wn * (8 * NT) + gid;
#pragma unroll
        for (int k4 = 0; k4 < DBK; k4 += 4) {
            double a[MT], b[NT];
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) a[mt] = as[(k4 + tig) * LDA + mt * 8];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) b[nt] = bs[(k4 + tig) * LDB + nt * 8];
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) mma_f64(acc[mt][nt], a[mt], b[nt]);
        }
    }
    cp_wait<0>();
    // an in-place row solve (C = A, the tile spans its columns) has read all of its rows
    __syncthreads();
    double *C = Cbase + tk.c_off;
    const int ib = i0 - da + wm * (8 * MT) + gid, jb = j0 - db + wn * (8 * NT) + tig * 2;
    auto live = [&](int mt, int nt, int e) {
        const int i = ib + mt * 8, j = jb + nt * 8 + e;
        return i >= 0 && i < tk.m && j >= 0 && j < tk.n && !(tk.lower && i < j);
    };
    auto at = [&](int mt, int nt, int e) { return C + int64_t(jb + nt * 8 + e) * tk.ldc + ib + mt * 8; };
    if (tk.mode == 0) {
        // half of the tile's C at a time (registers): every load before the first store
        constexpr int H = MT / 2;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            double c[H][NT][2];
#pragma unroll
            for (int m = 0; m < H; ++m)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        if (live(H * h + m, nt, e)) c[m][nt][e] = *at(H * h + m, nt, e);
#pragma unroll
            for (int m = 0; m < H; ++m)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        if (live(H * h + m, nt, e)) *at(H * h + m, nt, e) = c[m][nt][e] - acc[H * h + m][nt][e];
        }
    } else {
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int e = 0; e < 2; ++e)
                    if (live(mt, nt, e)) *at(mt, nt, e) = acc[mt][nt][e];
    }
}

}  // namespace

int gemm_tile_m(bool fp64) { return fp64 ? DBM : TBM; }
int gemm_tile_n(bool fp64) { return fp64 ? DBN : kTaskTileN32; }

template <>
void launch_gemm<float>(const GemmTask *tasks, int ntasks, int ntiles, const float *A, const float *B, float *C,
                        int split, int *err, cudaStream_t st) {
    if (ntiles <= 0) return;
    if (split == 1) {
        launch_gemm_tc(tasks, ntasks, ntiles, A, B, C, err, st);
        return;
    }
    ++g_kernel_launches;
    if (split == 3) {
        static PerDeviceOnce once3;
        once3([] { cudaFuncSetAttribute(gemm_tf32_kernel<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTF32Smem); });
        gemm_tf32_kernel<3><<<ntiles, 256, kTF32Smem, st>>>(tasks, ntasks, A, B, C);
    } else {
        static PerDeviceOnce once1;
        once1([] { cudaFuncSetAttribute(gemm_tf32_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTF32Smem); });
        gemm_tf32_kernel<1><<<ntiles, 256, kTF32Smem, st>>>(tasks, ntasks, A, B, C);
    }
}

template <>
void launch_gemm<double>(const GemmTask *tasks, int ntasks, int ntiles, const double *A, const double *B, double *C,
                         int split, int *err, cudaStream_t st) {
    (void)split;
    (void)err;
    if (ntiles <= 0) return;
    ++g_kernel_launches;
    static PerDeviceOnce once;
    once([] {
        cudaFuncSetAttribute(gemm_f64_kernel<DBM>, cudaFuncAttributeMaxDynamicSharedMemorySize, F64Tile<DBM>::SMEM);
        cudaFuncSetAttribute(gemm_f64_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, F64Tile<32>::SMEM);
    });
    if (ntiles <= kF64FewTiles)
        gemm_f64_kernel<32><<<ntiles * (DBM / 32), 256, F64Tile<32>::SMEM, st>>>(tasks, ntasks, A, B, C);
    else
        gemm_f64_kernel<DBM><<<ntiles, 256, F64Tile<DBM>::SMEM, st>>>(tasks, ntasks, A, B, C);
}

}  // namespace mfs
