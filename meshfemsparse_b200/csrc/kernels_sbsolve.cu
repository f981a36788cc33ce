// Triangular solves of the levels above the solve cut (K6): one persistent
// dataflow kernel per direction.
//
// Reference: SparseLDL::Solve (forward L y = b, backward L^T x = y; called at
// Solvers/CatamariFactorizer.cc:54,70) and its per-supernode kernels
// (trs_kernels::SolveLowerTri / MultiplyLowerBlock, solve_kernels::fused_forward /
// fused_backward, tests/test_catamari_solve_kernels.cc). The dependency chain of a
// front's L11 solve bounds the solve: a block of y cannot start before every
// earlier block is known. Here the chain runs over superblocks of SB = 256 rows:
// after the numeric factorization, sb_inverse_kernel writes inv(L_KK) of every
// superblock K of every front above the solve cut (dense, column-major, nrp x nrp
// with nrp = 64 * ceil(rows / 64), zeros above the diagonal), built from the
// 64 x 64 diagonal inverses by block forward substitution.
//
// Tasks (one CTA each; SbTask), v = right-hand side of the front's rows with the
// children's update vectors added in child order (pulled through the children's
// inverse row maps once their structure tasks have counted):
//   forward, diagonal   64-row part h of superblock K: a_h = v_h - sum_{J < K}
//             L(rows h, superblock J) y_J (J ascending, as J's count reaches its part
//             count), a_h to a scratch vector, count; once every part of K has
//             counted, y_h = inv(L_KK)(rows h, :) a_K, count;
//   forward, structure  64 rows of L21: u = v - sum_J L21(rows, superblock J) y_J, to
//             the solve arena, count (the parent waits for the front's total);
//   backward            64 columns h of superblock K: a_h = y_h - L21^T x_struct (as the
//             ancestors' superblocks are done) - sum_{J > K} L(superblock J, columns h)^T x_J (J
//             descending), then x_h = inv(L_KK)(:, columns h)^T a_K the same way.
// What bounds it: the chain of the large fronts (two hops between CTAs and two
// 64 x 256 products a superblock) and, between the levels, the pass from a front's last
// structure task to its parent's first part. One launch for all levels and both kinds
// of task instead of one to four launches a level: the next level's fronts start as
// soon as their own children are done, the structure products stream L21 while the
// chain runs, and no partial sums go through memory. One pass over the factor in FP64
// with one right-hand side (k = 40, 201,720 variables, 19 levels above the cut):
// 5.56 ms before (133 launches), 1.53 ms now; FP32 with 32 of them, refined in 4 iterations
// (k = 48, 345,744 variables): 146 ms before, 61 ms now.
//
// A CTA is 8 product warps and 8 warps that run ahead of them through the CTA's tasks, so
// that a small task costs its products and not its chain of dependent loads (a structure
// task of 64 rows x 33 columns took 4.1 us with the loads in line, 1.5 us this way):
//   copy warp     its lane 0 streams L and the inverses through shared memory in 32 KB
//                 chunks (64 rows x 128 FP32 / 64 FP64 columns forward, 128 / 64 rows x
//                 64 columns backward), one 2D TMA box per chunk through per-front /
//                 per-inverse tensor maps, across the borders of tasks: what a task reads
//                 after its last dependency arrives is already on chip;
//   vector warps  wait for the counts and bring y_J / x_J / x_struct, 256 rows at a time,
//                 into VS buffers;
//   gather warps  v of every task's own rows (forward: the children's counts, their row
//                 maps, their u);
//   count warp    publishes a structure task's results once all product warps have handed
//                 them over.
// Structure rows start at w rounded down to a multiple of 4 (TMA boxes start 16-byte
// aligned); the rows before w are not stored forward and cleared backward, and what a box
// holds past the front is zero.
//
// Launches are cooperative (all CTAs co-resident); every CTA walks its tasks in
// ascending order and a task waits only on lower-numbered tasks and on the other
// parts of its own superblock (adjacent task numbers, so on other CTAs), hence
// the lowest unfinished task can always proceed. Counts are zeroed before each
// solve: forward targets are eight (warps) times the superblock's part count, backward
// ones twice that. Waits are bounded in time: on expiry the kernel records an error and
// stops waiting; the host reports MFS_TIMEOUT. What a warp does and where it stores follows
// from the task list alone, never from what a wait was for, so that after an expiry only
// values are wrong; the product warps of a launch after one return at once. Sums run in a fixed
// order, so results are run-to-run identical. With an FP32 factor (the preconditioner of
// FP64 refinement) the products are FP32, summed in FP32 over at most 256 columns
// (forward) / 1024 rows (backward) and beyond that in FP64, and the inverse of the
// diagonal superblock is applied in FP64; an FP64 factor keeps FP64 throughout.
#include "device.h"

#include <algorithm>
#include <type_traits>

namespace mfs {

namespace {

constexpr int SB = kSuperBlock;
constexpr int kSbProducts = 256;                         // product threads (8 warps)
constexpr int kVecWarps = 4, kGatherWarps = 2;
constexpr int kSbThreads = kSbProducts + 32 * (2 + kVecWarps + kGatherWarps);
constexpr int kPubSlots = 4;                             // counts under way
constexpr int own_slots(int nr) { return nr > 4 ? 4 : 8; }   // tasks whose own rows are gathered ahead
// A gather warp's task `it` waits for the slot's task it - slots by the parity of its
// phase, which only tells that phase from the one before it; the warp's own last wait
// (for task it - warps - slots) covers the earlier ones as long as warps <= slots.
static_assert(kGatherWarps <= own_slots(8), "gather warps");
constexpr unsigned long long kWaitNs = 2000000000ull;    // 2 s per wait at most
static_assert(SB == kSbProducts, "one product thread per superblock row");

__device__ __forceinline__ int ld_acquire(const int *p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(int *p, int v) {
    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned long long gtimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Product type of the off-diagonal chunk sums: FP32 for an FP32 factor, FP64 otherwise.
template <typename T>
using PT = std::conditional_t<sizeof(T) == 4, float, double>;

// Chunks of 32 KB: forward 64 rows x FC columns (column-major, ld 64), backward
// FC rows x 64 columns (column-major, ld FC).
template <typename T>
struct SpChunk {
    static constexpr int FC = 32768 / (64 * int(sizeof(T)));   // 128 (FP32), 64 (FP64)
    static constexpr int ELEMS = 64 * FC;
    static constexpr int BYTES = ELEMS * int(sizeof(T));
};
// Shared memory: ring [NST][32 KB] | vp [VS][SB * NR] products' type (the vector warps'
// buffers) | red [8][NR][64] doubles (per-warp partial sums; its start also holds the
// exchanged a_K, [SB * NR] doubles) | own [own_slots][NR][64] doubles.
template <typename T, int NST, int NR, int VS>
struct SpLayout {
    static constexpr size_t vp_off = size_t(NST) * SpChunk<T>::BYTES;
    static constexpr size_t red_off = vp_off + size_t(VS) * NR * SB * sizeof(PT<T>);
    static constexpr size_t own_off = red_off + size_t(8) * NR * 64 * sizeof(double);
    static constexpr size_t bytes = own_off + size_t(own_slots(NR)) * NR * 64 * sizeof(double);
};

// Rows of superblock K of a front with w columns, and its 64-rounded extent.
__device__ __forceinline__ int sb_rows(int w, int K) { return min(SB, w - K * SB); }
__device__ __forceinline__ int sb_pad(int nr) { return (nr + 63) & ~63; }

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint32_t bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Bounded wait for the phase with the given parity; false on expiry (the error is
// recorded) or once another wait has expired: what follows is not trusted then.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int *err) {
    if (mbar_try(bar, parity)) return true;
    const unsigned long long t0 = gtimer();
    for (int it = 0;; ++it) {
        if (mbar_try(bar, parity)) return true;
        if ((it & 15) == 0) {                            // (at once: after an expiry every wait ends quickly)
            if (*(volatile int *)err) return false;
            if (gtimer() - t0 > kWaitNs) {
                atomicExch(err, 1);
                return false;
            }
        }
    }
}
// The product warps' barrier, and one that tells all of them whether any thread says so.
__device__ __forceinline__ void psync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
__device__ __forceinline__ bool psync_or(int pred) {
    int any;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.s32 p, %1, 0;\n\t"
        "bar.red.or.pred q, 1, 256, p;\n\t"
        "selp.s32 %0, 1, 0, q;\n\t}"
        : "=r"(any)
        : "r"(pred)
        : "memory");
    return any != 0;
}
// 2D tiled TMA load of one box of the tensor map at `map` (device memory written
// before the launch), box origin (x = row, y = column), completing on `bar`.
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const char *map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
        "[%4];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// The calling lanes wait until the count at p reaches target (bounded).
__device__ __forceinline__ void spin_count(const int *p, int target, int *err) {
    if (ld_acquire(p) >= target) return;
    const unsigned long long t0 = gtimer();
    for (int it = 1; ld_acquire(p) < target; ++it) {
        if (it & 31) continue;                           // (each look costs a round trip to L2)
        if (*(volatile int *)err) return;
        if (gtimer() - t0 > kWaitNs) {
            atomicExch(err, 1);
            return;
        }
    }
}
// N consecutive values from shared memory with 16-byte loads (N * sizeof(V) a multiple
// of 16, 16-byte aligned).
template <int N>
__device__ __forceinline__ void lds_vec(float (&x)[N], const float *p) {
#pragma unroll
    for (int k = 0; k < N / 4; ++k) {
        const float4 v = reinterpret_cast<const float4 *>(p)[k];
        x[4 * k] = v.x;
        x[4 * k + 1] = v.y;
        x[4 * k + 2] = v.z;
        x[4 * k + 3] = v.w;
    }
}
template <int N>
__device__ __forceinline__ void lds_vec(double (&x)[N], const double *p) {
#pragma unroll
    for (int k = 0; k < N / 2; ++k) {
        const double2 v = reinterpret_cast<const double2 *>(p)[k];
        x[2 * k] = v.x;
        x[2 * k + 1] = v.y;
    }
}

// Forward product of one chunk (64 rows x FC columns, column-major): the warp's FC / 8
// columns, two rows (2 lane, 2 lane + 1) per lane; v holds the vectors [r][SB].
template <typename T, typename V, int NR>
__device__ __forceinline__ void fwd_chunk(const T *ck, const V *v, V (&acc)[2][NR], int wp, int lane) {
    constexpr int QW = SpChunk<T>::FC / 8;
    using T2 = std::conditional_t<sizeof(T) == 4, float2, double2>;
    const T *a = ck + wp * QW * 64 + 2 * lane;
    const V *x = v + wp * QW;
#pragma unroll
    for (int j = 0; j < QW; j += 4) {
        T2 l[4];
        V xv[NR][4];
#pragma unroll
        for (int u = 0; u < 4; ++u) l[u] = *reinterpret_cast<const T2 *>(a + (j + u) * 64);
#pragma unroll
        for (int r = 0; r < NR; ++r) lds_vec(xv[r], x + r * SB + j);
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                acc[0][r] += V(l[u].x) * xv[r][u];
                acc[1][r] += V(l[u].y) * xv[r][u];
            }
    }
}

// Backward products: how a warp's lanes share a chunk's rows and the right-hand sides.
// With 8 right-hand sides the half-warps take 4 each (64 accumulators a lane otherwise).
template <typename T, int NR>
struct BwdLanes {
    static constexpr int RH = NR > 4 ? 2 : 1, NL = NR / RH;          // groups of lanes, right-hand sides each
    static constexpr int LN = 32 / RH, RV = SpChunk<T>::FC / LN;     // lanes of a group, rows per lane
    static constexpr int N = 8 * NL;                                 // a lane's accumulators (8 columns)
    static constexpr int NV = N > LN ? N / LN : 1;                   // sums a lane ends with
    static constexpr int VW = 16 / int(sizeof(T));                   // rows per 16-byte load
    // first of the chunk rows of vector load k of a lane (loads of a group are contiguous)
    static __device__ __forceinline__ int row(int lane, int k) { return (k * LN + (lane & (LN - 1))) * VW; }
};
// One chunk (FC rows x 64 columns, column-major) times v ([r][SB]): the warp's 8 columns
// from col0 on, rows below nrows.
template <typename T, typename V, int NR>
__device__ __forceinline__ void bwd_chunk(const T *ck, const V *v, V (&acc)[BwdLanes<T, NR>::N], int col0, int lane,
                                          int nrows) {
    using B = BwdLanes<T, NR>;
    constexpr int FC = SpChunk<T>::FC, VW = B::VW;
    const V *vr = v + (lane / B::LN) * B::NL * SB;
#pragma unroll
    for (int k = 0; k < B::RV / VW; ++k) {
        const int row = B::row(lane, k);
        if (row >= nrows) break;
        V xv[B::NL][VW];
#pragma unroll
        for (int r = 0; r < B::NL; ++r) lds_vec(xv[r], vr + r * SB + row);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            T l[VW];
            lds_vec(l, ck + (col0 + u) * FC + row);
#pragma unroll
            for (int e = 0; e < VW; ++e)
#pragma unroll
                for (int r = 0; r < B::NL; ++r) acc[u * B::NL + r] += V(l[e]) * xv[r][e];
        }
    }
}

// Sum N values (a power of two) over groups of LN lanes, spreading the sums: at each step
// a lane keeps one half of its values and hands the other to its partner. Lane `lane`
// ends with the sums spread_index, spread_index + 1, .. (N / LN of them; one, held by
// LN / N lanes, when N < LN).
template <int N, int LN, typename V>
__device__ __forceinline__ void spread_sum(V (&v)[N], int lane) {
    int n = N;
#pragma unroll
    for (int o = LN / 2; o > 0; o >>= 1) {
        if (n > 1) {
            n >>= 1;
            const bool up = lane & o;
#pragma unroll
            for (int k = 0; k < N / 2; ++k)
                if (k < n) {
                    const V give = up ? v[k] : v[k + n], keep = up ? v[k + n] : v[k];
                    v[k] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                }
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        }
    }
}
template <int N, int LN>
__device__ __forceinline__ int spread_index(int lane) {
    int idx = 0, n = N;
#pragma unroll
    for (int o = LN / 2; o > 0; o >>= 1)
        if (n > 1) {
            n >>= 1;
            if (lane & o) idx += n;
        }
    return idx;
}
// Whether this lane is the one that stores its value (N < LN: the first of its holders).
template <int N, int LN>
__device__ __forceinline__ bool spread_first(int lane) {
    return N >= LN || (lane & (LN / N - 1)) == 0;
}

// Barriers of a CTA: chunk ring, vector buffers, gathered own rows (full / empty each).
template <int NST, int VS, int OS>
struct SpBars {
    uint64_t full[NST], empty[NST], vfull[VS], vempty[VS], ofull[OS], oempty[OS], pfull[kPubSlots], pempty[kPubSlots];
};
struct SpRing {
    uint32_t full, empty, vfull, vempty, ofull, oempty, pfull, pempty;
};
template <int NST, int VS, int OS>
__device__ __forceinline__ SpRing init_bars(SpBars<NST, VS, OS> &b) {
    const SpRing rg{smem_u32(b.full),   smem_u32(b.empty), smem_u32(b.vfull),
                    smem_u32(b.vempty), smem_u32(b.ofull), smem_u32(b.oempty), smem_u32(b.pfull), smem_u32(b.pempty)};
    if (threadIdx.x == 0) {
        for (int k = 0; k < NST; ++k) {
            mbar_init(rg.full + 8 * k, 1);
            mbar_init(rg.empty + 8 * k, 8);
        }
        for (int k = 0; k < VS; ++k) {
            mbar_init(rg.vfull + 8 * k, 64);
            mbar_init(rg.vempty + 8 * k, 8);
        }
        for (int k = 0; k < OS; ++k) {
            mbar_init(rg.ofull + 8 * k, 32);
            mbar_init(rg.oempty + 8 * k, 8);
        }
        for (int k = 0; k < kPubSlots; ++k) {
            mbar_init(rg.pfull + 8 * k, 8);
            mbar_init(rg.pempty + 8 * k, 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    return rg;
}

// The product warps' tasks, by the last two bits of their number: four threads copy a task
// two ahead of its use, and a product barrier of the task in between makes it visible.
static_assert(sizeof(SbTask) == 64, "a task is four 16-byte copies");
__device__ __forceinline__ void fetch_task(SbTask (&meta)[4], int it, const SbTask *tasks, int t, int ntasks, int tid) {
    if (tid < 4 && t < ntasks)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_u32(&meta[it & 3]) + 16 * tid),
                     "l"(reinterpret_cast<const char *>(tasks + t) + 16 * tid)
                     : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
}
// (all but the newest copy have landed)
__device__ __forceinline__ void task_landed() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

// What a task streams. Forward: ndep chunks of earlier superblocks (diagonal tasks) or
// of the whole width (structure tasks, K < 0), then ninv chunks of the inverse.
template <typename T>
struct FwdShape {
    int w, f, R0, ndep, ninv, ngroups;
    __device__ __forceinline__ explicit FwdShape(const SbTask &tk) : w(tk.w), f(tk.f) {
        constexpr int FC = SpChunk<T>::FC;
        if (tk.K < 0) {
            R0 = (w & ~3) + tk.pad * 64;
            ndep = (w + FC - 1) / FC;
            ninv = 0;
            ngroups = (w + SB - 1) / SB;
        } else {
            R0 = tk.K * SB + tk.pad * 64;
            ndep = tk.K * (SB / FC);
            ninv = ((tk.pad + 1) * 64 + FC - 1) / FC;    // up to the rows' last nonzero column
            ngroups = tk.K;
        }
    }
};
// Backward: nstr chunks of L21 (groups of 256 rows from the last up), nql of the last superblock, then the others down to K + 1,
// then ninv of the inverse (from row 64 h on).
template <typename T>
struct BwdShape {
    static constexpr int FC = SpChunk<T>::FC, per = SB / FC;
    int w, f, nsb, C0, nstr, nsg, nql, ndep, ninv, irows;
    __device__ __forceinline__ explicit BwdShape(const SbTask &tk) : w(tk.w), f(tk.f) {
        nsb = (w + SB - 1) / SB;
        C0 = tk.K * SB + tk.pad * 64;
        nstr = f > w ? (f - (w & ~3) + FC - 1) / FC : 0;
        nsg = (nstr + per - 1) / per;
        nql = tk.K < nsb - 1 ? (sb_pad(sb_rows(w, nsb - 1)) + FC - 1) / FC : 0;
        ndep = nql > 0 ? nql + (nsb - 2 - tk.K) * per : 0;
        irows = sb_pad(sb_rows(w, tk.K)) - tk.pad * 64;
        ninv = (irows + FC - 1) / FC;
    }
    // chunk q of the superblock part: superblock J, chunk c of it
    __device__ __forceinline__ void dep(int q, int &J, int &c) const {
        if (q < nql) {
            J = nsb - 1;
            c = q;
        } else {
            J = nsb - 2 - (q - nql) / per;
            c = (q - nql) % per;
        }
    }
};

// Copy warp, lane 0: every chunk of the CTA's tasks in order into the ring.
template <typename T, int NST, bool FWD>
__device__ __forceinline__ void copy_chunks(const SbTask *tasks, int ntasks, const char *maps, T *ring,
                                            const SpRing &rg, int *err) {
    constexpr int FC = SpChunk<T>::FC, CE = SpChunk<T>::ELEMS;
    long long gq = 0;
    bool ok = true;
    auto load = [&](const char *map, int x, int y) {
        const int slot = int(gq % NST);
        // its last copy has landed (warps whose waits have expired hand slots back before
        // that, and a barrier takes one copy at a time), and it is read
        const uint32_t before = uint32_t((gq / NST) - 1) & 1u;
        if (gq >= NST && !(mbar_wait(rg.full + 8 * slot, before, err) && mbar_wait(rg.empty + 8 * slot, before, err)))
            ok = false;
        if (!ok) return;
        mbar_expect_tx(rg.full + 8 * slot, SpChunk<T>::BYTES);
        tma_load_2d(smem_u32(ring + slot * CE), map, x, y, rg.full + 8 * slot);
        ++gq;
    };
    for (int t = blockIdx.x; t < ntasks && ok; t += gridDim.x) {
        const SbTask tk = tasks[t];
        const char *pm = maps + size_t(tk.pmap + (FWD ? 0 : 1)) * kTensorMapBytes;
        const char *im = maps + size_t(tk.imap + (FWD ? 0 : 1)) * kTensorMapBytes;
        if constexpr (FWD) {
            const FwdShape<T> sh(tk);
            for (int q = 0; q < sh.ndep && ok; ++q) load(pm, sh.R0, q * FC);
            for (int c = 0; c < sh.ninv && ok; ++c) load(im, tk.pad * 64, c * FC);
        } else {
            const BwdShape<T> sh(tk);
            for (int g = sh.nsg - 1; g >= 0; --g)
                for (int c = g * (SB / FC); c < min(sh.nstr, (g + 1) * (SB / FC)) && ok; ++c)
                    load(pm, (sh.w & ~3) + c * FC, sh.C0);
            for (int q = 0; q < sh.ndep && ok; ++q) {
                int J, c;
                sh.dep(q, J, c);
                load(pm, J * SB + c * FC, sh.C0);
            }
            for (int c = 0; c < sh.ninv && ok; ++c) load(im, tk.pad * 64 + c * FC, tk.pad * 64);
        }
    }
    // whatever happened, the copies issued land before the CTA's shared memory goes away
    for (long long q = gq > NST ? gq - NST : 0; q < gq; ++q) {
        const uint32_t bar = rg.full + 8 * uint32_t(q % NST), par = uint32_t(q / NST) & 1u;
        const unsigned long long t0 = gtimer();
        while (!mbar_try(bar, par) && gtimer() - t0 < kWaitNs) {
        }
    }
}

// The warp's stores so far are published and counted (diagonal tasks: the chain waits, and
// eight warps releasing their own stores side by side are sooner done than one for all).
__device__ __forceinline__ void warp_count(int *p, int lane) {
    __syncwarp();
    if (lane == 0) asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(p) : "memory");
}
// Count warp, lane 0: once all product warps have handed over a structure task's stores,
// publish them to the GPU and count (a release waits for the stores to arrive, 0.8 us that
// the product warps would each spend otherwise: 1.5 instead of 2.15 us for a task of 64
// rows x 33 columns in FP64).
__device__ __forceinline__ void publish(const SbTask *tasks, int ntasks, const SpRing &rg, int *flags, int *err) {
    int e = 0;
    for (int t = blockIdx.x; t < ntasks; t += gridDim.x) {
        const SbTask tk = tasks[t];
        if (tk.K >= 0) continue;
        const int slot = e % kPubSlots;
        if (!mbar_wait(rg.pfull + 8 * slot, uint32_t(e / kPubSlots) & 1u, err)) return;
        asm volatile("fence.acq_rel.gpu;" ::: "memory");
        asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(flags + tk.flag0 + 2 * ((tk.w + SB - 1) / SB))
                     : "memory");
        mbar_arrive(rg.pempty + 8 * slot);
        ++e;
    }
}
// A product warp's side: its stores so far belong to the CTA's next count.
struct Handover {
    const SpRing &rg;
    int *err;
    int e = 0;
    __device__ __forceinline__ void operator()(int lane) {
        const int slot = e % kPubSlots;
        if (e >= kPubSlots) mbar_wait(rg.pempty + 8 * slot, uint32_t(e / kPubSlots - 1) & 1u, err);
        __syncwarp();
        if (lane == 0) mbar_arrive(rg.pfull + 8 * slot);
        ++e;
    }
};

// Vector warps: the vectors of every group of 256 rows, [r][256]. Two pairs take the groups
// in turn (a group costs a count's and a vector's round trip to L2, and small tasks have
// one each); a warp of a pair brings 128 rows. (A pair passes every second group, so its
// waits by parity are unambiguous with two buffers or more.)
constexpr int VR = SB / 2 / 32;                          // rows per lane

// Forward: y_J.
template <typename T, int NR, int VS>
__device__ __forceinline__ void fwd_vectors(const SbTask *tasks, int ntasks, const double *X,
                                            int64_t ldx, int nrhs, PT<T> *vp, const SpRing &rg, const int *flags,
                                            int *err, int me) {
    using P = PT<T>;
    const int pair = me >> 1, i0 = (me & 1) * (SB / 2) + (threadIdx.x & 31);
    long long gv = 0;
    for (int t = blockIdx.x; t < ntasks; t += gridDim.x) {
        const SbTask tk = tasks[t];
        const FwdShape<T> sh(tk);
        const int c0 = tk.c0;
        for (int J = 0; J < sh.ngroups; ++J, ++gv) {
            if (int(gv & 1) != pair) continue;
            const int slot = int(gv % VS);
            if (gv >= VS && !mbar_wait(rg.vempty + 8 * slot, uint32_t(gv / VS - 1) & 1u, err)) return;
            const int nrJ = sb_rows(sh.w, J);
            spin_count(flags + tk.flag0 + 2 * J, 8 * (sb_pad(nrJ) / 64), err);
            const double *xj = X + c0 + J * SB;
            P *dst = vp + slot * (NR * SB);
            double v[NR][VR];                      // (written by other CTAs: through L2)
#pragma unroll
            for (int r = 0; r < NR; ++r)
#pragma unroll
                for (int k = 0; k < VR; ++k) {
                    const int row = i0 + 32 * k;
                    v[r][k] = (row < nrJ && r < nrhs) ? __ldcg(xj + row + r * ldx) : 0.0;
                }
#pragma unroll
            for (int r = 0; r < NR; ++r)
#pragma unroll
                for (int k = 0; k < VR; ++k) dst[r * SB + i0 + 32 * k] = P(v[r][k]);
            mbar_arrive(rg.vfull + 8 * slot);
        }
    }
}

// Backward: x_struct from the last rows up (the ancestors are done from the root down, and
// each from its last superblock on, so that most of L21 is read while the parent's chain
// still runs), then x_J (J descending). A group's lowest row is the last to become final:
// rowcnt gives its superblock's count and parts.
template <typename T, int NR, int VS>
__device__ __forceinline__ void bwd_vectors(const SbTask *tasks, int ntasks, const SnDev &sd, const int32_t *rowcnt,
                                            const double *X, int64_t ldx, int nrhs, PT<T> *vp, const SpRing &rg,
                                            const int *flags, int *err, int me) {
    using P = PT<T>;
    const int pair = me >> 1, i0 = (me & 1) * (SB / 2) + (threadIdx.x & 31);
    const int vb = sd.vb;
    long long gv = 0;
    for (int t = blockIdx.x; t < ntasks; t += gridDim.x) {
        const SbTask tk = tasks[t];
        const BwdShape<T> sh(tk);
        const int c0 = tk.c0;
        const int32_t *rows = sd.struct_rows + sd.struct_ptr[tk.sn];
        const int nv = sh.nsg + (sh.nsb - 1 - tk.K);
        // the rows' places in X (-1: none) and the count to wait for, a group ahead of their use
        int64_t next[VR];
        int nflag = 0, nneed = 0;
        auto places = [&](int g) {
            if (g >= nv) return;
            if (g < sh.nsg) {
                const int base = (sh.w & ~3) + (sh.nsg - 1 - g) * SB;
                const int rc = rowcnt[rows[(max(base, sh.w) - sh.w) / vb]];
                nflag = rc >> 2;
                nneed = 16 * ((rc & 3) + 1);
#pragma unroll
                for (int k = 0; k < VR; ++k) {
                    const int row = base + i0 + 32 * k, li = row - sh.w;
                    next[k] = row >= sh.w && row < sh.f ? int64_t(rows[li / vb]) * vb + li % vb : -1;
                }
            } else {
                const int J = sh.nsb - 1 - (g - sh.nsg), nrJ = sb_rows(sh.w, J);
                nflag = tk.flag0 + 2 * J;
                nneed = 16 * (sb_pad(nrJ) / 64);
#pragma unroll
                for (int k = 0; k < VR; ++k) {
                    const int i = i0 + 32 * k;
                    next[k] = i < nrJ ? c0 + J * SB + i : -1;
                }
            }
        };
        places(int(gv & 1) == pair ? 0 : 1);
        for (int g = 0; g < nv; ++g, ++gv) {
            if (int(gv & 1) != pair) continue;
            const int slot = int(gv % VS);
            int64_t at[VR];
#pragma unroll
            for (int k = 0; k < VR; ++k) at[k] = next[k];
            const int flag = nflag, need = nneed;
            places(g + 2);
            if (gv >= VS && !mbar_wait(rg.vempty + 8 * slot, uint32_t(gv / VS - 1) & 1u, err)) return;
            spin_count(flags + flag, need, err);
            P *dst = vp + slot * (NR * SB);
            double v[NR][VR];
#pragma unroll
            for (int r = 0; r < NR; ++r)
#pragma unroll
                for (int k = 0; k < VR; ++k)
                    v[r][k] = (at[k] >= 0 && r < nrhs) ? __ldcg(X + at[k] + r * ldx) : 0.0;
#pragma unroll
            for (int r = 0; r < NR; ++r)
#pragma unroll
                for (int k = 0; k < VR; ++k) dst[r * SB + i0 + 32 * k] = P(v[r][k]);
            mbar_arrive(rg.vfull + 8 * slot);
        }
    }
}

// The own rows of a forward task of a front of ManyDev: its children are waited for, a lane
// each, then every row adds up its own list. (A call: rare, and inlined it costs the kernel
// registers.)
template <int NR>
__device__ __noinline__ void gather_many(const SbTask *task, int vb, const SbChild *children, const ManyDev &many,
                                         const double *X, int64_t ldx, int nrhs, const double *sol, const int *flags,
                                         int *err, double *o) {
    const int lane = threadIdx.x & 31, w = task->w, f = task->f, K = task->K;
    const ManyFront mf = many.fronts[task->many];
    for (int k = lane; k < mf.nwait; k += 32) {
        const SbChild &c = children[mf.child0 + k];
        if (c.flag >= 0) spin_count(flags + c.flag, c.need, err);
    }
    __syncwarp();
#pragma unroll 1
    for (int e = 0; e < 2; ++e) {
        const int row = (K < 0 ? (w & ~3) : K * SB) + task->pad * 64 + lane + 32 * e, brow = row / vb;
        const bool live = K < 0 ? (row >= w && row < f) : row < w;
        double v[NR];
#pragma unroll
        for (int r = 0; r < NR; ++r) v[r] = live && K >= 0 && r < nrhs ? X[task->c0 + row + r * ldx] : 0.0;
        const int64_t q1 = live ? many.ptr[mf.rows + brow + 1] : 0;
#pragma unroll 2
        for (int64_t q = live ? many.ptr[mf.rows + brow] : 0; q < q1; ++q) {
            const int2 en = many.ent[q];
            const SbChild &c = children[en.x];
            const double *uc = sol + c.sol * nrhs + en.y * vb + row - brow * vb;
            const int d = c.d;
#pragma unroll
            for (int r = 0; r < NR; ++r) v[r] += r < nrhs ? __ldcg(uc + int64_t(r) * d) : 0.0;
        }
#pragma unroll
        for (int r = 0; r < NR; ++r) o[r * 64 + lane + 32 * e] = v[r];
    }
}

// Gather warp `me`: every kGatherWarps-th task with its own rows, [r][64]. Forward: the
// right-hand side of a diagonal task's rows plus the children's update vectors, in child
// order; backward: y. What does not depend on a count (the task, its children, their row
// maps) is loaded a task ahead.
template <int NR, bool FWD, bool MANY>
__device__ __forceinline__ void gather_own(const SbTask *tasks, int ntasks, int vb, const SbChild *children,
                                           const int32_t *cmap, const ManyDev &many, const double *X, int64_t ldx, int nrhs,
                                           const double *sol, double *own, const SpRing &rg,
                                           const int *flags, int *err, int me) {
    constexpr int OS = own_slots(NR);
    const int lane = threadIdx.x & 31;
    struct Ahead {
        SbTask tk;
        SbChild ch[2];                                   // the first two children
        int m[2][2];                                     // [row][child]: block of the child's structure, or -1
    } nx;
    auto rows = [&](const SbTask &tk, int e, int &brow, int &off) {
        const int row = (tk.K < 0 ? (tk.w & ~3) : tk.K * SB) + tk.pad * 64 + lane + 32 * e;
        brow = row / vb;
        off = row - brow * vb;
        return tk.K < 0 ? (row >= tk.w && row < tk.f) : row < tk.w;
    };
    auto maps = [&](const SbTask &tk, int ci, SbChild (&ch)[2], int (&m)[2][2]) {
#pragma unroll
        for (int k = 0; k < 2; ++k)
            if (ci + k < tk.nchild) ch[k] = children[tk.child0 + ci + k];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            int brow, off;
            const bool live = rows(tk, e, brow, off);
#pragma unroll
            for (int k = 0; k < 2; ++k) m[e][k] = (ci + k < tk.nchild && live) ? cmap[ch[k].map + brow] : -1;
        }
    };
    auto ahead = [&](int t) {
        if (t >= ntasks) return;
        nx.tk = tasks[t];
        if constexpr (FWD) maps(nx.tk, 0, nx.ch, nx.m);
    };
    const int stride = gridDim.x * kGatherWarps;
    int it = me;
    ahead(blockIdx.x + me * int(gridDim.x));
    for (int t = blockIdx.x + me * gridDim.x; t < ntasks; t += stride, it += kGatherWarps) {
        const int slot = it % OS;
        const SbTask tk = nx.tk;
        double v[2][NR];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            int brow, off;
            const bool live = rows(tk, e, brow, off) && tk.K >= 0;
            const double *x = X + tk.c0 + brow * vb + off;
#pragma unroll
            for (int r = 0; r < NR; ++r) v[e][r] = (live && r < nrhs) ? x[r * ldx] : 0.0;
        }
        if constexpr (FWD) {
            SbChild ch[2] = {nx.ch[0], nx.ch[1]};
            int m[2][2] = {{nx.m[0][0], nx.m[0][1]}, {nx.m[1][0], nx.m[1][1]}};
            ahead(t + stride);
            if constexpr (MANY)
                if (tk.many >= 0) {
                    if (it >= OS && !mbar_wait(rg.oempty + 8 * slot, uint32_t(it / OS - 1) & 1u, err)) return;
                    gather_many<NR>(tasks + t, vb, children, many, X, ldx, nrhs, sol, flags, err,
                                    own + slot * (NR * 64));
                    mbar_arrive(rg.ofull + 8 * slot);
                    continue;
                }
            for (int ci = 0; ci < tk.nchild; ci += 2) {
                if (ci) maps(tk, ci, ch, m);
#pragma unroll
                for (int k = 0; k < 2; ++k)
                    if (ci + k < tk.nchild && ch[k].flag >= 0) spin_count(flags + ch[k].flag, ch[k].need, err);
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    double u[2][NR];
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        int brow, off;
                        rows(tk, e, brow, off);
                        const double *uc = sol + ch[k].sol * nrhs + m[e][k] * vb + off;
#pragma unroll
                        for (int r = 0; r < NR; ++r)
                            u[e][r] = (m[e][k] >= 0 && r < nrhs) ? __ldcg(uc + int64_t(r) * ch[k].d) : 0.0;
                    }
#pragma unroll
                    for (int e = 0; e < 2; ++e)
#pragma unroll
                        for (int r = 0; r < NR; ++r) v[e][r] += u[e][r];
                }
            }
        } else {
            ahead(t + stride);
        }
        if (it >= OS && !mbar_wait(rg.oempty + 8 * slot, uint32_t(it / OS - 1) & 1u, err)) return;
        double *o = own + slot * (NR * 64);
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int r = 0; r < NR; ++r) o[r * 64 + lane + 32 * e] = v[e][r];
        mbar_arrive(rg.ofull + 8 * slot);
    }
}

// MANY: some front has more than kManyChildren children (the branch alone costs the eight-wide
// form registers: 32 right-hand sides at k = 48 62.3 ms with it, 61.4 ms without).
template <typename T, int NST, int NR, int VS, bool MANY>
__global__ void __launch_bounds__(kSbThreads, 1)
    sp_fwd_kernel(const SbTask *__restrict__ tasks, int ntasks, SnDev sd, const char *__restrict__ maps,
                  const SbChild *__restrict__ children, ManyDev many, const int32_t *__restrict__ cmap, double *X,
                  int64_t ldx, int nrhs, double *sol, double *scratch, int *flags, int *err) {
    using Lay = SpLayout<T, NST, NR, VS>;
    using P = PT<T>;
    constexpr int FC = SpChunk<T>::FC, CE = SpChunk<T>::ELEMS, per = SB / FC;
    constexpr int NO = (NR + 3) / 4;
    extern __shared__ __align__(128) unsigned char sp_dyn[];
    constexpr int OS = own_slots(NR);
    __shared__ __align__(8) SpBars<NST, VS, OS> bars;
    __shared__ __align__(16) SbTask meta[4];
    // TMA destinations: 128-byte aligned (the launch adds 128 bytes for this)
    unsigned char *sp_raw = sp_dyn + ((128u - (smem_u32(sp_dyn) & 127u)) & 127u);
    T *ring = reinterpret_cast<T *>(sp_raw);
    P *vp = reinterpret_cast<P *>(sp_raw + Lay::vp_off);
    double *red = reinterpret_cast<double *>(sp_raw + Lay::red_off);
    double *vec = red;
    double *owns = reinterpret_cast<double *>(sp_raw + Lay::own_off);
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    const int expired = tid == 0 ? *(volatile int *)err : 0;   // a wait of an earlier launch
    fetch_task(meta, 0, tasks, blockIdx.x, ntasks, tid);
    fetch_task(meta, 1, tasks, blockIdx.x + gridDim.x, ntasks, tid);
    const SpRing rg = init_bars(bars);
    if (wp == 8) {
        if (lane == 0) copy_chunks<T, NST, true>(tasks, ntasks, maps, ring, rg, err);
        return;
    }
    if (wp > 8 && wp <= 8 + kVecWarps) {
        fwd_vectors<T, NR, VS>(tasks, ntasks, X, ldx, nrhs, vp, rg, flags, err, wp - 9);
        return;
    }
    if (wp == 9 + kVecWarps + kGatherWarps) {
        if (lane == 0) publish(tasks, ntasks, rg, flags, err);
        return;
    }
    if (wp > 8) {
        gather_own<NR, true, MANY>(tasks, ntasks, sd.vb, children, cmap, many, X, ldx, nrhs, sol, owns, rg, flags, err,
                              wp - 9 - kVecWarps);
        return;
    }
    task_landed();
    if (psync_or(expired)) return;                       // (the other warps' waits end too)
    const int i = tid & 63, part = tid >> 6;             // combining thread: row i, right-hand sides part + 4 o
    long long gq = 0, gv = 0;
    Handover handover{rg, err};
    auto chunk = [&]() -> const T * {
        const int slot = int(gq % NST);
        mbar_wait(rg.full + 8 * slot, uint32_t(gq / NST) & 1u, err);
        return ring + slot * CE;
    };
    auto release = [&]() {
        __syncwarp();
        if (lane == 0) mbar_arrive(rg.empty + 8 * uint32_t(gq % NST));
        ++gq;
    };
    // per-warp partial sums to shared memory, then the sum over warps of this thread's entries
    auto combine = [&](const double (&d)[2][NR], double (&out)[NO]) {
        psync();                                         // red / vec of before is read
#pragma unroll
        for (int r = 0; r < NR; ++r)
            *reinterpret_cast<double2 *>(red + (wp * NR + r) * 64 + 2 * lane) = make_double2(d[0][r], d[1][r]);
        psync();
#pragma unroll
        for (int o = 0; o < NO; ++o) {
            const int r = part + 4 * o;
            double s = 0.0;
            if (r < NR)
#pragma unroll
                for (int k = 0; k < 8; ++k) s += red[(k * NR + r) * 64 + i];
            out[o] = s;
        }
    };
    int it = 0;
    for (int t = blockIdx.x; t < ntasks; t += gridDim.x, ++it) {
        const int os = it % OS;
        fetch_task(meta, it + 2, tasks, t + 2 * gridDim.x, ntasks, tid);
        const SbTask tk = meta[it & 3];
        mbar_wait(rg.ofull + 8 * os, uint32_t(it / OS) & 1u, err);
        const int c0 = tk.c0;
        const FwdShape<T> sh(tk);
        const int w = sh.w, K = tk.K;
        const int row = sh.R0 + i;                       // front row of this thread's entries
        const bool live = K < 0 ? (row >= w && row < sh.f) : row < w;
        int *cnt = flags + tk.flag0;
        double own[NO];
#pragma unroll
        for (int o = 0; o < NO; ++o) own[o] = part + 4 * o < NR ? owns[(os * NR + part + 4 * o) * 64 + i] : 0.0;
        __syncwarp();
        if (lane == 0) mbar_arrive(rg.oempty + 8 * os);
        double dacc[2][NR];
#pragma unroll
        for (int r = 0; r < NR; ++r) dacc[0][r] = dacc[1][r] = 0.0;
        for (int J = 0, q = 0; J < sh.ngroups; ++J, ++gv) {
            const int slot = int(gv % VS), qe = min(sh.ndep, q + per);
            mbar_wait(rg.vfull + 8 * slot, uint32_t(gv / VS) & 1u, err);
            P pacc[2][NR];
#pragma unroll
            for (int r = 0; r < NR; ++r) pacc[0][r] = pacc[1][r] = P(0);
            for (int c = 0; q < qe; ++q, ++c) {
                const T *ck = chunk();
                if (J * SB + c * FC + wp * (FC / 8) < w)
                    fwd_chunk<T, P, NR>(ck, vp + slot * (NR * SB) + c * FC, pacc, wp, lane);
                release();
            }
            if (lane == 0) mbar_arrive(rg.vempty + 8 * slot);   // (after release's __syncwarp)
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                dacc[0][r] += double(pacc[0][r]);
                dacc[1][r] += double(pacc[1][r]);
            }
        }
        task_landed();
        double sum[NO];
        combine(dacc, sum);
        if (K < 0) {
#pragma unroll
            for (int o = 0; o < NO; ++o) {
                const int r = part + 4 * o;
                if (live && r < nrhs) sol[tk.sol * nrhs + (row - w) + int64_t(r) * (sh.f - w)] = own[o] - sum[o];
            }
            handover(lane);
            continue;
        }
        // a_h; exchanged with the other parts of K through the scratch vector
        const int nrK = sb_rows(w, K), nhK = sb_pad(nrK) / 64;
        if (nhK > 1) {
#pragma unroll
            for (int o = 0; o < NO; ++o) {
                const int r = part + 4 * o;
                if (live && r < nrhs) scratch[c0 + row + r * ldx] = own[o] - sum[o];
            }
            // (this CTA's eight warps are among the counted: all have read red then)
            warp_count(cnt + 2 * K + 1, lane);
            spin_count(cnt + 2 * K + 1, 8 * nhK, err);
#pragma unroll
            for (int r = 0; r < NR; ++r)
                vec[r * SB + tid] = (r < nrhs && tid < nrK) ? __ldcg(&scratch[c0 + K * SB + tid + r * ldx]) : 0.0;
        } else {
            psync();                                     // red is read, vec may be written
#pragma unroll
            for (int o = 0; o < NO; ++o) {
                const int r = part + 4 * o;
                if (r < NR) vec[r * SB + i] = (live && r < nrhs) ? own[o] - sum[o] : 0.0;
            }
        }
        psync();
#pragma unroll
        for (int r = 0; r < NR; ++r) dacc[0][r] = dacc[1][r] = 0.0;
        for (int c = 0; c < sh.ninv; ++c) {
            const T *ck = chunk();
            if (c * FC + wp * (FC / 8) < (tk.pad + 1) * 64)
                fwd_chunk<T, double, NR>(ck, vec + c * FC, dacc, wp, lane);
            release();
        }
        combine(dacc, sum);
#pragma unroll
        for (int o = 0; o < NO; ++o) {
            const int r = part + 4 * o;
            if (live && r < nrhs) X[c0 + row + r * ldx] = sum[o];
        }
        warp_count(cnt + 2 * K, lane);
    }
}

template <typename T, int NST, int NR, int VS>
__global__ void __launch_bounds__(kSbThreads, 1)
    sp_bwd_kernel(const SbTask *__restrict__ tasks, int ntasks, SnDev sd, const char *__restrict__ maps,
                  const SbChild *__restrict__ children, ManyDev many, const int32_t *__restrict__ rowcnt, double *X,
                  int64_t ldx, int nrhs, double *sol, double *scratch, int *flags, int *err) {
    using Lay = SpLayout<T, NST, NR, VS>;
    using P = PT<T>;
    using B = BwdLanes<T, NR>;
    constexpr int FC = SpChunk<T>::FC, CE = SpChunk<T>::ELEMS, per = SB / FC;
    constexpr int N = B::N, NV = B::NV;
    constexpr int kFlush = sizeof(T) == 4 ? 1024 / FC : 1 << 30;   // chunks between FP64 sums
    extern __shared__ __align__(128) unsigned char sp_dyn[];
    constexpr int OS = own_slots(NR);
    __shared__ __align__(8) SpBars<NST, VS, OS> bars;
    __shared__ __align__(16) SbTask meta[4];
    unsigned char *sp_raw = sp_dyn + ((128u - (smem_u32(sp_dyn) & 127u)) & 127u);
    T *ring = reinterpret_cast<T *>(sp_raw);
    P *vp = reinterpret_cast<P *>(sp_raw + Lay::vp_off);
    double *vec = reinterpret_cast<double *>(sp_raw + Lay::red_off);   // a_K, [r][SB]
    double *owns = reinterpret_cast<double *>(sp_raw + Lay::own_off);
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    const int expired = tid == 0 ? *(volatile int *)err : 0;   // a wait of an earlier launch
    fetch_task(meta, 0, tasks, blockIdx.x, ntasks, tid);
    fetch_task(meta, 1, tasks, blockIdx.x + gridDim.x, ntasks, tid);
    const SpRing rg = init_bars(bars);
    if (wp == 8) {
        if (lane == 0) copy_chunks<T, NST, false>(tasks, ntasks, maps, ring, rg, err);
        return;
    }
    if (wp > 8 && wp <= 8 + kVecWarps) {
        bwd_vectors<T, NR, VS>(tasks, ntasks, sd, rowcnt, X, ldx, nrhs, vp, rg, flags, err, wp - 9);
        return;
    }
    if (wp == 9 + kVecWarps + kGatherWarps) return;      // (forward only)
    if (wp > 8) {
        gather_own<NR, false, false>(tasks, ntasks, sd.vb, children, nullptr, many, X, ldx, nrhs, sol, owns, rg, flags, err,
                               wp - 9 - kVecWarps);
        return;
    }
    task_landed();
    if (psync_or(expired)) return;                       // (the other warps' waits end too)
    long long gq = 0, gv = 0;
    auto chunk = [&]() -> const T * {
        const int slot = int(gq % NST);
        mbar_wait(rg.full + 8 * slot, uint32_t(gq / NST) & 1u, err);
        return ring + slot * CE;
    };
    auto release = [&]() {
        __syncwarp();
        if (lane == 0) mbar_arrive(rg.empty + 8 * uint32_t(gq % NST));
        ++gq;
    };
    // the sums this lane ends with: columns and right-hand sides
    int scol[NV], srhs[NV];
    const bool first = spread_first<N, B::LN>(lane);
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int e = spread_index<N, B::LN>(lane) + k;
        scol[k] = wp * 8 + e / B::NL;
        srhs[k] = (lane / B::LN) * B::NL + e % B::NL;
    }
    int it = 0;
    for (int t = blockIdx.x; t < ntasks; t += gridDim.x, ++it) {
        const int os = it % OS;
        fetch_task(meta, it + 2, tasks, t + 2 * gridDim.x, ntasks, tid);
        const SbTask tk = meta[it & 3];
        mbar_wait(rg.ofull + 8 * os, uint32_t(it / OS) & 1u, err);
        const int c0 = tk.c0, K = tk.K;
        const BwdShape<T> sh(tk);
        const int w = sh.w;
        const int nch = min(64, w - sh.C0), nrK = sb_rows(w, K), nhK = sb_pad(nrK) / 64;
        int *cnt = flags + tk.flag0;
        double *xs = X + c0 + sh.C0;
        double own[NV], sum[NV];
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            own[k] = owns[(os * NR + srhs[k]) * 64 + scol[k]];
            sum[k] = 0.0;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(rg.oempty + 8 * os);
        P pacc[N];
#pragma unroll
        for (int k = 0; k < N; ++k) pacc[k] = P(0);
        int held = 0;
        auto flush = [&]() {
            spread_sum<N, B::LN>(pacc, lane);
#pragma unroll
            for (int k = 0; k < NV; ++k) sum[k] += double(pacc[k]);
#pragma unroll
            for (int k = 0; k < N; ++k) pacc[k] = P(0);
            held = 0;
        };
        // one vector buffer at a time: its chunks
        const int ngroups = sh.nsg + (sh.nsb - 1 - K);
        for (int g = 0; g < ngroups; ++g, ++gv) {
            const int slot = int(gv % VS);
            const int nc = g < sh.nsg ? min(per, sh.nstr - (sh.nsg - 1 - g) * per) : g == sh.nsg ? sh.nql : per;
            mbar_wait(rg.vfull + 8 * slot, uint32_t(gv / VS) & 1u, err);
            for (int c = 0; c < nc; ++c) {
                const T *ck = chunk();
                if (g == sh.nsg - 1 && c == 0 && (w & 3)) {
                    // L11's last rows, for the boxes' alignment: they meet zeros, but an infinite
                    // pivot among them does not (each warp clears the columns that it reads)
                    T *own_cols = ring + int(gq % NST) * CE + (wp * 8 + (lane & 7)) * FC;
                    if (lane < 8)
                        for (int e = 0; e < (w & 3); ++e) own_cols[e] = T(0);
                    // (before the slot's next copy)
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                }
                bwd_chunk<T, P, NR>(ck, vp + slot * (NR * SB) + c * FC, pacc, wp * 8, lane, FC);
                release();
                if (++held == kFlush) flush();
            }
            if (lane == 0) mbar_arrive(rg.vempty + 8 * slot);   // (after release's __syncwarp)
        }
        if (held > 0) flush();
        task_landed();
        // a_h; exchanged with the other parts of K through the scratch vector
        if (nhK > 1) {
#pragma unroll
            for (int k = 0; k < NV; ++k)
                if (first && srhs[k] < nrhs && scol[k] < nch)
                    scratch[c0 + sh.C0 + scol[k] + srhs[k] * ldx] = own[k] - sum[k];
            // (this CTA's eight warps are among the counted: all are done with the vec of before)
            warp_count(cnt + 2 * K + 1, lane);
            spin_count(cnt + 2 * K + 1, 16 * nhK, err);
#pragma unroll
            for (int r = 0; r < NR; ++r)
                vec[r * SB + tid] = (r < nrhs && tid < nrK) ? __ldcg(&scratch[c0 + K * SB + tid + r * ldx]) : 0.0;
        } else {
            psync();                                     // vec of before is read
#pragma unroll
            for (int k = 0; k < NV; ++k)
                if (first)
                    vec[srhs[k] * SB + scol[k]] = (srhs[k] < nrhs && scol[k] < nch) ? own[k] - sum[k] : 0.0;
        }
        psync();
        double dacc[N];
#pragma unroll
        for (int k = 0; k < N; ++k) dacc[k] = 0.0;
        for (int c = 0; c < sh.ninv; ++c) {
            const T *ck = chunk();
            bwd_chunk<T, double, NR>(ck, vec + tk.pad * 64 + c * FC, dacc, wp * 8, lane, sh.irows - c * FC);
            release();
        }
        spread_sum<N, B::LN>(dacc, lane);
#pragma unroll
        for (int k = 0; k < NV; ++k)
            if (first && srhs[k] < nrhs && scol[k] < nch) xs[scol[k] + srhs[k] * ldx] = dacc[k];
        warp_count(cnt + 2 * K, lane);
    }
}

// inv(L_KK) of superblock K of front s (nr rows), nrp x nrp column-major at
// factor + tk.inv, one CTA per NC columns of it (blockIdx.y; columns of 64-column block b):
//   X_bb = D_b, X_ab = -D_a sum_{c=b}^{a-1} L_ac X_cb for a > b, X_ab = 0 for a < b,
// with D_a = inv(L_aa) the 64 x 64 diagonal inverses: the panel kernel's stored ones when
// the front has them, else (given) what sb_diagonal_kernel left in place, else by
// substitution on L_aa (all threads, a barrier a row). The
// columns' blocks X_cb stay in shared memory; each L_ac and D_a is loaded into registers
// while the product before runs and staged there for its own 64 x 64 x NC one (thread = row
// i, NC / 4 columns).
// NC: few superblocks are bound by the chain of up to nine products, which 16 columns make the
// shortest (with 64 columns, no loads ahead and one thread per column in the substitution
// 90 us for the 7-sided cube and 120 us for the 20-sided one in FP64, 34 and 74 us this
// way). More than kSbInverseMany of them fill the SMs and are bound by the blocks' loads and
// staging, which 32 columns halve: FP32, 16 and 32 columns, 166 superblocks 29 and 36 us,
// 276 41 and 49, 453 54 and 54, 872 99 and 68, 936 127 and 87 us, a batch of 48 cubes 854 and
// 553 us, the 64-sided cube 1,572 and 1,046 us. 64 columns are one CTA an SM (615 us for the
// batch). In FP64 32 columns are one CTA an SM, too: the 48-sided cube 996 and 1,052 us.
constexpr int kSbInverseMany = 512;
template <typename T, int NC>
__global__ void __launch_bounds__(256) sb_inverse_kernel(const SbTask *__restrict__ tasks, SnDev sd, bool given,
                                                         T *factor) {
    constexpr int LD = 65, U = NC / 4;                    // columns a thread
    extern __shared__ __align__(16) double inv_smem[];
    T *Xc = reinterpret_cast<T *>(inv_smem);              // [4][NC][LD]: X_cb, c = b .. nbk - 1
    T *Tt = Xc + 4 * NC * LD;                             // [NC][LD]: sum L_ac X_cb
    T *Ls = Tt + NC * LD;                                 // [64][LD]: L_ac
    T *Ds = Ls + 64 * LD;                                 // [64][LD]: D_a, or L_aa
    const SbTask tk = tasks[blockIdx.x];
    const int s = tk.sn, K = tk.K, b = blockIdx.y / (64 / NC), j0 = (blockIdx.y % (64 / NC)) * NC;
    const int w = sd.w[s], ld = sd.ld[s];
    const T *pan = factor + sd.pan_off[s];
    T *out = factor + tk.inv;
    const int nr = sb_rows(w, K), nrp = sb_pad(nr), nbk = nrp / 64;
    if (b >= nbk) return;
    const int r0 = K * SB;
    const int tid = threadIdx.x, i = tid & 63, jg = tid >> 6;
    const int64_t dinv = sd.inv_off[s];
    // block (a, c) of L_KK, or D_a for a == c when it is there: a column a quarter, lane = row
    T v[16];
    auto fetch = [&](int a, int c) {
        if (a >= nbk) return;
        const bool stored = a == c && (dinv >= 0 || given);
        const T *src = dinv >= 0 ? factor + dinv + int64_t(K * (SB / 64) + a) * 4096 : out + int64_t(a * 64) * nrp + a * 64;
        const int lds = dinv >= 0 ? 64 : nrp;
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            const int m = jg + 4 * u, gi = a * 64 + i, gj = c * 64 + m;
            v[u] = T(0);
            if (gi < nr && gj < nr) v[u] = stored ? src[m * lds + i] : pan[int64_t(r0 + gj) * ld + r0 + gi];
        }
    };
    auto stage = [&](T *dst) {
#pragma unroll
        for (int u = 0; u < 16; ++u) dst[(jg + 4 * u) * LD + i] = v[u];
    };
    // D_a from the staged block in Ds: itself, or by substitution into Ls
    auto diagonal = [&](int a) -> const T * {
        __syncthreads();
        if (dinv >= 0 || given) return Ds;
        // rows k in order: every thread has column j and every fourth row below; row k stays
        // unscaled until the end, so that a step needs one barrier
        const int nb = min(64, nr - a * 64), j = i;
        for (int q = tid; q < 4096; q += 256) Ls[(q >> 6) * LD + (q & 63)] = (q >> 6) == (q & 63) ? T(1) : T(0);
        __syncthreads();
        for (int k = 0; k < nb; ++k) {
            if (j <= k) {
                const T y = Ls[j * LD + k] / Ds[k * LD + k];
                for (int m = k + 1 + jg; m < nb; m += 4) Ls[j * LD + m] -= Ds[k * LD + m] * y;
            }
            __syncthreads();
        }
        for (int q = tid; q < 4096; q += 256) {
            const int jj = q >> 6, ii = q & 63;
            Ls[jj * LD + ii] = ii < nb && jj < nb ? Ls[jj * LD + ii] / Ds[ii * LD + ii] : T(0);
        }
        __syncthreads();
        return Ls;
    };
    fetch(b, b);
    // the strict upper blocks of these columns are zero
    for (int q = tid; q < NC * b * 64; q += 256) {
        const int jj = q / (b * 64), ii = q - jj * (b * 64);
        out[int64_t(b * 64 + j0 + jj) * nrp + ii] = T(0);
    }
    stage(Ds);
    fetch(b + 1, b);
    // X_bb = D_b
    {
        const T *D = diagonal(b);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = jg * U + u;
            const T x = D[(j0 + j) * LD + i];
            Xc[j * LD + i] = x;
            if (dinv >= 0 || !given) out[int64_t(b * 64 + j0 + j) * nrp + b * 64 + i] = x;
        }
    }
    for (int a = b + 1; a < nbk; ++a) {
        T acc[U];
#pragma unroll
        for (int u = 0; u < U; ++u) acc[u] = T(0);
        for (int c = b; c < a; ++c) {
            __syncthreads();                               // Ls is free
            stage(Ls);
            fetch(a, c + 1);
            __syncthreads();
            const T *X = Xc + ((c - b) * NC + jg * U) * LD;
#pragma unroll 8
            for (int m = 0; m < 64; ++m) {
                const T l = Ls[m * LD + i];
#pragma unroll
                for (int u = 0; u < U; ++u) acc[u] += l * X[u * LD + m];
            }
        }
        __syncthreads();                                   // Ls, Ds and Tt are free
#pragma unroll
        for (int u = 0; u < U; ++u) Tt[(jg * U + u) * LD + i] = acc[u];
        stage(Ds);
        fetch(a + 1, b);
        const T *D = diagonal(a);
        const T *Tj = Tt + jg * U * LD;
#pragma unroll
        for (int u = 0; u < U; ++u) acc[u] = T(0);
#pragma unroll 8
        for (int m = 0; m < 64; ++m) {
            const T dv = D[m * LD + i];
#pragma unroll
            for (int u = 0; u < U; ++u) acc[u] -= dv * Tj[u * LD + m];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = jg * U + u;
            Xc[((a - b) * NC + j) * LD + i] = acc[u];
            out[int64_t(b * 64 + j0 + j) * nrp + a * 64 + i] = acc[u];
        }
    }
}

// Diagonal block `pad` of a superblock without stored 64 x 64 inverses, inverted to its place
// in inv(L_KK): four threads a column, rows in order. For many of them (fronts factored whole
// above the cut: forests of small systems), since the kernel above substitutes again for every
// 16 columns. Whole factorizations of 5,000 fronts of 15 rows: 613 us in FP32 and 711 us in
// FP64 without it (271 and 498 us with 64 columns a CTA there), 121 and 162 us with it; 3,000
// fronts of 120 rows 4.46 and 5.52 ms (3.89 and 6.37 ms), 1.74 and 2.54 ms with it.
template <typename T>
__global__ void __launch_bounds__(256) sb_diagonal_kernel(const SbTask *__restrict__ tasks, SnDev sd, int LD,
                                                          T *factor) {
    extern __shared__ __align__(16) double inv_smem[];
    T *Ls = reinterpret_cast<T *>(inv_smem);              // [LD][LD]: the block of L, column-major
    T *Y = Ls + LD * LD;                                  // [LD][LD]: its inverse, row-major
    const SbTask tk = tasks[blockIdx.x];
    const int s = tk.sn, ld = sd.ld[s], a0 = 64 * tk.pad, r0 = tk.K * SB + a0;
    const int rows = sb_rows(sd.w[s], tk.K), nrp = sb_pad(rows), nr = min(64, rows - a0);
    const int tid = threadIdx.x, i = tid & 63;
    const T *pan = factor + sd.pan_off[s] + int64_t(r0) * ld + r0;
    T *out = factor + tk.inv + int64_t(a0) * nrp + a0;
#pragma unroll 4
    for (int c = tid >> 6; c < nr; c += 4)
        if (i >= c && i < nr) Ls[c * LD + i] = pan[int64_t(c) * ld + i];
    __syncthreads();
    const int j = tid >> 2, part = tid & 3, j0 = j & ~7;   // a warp has eight columns
    if (j0 < nr)
        for (int k = j0; k < nr; ++k) {
            T y = T(0);
#pragma unroll 2
            for (int m = j0 + part; m < k; m += 4)
                if (m >= j && j < nr) y -= Ls[m * LD + k] * Y[m * LD + j];
            y += __shfl_xor_sync(0xffffffffu, y, 1);
            y += __shfl_xor_sync(0xffffffffu, y, 2);
            if (k == j) y = T(1);
            if (part == 0 && j < nr) Y[k * LD + j] = k >= j ? y / Ls[k * LD + k] : T(0);
            __syncwarp();
        }
    __syncthreads();
    for (int c = tid >> 6; c < 64; c += 4) out[int64_t(c) * nrp + i] = i >= c && i < nr ? Y[i * LD + c] : T(0);
}

// NR: the right-hand sides the vectors hold (nrhs <= NR)
template <typename T, int NST, int NR, int VS>
cudaError_t launch_sp_impl(bool forward, const SbTask *tasks, int ntasks, SnDev sd, const char *maps,
                           const SbChild *children, ManyDev many, const int32_t *cmap, const int32_t *rowcnt, double *X,
                           int64_t ldx, int nrhs, double *sol, double *scratch, int *flags, int *err, cudaStream_t st) {
    using L = SpLayout<T, NST, NR, VS>;
    constexpr size_t smem = L::bytes + 128;
    static_assert(smem + 1024 <= size_t(kMaxSmemOptin), "superblock solve shared memory");
    void *kern = !forward      ? (void *)sp_bwd_kernel<T, NST, NR, VS>
                 : many.fronts ? (void *)sp_fwd_kernel<T, NST, NR, VS, true>
                               : (void *)sp_fwd_kernel<T, NST, NR, VS, false>;
    static PerDeviceOnce once;
    once([] {
        cudaFuncSetAttribute(sp_fwd_kernel<T, NST, NR, VS, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        cudaFuncSetAttribute(sp_fwd_kernel<T, NST, NR, VS, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        cudaFuncSetAttribute(sp_bwd_kernel<T, NST, NR, VS>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    });
    // one CTA per SM (its shared memory); the parts of a superblock (at most four) must be
    // on different CTAs, which a grid of min(SMs, tasks) gives
    const int grid = std::min(device_sm_count(), ntasks);
    // (the kernels differ in this one argument)
    const int32_t **rows = forward ? &cmap : &rowcnt;
    void *args[] = {(void *)&tasks, (void *)&ntasks, (void *)&sd,  (void *)&maps, (void *)&children,
                    (void *)&many,  (void *)rows,    (void *)&X,   (void *)&ldx,  (void *)&nrhs,
                    (void *)&sol,   (void *)&scratch, (void *)&flags, (void *)&err};
    ++g_kernel_launches;
    return cudaLaunchCooperativeKernel(kern, dim3(grid), dim3(kSbThreads), args, smem, st);
}

// Inverse row map of one child (blockIdx.x) of the assembly forest in its parent's front.
__global__ void child_map_kernel(const int32_t *__restrict__ parent, const int64_t *__restrict__ off, SnDev sd,
                                 int32_t *__restrict__ map) {
    const int c = blockIdx.x, p = parent[c];
    if (p < 0) return;
    const int vb = sd.vb, nf = sd.f[p] / vb, nc = sd.d[c] / vb;
    int32_t *m = map + off[c];
    const int32_t *rel = sd.rel + sd.struct_ptr[c];
    for (int k = threadIdx.x; k < nf; k += blockDim.x) m[k] = -1;
    __syncthreads();
    for (int k = threadIdx.x; k < nc; k += blockDim.x) m[rel[k] / vb] = k;
}

}  // namespace

void launch_child_maps(const int32_t *parent, const int64_t *off, int nsn, SnDev sd, int32_t *map, cudaStream_t st) {
    if (nsn <= 0) return;
    ++g_kernel_launches;
    child_map_kernel<<<nsn, 128, 0, st>>>(parent, off, sd, map);
}

template <typename T>
cudaError_t launch_sb_solve(bool forward, const SbTask *tasks, int ntasks, SnDev sd, const void *maps,
                            const SbChild *children, const int32_t *cmap, ManyDev many, const int32_t *rowcnt,
                            double *X, int64_t ldx, int nrhs, double *sol, double *scratch, int *flags, int *err,
                            cudaStream_t st) {
    const char *mp = static_cast<const char *>(maps);
    if (ntasks <= 0) return cudaSuccess;
    if (nrhs > kSbMaxRhs) return cudaErrorInvalidValue;
    auto go = [&](auto impl) {
        return impl(forward, tasks, ntasks, sd, mp, children, many, cmap, rowcnt, X, ldx, nrhs, sol, scratch, flags, err,
                    st);
    };
    // ring depth and vector buffers: the most that fit beside the sums of nrhs right-hand sides
    if (nrhs == 1) return go(launch_sp_impl<T, 6, 1, 4>);
    if (nrhs == 2) return go(launch_sp_impl<T, 6, 2, 4>);
    if (nrhs <= 4) return go(launch_sp_impl<T, 5, 4, 4>);
    return go(launch_sp_impl<T, sizeof(T) == 4 ? 5 : 4, kSbMaxRhs, 2>);
}

template <typename T>
void launch_sb_inverse(const SbTask *tasks, int ntasks, int max_rows, int ndiag, int diag_rows, SnDev sd, T *factor,
                       cudaStream_t st) {
    if (ndiag > 0) {
        const int ld = diag_rows | 1;
        const size_t smem = size_t(2) * ld * ld * sizeof(T);
        static PerDeviceOnce once;
        once([] {
            cudaFuncSetAttribute(sb_diagonal_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 int(2 * 65 * 65 * sizeof(T)));
        });
        ++g_kernel_launches;
        sb_diagonal_kernel<T><<<ndiag, 256, smem, st>>>(tasks + ntasks, sd, ld, factor);
    }
    if (ntasks <= 0) return;
    auto go = [&](auto cols, PerDeviceOnce &once) {
        constexpr int NC = decltype(cols)::value;
        constexpr size_t smem = size_t(5 * NC + 2 * 64) * 65 * sizeof(T);
        once([] {
            cudaFuncSetAttribute(sb_inverse_kernel<T, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        });
        ++g_kernel_launches;
        sb_inverse_kernel<T, NC><<<dim3(ntasks, 64 / NC * ((max_rows + 63) / 64)), 256, smem, st>>>(tasks, sd, ndiag > 0,
                                                                                                   factor);
    };
    static PerDeviceOnce once16, once32;
    if constexpr (sizeof(T) == 4)
        if (ntasks > kSbInverseMany) return go(std::integral_constant<int, 32>{}, once32);
    go(std::integral_constant<int, 16>{}, once16);
}

#define MFS_SB_INSTANTIATE(T)                                                                                      \
    template cudaError_t launch_sb_solve<T>(bool, const SbTask *, int, SnDev, const void *, const SbChild *,       \
                                            const int32_t *, ManyDev, const int32_t *, double *, int64_t, int,     \
                                            double *, double *, int *, int *, cudaStream_t);
MFS_SB_INSTANTIATE(float)
MFS_SB_INSTANTIATE(double)
template void launch_sb_inverse<float>(const SbTask *, int, int, int, int, SnDev, float *, cudaStream_t);
template void launch_sb_inverse<double>(const SbTask *, int, int, int, int, SnDev, double *, cudaStream_t);

}  // namespace mfs
