// Standalone SBP operator application: SbpOperator2d::diffxi/diffeta and
// UpwindOperator2d::dissxi/disseta on device arrays (sbp/src/operators.rs:55-106).
// Compiled with -fmad=false: results are bit-identical to the reference's row path
// (xi) and column path (eta) in the same dtype.
//
// One tile per CTA, every input row segment of the tile (with its halo or closure region) brought
// into shared memory by one cp.async.bulk copy that completes on an mbarrier, so a CTA has its
// whole tile in flight at once and no thread spends instructions on the loads.  Rows need not
// start on 16-byte boundaries (odd lengths, offset pointers): a segment is widened to 16-byte
// boundaries, which stays inside the array except at its first and last bytes, where the copy is
// narrowed instead and a lane fetches the few elements left over (fetch_row).
//
// Row tiles: 16 or 4 rows x 2 KB.  A thread's outputs are one 16-byte vector of the row in
// memory (a column is counted from the 16-byte boundary at or before its row's start), so window loads
// from shared memory and stores are 16 bytes wide on every row, whatever its alignment; outputs
// of the boundary closures and of the vectors that a row's ends cut are taken one by one
// afterwards, with the closure coefficients gathered from global memory.
//
// Arrays whose rows all start on 16-byte boundaries take instantiations (ALIGNED) in which that is
// known: the bookkeeping of the general form costs 6% on 4 fields of 4096 x 4096.
//
// Column tiles: TR rows x TC adjacent columns (launch_t), each thread one column over its share of the rows
// with the D-tap window in a register ring.  The reference's fused / unfused column split falls on a
// multiple of 8 (f64) or 16 (f32) columns.
//
// Bound by memory: one read and one write of the field.  Upwind9, 4 fields of 1021 x 1533 f64 (rows off
// the 16-byte boundaries): 26 us each direction and kind, from 41 (row) and 69 (column) with a scalar load per
// element; 64 x 64 f64 Upwind4: 10.8 to 5.3 (row) and 6.4 to 4.6 us (column).
//
// Dependent launches (dependent_launch.cuh): an application starts, and sets its barrier up, while the
// previous kernel of the stream drains, and waits for it before it touches global memory.  The four
// applications in a row on 64 x 64 f64 Upwind4: 21.4 to 19.3 us; on 4 fields of 1021 x 1533 f64 Upwind9:
// 112 to 104 us; the two of SBP8 on 4 fields of 1537 x 2047 f32: 64 to 60 us; the four of Upwind9 on 4
// fields of 4096 x 4096 f64: 813 to 796 us (781 with the WIDE rows of op_xi_kernel).
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "bulk_copy.cuh"
#include "dependent_launch.cuh"
#include "dynamic_smem.h"
#include "op_apply.h"
#include "sbp_ops.cuh"

namespace sbp {

namespace {

constexpr int kThreads = 256;

template <class T>
struct Vec;
template <>
struct Vec<double> {
    using type = double2;
};
template <>
struct Vec<float> {
    using type = float4;
};

// Closure-block rows (start blocks) in global memory: the row kernel's lanes read different rows of
// them, which constant memory would serialise.
template <int OP, int KIND, class T>
struct GatherCoef;
#define SBP_GATHER(OP, TAG, KINDV, KINDN, T, LIT, SUF)                                                          \
    static __device__ const T g_##TAG##_##KINDN##_START_##SUF[] = {SBPC_##TAG##_##KINDN##_START(LIT)};           \
    template <>                                                                                                 \
    struct GatherCoef<OP, KINDV, T> {                                                                           \
        __device__ __forceinline__ static T start(int i) { return __ldg(g_##TAG##_##KINDN##_START_##SUF + i); } \
    };
#define SBP_GATHER2(OP, TAG, KINDV, KINDN)                    \
    SBP_GATHER(OP, TAG, KINDV, KINDN, double, SBPC_LIT_F64, D) \
    SBP_GATHER(OP, TAG, KINDV, KINDN, float, SBPC_LIT_F32, F)
SBP_GATHER2(UPWIND4, UPWIND4, DIFF, DIFF)
SBP_GATHER2(UPWIND4H2, UPWIND4H2, DIFF, DIFF)
SBP_GATHER2(UPWIND9, UPWIND9, DIFF, DIFF)
SBP_GATHER2(UPWIND9H2, UPWIND9H2, DIFF, DIFF)
SBP_GATHER2(SBP4, SBP4, DIFF, DIFF)
SBP_GATHER2(SBP8, SBP8, DIFF, DIFF)
SBP_GATHER2(UPWIND4, UPWIND4, DISS, DISS)
SBP_GATHER2(UPWIND4H2, UPWIND4H2, DISS, DISS)
SBP_GATHER2(UPWIND9, UPWIND9, DISS, DISS)
SBP_GATHER2(UPWIND9H2, UPWIND9H2, DISS, DISS)
#undef SBP_GATHER
#undef SBP_GATHER2

// sum_unfused (sbp_ops.cuh) with gathered closure coefficients: the same sum in the same order.
template <int OP, int KIND, class T, class P>
__device__ __forceinline__ T sum_gathered(int i, int n, P&& p) {
    constexpr int M = OpShape<OP>::M, N = OpShape<OP>::N, H = OpShape<OP>::H;
    using C = GatherCoef<OP, KIND, T>;
    if (i >= M && i < n - M) return diag_unfused<OP, KIND, T>([&](int d) { return p(i - H + d); });
    const bool right = i >= n - M;
    const int b = right ? n - N : 0;
    auto coef = [&](int k) {
        const T v = C::start(right ? (n - 1 - i) * N + (N - 1 - k) : i * N + k);
        return right && KIND == DIFF ? -v : v;
    };
    T t = coef(0) * p(b);
#pragma unroll
    for (int k = 1; k < N; ++k) t = t + coef(k) * p(b + k);
    return t;
}

// Elements of a row's first element past the 16-byte boundary at or before it.
template <class T>
__device__ __forceinline__ int parity_of(const T* p) {
    return (int)((reinterpret_cast<uintptr_t>(p) & 15) / sizeof(T));
}

// The extent of the whole input array in memory.
struct Extent {
    uintptr_t begin, end;
};

// Bytes that the bulk copy of `w` elements at `src` takes, and its first byte: widened to 16-byte
// boundaries, or narrowed at an end where that would leave the array.
template <class T>
__device__ __forceinline__ uint32_t row_span(const T* src, int w, const Extent& A, uintptr_t& first) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(src), b = a + (uintptr_t)w * sizeof(T);
    uintptr_t lo = a & ~(uintptr_t)15, hi = (b + 15) & ~(uintptr_t)15;
    if (lo < A.begin) lo += 16;
    if (hi > A.end) hi -= 16;
    first = lo;
    return hi > lo ? (uint32_t)(hi - lo) : 0u;
}

// Fetches `nrows` row segments, `w(r)` elements at `src(r)` into `dst(r)` (16-byte aligned; element 0
// lands parity_of(src) elements in), by the calling warp.  Announces the bytes on `bar` (count 1)
// after the elements that the copies leave out have been written.
template <class T, class SRC, class W, class DST>
__device__ __forceinline__ void fetch_rows(int nrows, const SRC& src, const W& w, const DST& dst, const Extent& A,
                                           uint64_t* bar) {
    const int lane = threadIdx.x & 31;
    uint32_t bytes = 0;
    for (int r = lane; r < nrows; r += 32) {
        uintptr_t first;
        const T* s = src(r);
        const int n = w(r);
        const uint32_t b = row_span(s, n, A, first);
        bytes += b;
        const uintptr_t a = reinterpret_cast<uintptr_t>(s), last = first + b;
        if (first > a || last < a + (uintptr_t)n * sizeof(T)) {
            T* d = dst(r) + parity_of(s);
            for (int k = 0; k < n; ++k) {
                const uintptr_t e = a + (uintptr_t)k * sizeof(T);
                if (e >= first && e < last) k = (int)((last - a) / sizeof(T)) - 1;  // copied in bulk
                else d[k] = s[k];
            }
        }
    }
    bytes = __reduce_add_sync(0xffffffffu, bytes);
    __syncwarp();
    if (lane == 0) bulk_expect(bar, bytes);
    __syncwarp();
    for (int r = lane; r < nrows; r += 32) {
        uintptr_t first;
        const T* s = src(r);
        const uint32_t b = row_span(s, w(r), A, first);
        if (b)
            bulk_g2s(reinterpret_cast<unsigned char*>(dst(r)) + (first - (reinterpret_cast<uintptr_t>(s) & ~(uintptr_t)15)),
                     reinterpret_cast<const void*>(first), b, bar);
    }
}

// A staged row again, by plain loads, for a thread that gave up waiting for the copies.  An application is
// asynchronous and has no status to report, so a wait that runs out costs time and not the result.  Every
// such thread fetches the whole tile (others may have seen the copies arrive, so it cannot count on
// them); copies that still arrive write the same values.  They are waited for once more, with a limit, as
// they end in the CTA's shared memory.  Out of line: within the kernels this cost 3% of a large odd field.
template <class T>
__device__ __forceinline__ void fetch_plainly(const T* __restrict__ s, T* d, int n) {
#pragma unroll 1
    for (int k = 0; k < n; ++k) d[k] = s[k];
}

constexpr int kXiRows = 16;  // most rows of a row tile
template <class T>
constexpr int xi_cols() { return 128 * (16 / (int)sizeof(T)); }
template <class T>
constexpr int xi_pitch() { return xi_cols<T>() + 32; }  // covers the halo, closures and alignment
template <class T>
constexpr size_t xi_smem(int rows) { return (size_t)rows * xi_pitch<T>() * sizeof(T) + 16; }

// Columns [lo, hi) of a row of parity `par` that the outputs of its tile at u0 read (aligned: whole vectors).
template <int OP, class T, bool ALIGNED>
__device__ __forceinline__ void xi_segment(int u0, int par, int nx, int& lo, int& hi) {
    constexpr int TC = xi_cols<T>(), K = 16 / sizeof(T);
    lo = hi = 0;
    if constexpr (ALIGNED) {
        region_of<OP>(u0, min(nx, u0 + TC), nx, lo, hi);
        lo &= ~(K - 1);
        hi = min(nx, (hi + K - 1) & ~(K - 1));
    } else {
        const int c0 = max(0, u0 - par), c1 = min(nx, u0 + TC - par);
        if (c0 < c1) region_of<OP>(c0, c1, nx, lo, hi);
    }
}

template <int OP, class T, bool ALIGNED>
__device__ __noinline__ void xi_fetch_plainly(const T* __restrict__ src, T* buf, int nrows, int nx, int u0, uint64_t* bar) {
#pragma unroll 1
    for (int r = 0; r < nrows; ++r) {
        const T* row = src + (int64_t)r * nx;
        int lo, hi;
        xi_segment<OP, T, ALIGNED>(u0, ALIGNED ? 0 : parity_of(row), nx, lo, hi);
        fetch_plainly(row + lo, buf + r * xi_pitch<T>() + (ALIGNED ? 0 : parity_of(row + lo)), hi - lo);
    }
    bulk_wait(bar, 0, kBulkWaitPolls);
}

// Row direction (see the file comment): `tr` rows per tile, 2^lpr threads per row.  WIDE: 16 rows and 128
// threads, known to the compiler, which saves a large aligned field of the lighter operators its loop over
// a row's vectors: SBP4 on 1874 x 856 f64 8.1 to 7.0 us and on 20 x 1,000,000 f32 31.6 to 27.2, Upwind9 on 4 fields
// of 4096 x 4096 f64 179 to 167 and f32 98 to 89.  u counts elements
// from the 16-byte boundary at or before a row's start; tile cb covers u in [cb TC, cb TC + TC).
// vec_out: output rows have the alignment of the input rows, so vectors are stored whole.
template <int OP, int KIND, class T, bool ALIGNED, bool WIDE>
__global__ void __launch_bounds__(kThreads)
    op_xi_kernel(const T* __restrict__ in, T* __restrict__ out, int ny, int nx, int64_t bstride, T idx, int ncb, int rows,
                 int lanes, bool vec_out, Extent A, int polls) {
    const int tr = WIDE ? kXiRows : rows, lpr = WIDE ? 7 : lanes;
    constexpr int M = OpShape<OP>::M, H = OpShape<OP>::H;
    constexpr int K = 16 / sizeof(T);
    constexpr int TC = xi_cols<T>(), P = xi_pitch<T>();
    constexpr int PAD = ((H + K - 1) / K) * K;
    constexpr int NV = (K + 2 * PAD) / K;
    using V = typename Vec<T>::type;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    T* buf = reinterpret_cast<T*>(smem_raw);
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw + (size_t)tr * P * sizeof(T));
    const int nrg = (ny + tr - 1) / tr;
    int64_t it = blockIdx.x;
    const int cb = (int)(it % ncb);
    it /= ncb;
    const int rg = (int)(it % nrg);
    const int64_t off = (it / nrg) * bstride + (int64_t)rg * tr * nx;  // the tile's first row
    const int nrows = min(tr, ny - rg * tr), u0 = cb * TC;
    const T* src = in + off;
    T* dst = out + off;
    auto row_parity = [&](int r) { return ALIGNED ? 0 : parity_of(src + (int64_t)r * nx); };
    int lo_a = 0, hi_a = 0;  // aligned: the segment of every row
    if constexpr (ALIGNED) xi_segment<OP, T, true>(u0, 0, nx, lo_a, hi_a);
    auto seg = [&](int r, int& lo, int& hi) {
        lo = lo_a;
        hi = hi_a;
        if constexpr (!ALIGNED) xi_segment<OP, T, false>(u0, row_parity(r), nx, lo, hi);
    };
    if (threadIdx.x == 0) bulk_mbar_init(bar, 1);
    __syncthreads();
    dependency_wait();
    if (threadIdx.x < 32) {
        if constexpr (ALIGNED) {
            const uint32_t row_bytes = (uint32_t)(hi_a - lo_a) * (uint32_t)sizeof(T);
            if (threadIdx.x == 0) bulk_expect(bar, row_bytes * (uint32_t)nrows);
            for (int r = threadIdx.x; r < nrows; r += 32)
                bulk_g2s(buf + r * P, src + (int64_t)r * nx + lo_a, row_bytes, bar);
        } else {
            int lo, hi;
            fetch_rows<T>(
                nrows,
                [&](int r) {
                    seg(r, lo, hi);
                    return src + (int64_t)r * nx + lo;
                },
                [&](int r) {
                    seg(r, lo, hi);
                    return hi - lo;
                },
                [&](int r) { return buf + r * P; }, A, bar);
        }
    }
    if (!bulk_wait(bar, 0, polls)) xi_fetch_plainly<OP, T, ALIGNED>(src, buf, nrows, nx, u0, bar);
    const int v = threadIdx.x & ((1 << lpr) - 1);
    for (int r = threadIdx.x >> lpr; r < nrows; r += kThreads >> lpr) {
        const int par = row_parity(r);
        int lo, hi;
        seg(r, lo, hi);
        const int su = (lo + par) & ~(K - 1);  // u of the segment's first staged element
        for (int u = u0 + K * v; u < u0 + TC; u += K << lpr) {
            const int c = u - par;
            if (c < M || c + K - 1 >= nx - M) continue;
            T w[K + 2 * PAD];  // w[j] holds column c - PAD + j
            const V* bv = reinterpret_cast<const V*>(buf + r * P + (u - PAD - su));
#pragma unroll
            for (int q = 0; q < NV; ++q) reinterpret_cast<V*>(w)[q] = bv[q];
            T o[K];
#pragma unroll
            for (int j = 0; j < K; ++j)
                o[j] = diag_unfused<OP, KIND, T>([&](int d) { return w[j + d + PAD - H]; }) * idx;
            T* d = dst + (int64_t)r * nx + c;
            if (vec_out) {
                *reinterpret_cast<V*>(d) = *reinterpret_cast<V*>(o);
            } else {
#pragma unroll
                for (int j = 0; j < K; ++j) d[j] = o[j];
            }
        }
    }
    // the ends of the rows: columns whose vector is not interior, one output per thread
    constexpr int E = M + K - 1;
    const bool any_left = u0 < E + K, any_right = u0 + TC > nx - E;
    if (!any_left && !any_right) return;
    for (int i = threadIdx.x; i < nrows * 2 * E; i += kThreads) {
        const int r = i / (2 * E), k = i % (2 * E);
        const int c = k < E ? k : nx - 1 - (k - E);
        if (k < E ? c >= nx - E : c < 0) continue;  // the two ends meet on short rows: the right one takes it
        const int par = row_parity(r), u = c + par;
        if (u < u0 || u >= u0 + TC) continue;
        const int cv = (u & ~(K - 1)) - par;
        if (cv >= M && cv + K - 1 < nx - M) continue;  // done above
        int lo, hi;
        seg(r, lo, hi);
        const T* rb = buf + r * P + (par - ((lo + par) & ~(K - 1)));  // column 0 of the row
        dst[(int64_t)r * nx + c] = sum_gathered<OP, KIND, T>(c, nx, [&](int kk) { return rb[kk]; }) * idx;
    }
}

template <int OP, int TR>
constexpr int eta_region() {  // input rows a column tile can need (region_of's extent)
    constexpr int M = OpShape<OP>::M, N = OpShape<OP>::N, H = OpShape<OP>::H;
    constexpr int a = TR + H + (H > M - 1 ? H : M - 1);
    return a > N ? a : N;
}
template <class T, int TC, bool ALIGNED>
constexpr int eta_pitch() { return TC + (ALIGNED ? 0 : 2 * (16 / (int)sizeof(T))); }  // room for the widened ends
template <int OP, class T, int TR, int TC, bool ALIGNED>
constexpr size_t eta_smem() { return (size_t)eta_region<OP, TR>() * eta_pitch<T, TC, ALIGNED>() * sizeof(T) + 16; }

template <class T, int P, bool ALIGNED>
__device__ __noinline__ void eta_fetch_plainly(const T* __restrict__ src, T* buf, int nrows, int nx, int tw, uint64_t* bar) {
#pragma unroll 1
    for (int r = 0; r < nrows; ++r) {
        const T* row = src + (int64_t)r * nx;
        fetch_plainly(row, buf + r * P + (ALIGNED ? 0 : parity_of(row)), tw);
    }
    bulk_wait(bar, 0, kBulkWaitPolls);
}

// Column direction (see the file comment).
template <int OP, int KIND, class T, int TR, int TC, bool ALIGNED>
__global__ void __launch_bounds__(kThreads)
    op_eta_kernel(const T* __restrict__ in, T* __restrict__ out, int ny, int nx, int64_t bstride, T idx, int simd,
                  Extent A, int polls) {
    constexpr int M = OpShape<OP>::M, D = OpShape<OP>::D, H = OpShape<OP>::H;
    constexpr int K = 16 / sizeof(T), P = eta_pitch<T, TC, ALIGNED>();
    constexpr int GROUPS = kThreads / TC;  // row groups
    constexpr int RG = TR / GROUPS;        // rows of one thread
    extern __shared__ __align__(128) unsigned char smem_raw[];
    T* buf = reinterpret_cast<T*>(smem_raw);
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw + (size_t)eta_region<OP, TR>() * P * sizeof(T));
    const int ncb = (nx + TC - 1) / TC, nrc = (ny + TR - 1) / TR;
    int64_t it = blockIdx.x;  // vertically adjacent tiles are adjacent in launch order (shared halos in L2)
    const int rc = (int)(it % nrc);
    it /= nrc;
    const int cb = (int)(it % ncb);
    const int64_t b = it / ncb;
    const int y0 = rc * TR, y1 = min(ny, y0 + TR), c0 = cb * TC, tw = min(TC, nx - c0);
    int lo, hi;
    region_of<OP>(y0, y1, ny, lo, hi);
    const T* src = in + b * bstride + (int64_t)lo * nx + c0;
    if (threadIdx.x == 0) bulk_mbar_init(bar, 1);
    __syncthreads();
    dependency_wait();
    if (threadIdx.x < 32) {
        if constexpr (ALIGNED) {
            const int nrows = hi - lo;
            const uint32_t row_bytes = (uint32_t)tw * (uint32_t)sizeof(T);
            if (threadIdx.x == 0) bulk_expect(bar, row_bytes * (uint32_t)nrows);
            for (int r = threadIdx.x; r < nrows; r += 32) bulk_g2s(buf + r * P, src + (int64_t)r * nx, row_bytes, bar);
        } else {
            fetch_rows<T>(
                hi - lo, [&](int r) { return src + (int64_t)r * nx; }, [&](int) { return tw; },
                [&](int r) { return buf + r * P; }, A, bar);
        }
    }
    if (!bulk_wait(bar, 0, polls)) eta_fetch_plainly<T, P, ALIGNED>(src, buf, hi - lo, nx, tw, bar);
    const int j = threadIdx.x % TC, g = threadIdx.x / TC;
    if (j >= tw) return;
    const int col = c0 + j;
    const bool fused = col < simd;
    T* dst = out + b * bstride + col;
    // row r of the array starts (p0 + (r - lo) nx) mod K elements past a 16-byte boundary
    const int p0 = parity_of(src), step = nx & (K - 1);
    auto at = [&](int r) { return buf[(r - lo) * P + (ALIGNED ? 0 : (p0 + (r - lo) * step) & (K - 1)) + j]; };
    const int ra = y0 + g * RG, rb = min(y1, ra + RG);
    for (int r = ra; r < rb && r < M; ++r) dst[(int64_t)r * nx] = sum_column<OP, KIND, T>(fused, r, ny, at) * idx;
    for (int r = max(ra, ny - M); r < rb; ++r) dst[(int64_t)r * nx] = sum_column<OP, KIND, T>(fused, r, ny, at) * idx;
    const int i0 = max(ra, M), i1 = min(rb, ny - M);
    if (i0 >= i1) return;
    T w[D];
#pragma unroll
    for (int k = 0; k < D - 1; ++k) w[k] = at(i0 - H + k);
    int r = i0;
    for (; r + D <= i1; r += D) {
#pragma unroll
        for (int u = 0; u < D; ++u) {
            w[(u + D - 1) % D] = at(r + u + H);
            T f = T(0);
            if (fused) {
#pragma unroll
                for (int k = 0; k < D; ++k) f = fma_rn(w[(u + k) % D], Coef<OP, KIND, T>::diag(k), f);
            } else {
#pragma unroll
                for (int k = 0; k < D; ++k) f = f + Coef<OP, KIND, T>::diag(k) * w[(u + k) % D];
            }
            dst[(int64_t)(r + u) * nx] = f * idx;
        }
    }
    for (; r < i1; ++r) dst[(int64_t)r * nx] = sum_column<OP, KIND, T>(fused, r, ny, at) * idx;
}

constexpr int kSms = 148;

template <int OP, int KIND, class T, int TR, int TC, bool ALIGNED>
cudaError_t launch_eta(const T* in, T* out, int64_t ny, int64_t nx, int64_t nbatch, int64_t bstride, const Extent& A,
                       cudaStream_t st, int polls) {
    constexpr size_t smem = eta_smem<OP, T, TR, TC, ALIGNED>();
    if constexpr (smem > 48 * 1024) {
        static DynamicSmem opt_in;
        const cudaError_t e = opt_in.allow(reinterpret_cast<const void*>(&op_eta_kernel<OP, KIND, T, TR, TC, ALIGNED>), smem);
        if (e != cudaSuccess) return e;
    }
    const T idx = inv_spacing<T>(OpShape<OP>::h2, ny);
    const int simd = (int)(simd_lanes<T>() * (nx / simd_lanes<T>()));
    const int64_t items = nbatch * ((ny + TR - 1) / TR) * ((nx + TC - 1) / TC);
    return launch_after(op_eta_kernel<OP, KIND, T, TR, TC, ALIGNED>, (unsigned)items, kThreads, smem, st, in, out, (int)ny,
                        (int)nx, bstride, idx, simd, A, polls);
}

template <int OP, int KIND, class T, bool ALIGNED>
cudaError_t launch_t(int dir, const T* in, T* out, int64_t ny, int64_t nx, int64_t nbatch, int64_t bstride,
                     cudaStream_t st, int polls) {
    constexpr int K = 16 / sizeof(T);
    const uintptr_t a = reinterpret_cast<uintptr_t>(in);
    const Extent A{a, a + ((uintptr_t)(nbatch - 1) * bstride + (uintptr_t)ny * nx) * sizeof(T)};
    if (dir == 1) {
        // Tiles of 16 rows x 32 columns, two rows per thread, while all of them fit the SMs at once; beyond that
        // taller and wider ones, which load fewer halo rows (Upwind9 f64, us, tiles of 16 x 32, 24 rows x 1 KB, 48
        // rows x 1 KB: 257 x 255 3.6, 5.5, 8.3; 768 x 768 7.1, 4.8, 6.6; 2048 x 2048 40, 15.4, 13.4).  f64 takes 48 rows
        // once they give every SM a tile (467 x 1730 6.3, 24 rows 5.0; 756 x 998 x 2 7.9, 8.3); f32 keeps 24, whose
        // shared memory lets more CTAs run (2049 x 2047 SBP4 8.9, 48 rows 12.1; 4096 x 4096 Upwind9 31.9, 33.9).
        // Fields no wider than half of a tile take half the width, so that fewer threads are without a column
        // (100,000 x 17 Upwind9 f64 28 instead of 35 us, 2000 fields of 17 x 19 f32 19 instead of 29).
        constexpr int TC = 1024 / sizeof(T), TR = 6 * sizeof(T);
        auto tiles = [&](int tr, int tc) { return nbatch * ((ny + tr - 1) / tr) * ((nx + tc - 1) / tc); };
        if (tiles(16, 32) <= 5 * kSms)
            return launch_eta<OP, KIND, T, 16, 32, ALIGNED>(in, out, ny, nx, nbatch, bstride, A, st, polls);
        if (nx <= TC / 2)
            return launch_eta<OP, KIND, T, TR, TC / 2, ALIGNED>(in, out, ny, nx, nbatch, bstride, A, st, polls);
        if (TR > 24 && tiles(TR, TC) >= kSms)
            return launch_eta<OP, KIND, T, TR, TC, ALIGNED>(in, out, ny, nx, nbatch, bstride, A, st, polls);
        return launch_eta<OP, KIND, T, 24, TC, ALIGNED>(in, out, ny, nx, nbatch, bstride, A, st, polls);
    }
    constexpr int TC = xi_cols<T>();
    const int64_t ncb = (nx + (ALIGNED ? 0 : K - 1) + TC - 1) / TC;
    // 16 rows a tile, or 4 where that would leave SMs without a tile; as many threads per row as its
    // vectors need, so that narrow fields take several rows at once
    int tr = kXiRows;
    if (nbatch * ((ny + tr - 1) / tr) * ncb < kSms) tr = 4;
    int lpr = 7;
    while (lpr > 3 && (K << (lpr - 1)) >= nx + K - 1) --lpr;
    const bool vec_out = (a - reinterpret_cast<uintptr_t>(out)) % 16 == 0;
    const T idx = inv_spacing<T>(OpShape<OP>::h2, nx);
    const int64_t items = nbatch * ((ny + tr - 1) / tr) * ncb;
    auto launch = [&](auto kernel) {
        return launch_after(kernel, (unsigned)items, kThreads, xi_smem<T>(tr), st, in, out, (int)ny, (int)nx, bstride, idx,
                            (int)ncb, tr, lpr, vec_out, A, polls);
    };
    if constexpr (ALIGNED)
        if (tr == kXiRows && lpr == 7) return launch(op_xi_kernel<OP, KIND, T, ALIGNED, true>);
    return launch(op_xi_kernel<OP, KIND, T, ALIGNED, false>);
}

template <int OP, class T>
cudaError_t launch_kind(int dir, int kind, const void* in, void* out, int64_t ny, int64_t nx, int64_t nbatch,
                        int64_t bstride, cudaStream_t st, int polls) {
    const T* i = static_cast<const T*>(in);
    T* o = static_cast<T*>(out);
    constexpr int K = 16 / sizeof(T);
    const bool aligned = nx % K == 0 && bstride % K == 0 && reinterpret_cast<uintptr_t>(in) % 16 == 0;
    auto launch = [&](auto k) {
        return aligned ? launch_t<OP, decltype(k)::value, T, true>(dir, i, o, ny, nx, nbatch, bstride, st, polls)
                       : launch_t<OP, decltype(k)::value, T, false>(dir, i, o, ny, nx, nbatch, bstride, st, polls);
    };
    if (kind == DIFF) return launch(std::integral_constant<int, DIFF>{});
    if constexpr (OpShape<OP>::upwind) return launch(std::integral_constant<int, DISS>{});
    return cudaErrorInvalidValue;
}

template <class T>
cudaError_t launch_op(int op, int dir, int kind, const void* in, void* out, int64_t ny, int64_t nx, int64_t nbatch,
                      int64_t bstride, cudaStream_t st, int polls) {
    switch (op) {
        case UPWIND4: return launch_kind<UPWIND4, T>(dir, kind, in, out, ny, nx, nbatch, bstride, st, polls);
        case UPWIND4H2: return launch_kind<UPWIND4H2, T>(dir, kind, in, out, ny, nx, nbatch, bstride, st, polls);
        case UPWIND9: return launch_kind<UPWIND9, T>(dir, kind, in, out, ny, nx, nbatch, bstride, st, polls);
        case UPWIND9H2: return launch_kind<UPWIND9H2, T>(dir, kind, in, out, ny, nx, nbatch, bstride, st, polls);
        case SBP4: return launch_kind<SBP4, T>(dir, kind, in, out, ny, nx, nbatch, bstride, st, polls);
        case SBP8: return launch_kind<SBP8, T>(dir, kind, in, out, ny, nx, nbatch, bstride, st, polls);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace

cudaError_t op_apply(int op, int dir, int kind, int dtype, const void* in, void* out, int64_t ny, int64_t nx,
                     int64_t nbatch, int64_t bstride, cudaStream_t st, int polls) {
    if (dtype == 0) return launch_op<double>(op, dir, kind, in, out, ny, nx, nbatch, bstride, st, polls);
    return launch_op<float>(op, dir, kind, in, out, ny, nx, nbatch, bstride, st, polls);
}

}  // namespace sbp
