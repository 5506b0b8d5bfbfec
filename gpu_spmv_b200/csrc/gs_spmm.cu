// gs_spmm.cu -- multi-RHS K1 products and the adjoint of y = A(v) x.
//
// Forward: Y = A X for k right-hand sides (X row-major [ncols][k], Y row-major [nrows][k],
// k in {1, 2, 4, 8, 16, 32}) on the K1 layout.  Each lane owns one sorted row, as in the
// single-RHS kernel (gs_spmv_k1.cu), and one gather of a column fetches all k values of
// X's row at once (32 bytes for k = 8 in FP32), so the gather cost is paid once per
// stored element for every right-hand side.  Long chunks are cut into the same kK1Split-step
// pieces, whose partial sums meet in scratch memory in piece order.
//
// Adjoint, for a loss L(Y) with Ybar = dL/dY:
//   Xbar = A^T Ybar                      (ncols x k)
//   vbar_e = sum_r Ybar[row_e][r] X[col_e][r]   for every stored element e (CSR order)
// Deterministic mode: the transpose is stored as its own K1 layout, built once by
// gs_matrix_prepare_adjoint (columns of A sorted by decreasing length, each transposed slot
// remembering the CSR index of its element and its row), and Xbar is the forward kernel run
// on it.  vbar in CSR order is a pass of its own over the elements (k_vbar); in the transposed
// layout's slot order the pass that gathers Ybar[row_e] for Xbar also forms vbar_e against
// X[col] held in registers.  Atomic mode: the forward layout, with Xbar accumulated by atomic
// adds (its rounding order varies between runs).
//
// The reference has no multi-RHS product and no adjoint; these extend its K1 format.
#include <algorithm>
#include <mutex>
#include <type_traits>

#include "gs_k1_fill.cuh"
#include "gs_mm.cuh"

namespace gs {

namespace {

using namespace mm;

// Blocks of 2 warps (a place on the SM is free when two units end: FP32 k = 8 on a 524,288-row
// power-law 53.9 us in blocks of 8, 52.0 in blocks of 2), and registers for the rows in flight
// before warps: the gathers are bound by the L1's line requests, which 16 warps of 4 to 8 rows in
// flight per lane keep busy (32 warps capped at 64 registers 52.0 us, 24 49.6, 16 48.0, before the
// streams loaded ahead 58.4; k = 4 101 -> 46, FP64 k = 2 118 -> 44).  On 1,048,576 rows the same
// product gains 2 % in all: 88 -> 86 us.
constexpr int kMMThreads = 64;
// One right-hand side streams: 32 warps (FP64 on a 27-point stencil 80^3 33.6 -> 31.1 us; with 16
// 40.3).  Rows of 64 bytes (FP32 k = 16; the adjoint's FP64 k = 8) hold to 24, as FP64 k = 8 did
// before it went by several lanes (a band 62.5 -> 60.4 us; with 16 64.6).
// The adjoint with its value gradient holds a row of X besides and takes the warps that leave it its
// registers: with the product's 24 warps it spilled 0.1 to 2.3 KB a thread from rows of 128 bytes on
// (slot order on a 524,288-row power-law, FP64 k = 16 / 32: 323 / 1043 us, 204 / 397 here; FP32 k =
// 32: 338, 201; FP64 k = 1 with 32 warps 69, with 24 55).
template <class T, int K, bool ADJ> constexpr int mm_warps()
{
    constexpr int row = K * (int)sizeof(T);
    if (K == 1) return ADJ && sizeof(T) == 8 ? 24 : 32;
    if (ADJ && row >= 128) return row >= 256 ? 8 : 16;
    return row >= 64 ? 24 : 16;
}

template <class T, int K, bool ADJ>
__global__ void __launch_bounds__(kMMThreads, mm_warps<T, K, ADJ>() * 32 / kMMThreads) k_k1_mm(const MMArgs a)
{
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t u = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); u < a.units;
         u += warps)
        mm_unit<T, K, ADJ>(a, u, 0);
}

// Atomic-mode adjoint on the forward layout, over the same kK1Split-step work units: lane = row
// r of A with Ybar[r] in registers; per stored element e: Xbar[col_e] += v_e Ybar[r] (atomic
// adds; Xbar zeroed first) and, when vbar is wanted, vbar_e = Ybar[r] . X[col_e] (one more
// gather of X's row per element).
struct AtomicArgs {
    uint32_t nrows;
    const uint32_t *permi, *chp, *klen, *col, *unit_chunk, *unit_base;
    uint32_t units;
    const void *val, *x, *ybar;
    void *xbar, *vbar;  // vbar (or nullptr) in forward slot order
};

template <class T, int K>
__device__ __forceinline__ void red_row(T *__restrict__ X, uint32_t r, const T (&v)[K])
{
    T *p = X + (size_t)r * K;
    if constexpr (sizeof(T) == 4 && K % 4 == 0) {
#pragma unroll
        for (int i = 0; i < K / 4; i++)
            atomicAdd(reinterpret_cast<float4 *>(p) + i,
                      make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]));
    } else {
#pragma unroll
        for (int k = 0; k < K; k++) atomicAdd(p + k, v[k]);
    }
}

template <class T, int K>
__global__ void __launch_bounds__(256) k_k1_adj_atomic(const AtomicArgs a)
{
    using A = Arith<T>;
    constexpr int B = mm_batch<T, K>();
    const T *__restrict__ val = static_cast<const T *>(a.val);
    const T *__restrict__ x = static_cast<const T *>(a.x);
    T *__restrict__ vbar = static_cast<T *>(a.vbar);
    const int lane = threadIdx.x & 31;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t u = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); u < a.units;
         u += warps) {
        const uint32_t c = __ldg(a.unit_chunk + u);
        const uint32_t piece = u - __ldg(a.unit_base + c);
        const uint32_t g = 32u * c + (uint32_t)lane;
        const uint32_t len = g < a.nrows ? __ldg(a.klen + g) : 0u;
        const uint32_t j0 = piece * kK1Split;
        const uint32_t j1 = min(len, j0 + kK1Split);
        if (j0 >= j1) continue;
        T yb[K];
        load_row<T, K>(static_cast<const T *>(a.ybar), __ldg(a.permi + g), K, yb);
        const uint32_t base = __ldg(a.chp + c) + (uint32_t)lane;
        for (uint32_t j = j0; j < j1; j += B) {
            T v[B], xg[B][K];
            uint32_t cc[B], sr[B];
#pragma unroll
            for (int b = 0; b < B; b++) {
                const bool in = j + b < j1;
                const uint32_t pos = base + 32u * (j + b);
                v[b] = in ? __ldcs(val + pos) : T(0);
                cc[b] = in ? __ldcs(a.col + pos) : 0u;
                sr[b] = pos;  // vbar in forward slot order
            }
            if (vbar) {
#pragma unroll
                for (int b = 0; b < B; b++) {
                    if (j + b < j1) load_row<T, K>(x, cc[b], K, xg[b]);
                }
            }
#pragma unroll
            for (int b = 0; b < B; b++) {
                if (j + b < j1) {
                    T contrib[K];
#pragma unroll
                    for (int k = 0; k < K; k++) contrib[k] = A::mul(v[b], yb[k]);
                    if (vbar) {
                        T d = T(0);
#pragma unroll
                        for (int k = 0; k < K; k++) d = A::add(d, A::mul(yb[k], xg[b][k]));
                        vbar[sr[b]] = d;
                    }
                    red_row<T, K>(static_cast<T *>(a.xbar), cc[b], contrib);
                }
            }
        }
    }
}

// ------------------------------------------------------------------ value gradient
// vbar_e = Ybar[row_e] . X[col_e] in CSR order, from the elements' rows and columns: L lanes of
// VEC columns (32 bytes at most) per element.  A row's elements are neighbours, so Ybar's rows come
// from L1 and the X gathers set the pace, one line request an element (FP32 k = 8, 16.8M elements:
// 60 us at the rate of bare gathers, 93 us here; the indices of the next step load while this
// one's rows are gathered, without which it took 145).  Before, the transposed pass formed vbar
// beside Xbar in its own slot order and another kernel permuted it: 122 + 83 us, where Xbar alone
// is 84 us.
struct VbarArgs {
    uint32_t nnz;
    uint32_t k, ldx, ldy;  // right-hand sides, row strides of X and Ybar
    const uint32_t *row, *col;
    const void *x, *ybar;
    void *vbar;
};

constexpr int kVbarThreads = 64;
constexpr int kVbarSteps = 8;  // steps of a warp, over consecutive elements (32: 2 % slower)
constexpr int kVbarUnroll = 2;  // elements per lane and step (1 / 4: 4 / 2 % slower in all)
// CHAIN: L * VEC = k, and the sum goes from lane to lane in the order of the right-hand sides, as
// in the transposed pass; else the lanes' sums meet in a tree.
template <class T, int VEC, int L, bool CHAIN>
__global__ void __launch_bounds__(kVbarThreads, 12) k_vbar(const VbarArgs a)
{
    using A = Arith<T>;
    constexpr int U = kVbarUnroll, E = 32 / L * U;  // elements per step
    const int lane = threadIdx.x & 31, li = lane % L;
    const uint64_t warp = blockIdx.x * (uint64_t)(kVbarThreads / 32) + (threadIdx.x >> 5);
    const T *__restrict__ x = static_cast<const T *>(a.x) + li * VEC;
    const T *__restrict__ yb = static_cast<const T *>(a.ybar) + li * VEC;
    T *__restrict__ vbar = static_cast<T *>(a.vbar);
    const bool act = CHAIN || (uint32_t)(li * VEC) < a.k;
    uint64_t e0 = warp * (uint64_t)(E * kVbarSteps) + (uint64_t)(lane / L);
    uint32_t r[U], c[U];
    auto indices = [&](uint64_t e, uint32_t(&ri)[U], uint32_t(&ci)[U]) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            const bool in = e + (uint64_t)(u * (32 / L)) < a.nnz;
            ri[u] = in ? __ldcs(a.row + e + u * (32 / L)) : 0u;
            ci[u] = in ? __ldcs(a.col + e + u * (32 / L)) : 0u;
        }
    };
    indices(e0, r, c);
    for (int t = 0; t < kVbarSteps; t++, e0 += E) {
        if (e0 - (uint64_t)(lane / L) >= a.nnz) break;  // the whole warp
        T xs[U][VEC], ys[U][VEC];
        uint32_t rn[U], cn[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (act && e0 + (uint64_t)(u * (32 / L)) < a.nnz) {
                load_slice<T, VEC>(x + (size_t)c[u] * a.ldx, xs[u]);
                load_slice<T, VEC>(yb + (size_t)r[u] * a.ldy, ys[u]);
            }
        }
        // the next step's indices load while this one's rows are gathered
        if (t + 1 < kVbarSteps) indices(e0 + E, rn, cn);
#pragma unroll
        for (int u = 0; u < U; u++) {
            const uint64_t e = e0 + (uint64_t)(u * (32 / L));
            T d = T(0);
            if constexpr (CHAIN) {
#pragma unroll
                for (int st = 0; st < L; st++) {
                    T q = st ? __shfl_up_sync(0xffffffffu, d, 1) : T(0);
                    if (e < a.nnz) {
#pragma unroll
                        for (int k = 0; k < VEC; k++) q = A::add(q, A::mul(ys[u][k], xs[u][k]));
                    }
                    if (li == st) d = q;
                }
                if (li == L - 1 && e < a.nnz) __stcs(vbar + e, d);
            } else {
                if (act && e < a.nnz) {
#pragma unroll
                    for (int k = 0; k < VEC; k++)
                        if ((uint32_t)(li * VEC + k) < a.k)
                            d = A::add(d, A::mul(ys[u][k], xs[u][k]));
                }
#pragma unroll
                for (int o = L / 2; o; o >>= 1)
                    d = A::add(d, __shfl_xor_sync(0xffffffffu, d, o));
                if (li == 0 && e < a.nnz) __stcs(vbar + e, d);
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) r[u] = rn[u], c[u] = cn[u];
    }
}

template <class T, int VEC, int L, bool CHAIN>
gs_status launch_vbar_t(const VbarArgs &a, cudaStream_t s)
{
    if (!a.nnz) return GS_OK;
    const uint32_t per = (uint32_t)(kVbarThreads / 32 * kVbarSteps * kVbarUnroll * (32 / L));
    k_vbar<T, VEC, L, CHAIN><<<(a.nnz - 1u) / per + 1u, kVbarThreads, 0, s>>>(a);
    GS_CHECK_LAUNCH();
    return GS_OK;
}

// k a power of two, rows contiguous and 32-byte aligned
template <class T> gs_status launch_vbar(const VbarArgs &a, uint32_t k, cudaStream_t s)
{
#define GS_V(K_)                                                                             \
    case K_: {                                                                               \
        constexpr int l = K_ * (int)sizeof(T) > 32 ? K_ * (int)sizeof(T) / 32 : 1;           \
        return launch_vbar_t<T, K_ / l, l, true>(a, s);                                      \
    }
    switch (k) {
        GS_V(1) GS_V(2) GS_V(4) GS_V(8) GS_V(16) GS_V(32)
    default: return fail(GS_ERR_UNSUPPORTED, "k = %u right-hand sides (1, 2, 4, 8, 16, 32)", k);
    }
#undef GS_V
}

// ------------------------------------------------------------------ any k, any row strides
// Registers before warps, as for k_k1_mm: 12 warps per SM hold the 192 and 256 bytes of sums a lane
// of FP64 k = 24 / 32 has (397 / 395 us with 16 and spills, 280 / 297 with 12).
template <class T, int VEC, int L>
constexpr int kWideBlocks = (L * VEC * (int)sizeof(T) >= 192
                                 ? 12
                                 : (L * VEC * (int)sizeof(T) >= 64 ? 16 : 24)) / 2;
template <class T, int VEC, int L>
__global__ void __launch_bounds__(kMMThreads, kWideBlocks<T, VEC, L>)
    k_k1_mm_wide(const MMArgs a)
{
    const uint32_t u = blockIdx.x * (kMMThreads / 32) + (threadIdx.x >> 5);
    if (u < a.units) mm_unit_wide<T, VEC, L>(a, u);
}

// f(VEC, L) for k right-hand sides in rows that are readable up to column `cols` and whose slices
// may start at multiples of `align` bytes: the widest slice up to 32 bytes, lanes a power of two
template <class T, class F> gs_status with_slices(uint32_t k, uint32_t cols, uint32_t align, F f)
{
    auto pick = [&](auto vec) -> gs_status {
        constexpr int V = decltype(vec)::value;
        const uint32_t need = (k + V - 1) / V;
        if (need <= 1) return f(vec, std::integral_constant<int, 1>());
        if (need <= 2) return f(vec, std::integral_constant<int, 2>());
        if (need <= 4) return f(vec, std::integral_constant<int, 4>());
        if constexpr (32 / V >= 8)
            if (need <= 8) return f(vec, std::integral_constant<int, 8>());
        if constexpr (32 / V >= 16)
            if (need <= 16) return f(vec, std::integral_constant<int, 16>());
        if constexpr (32 / V >= 32) return f(vec, std::integral_constant<int, 32>());
        return fail(GS_ERR_UNSUPPORTED, "k = %u right-hand sides (1..32)", k);
    };
    auto fits = [&](uint32_t v) {
        return v <= k && align % (v * sizeof(T)) == 0 && (k + v - 1) / v * v <= cols;
    };
    if constexpr (sizeof(T) == 4)
        if (fits(8) || (k > 4 && align % 32 == 0 && cols >= 8 && (k + 7) / 8 * 8 <= cols))
            return pick(std::integral_constant<int, 8>());
    if (fits(4) || (k == 3 && align % (4 * sizeof(T)) == 0 && cols >= 4))
        return pick(std::integral_constant<int, 4>());
    if (fits(2)) return pick(std::integral_constant<int, 2>());
    return pick(std::integral_constant<int, 1>());
}

// largest power of two up to 32 that divides a pointer and a row stride in bytes
uint32_t row_align(const void *p, size_t stride)
{
    const uintptr_t x = reinterpret_cast<uintptr_t>(p) | stride | 32u;
    return (uint32_t)(x & (~x + 1));
}

template <class T> gs_status launch_mm_wide(const MMArgs &a, uint32_t cols, cudaStream_t s)
{
    if (!a.units) return GS_OK;
    const uint32_t align = row_align(a.xin, (size_t)a.ldx * sizeof(T));
    return with_slices<T>(a.k, cols, align, [&](auto vec, auto lanes) -> gs_status {
        k_k1_mm_wide<T, decltype(vec)::value, decltype(lanes)::value>
            <<<(a.units + kMMThreads / 32 - 1) / (kMMThreads / 32), kMMThreads, 0, s>>>(a);
        GS_CHECK_LAUNCH();
        return GS_OK;
    });
}

template <class T> gs_status launch_vbar_wide(const VbarArgs &a, uint32_t cols, cudaStream_t s)
{
    const uint32_t align = std::min(row_align(a.x, (size_t)a.ldx * sizeof(T)),
                                    row_align(a.ybar, (size_t)a.ldy * sizeof(T)));
    return with_slices<T>(a.k, cols, align, [&](auto vec, auto lanes) -> gs_status {
        return launch_vbar_t<T, decltype(vec)::value, decltype(lanes)::value, false>(a, s);
    });
}

// ------------------------------------------------------------------ layout helpers
// out[i] = v[src[i]], 0 where src is kNoSrc.  Four neighbours a thread, so that four gathers are in
// flight where one was (16.8M FP32 values in random order 90 -> 82 us, 60 at the line rate);
// n4 groups of four, for arrays whose out is 16-byte aligned.
template <class T>
__global__ void __launch_bounds__(256) k_gather_vals4(size_t n4, const uint4 *__restrict__ src,
                                                      const T *__restrict__ v,
                                                      T *__restrict__ out)
{
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= n4) return;
    const uint4 q = __ldcs(src + i);
    const uint32_t s[4] = {q.x, q.y, q.z, q.w};
    T w[4];
#pragma unroll
    for (int k = 0; k < 4; k++) w[k] = s[k] == kNoSrc ? T(0) : __ldg(v + s[k]);
    if constexpr (sizeof(T) == 4) {
        __stcs(reinterpret_cast<float4 *>(out) + i, make_float4(w[0], w[1], w[2], w[3]));
    } else {
        __stcs(reinterpret_cast<double2 *>(out) + 2 * i, make_double2(w[0], w[1]));
        __stcs(reinterpret_cast<double2 *>(out) + 2 * i + 1, make_double2(w[2], w[3]));
    }
}

template <class T>
__global__ void k_gather_vals(size_t nslots, const uint32_t *src, const T *v, T *out)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nslots;
         i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t s = src[i];
        out[i] = s == kNoSrc ? T(0) : v[s];
    }
}

template <class T>
__global__ void k_scatter_vals(size_t nslots, const uint32_t *src, const T *v, T *out)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nslots;
         i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t s = src[i];
        if (s != kNoSrc) out[s] = v[i];
    }
}

// Sorted row g: its first CSR element; and the way back from the row
__global__ void k_row_places(uint32_t n, const uint32_t *row, const uint32_t *perm,
                             uint32_t *start, uint32_t *inv)
{
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n) return;
    start[g] = row[perm[g]];
    inv[perm[g]] = g;
}

// place[e] = row and forward slot of CSR element e (its row at sorted place inv[row])
__global__ void k_forward_slots(uint32_t nnz, const uint32_t *__restrict__ vrow,
                                const uint32_t *__restrict__ rowptr,
                                const uint32_t *__restrict__ inv,
                                const uint32_t *__restrict__ chp, uint2 *__restrict__ place)
{
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nnz) return;
    const uint32_t r = vrow[e], g = __ldg(inv + r);
    place[e] = make_uint2(r, __ldg(chp + (g >> 5)) + 32u * (e - __ldg(rowptr + r)) + (g & 31u));
}

// The adjoint layout's slots, from the CSR index tsrc of each: the row and the stored value of the
// element, its forward slot and the way back from there; padding slots 0, 0, none
template <class T>
__global__ void k_t_maps(uint32_t nslots, const uint32_t *__restrict__ tsrc,
                         const uint2 *__restrict__ place, const T *__restrict__ val,
                         uint32_t *__restrict__ trow, T *__restrict__ tval,
                         uint32_t *__restrict__ t2f, uint32_t *__restrict__ ftslot)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nslots) return;
    const uint32_t e = tsrc[i];
    const bool in = e != kNoSrc;
    const uint2 at = in ? __ldg(place + e) : make_uint2(0u, kNoSrc);
    trow[i] = at.x;
    t2f[i] = at.y;
    tval[i] = in ? __ldg(val + at.y) : T(0);
    if (in) ftslot[at.y] = i;
}

// rowidx[e] = row of CSR element e: a warp per 32 rows, in element order (coalesced writes; the
// row by a search of the 32 row pointers the lanes hold).  One thread per row wrote 4.2M elements
// in 69 us.
__global__ void k_expand_rows(uint32_t n, const uint32_t *__restrict__ row,
                              uint32_t *__restrict__ rowidx)
{
    const uint32_t r0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 32u;
    if (r0 >= n) return;
    const uint32_t lane = threadIdx.x & 31u, nr = min(32u, n - r0);
    const uint32_t b = row[r0], tot = row[r0 + nr] - b;
    const uint32_t st = row[min(r0 + lane, n)] - b;  // start of row r0 + lane
    for (uint32_t t = 0; t < tot; t += 32u) {
        const uint32_t e = t + lane;
        uint32_t r = 0;  // last of the nr rows that starts at or before e
#pragma unroll
        for (uint32_t d = 16; d; d >>= 1) {
            const uint32_t s = __shfl_sync(0xffffffffu, st, (int)min(r + d, 31u));
            if (r + d < nr && s <= e) r += d;
        }
        if (e < tot) rowidx[b + e] = r0 + r;
    }
}

// cptr[j] = first place of a column >= j among the sorted columns, j = 0 .. m (a search per column:
// no counting by atomics, and columns without elements cost no more than others)
__global__ void k_col_starts(uint32_t nnz, uint32_t m, const uint32_t *__restrict__ sorted,
                             uint32_t *__restrict__ cptr)
{
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j > m) return;
    uint32_t lo = 0, hi = nnz;
    while (lo < hi) {
        const uint32_t mid = lo + (hi - lo) / 2;
        if (__ldg(sorted + mid) < j) lo = mid + 1;
        else hi = mid;
    }
    cptr[j] = lo;
}

__global__ void k_t_meta(uint32_t m, const uint32_t *cptr, const uint32_t *tperm, uint32_t *nmc,
                         uint32_t *tlen, uint32_t *tstart)
{
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= m) return;
    const uint32_t j = tperm[g], b = cptr[j], l = cptr[j + 1] - b;
    tlen[g] = l;
    tstart[g] = b;
    if ((g & 31) == 0) nmc[g >> 5] = l;
}

unsigned blocks_of(size_t n) { return (unsigned)((n + 255) / 256); }

template <class T>
gs_status gather_vals(size_t n, const DevBuf &src, const T *v, T *out, cudaStream_t s)
{
    if (!n) return GS_OK;
    if (n % 4 == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0)
        k_gather_vals4<T><<<blocks_of(n / 4), 256, 0, s>>>(n / 4, src.as<uint4>(), v, out);
    else
        k_gather_vals<T><<<148u * 16u, 256, 0, s>>>(n, src.as<uint32_t>(), v, out);
    GS_CHECK_LAUNCH();
    return GS_OK;
}

// adjoint-layout slots -> CSR order
template <class T>
gs_status scatter_vals(const gs_matrix *A, const T *v, T *out, cudaStream_t s)
{
    k_scatter_vals<T><<<148u * 16u, 256, 0, s>>>(A->tlenVC, A->tsrc.as<uint32_t>(), v, out);
    GS_CHECK_LAUNCH();
    return GS_OK;
}

// Rows of 64 bytes and more go by several lanes per row (FP64 k = 8 / 16 / 32, a band 60 / 138 / 293
// -> 46 / 87 / 141 us, a 524,288-row power-law 96 / 246 / 400 -> 75 / 194 / 300; FP32 k = 32 140 ->
// 83 and 264 -> 200), but for FP32 k = 16, whose two lanes a row lose on a 27-point stencil 80^3 (81
// -> 99; a band 60 -> 53, the power-law 96 -> 96).
template <class T> constexpr bool several_lanes(uint32_t k)
{
    return sizeof(T) == 8 ? k >= 8 : k > 16;
}

// The products of one lane a row, and the adjoint with its value gradient at every width
template <class T, int K, bool ADJ> gs_status launch_mm_k(const MMArgs &a, cudaStream_t s)
{
    if constexpr (ADJ || !several_lanes<T>(K)) {
        const uint32_t blocks = (a.units + kMMThreads / 32 - 1) / (kMMThreads / 32);
        k_k1_mm<T, K, ADJ><<<blocks, kMMThreads, 0, s>>>(a);
        GS_CHECK_LAUNCH();
        return GS_OK;
    } else {
        return launch_mm_wide<T>(a, K, s);
    }
}

template <class T, bool ADJ>
gs_status launch_mm(const MMArgs &a, uint32_t k, cudaStream_t s)
{
    if (!a.units) return GS_OK;
    switch (k) {
    case 1: return launch_mm_k<T, 1, ADJ>(a, s);
    case 2: return launch_mm_k<T, 2, ADJ>(a, s);
    case 4: return launch_mm_k<T, 4, ADJ>(a, s);
    case 8: return launch_mm_k<T, 8, ADJ>(a, s);
    case 16: return launch_mm_k<T, 16, ADJ>(a, s);
    case 32: return launch_mm_k<T, 32, ADJ>(a, s);
    default: return fail(GS_ERR_UNSUPPORTED, "k = %u right-hand sides (1, 2, 4, 8, 16, 32)", k);
    }
}

template <class T>
gs_status launch_atomic(const AtomicArgs &a, uint32_t k, cudaStream_t s)
{
    if (!a.units) return GS_OK;
    const uint32_t blocks = min((a.units + 7) / 8, 148u * 64u);
    switch (k) {
    case 1: k_k1_adj_atomic<T, 1><<<blocks, 256, 0, s>>>(a); break;
    case 2: k_k1_adj_atomic<T, 2><<<blocks, 256, 0, s>>>(a); break;
    case 4: k_k1_adj_atomic<T, 4><<<blocks, 256, 0, s>>>(a); break;
    case 8: k_k1_adj_atomic<T, 8><<<blocks, 256, 0, s>>>(a); break;
    case 16: k_k1_adj_atomic<T, 16><<<blocks, 256, 0, s>>>(a); break;
    case 32: k_k1_adj_atomic<T, 32><<<blocks, 256, 0, s>>>(a); break;
    default: return fail(GS_ERR_UNSUPPORTED, "k = %u right-hand sides (1, 2, 4, 8, 16, 32)", k);
    }
    GS_CHECK_LAUNCH();
    return GS_OK;
}

bool valid_k(uint32_t k) { return k == 1 || k == 2 || k == 4 || k == 8 || k == 16 || k == 32; }

gs_status check_mm_matrix(const gs_matrix *A)
{
    if (A->p.format != GS_FMT_K1)
        return fail(GS_ERR_UNSUPPORTED, "multi-RHS products and adjoints run on K1 matrices");
    if (A->p.vtype != GS_F64 && A->p.vtype != GS_F32)
        return fail(GS_ERR_UNSUPPORTED, "multi-RHS products take FP64 or FP32 values");
    if (A->p.itype != GS_IDX_U32)
        return fail(GS_ERR_UNSUPPORTED, "multi-RHS products take 32-bit columns");
    return GS_OK;
}

bool aligned32(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 31u) == 0; }

std::mutex g_mm_mutex;  // guards the lazily sized multi-RHS scratch of a matrix

gs_status ensure_mm_scratch(gs_matrix *A, cudaStream_t s)
{
    std::lock_guard<std::mutex> lock(g_mm_mutex);
    if (A->mm_ready) return GS_OK;
    GS_TRY(A->mmpartial.alloc((size_t)A->k1split_units * 32 * 32 * 8 + 8, s));
    GS_CUDA(cudaStreamSynchronize(s));  // from here on any stream may use it
    A->mm_ready = true;
    return GS_OK;
}

// CSR order -> forward slots
k1fill::Args forward_fill(const gs_matrix *A)
{
    k1fill::Args f{};
    f.n = A->nrows;
    f.units = A->k1units;
    f.unit_chunk = A->k1unit_chunk.as<uint32_t>();
    f.unit_base = A->k1unit_base.as<uint32_t>();
    f.nmc = A->nmc.as<uint32_t>();
    f.chp = A->chp.as<uint32_t>();
    f.start = A->kstart.as<uint32_t>();
    f.len = A->k1len.as<uint32_t>();
    return f;
}

template <class T>
gs_status refresh_values(gs_matrix *A, const T *v, gs_value_order order, cudaStream_t s)
{
    if (order == GS_VALUES_CSR) {
        k1fill::Args f = forward_fill(A);
        f.val = v;
        f.oval = A->val.p;
        GS_TRY((k1fill::fill<T, T, false>(f, T(0), s)));
        GS_TRY(gather_vals<T>(A->tlenVC, A->tsrc, v, A->tval.as<T>(), s));
    } else {
        GS_TRY(gather_vals<T>(A->lenVC, A->ftslot, v, A->val.as<T>(), s));
        GS_CUDA(cudaMemcpyAsync(A->tval.p, v, (size_t)A->tlenVC * sizeof(T),
                                cudaMemcpyDeviceToDevice, s));
    }
    GS_CHECK_LAUNCH();
    return GS_OK;
}

// The forward layout and its plan; Y = A X
MMArgs forward_args(const gs_matrix *A, const void *x, void *y)
{
    MMArgs a{};
    a.nrows = A->nrows;
    a.permi = A->permi.as<uint32_t>();
    a.nmc = A->nmc.as<uint32_t>();
    a.chp = A->chp.as<uint32_t>();
    a.klen = A->k1len.as<uint32_t>();
    a.val = A->val.p;
    a.col = A->col.as<uint32_t>();
    a.xin = x;
    a.yout = y;
    a.unit_chunk = A->k1unit_chunk.as<uint32_t>();
    a.unit_base = A->k1unit_base.as<uint32_t>();
    a.units = A->k1units;
    a.split_units = A->k1split_units;
    a.split_extra = A->k1units - A->chunkNum;
    a.partial = A->mmpartial.p;
    a.count = A->k1count.as<uint32_t>();
    a.nrb = 1;
    return a;
}

// The transposed layout and its plan; Xbar = A^T Ybar
MMArgs adjoint_args(const gs_matrix *A, const void *ybar, void *xbar)
{
    MMArgs a{};
    a.nrows = A->ncols;
    a.permi = A->tpermi.as<uint32_t>();
    a.nmc = A->tnmc.as<uint32_t>();
    a.chp = A->tchp.as<uint32_t>();
    a.klen = A->tlen.as<uint32_t>();
    a.val = A->tval.p;
    a.col = A->trow.as<uint32_t>();
    a.xin = ybar;
    a.yout = xbar;
    a.unit_chunk = A->tunit_chunk.as<uint32_t>();
    a.unit_base = A->tunit_base.as<uint32_t>();
    a.units = A->tunits;
    a.split_units = A->tsplit_units;
    a.split_extra = A->tunits - A->tchunkNum;
    a.partial = A->tpartial.p;
    a.count = A->tcount.as<uint32_t>();
    a.nrb = 1;
    return a;
}

gs_status check_strided(const gs_matrix *A, gs_dtype dtype, uint32_t k, uint32_t cols)
{
    GS_TRY(check_mm_matrix(A));
    if (dtype != A->p.vtype) return fail(GS_ERR_UNSUPPORTED, "operands take the value type");
    if (k < 1 || k > 32) return fail(GS_ERR_UNSUPPORTED, "k = %u right-hand sides (1..32)", k);
    if (cols < k) return fail(GS_ERR_INVALID, "%u readable columns for k = %u", cols, k);
    return GS_OK;
}
// rows of k entries, `ld` apart, each entry aligned to its size
gs_status check_rows(const char *what, const void *p, uint32_t ld, uint32_t k, gs_dtype dtype)
{
    if (ld < k) return fail(GS_ERR_INVALID, "%s: row stride %u below %u columns", what, ld, k);
    if (reinterpret_cast<uintptr_t>(p) % dtype_size(dtype))
        return fail(GS_ERR_INVALID, "%s is not aligned to its entries", what);
    return GS_OK;
}

}  // namespace

gs_status prepare_mm_scratch(gs_matrix *A, cudaStream_t s) { return ensure_mm_scratch(A, s); }

}  // namespace gs

using namespace gs;

extern "C" {

gs_status gs_spmm(gs_matrix *A, const void *d_X, void *d_Y, gs_dtype dtype, UIN k,
                  gs_stream stream)
{
    if (!A || !d_X || !d_Y) return fail(GS_ERR_INVALID, "NULL argument");
    GS_TRY(check_mm_matrix(A));
    if (dtype != A->p.vtype) return fail(GS_ERR_UNSUPPORTED, "X and Y take the value type");
    if (!valid_k(k)) return fail(GS_ERR_UNSUPPORTED, "k = %u right-hand sides (1, 2, 4, 8, 16, 32)", k);
    if (!aligned32(d_X) || !aligned32(d_Y)) return fail(GS_ERR_INVALID, "X and Y must be 32-byte aligned");
    cudaStream_t s = cs(stream);
    GS_TRY(ensure_mm_scratch(A, s));
    MMArgs a = forward_args(A, d_X, d_Y);
    a.ld = a.k = a.ldx = a.ldy = k;
    if (A->p.vtype == GS_F64) return launch_mm<double, false>(a, k, s);
    return launch_mm<float, false>(a, k, s);
}

gs_status gs_matrix_prepare_adjoint(gs_matrix *A, const UIN *d_row, const UIN *d_col,
                                    gs_stream stream)
{
    if (!A || !d_row || (A->nnz && !d_col)) return fail(GS_ERR_INVALID, "NULL argument");
    GS_TRY(check_mm_matrix(A));
    cudaStream_t s = cs(stream);
    GS_TRY(ensure_mm_scratch(A, s));
    if (A->adj_ready) return GS_OK;
    const uint32_t n = A->nrows, m = A->ncols, nnz = A->nnz;
    GS_TRY(A->kstart.alloc((size_t)n * 4, s));
    // row and column of each element, for value gradients in CSR order
    GS_TRY(A->vrow.alloc((size_t)nnz * 4, s));
    GS_TRY(A->vcol.alloc((size_t)nnz * 4, s));
    // CSC order of the elements: stable sort of CSR indices by ascending column
    StreamBuf ccount(s), csc(s), csorted(s), cptr(s), place(s), inv(s);
    GS_TRY(ccount.alloc((size_t)m * 4));
    GS_TRY(csc.alloc((size_t)nnz * 4));
    GS_TRY(csorted.alloc((size_t)nnz * 4));
    GS_TRY(place.alloc((size_t)nnz * 8));
    GS_TRY(inv.alloc((size_t)n * 4));
    if (n) {
        k_expand_rows<<<blocks_of(n), 256, 0, s>>>(n, d_row, A->vrow.as<uint32_t>());
        k_row_places<<<blocks_of(n), 256, 0, s>>>(n, d_row, A->permi.as<uint32_t>(),
                                                  A->kstart.as<uint32_t>(), inv.as<uint32_t>());
        GS_CHECK_LAUNCH();
    }
    if (nnz) {
        GS_CUDA(cudaMemcpyAsync(A->vcol.p, d_col, (size_t)nnz * 4, cudaMemcpyDeviceToDevice, s));
        k_forward_slots<<<blocks_of(nnz), 256, 0, s>>>(
            nnz, A->vrow.as<uint32_t>(), d_row, inv.as<uint32_t>(),
            A->chp.as<uint32_t>(), place.as<uint2>());
        GS_CHECK_LAUNCH();
        GS_TRY(stable_sort_asc(d_col, nnz, m ? m - 1 : 0, csc.as<uint32_t>(),
                               csorted.as<uint32_t>(), s));
    }
    GS_TRY(cptr.alloc(((size_t)m + 1) * 4));
    k_col_starts<<<m / 256 + 1, 256, 0, s>>>(nnz, m, csorted.as<uint32_t>(), cptr.as<uint32_t>());
    GS_CHECK_LAUNCH();
    // K1 layout of A^T: columns of A sorted by decreasing length
    const uint32_t tchunks = (m + 31) / 32;
    A->tchunkNum = tchunks;
    uint32_t top[2] = {0, 0};  // (check), longest column
    {
        StreamBuf out(s);
        GS_TRY(out.alloc_zero(8));
        GS_TRY(row_lengths(m, cptr.as<uint32_t>(), nnz, ccount.as<uint32_t>(), out.as<uint32_t>(), s));
        GS_CUDA(cudaMemcpyAsync(top, out.p, 8, cudaMemcpyDeviceToHost, s));
        GS_CUDA(cudaStreamSynchronize(s));
    }
    const uint32_t maxlen = top[1];
    GS_TRY(A->tpermi.alloc_zero(((size_t)tchunks + 1) * 32 * 4, s));
    GS_TRY(stable_sort_desc(ccount.as<uint32_t>(), m, maxlen, A->tpermi.as<uint32_t>(), s));
    GS_TRY(A->tnmc.alloc_zero((size_t)tchunks * 4 + 4, s));
    GS_TRY(A->tlen.alloc((size_t)m * 4 + 4, s));
    StreamBuf tstart(s);
    GS_TRY(tstart.alloc((size_t)m * 4));
    if (m) {
        k_t_meta<<<blocks_of(m), 256, 0, s>>>(m, cptr.as<uint32_t>(), A->tpermi.as<uint32_t>(),
                                              A->tnmc.as<uint32_t>(), A->tlen.as<uint32_t>(),
                                              tstart.as<uint32_t>());
        GS_CHECK_LAUNCH();
    }
    GS_TRY(A->tchp.alloc((size_t)tchunks * 4 + 4, s));
    GS_TRY(A->tunit_base.alloc(((size_t)tchunks + 1) * 4, s));
    uint64_t total[3] = {0, 0, 0};
    GS_TRY(k1_layout_scan(A->tnmc.as<uint32_t>(), tchunks, A->tchp.as<uint32_t>(),
                          A->tunit_base.as<uint32_t>(), total, s));
    if (total[0] > 0xffffffffull) return fail(GS_ERR_OVERFLOW, "transposed K1 exceeds 32-bit slots");
    if (total[1] >= 0xffffffffull) return fail(GS_ERR_OVERFLOW, "K1 plan too large");
    A->tlenVC = (uint32_t)total[0];
    A->tunits = (uint32_t)total[1];
    A->tsplit_units = (uint32_t)total[2];
    const size_t vsz = A->p.vtype == GS_F64 ? 8 : 4;
    GS_TRY(build_k1_units(A->tunit_base.as<uint32_t>(), tchunks, A->tunits, A->tunit_chunk,
                          nullptr, A->tcount, s));
    GS_TRY(A->tpartial.alloc((size_t)A->tsplit_units * 32 * 32 * 8 + 8, s));
    GS_TRY(A->trow.alloc((size_t)A->tlenVC * 4, s));
    GS_TRY(A->tsrc.alloc((size_t)A->tlenVC * 4, s));
    GS_TRY(A->tval.alloc((size_t)A->tlenVC * vsz, s));
    GS_TRY(A->t2f.alloc((size_t)A->tlenVC * 4 + 4, s));
    GS_TRY(A->ftslot.alloc((size_t)A->lenVC * 4 + 4, s));  // forward slot -> adjoint-layout slot
    // adjoint-layout slot -> CSR index
    k1fill::Args tf{};
    tf.n = m;
    tf.units = A->tunits;
    tf.unit_chunk = A->tunit_chunk.as<uint32_t>();
    tf.unit_base = A->tunit_base.as<uint32_t>();
    tf.nmc = A->tnmc.as<uint32_t>();
    tf.chp = A->tchp.as<uint32_t>();
    tf.start = tstart.as<uint32_t>();
    tf.len = A->tlen.as<uint32_t>();
    tf.val = csc.p;
    tf.oval = A->tsrc.p;
    GS_TRY((k1fill::fill<uint32_t, uint32_t, false>(tf, kNoSrc, s)));
    GS_CUDA(cudaMemsetAsync(A->ftslot.p, 0xff, (size_t)A->lenVC * 4, s));  // kNoSrc
    if (A->tlenVC) {
        if (A->p.vtype == GS_F64)
            k_t_maps<double><<<blocks_of(A->tlenVC), 256, 0, s>>>(
                A->tlenVC, A->tsrc.as<uint32_t>(), place.as<uint2>(), A->val.as<double>(),
                A->trow.as<uint32_t>(), A->tval.as<double>(), A->t2f.as<uint32_t>(),
                A->ftslot.as<uint32_t>());
        else
            k_t_maps<float><<<blocks_of(A->tlenVC), 256, 0, s>>>(
                A->tlenVC, A->tsrc.as<uint32_t>(), place.as<uint2>(), A->val.as<float>(),
                A->trow.as<uint32_t>(), A->tval.as<float>(), A->t2f.as<uint32_t>(),
                A->ftslot.as<uint32_t>());
        GS_CHECK_LAUNCH();
    }
    GS_TRY(A->vslots.alloc((size_t)max(A->lenVC, A->tlenVC) * vsz + 8, s));
    A->adj_ready = true;
    GS_CUDA(cudaStreamSynchronize(s));
    return GS_OK;
}

gs_status gs_matrix_set_values(gs_matrix *A, const void *d_val, gs_dtype dtype,
                               gs_value_order order, gs_stream stream)
{
    if (!A || (A->nnz && !d_val)) return fail(GS_ERR_INVALID, "NULL argument");
    GS_TRY(check_mm_matrix(A));
    if (!A->adj_ready)
        return fail(GS_ERR_INVALID, "gs_matrix_prepare_adjoint must run first");
    if (dtype != A->p.vtype) return fail(GS_ERR_UNSUPPORTED, "values take the matrix value type");
    if (order != GS_VALUES_CSR && order != GS_VALUES_SLOTS)
        return fail(GS_ERR_INVALID, "unknown value order %d", (int)order);
    cudaStream_t s = cs(stream);
    if (dtype == GS_F64) return refresh_values(A, static_cast<const double *>(d_val), order, s);
    return refresh_values(A, static_cast<const float *>(d_val), order, s);
}

gs_status gs_matrix_value_slots(const gs_matrix *A, UIN *nslots)
{
    if (!A || !nslots) return fail(GS_ERR_INVALID, "NULL argument");
    if (!A->adj_ready) return fail(GS_ERR_INVALID, "gs_matrix_prepare_adjoint must run first");
    *nslots = A->tlenVC;
    return GS_OK;
}

gs_status gs_matrix_convert_values(const gs_matrix *A, const void *d_in, gs_value_order in_order,
                                   void *d_out, gs_dtype dtype, gs_stream stream)
{
    if (!A || !d_in || !d_out) return fail(GS_ERR_INVALID, "NULL argument");
    if (!A->adj_ready) return fail(GS_ERR_INVALID, "gs_matrix_prepare_adjoint must run first");
    if (dtype != A->p.vtype) return fail(GS_ERR_UNSUPPORTED, "values take the matrix value type");
    cudaStream_t s = cs(stream);
    const bool f64 = dtype == GS_F64;
    if (in_order == GS_VALUES_CSR) {  // slots[t] = csr[tsrc[t]], padding 0
        return f64 ? gather_vals<double>(A->tlenVC, A->tsrc, static_cast<const double *>(d_in),
                                         static_cast<double *>(d_out), s)
                   : gather_vals<float>(A->tlenVC, A->tsrc, static_cast<const float *>(d_in),
                                        static_cast<float *>(d_out), s);
    }
    if (in_order == GS_VALUES_SLOTS) {  // csr[tsrc[t]] = slots[t]
        return f64 ? scatter_vals(A, static_cast<const double *>(d_in),
                                  static_cast<double *>(d_out), s)
                   : scatter_vals(A, static_cast<const float *>(d_in),
                                  static_cast<float *>(d_out), s);
    }
    return fail(GS_ERR_INVALID, "unknown value order %d", (int)in_order);
}

gs_status gs_spmm_adjoint(gs_matrix *A, const void *d_Ybar, const void *d_X, void *d_Xbar,
                          void *d_vbar, gs_dtype dtype, UIN k, gs_adjoint_mode mode,
                          gs_value_order vbar_order, gs_stream stream)
{
    if (vbar_order != GS_VALUES_CSR && vbar_order != GS_VALUES_SLOTS)
        return fail(GS_ERR_INVALID, "unknown value order %d", (int)vbar_order);
    if (!A || !d_Ybar || !d_Xbar || (d_vbar && !d_X)) return fail(GS_ERR_INVALID, "NULL argument");
    GS_TRY(check_mm_matrix(A));
    if (!A->adj_ready)
        return fail(GS_ERR_INVALID, "gs_matrix_prepare_adjoint must run first");
    if (dtype != A->p.vtype) return fail(GS_ERR_UNSUPPORTED, "operands take the value type");
    if (!valid_k(k)) return fail(GS_ERR_UNSUPPORTED, "k = %u right-hand sides (1, 2, 4, 8, 16, 32)", k);
    if (!aligned32(d_Ybar) || !aligned32(d_Xbar) || (d_X && !aligned32(d_X)))
        return fail(GS_ERR_INVALID, "Ybar, X and Xbar must be 32-byte aligned");
    cudaStream_t s = cs(stream);
    const bool f64 = A->p.vtype == GS_F64;
    if (mode != GS_ADJ_ATOMIC && mode != GS_ADJ_DETERMINISTIC)
        return fail(GS_ERR_INVALID, "unknown adjoint mode %d", (int)mode);
    // a value gradient in CSR order has its own kernel; one in slot order comes with Xbar.  With 32
    // right-hand sides the own kernel gathers two more rows of 128 or 256 bytes an element than the
    // pass that forms both, which then leads also in CSR order, its gradient scattered (FP64 on a
    // 524,288-row power-law / a band / a 27-point stencil 80^3 667 / 452 / 882 us with the own
    // kernel, 519 / 399 / 761 so; FP32 300 / 215 / 422 and 279 / 218 / 364)
    const bool scatter = d_vbar && vbar_order == GS_VALUES_CSR && k == 32 &&
                         mode == GS_ADJ_DETERMINISTIC;
    const bool csr_vbar = d_vbar && vbar_order == GS_VALUES_CSR && !scatter;
    if (csr_vbar) {
        VbarArgs v{};
        v.nnz = A->nnz;
        v.k = v.ldx = v.ldy = k;
        v.row = A->vrow.as<uint32_t>();
        v.col = A->vcol.as<uint32_t>();
        v.x = d_X;
        v.ybar = d_Ybar;
        v.vbar = d_vbar;
        GS_TRY((f64 ? launch_vbar<double>(v, k, s) : launch_vbar<float>(v, k, s)));
    }
    if (mode == GS_ADJ_ATOMIC) {
        GS_CUDA(cudaMemsetAsync(d_Xbar, 0, (size_t)A->ncols * k * (f64 ? 8 : 4), s));
        AtomicArgs a{};
        a.nrows = A->nrows;
        a.permi = A->permi.as<uint32_t>();
        a.chp = A->chp.as<uint32_t>();
        a.klen = A->k1len.as<uint32_t>();
        a.col = A->col.as<uint32_t>();
        // vbar in forward slot order first (coalesced), then gathered into the adjoint layout's
        const bool via_slots = d_vbar && !csr_vbar;
        a.unit_chunk = A->k1unit_chunk.as<uint32_t>();
        a.unit_base = A->k1unit_base.as<uint32_t>();
        a.units = A->k1units;
        a.val = A->val.p;
        a.x = d_X;
        a.ybar = d_Ybar;
        a.xbar = d_Xbar;
        a.vbar = via_slots ? A->vslots.p : nullptr;
        GS_TRY((f64 ? launch_atomic<double>(a, k, s) : launch_atomic<float>(a, k, s)));
        if (via_slots) {
            GS_TRY((f64 ? gather_vals<double>(A->tlenVC, A->t2f, A->vslots.as<double>(),
                                              static_cast<double *>(d_vbar), s)
                        : gather_vals<float>(A->tlenVC, A->t2f, A->vslots.as<float>(),
                                             static_cast<float *>(d_vbar), s)));
        }
        return GS_OK;
    }
    MMArgs a = adjoint_args(A, d_Ybar, d_Xbar);
    a.xrow = d_X;
    a.vbar = csr_vbar ? nullptr : scatter ? A->vslots.p : d_vbar;
    a.ld = a.k = a.ldx = a.ldy = k;
    if (a.vbar) {
        GS_TRY((f64 ? launch_mm<double, true>(a, k, s) : launch_mm<float, true>(a, k, s)));
        if (!scatter) return GS_OK;
        return f64 ? scatter_vals(A, A->vslots.as<double>(), static_cast<double *>(d_vbar), s)
                   : scatter_vals(A, A->vslots.as<float>(), static_cast<float *>(d_vbar), s);
    }
    return f64 ? launch_mm<double, false>(a, k, s) : launch_mm<float, false>(a, k, s);
}

gs_status gs_spmm_strided(gs_matrix *A, const void *d_X, UIN ldx, void *d_Y, UIN ldy,
                          gs_dtype dtype, UIN k, UIN cols, gs_stream stream)
{
    if (!A || !d_X || !d_Y) return fail(GS_ERR_INVALID, "NULL argument");
    GS_TRY(check_strided(A, dtype, k, cols));
    GS_TRY(check_rows("X", d_X, ldx, cols, dtype));
    GS_TRY(check_rows("Y", d_Y, ldy, k, dtype));
    if (ldx == k && ldy == k && valid_k(k) && aligned32(d_X) && aligned32(d_Y))
        return gs_spmm(A, d_X, d_Y, dtype, k, stream);
    cudaStream_t s = cs(stream);
    GS_TRY(ensure_mm_scratch(A, s));
    MMArgs a = forward_args(A, d_X, d_Y);
    a.k = k;
    a.ldx = ldx;
    a.ldy = ldy;
    return dtype == GS_F64 ? launch_mm_wide<double>(a, cols, s) : launch_mm_wide<float>(a, cols, s);
}

gs_status gs_spmm_adjoint_strided(gs_matrix *A, const void *d_Ybar, UIN ldyb, const void *d_X,
                                  UIN ldx, void *d_Xbar, UIN ldxb, void *d_vbar, gs_dtype dtype,
                                  UIN k, UIN cols, gs_stream stream)
{
    if (!A || !d_Ybar || !d_Xbar || (d_vbar && !d_X)) return fail(GS_ERR_INVALID, "NULL argument");
    GS_TRY(check_strided(A, dtype, k, cols));
    GS_TRY(check_rows("Ybar", d_Ybar, ldyb, cols, dtype));
    GS_TRY(check_rows("Xbar", d_Xbar, ldxb, k, dtype));
    if (d_vbar) GS_TRY(check_rows("X", d_X, ldx, cols, dtype));
    if (!A->adj_ready)
        return fail(GS_ERR_INVALID, "gs_matrix_prepare_adjoint must run first");
    if (ldyb == k && ldxb == k && valid_k(k) && aligned32(d_Ybar) && aligned32(d_Xbar) &&
        (!d_vbar || (ldx == k && aligned32(d_X))))
        return gs_spmm_adjoint(A, d_Ybar, d_X, d_Xbar, d_vbar, dtype, k, GS_ADJ_DETERMINISTIC,
                               GS_VALUES_CSR, stream);
    cudaStream_t s = cs(stream);
    const bool f64 = dtype == GS_F64;
    if (d_vbar) {
        VbarArgs v{};
        v.nnz = A->nnz;
        v.k = k;
        v.ldx = ldx;
        v.ldy = ldyb;
        v.row = A->vrow.as<uint32_t>();
        v.col = A->vcol.as<uint32_t>();
        v.x = d_X;
        v.ybar = d_Ybar;
        v.vbar = d_vbar;
        GS_TRY((f64 ? launch_vbar_wide<double>(v, cols, s) : launch_vbar_wide<float>(v, cols, s)));
    }
    MMArgs a = adjoint_args(A, d_Ybar, d_Xbar);
    a.k = k;
    a.ldx = ldyb;
    a.ldy = ldxb;
    return f64 ? launch_mm_wide<double>(a, cols, s) : launch_mm_wide<float>(a, cols, s);
}

}  // extern "C"
