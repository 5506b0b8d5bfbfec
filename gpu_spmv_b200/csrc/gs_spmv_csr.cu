// gs_spmv_csr.cu -- the CSR product (CSR, COM tileH = 1) for matrices of local columns, and for
// CSR arrays that are multiplied once: straight from the row pointers, with no plan.
//
// Reference: gcsr (cudaSpmv.cu:531-543), one thread per row.  Here a warp owns G consecutive
// rows (4 to 128), as many as fill a window of some 5 KB of shared memory.  It copies their
// values and columns there with 16-byte asynchronous copies, in position order and whole lines;
// then 32 / G lanes walk each row from there, gathering x as they go, and add their sums in a
// shuffle tree.
// Neighbouring rows of a mesh or a band read neighbouring x, so the gathers of a step fall into
// few lines, where 32 consecutive elements of one row fall into as many as the row has runs.
// Rows that do not fit the window together are taken as many at a time as do, and a row longer
// than the window alone, by the whole warp, in several.  Every y entry is written once, by a
// fixed order of sums: no atomics, deterministic.  Sums are FP64 for every stored type.
//
// What bounds it: HBM on local columns.  The row-stream kernel that ran here before (start-bit
// ranks and a segmented warp scan per window, gs_spmv_rows.cu) spends 64 instructions a stored
// element (BF16 values, 16-bit columns, 27-point stencil 131^3: 69 % of the issue slots, DRAM
// 28 %).  Both kernels, us per product, row-stream -> this one:
//   FP64   27-point 160^3 309 -> 229 (6.1 TB/s of algorithmic bytes, 0.93 of the measured copy),
//          60^3 21.8 -> 11.0; Laplacian 2048^2 76.2 -> 58.5, 512^2 (in L2) 9.95 -> 4.75; band of
//          half-width 256 with 5 to 60 a row, 200,000 rows 24.8 -> 22
//   FP32   27-point 131^3 125 -> 86.5, Laplacian 2048^2 57.6 -> 46
//   BF16, 16-bit columns  27-point 131^3 124 -> 64, Laplacian 2048^2 50 -> 44
// Random columns stay on the row-stream kernel (power-law 4.2M rows: 326 us against 410 for
// products staged in position order), and so do rows of very uneven length, which leave lanes
// idle here (lognormal lengths of sigma 1.2, local columns, 24.5M elements: FP64 107 against 120
// us, BF16 60 against 133), few long rows (csr_enough_rows) and long rows side by side:
// gs_matrix_create looks at the matrix (csr_suits).  A product straight from CSR arrays runs here
// without that look, whose read-back would cost more than it saves (27-point 101^3 180 us with the
// row-stream kernel and its plan's kernels, 79 us here), until a warp meets long rows side by side
// (kCsrOverlong).
#include <cmath>

#include "gs_internal.cuh"

namespace gs {

namespace {

constexpr int kCsrWarps = 2;  // warps per block: its place is free when two warps end
constexpr unsigned kFull = 0xffffffffu;
// With CsrArgs::overlong: elements beside its longest row from which on a warp leaves its rows
// undone and says so.  One warp walks 150 (rows one by one) to 300 a microsecond, so this is about
// the time that the row-stream kernel's plan takes (30 rows of 12,000, 36,000 beside the longest:
// 325 us here, 367 with the plan; 1M rows of 27 and 128 of 30,000 side by side: 1457, 533).
constexpr uint32_t kCsrOverlong = 49152;

// Shared-memory index of position p for elements of B bytes: as it is, or (PAD) with a gap of 16
// bytes after every 128, for rows of about 8 m elements, whose lanes would otherwise meet in the
// same banks (FP64, 8 a row: 33.1 -> 23.4 us).
template <bool PAD, int B> __device__ __forceinline__ uint32_t csr_pad(uint32_t p)
{
    return PAD ? p + p / (128 / B) * (16 / B) : p;
}
template <bool PAD, int B, int CAP> constexpr int kCsrRoom =
    PAD ? CAP + (CAP + 128 / B - 1) / (128 / B) * (16 / B) : CAP;

__device__ __forceinline__ void copy16(void *d, const void *g)
{
    const uint32_t sa = (uint32_t)__cvta_generic_to_shared(d);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(g) : "memory");
}

// Positions 0 .. lim - 1 of a stream from g on (16-byte aligned) into s; `avail` exist
template <class T, int CAP, bool PAD>
__device__ __forceinline__ void csr_stage(T *s, const T *g, uint32_t lim, uint32_t avail, int lane)
{
    constexpr uint32_t P = 16 / sizeof(T);
    if (lim + P <= avail) {
#pragma unroll
        for (uint32_t i = 0; i < (CAP + 32 * P - 1) / (32 * P); i++) {
            const uint32_t q = (i * 32u + (uint32_t)lane) * P;
            if (q < lim) copy16(s + csr_pad<PAD, sizeof(T)>(q), g + q);
        }
    } else {  // the stream's end
        for (uint32_t q = (uint32_t)lane; q < lim; q += 32u) s[csr_pad<PAD, sizeof(T)>(q)] = g[q];
    }
}

// FP64: fused, one rounding less than the CPU loop.  With the four interleaved sums below, the
// relative error of y against 64-bit products summed exactly, row-stream kernel -> here: Laplacian
// 512^2 7.5e-17 -> 6.5e-17, 27-point 101^3 1.35e-16 -> 1.05e-16, band of half-width 256 1.41e-16 ->
// 1.19e-16 (one fused sum in row order: 7.7e-17, 1.31e-16, 1.32e-16).  FP32 / BF16: the product
// rounded to FP32 as everywhere in the engine, the sum FP64.
template <class VT, class XT> __device__ __forceinline__ double csr_add(double sum, VT v, XT x)
{
    if constexpr (sizeof(VT) == 8) return __fma_rn(v, x, sum);
    else return __dadd_rn(sum, (double)__fmul_rn(ValTraits<VT>::to_f32(v), x));
}

// Sum of the staged positions j, j + L, .. < e of one lane: four interleaved sums, then a tree
template <bool PAD, class VT, class IT, class XT>
__device__ __forceinline__ double csr_walk(const VT *sv, const IT *sc, const uint32_t *sb,
                                           uint32_t b0, const XT *__restrict__ x, uint32_t j,
                                           uint32_t e, uint32_t L)
{
    constexpr int U = 4;  // gathers in flight per lane
    auto gather = [&](uint32_t q) {
        uint32_t c = (uint32_t)sc[csr_pad<PAD, sizeof(IT)>(q)];
        if constexpr (sizeof(IT) == 2) c += sb[(b0 + q) >> 8];
        return __ldg(x + c);
    };
    double acc[U] = {0.0, 0.0, 0.0, 0.0};
    for (; j + (U - 1) * L < e; j += U * L) {
        XT xv[U];
#pragma unroll
        for (int k = 0; k < U; k++) xv[k] = gather(j + k * L);
#pragma unroll
        for (int k = 0; k < U; k++)
            acc[k] = csr_add<VT, XT>(acc[k], sv[csr_pad<PAD, sizeof(VT)>(j + k * L)], xv[k]);
    }
    if (j < e) {
        XT xv[U - 1];
#pragma unroll
        for (int k = 0; k < U - 1; k++)
            if (j + k * L < e) xv[k] = gather(j + k * L);
#pragma unroll
        for (int k = 0; k < U - 1; k++)
            if (j + k * L < e)
                acc[k] = csr_add<VT, XT>(acc[k], sv[csr_pad<PAD, sizeof(VT)>(j + k * L)], xv[k]);
    }
    return __dadd_rn(__dadd_rn(acc[0], acc[1]), __dadd_rn(acc[2], acc[3]));
}

template <class VT, class IT, int CAP, int G, bool PAD>
__global__ void __launch_bounds__(kCsrWarps * 32) k_csr(const CsrArgs a)
{
    using XT = typename std::conditional<sizeof(VT) == 8, double, float>::type;
    constexpr int L = G < 32 ? 32 / G : 1;  // lanes per row when the G rows fit the window
    constexpr int R = G > 32 ? G / 32 : 1;  // rows per lane
    constexpr int W = 32 / L;               // rows per step of the warp
    __shared__ __align__(16) VT sval[kCsrWarps][kCsrRoom<PAD, sizeof(VT), CAP>];
    __shared__ __align__(16) IT scol[kCsrWarps][kCsrRoom<PAD, sizeof(IT), CAP>];
    __shared__ uint32_t sbase[kCsrWarps][sizeof(IT) == 2 ? CAP / 256 + 2 : 1];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t r0 = (blockIdx.x * kCsrWarps + (uint32_t)wid) * (uint32_t)G;
    if (r0 >= a.n) return;
    const VT *__restrict__ val = static_cast<const VT *>(a.val);
    const IT *__restrict__ col = static_cast<const IT *>(a.col);
    const XT *__restrict__ x = static_cast<const XT *>(a.x);
    auto put = [&](uint32_t row, double v) {
        if (sizeof(VT) == 8 || a.y64) static_cast<double *>(a.y)[row] = v;
        else static_cast<float *>(a.y)[row] = (float)v;
    };
    VT *const sv = sval[wid];
    IT *const sc = scol[wid];
    uint32_t *const sb = sbase[wid];
    uint32_t rp[R], re[R];  // of rows r0 + W k + lane / L
#pragma unroll
    for (int k = 0; k < R; k++) {
        const uint32_t r = min(r0 + (uint32_t)(W * k + lane / L), a.n);
        rp[k] = min(__ldg(a.row + r), a.nnz);
        re[k] = min(__ldg(a.row + min(r + 1u, a.n)), a.nnz);
    }
    // positions c0 .. c0 + lim - 1 into shared memory
    auto stage = [&](uint32_t c0, uint32_t lim) {
        csr_stage<VT, CAP, PAD>(sv, val + c0, lim, a.nnz - c0, lane);
        csr_stage<IT, CAP, PAD>(sc, col + c0, lim, a.nnz - c0, lane);
        if constexpr (sizeof(IT) == 2) {
            const uint32_t b = (c0 >> 8) + (uint32_t)lane;
            if (lim && b <= (c0 + lim - 1u) >> 8) sb[lane] = __ldg(a.colbase + b);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
    };
    const uint32_t c0 = __shfl_sync(kFull, rp[0], 0) & ~7u, end = __shfl_sync(kFull, re[R - 1], 31);
    if (end >= c0 && end - c0 <= (uint32_t)CAP) {
        stage(c0, end - c0);
#pragma unroll
        for (int k = 0; k < R; k++) {
            double sum = csr_walk<PAD, VT, IT, XT>(sv, sc, sb, c0 & 255u, x,
                                                   rp[k] - c0 + (uint32_t)(lane % L),
                                                   min(re[k] - c0, end - c0), L);
#pragma unroll
            for (int d = L / 2; d; d >>= 1) sum = __dadd_rn(sum, __shfl_xor_sync(kFull, sum, d));
            const uint32_t r = r0 + (uint32_t)(W * k + lane / L);
            if (lane % L == 0 && r < a.n) put(r, sum);
        }
        return;
    }
    // too long for one window: as many rows at a time as fit, a longer row alone in windows
    if (a.overlong && end > c0) {
        uint32_t longest = 0;
#pragma unroll
        for (int k = 0; k < R; k++) longest = max(longest, re[k] > rp[k] ? re[k] - rp[k] : 0u);
        longest = __reduce_max_sync(kFull, longest);
        if (end - c0 > longest && end - c0 - longest > kCsrOverlong) {
            if (lane == 0) *static_cast<volatile uint32_t *>(a.overlong) = 1u;
            return;
        }
    }
#pragma unroll 1
    for (int k = 0; k < R; k++) {
        const uint32_t b0 = r0 + (uint32_t)(W * k);
        const uint32_t p = rp[R == 1 ? 0 : k], q = re[R == 1 ? 0 : k];
        for (int i = 0; i < W && b0 + (uint32_t)i < a.n;) {
            const uint32_t ps = __shfl_sync(kFull, p, i * L), w0 = ps & ~7u;
            const unsigned fit =
                __ballot_sync(kFull, lane >= i * L && q >= ps && q - w0 <= (uint32_t)CAP);
            // rows i .. i + cnt - 1 (a run: the pointers ascend)
            const int cnt = fit ? min((__popc(fit) + L - 1) / L, W - i) : 1;
            const uint32_t pe = __shfl_sync(kFull, q, (i + cnt - 1) * L);
            const int lg = cnt <= 1 ? 5 : __clz(cnt - 1) - 27;
            const int gi = lane >> lg, src = min((i + gi) * L, 31);
            const uint32_t s = __shfl_sync(kFull, p, src), e = __shfl_sync(kFull, q, src);
            double sum = 0.0;
            for (uint32_t w = w0; w < pe; w += (uint32_t)CAP) {
                const uint32_t lim = min(pe - w, (uint32_t)CAP);
                __syncwarp();
                stage(w, lim);
                if (gi < cnt) {
                    const uint32_t j = (s > w ? s - w : 0u) + ((uint32_t)lane & ((1u << lg) - 1u));
                    sum = __dadd_rn(sum, csr_walk<PAD, VT, IT, XT>(sv, sc, sb, w & 255u, x, j,
                                                                   e > w ? min(e - w, lim) : 0u,
                                                                   1u << lg));
                }
                if (pe - w <= (uint32_t)CAP) break;
            }
            for (int d = (1 << lg) >> 1; d; d >>= 1)
                sum = __dadd_rn(sum, __shfl_xor_sync(kFull, sum, d));
            const uint32_t r = b0 + (uint32_t)(i + gi);
            if (gi < cnt && (lane & ((1 << lg) - 1)) == 0 && r < a.n) put(r, sum);
            i += cnt;
        }
    }
}

template <class VT, class IT, int CAP, int G, bool PAD>
gs_status launch_csr_g(const CsrArgs &a, cudaStream_t s)
{
    const uint64_t rows = (uint64_t)kCsrWarps * G;
    k_csr<VT, IT, CAP, G, PAD>
        <<<(uint32_t)((a.n + rows - 1) / rows), kCsrWarps * 32, 0, s>>>(a);
    GS_CHECK_LAUNCH();
    return GS_OK;
}

// The window `cap` and the rows G per warp, from the average row length with 5 % to spare: two or
// four rows per lane when they fit and leave an SM 32 warps (Laplacian 2048^2 67 -> 58.5 us, FP32
// 59.5 -> 46), else 32 rows in the smallest window that holds them (288 positions instead of 480
// for the Laplacian 2048^2: 72 -> 67 us, more warps per SM; BF16 27-point with 1024 instead of
// 480: 80 -> 68 us), else fewer rows in the largest, which is 5.8 KB of FP64 values and columns
// (27-point 160^3 with 256, 480, 640, 920 positions: 260, 229, 253, 224 us; 101^3 with its
// launch and synchronisation 85, 79, 86, 79).
struct CsrShape {
    int cap, rows;
};

CsrShape csr_shape(uint32_t n, uint32_t nnz, bool f64)
{
    const int big = f64 ? 480 : 1024;
    const double avg = (double)nnz / n;
    auto fits = [&](int rows, int cap) { return avg * rows <= (cap - 8) / 1.05; };
    if (fits(64, 480) && n / 64 >= 148u * 32u)
        return {480, fits(128, 480) && n / 128 >= 148u * 32u ? 128 : 64};
    if (fits(32, 288)) return {288, 32};
    if (fits(32, 480)) return {480, 32};
    for (int rows = 32; rows > 4; rows /= 2)
        if (fits(rows, big)) return {big, rows};
    return {big, 4};
}

template <class VT, class IT, bool PAD>
gs_status launch_csr_t(const CsrArgs &a, cudaStream_t s)
{
    constexpr int BIG = sizeof(VT) == 8 ? 480 : 1024;
    const CsrShape c = csr_shape(a.n, a.nnz, sizeof(VT) == 8);
    if (c.cap == 288) return launch_csr_g<VT, IT, 288, 32, PAD>(a, s);
    if constexpr (!PAD) {  // 64 rows a warp average 7 elements at most
        if (c.rows == 128) return launch_csr_g<VT, IT, 480, 128, PAD>(a, s);
        if (c.rows == 64) return launch_csr_g<VT, IT, 480, 64, PAD>(a, s);
    }
    if (c.rows == 32 && c.cap == 480) return launch_csr_g<VT, IT, 480, 32, PAD>(a, s);
    if (c.rows == 32) return launch_csr_g<VT, IT, BIG, 32, PAD>(a, s);
    if (c.rows == 16) return launch_csr_g<VT, IT, BIG, 16, PAD>(a, s);
    if (c.rows == 8) return launch_csr_g<VT, IT, BIG, 8, PAD>(a, s);
    return launch_csr_g<VT, IT, BIG, 4, PAD>(a, s);
}

template <class VT, class IT> gs_status launch_csr_v(const CsrArgs &a, cudaStream_t s)
{
    // rows of 8, 16, 24 .. elements nearly all: padded windows
    const double avg = (double)a.nnz / a.n;
    const long m = lround(avg);
    if (m && m % 8 == 0 && fabs(avg - (double)m) < 0.5) return launch_csr_t<VT, IT, true>(a, s);
    return launch_csr_t<VT, IT, false>(a, s);
}

}  // namespace

// A warp walks its four rows one after the other where they do not fit a window together (112
// elements on average for FP64, 241 for the reduced types), and the row-stream kernel cuts the
// stream into equal ranges whatever the rows: few rows of that length leave most of the chip idle
// here.  us per product, row-stream -> this kernel, FP64: rows of 200 elements, 1,000 / 3,000 /
// 6,000 / 10,000 of them 4.6 -> 7.8, 5.7 -> 7.9, 8.0 -> 8.5, 12.1 -> 9.5; of 300 6.0 -> 8.2, 7.9 ->
// 8.4, 12.8 -> 8.9, 17.5 -> 11.2; of 1,000 9.7 -> 19, 18 -> 25, 29 -> 34, 44 -> 48 (20,000: 81 -> 78);
// 30 rows of 100,000 534 -> 2519.  FP32: 300 5.4 -> 6.9, 6.2 -> 6.9, 8.9 -> 7.2, 13 -> 8.1.  So rows up
// to a window long from 6,000 of them on, longer ones from 20,000.
bool csr_enough_rows(uint32_t n, uint32_t nnz, gs_dtype vtype)
{
    const CsrShape c = csr_shape(n, nnz, vtype == GS_F64);
    const double avg = (double)nnz / n;
    if (avg * c.rows <= (c.cap - 8) / 1.05) return true;
    return n >= (avg <= c.cap ? 6000u : 20000u);
}

// Row lengths, for csr_suits: over `take` groups of 32 rows, `stride` groups apart, out[0] += 32
// times the longest row, out[1] += elements; out[2] = the longest row (where `rows` is n; 0 rows: it
// is known), and over all groups of G rows out[3] = the most elements (out cleared before).
__global__ void __launch_bounds__(256) k_row_shape(const uint32_t *__restrict__ row, uint32_t n,
                                                   uint32_t stride, uint32_t take, uint32_t G,
                                                   uint32_t rows, unsigned long long *out)
{
    __shared__ unsigned long long part[4];  // one atomic a block and number (a warp each: 10 us)
    if (threadIdx.x < 4) part[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t t = blockIdx.x * 256ull + threadIdx.x, all = gridDim.x * 256ull;
    for (uint64_t w = t >> 5; w < take; w += all >> 5) {
        const uint32_t r = (uint32_t)w * stride * 32u + lane;
        const uint32_t len = row[r + 1] - row[r];
        const uint32_t top = __reduce_max_sync(kFull, len), sum = __reduce_add_sync(kFull, len);
        if (lane == 0) {
            atomicAdd(part, 32ull * top);
            atomicAdd(part + 1, (unsigned long long)sum);
        }
    }
    uint32_t longest = 0, heaviest = 0;
    for (uint64_t r = t; r < rows; r += all) longest = max(longest, row[r + 1] - row[r]);
    for (uint64_t r = t * G; r < n; r += all * G)
        heaviest = max(heaviest, row[min(r + G, (uint64_t)n)] - row[r]);
    longest = __reduce_max_sync(kFull, longest);
    heaviest = __reduce_max_sync(kFull, heaviest);
    if (lane == 0) {
        atomicMax(part + 2, (unsigned long long)longest);
        atomicMax(part + 3, (unsigned long long)heaviest);
    }
    __syncthreads();
    if (threadIdx.x < 2 && part[threadIdx.x]) atomicAdd(out + threadIdx.x, part[threadIdx.x]);
    if ((threadIdx.x == 2 || threadIdx.x == 3) && part[threadIdx.x])
        atomicMax(out + threadIdx.x, part[threadIdx.x]);
}

// Whether a matrix's products run on k_csr rather than on the row-stream kernel: local columns;
// rows of even length (over a sample of groups of 32 rows, 32 times the longest at most 2.5 times
// the elements); rows of 2.5 elements or more on average (FP64, 3M rows of 1 / 2 / 3: 18.7 / 25.7 /
// 45.4 us on the row-stream kernel, 22.8 / 31.0 / 35.1 here; FP32, 12M: 66 / 66 / 92 and 77 / 77 /
// 85), for the reduced types of 4.5 unless they are nearly all the same (32 times the longest at
// most 1.25 times the elements; 12M rows of 4 in the four reduced types 108 / 94 / 96 / 93 us and
// 104 / 99 / 104 / 93, of 1 to 5 92 / 87 / 88 / 84 and 99 / 96 / 104 / 103, of 1 to 8 122 / 118 / 121
// / 119 and 125 / 124 / 137 / 130, of 5 137 / 132 / 134 / 131 and 116 / 110 / 118 / 107, of 1 to 9
// level); enough of them; and no group of a warp's rows that the warp would still be walking when
// the others are done.  A single long row is none (one warp walks it in either kernel: 300,000 rows
// of 5 and one of 30,000 288 us there, 141 here), nor a group of 1 1/4 windows (of 480 at least),
// nor one within 1/8000 of the elements (some 10 % of the product's time); several long rows side
// by side are (1M rows of 27, 16 of 2,000 among them 81 us there and 166 here, 64 of 10,000 123 and
// 946; 300,000 of 5 with 128 of 300 11 and 49).
static bool csr_suits(uint32_t n, uint32_t nnz, gs_dtype vtype, const unsigned long long steps[2],
                      const unsigned long long shape[4])
{
    const bool f64 = vtype == GS_F64, random = steps[1] * 4 < steps[0];
    if (random || shape[0] * 2 > shape[1] * 5) return false;
    if ((double)nnz < 2.5 * n) return false;
    if (!f64 && (double)nnz < 4.5 * n && shape[0] * 4 > shape[1] * 5) return false;
    if (!csr_enough_rows(n, nnz, vtype)) return false;
    const CsrShape c = csr_shape(n, nnz, f64);
    const double own = 1.25 * c.rows * (double)nnz / n;
    return shape[3] <= (c.cap > 480 ? 1280u : 600u) || shape[3] <= nnz / 8000u ||
           (double)shape[3] <= (double)shape[2] + own;
}

gs_status csr_choice(const uint32_t *d_row, const uint32_t *d_col, uint32_t n, uint32_t nnz,
                     gs_dtype vtype, uint32_t longest, CsrChoice *out, cudaStream_t s)
{
    *out = CsrChoice();
    if (n == 0) return GS_OK;
    StreamBuf cnt(s);
    GS_TRY(cnt.alloc_zero(48));
    unsigned long long *c = cnt.as<unsigned long long>();
    GS_TRY(sample_col_steps(d_row, d_col, n, c, s));
    const uint32_t groups = n / 32, take = groups < 4096u ? groups : 4096u;
    const uint32_t blocks = (n - 1) / 256 + 1;
    k_row_shape<<<blocks < 592u ? blocks : 592u, 256, 0, s>>>(
        d_row, n, take ? groups / take : 0u, take,
        (uint32_t)csr_shape(n, nnz, vtype == GS_F64).rows, longest ? 0u : n, c + 2);
    GS_CHECK_LAUNCH();
    unsigned long long h[6] = {0, 0, 0, 0, 0, 0};
    GS_CUDA(cudaMemcpyAsync(h, c, 48, cudaMemcpyDeviceToHost, s));
    GS_CUDA(cudaStreamSynchronize(s));
    if (longest) h[4] = longest;
    out->random = h[1] * 4 < h[0];
    out->local = csr_suits(n, nnz, vtype, h, h + 2);
    return GS_OK;
}

gs_status launch_csr(const CsrArgs &a0, gs_dtype vtype, gs_itype itype, gs_dtype ytype,
                     cudaStream_t s)
{
    CsrArgs a = a0;
    if (!a.n) return GS_OK;
    a.y64 = ytype == GS_F64;
    if (vtype == GS_F64) {
        if (ytype != GS_F64 || itype != GS_IDX_U32)
            return fail(GS_ERR_UNSUPPORTED, "FP64 matrices take FP64 y and 32-bit columns");
        return launch_csr_v<double, uint32_t>(a, s);
    }
    if (vtype == GS_F32 && itype == GS_IDX_U32) return launch_csr_v<float, uint32_t>(a, s);
    if (vtype == GS_F32 && itype == GS_IDX_U16) return launch_csr_v<float, uint16_t>(a, s);
    if (vtype == GS_BF16 && itype == GS_IDX_U32) return launch_csr_v<__nv_bfloat16, uint32_t>(a, s);
    if (vtype == GS_BF16 && itype == GS_IDX_U16) return launch_csr_v<__nv_bfloat16, uint16_t>(a, s);
    return fail(GS_ERR_UNSUPPORTED, "value type %d / index type %d not supported", (int)vtype,
                (int)itype);
}

}  // namespace gs
