// gs_scan.cu -- error state, device buffers and the device scan / sort primitives used by
// the format converters.
//
// The reference builds every format on the CPU with serial prefix loops (row pointers of
// AXC cudaSpmv.cu:937-948, AXT con cudaSpmv.cu:1158-1201, K1 chunk pointers 741-754) and a
// qsort for the K1 permutation (716-737); its block-local scan micro-benchmark (scan.cu)
// has no carry between blocks.  Here those become one device-wide exclusive scan
// (reduce / scan-of-block-sums / down-sweep, 64-bit offsets so 32-bit overflow is
// detected, no inter-block waiting) and a stable LSD radix sort of up to 8 bits a pass.
#include <cuda.h>

#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <utility>

#include "gs_internal.cuh"

namespace gs {

// ------------------------------------------------------------------ errors
static thread_local char g_err[512] = "";

gs_status fail(gs_status st, const char *fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    return st;
}
void clear_error() { g_err[0] = 0; }
const char *last_error_text() { return g_err; }

// ------------------------------------------------------------------ device memory
struct DevPool {
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;  // orders allocations and frees that belong to no stream
    int dev = -1;
    uint64_t ctx = 0;
    size_t live = 0, kept_for = 0;  // bytes in buffers; the value of `live` the pool was told
};

uint64_t context_id()
{
    using Get = CUresult (*)(CUcontext, unsigned long long *);
    static const Get get = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &r) !=
                cudaSuccess || r != cudaDriverEntryPointSuccess)
            f = nullptr;
        return reinterpret_cast<Get>(f);
    }();
    if (!get) return 1;
    unsigned long long id = 0;
    if (get(nullptr, &id) == CUDA_SUCCESS && id) return id;
    if (cudaFree(nullptr) != cudaSuccess) return 0;  // makes the context the thread's current one
    return get(nullptr, &id) == CUDA_SUCCESS ? id : 0;
}

namespace {

std::mutex g_pool_mutex;
// by device and context; never destroyed, since buffers may be reset while the process ends
auto &g_pools = *new std::map<std::pair<int, uint64_t>, DevPool>;

thread_local int t_idle_device = -1;  // DeviceIdle

gs_status pool_of(DevPool **out) try
{
    int dev = -1;
    GS_CUDA(cudaGetDevice(&dev));
    const uint64_t ctx = context_id();
    if (!ctx) return fail(GS_ERR_CUDA, "no context on device %d", dev);
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    DevPool &P = g_pools[{dev, ctx}];
    if (!P.pool) {
        P.dev = dev;
        P.ctx = ctx;
        if (!P.stream) GS_CUDA(cudaStreamCreateWithFlags(&P.stream, cudaStreamNonBlocking));
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t p = nullptr;
        GS_CUDA(cudaMemPoolCreate(&p, &props));
        uint64_t keep = kPoolIdle;
        GS_CUDA(cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep));
        P.pool = p;
    }
    *out = &P;
    return GS_OK;
} catch (const std::bad_alloc &) {
    return fail(GS_ERR_ALLOC, "host allocation failed");
}

// The pool holds on to what its buffers use and kPoolIdle more; it is told again when the use
// has moved by an eighth of that.
void pool_use(DevPool &P, size_t add, size_t sub)
{
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    P.live = P.live + add - sub;
    const size_t d = P.live > P.kept_for ? P.live - P.kept_for : P.kept_for - P.live;
    if (d >= kPoolIdle / 8) {
        uint64_t keep = P.live + kPoolIdle;
        cudaMemPoolSetAttribute(P.pool, cudaMemPoolAttrReleaseThreshold, &keep);
        P.kept_for = P.live;
    }
}

size_t rounded(size_t nbytes)  // slack: vector loads may touch the tail
{
    return ((nbytes + 255) / 256) * 256 + 256;
}

// n bytes ordered on s, or on the pool's own stream (own)
gs_status pool_alloc(size_t n, cudaStream_t s, bool own, void **p, DevPool **pool)
{
    GS_TRY(pool_of(pool));
    if (own) s = (*pool)->stream;
    // a captured allocation would belong to the graph, not to the buffer
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    GS_CUDA(cudaStreamIsCapturing(s, &cap));
    if (cap != cudaStreamCaptureStatusNone)
        return fail(GS_ERR_CUDA, "device memory is needed on a stream under capture");
    cudaError_t e = cudaMallocFromPoolAsync(p, n, (*pool)->pool, s);
    if (e == cudaSuccess && own && (e = cudaStreamSynchronize(s)) != cudaSuccess)
        cudaFreeAsync(*p, s);
    if (e != cudaSuccess) {
        *p = nullptr;
        cudaGetLastError();
        return fail(GS_ERR_ALLOC, "allocation of %zu bytes failed: %s", n, cudaGetErrorString(e));
    }
    pool_use(**pool, n, 0);
    return GS_OK;
}

}  // namespace

gs_status DevBuf::alloc(size_t nbytes)
{
    reset();
    GS_TRY(pool_alloc(rounded(nbytes), nullptr, true, &p, &pool));
    reserved = rounded(nbytes);
    bytes = nbytes;
    return GS_OK;
}

gs_status DevBuf::alloc(size_t nbytes, cudaStream_t s)
{
    reset();
    GS_TRY(pool_alloc(rounded(nbytes), s, false, &p, &pool));
    reserved = rounded(nbytes);
    bytes = nbytes;
    return GS_OK;
}

gs_status DevBuf::alloc_zero(size_t nbytes, cudaStream_t s)
{
    GS_TRY(alloc(nbytes, s));
    GS_CUDA(cudaMemsetAsync(p, 0, reserved, s));
    return GS_OK;
}

void DevBuf::reset()
{
    if (!p) return;
    int cur = -1;
    cudaGetDevice(&cur);
    if (cur != pool->dev) cudaSetDevice(pool->dev);
    // kernels of any stream may still read it; memory of a device that cannot be waited for
    // stays allocated, and that of an ended context has gone with it
    if (context_id() == pool->ctx &&
        (t_idle_device == pool->dev || cudaDeviceSynchronize() == cudaSuccess)) {
        cudaFreeAsync(p, pool->stream);
        pool_use(*pool, 0, reserved);
    }
    if (cur != pool->dev) cudaSetDevice(cur);
    p = nullptr;
    bytes = 0;
}

DeviceIdle::DeviceIdle() : outer(t_idle_device)
{
    int dev = -1;
    if (cudaDeviceSynchronize() == cudaSuccess) cudaGetDevice(&dev);
    t_idle_device = dev;
}
DeviceIdle::~DeviceIdle() { t_idle_device = outer; }

gs_status StreamBuf::alloc(size_t nbytes)
{
    GS_TRY(pool_alloc(rounded(nbytes), s, false, &p, &pool));
    reserved = rounded(nbytes);
    return GS_OK;
}

gs_status StreamBuf::alloc_zero(size_t nbytes)
{
    GS_TRY(alloc(nbytes));
    GS_CUDA(cudaMemsetAsync(p, 0, reserved, s));
    return GS_OK;
}

StreamBuf::~StreamBuf()
{
    if (!p) return;
    cudaFreeAsync(p, s);
    pool_use(*pool, 0, reserved);
}

gs_status release_cached()
{
    DevPool *P = nullptr;
    GS_TRY(pool_of(&P));
    GS_CUDA(cudaDeviceSynchronize());
    GS_CUDA(cudaMemPoolTrimTo(P->pool, 0));
    return GS_OK;
}

// ------------------------------------------------------------------ scan
// kind follows CountKind's order.
struct CountDev {
    int kind;
    const uint32_t *row;
    const uint32_t *arr;
    uint32_t a;
    __device__ __forceinline__ uint64_t operator()(size_t i) const
    {
        switch (kind) {
        case 0: {
            uint32_t l = row[i + 1] - row[i];
            return (uint64_t)((l + a - 1) / a);
        }
        case 1: return (uint64_t)arr[i];
        case 2: {
            uint64_t c = 0;
            for (uint32_t j = 0; j < a; j++) c += __popc(arr[i * a + j]);
            return c;
        }
        default: return (uint64_t)(row[i + 1] > row[i]);
        }
    }
};

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ uint64_t warp_incl_scan_u64(uint64_t v)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        uint64_t u = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += u;
    }
    return v;
}

// Block-wide exclusive scan of one value per thread; returns the exclusive prefix and the
// block total through *total.
__device__ __forceinline__ uint64_t block_excl_scan_u64(uint64_t v, uint64_t *total)
{
    __shared__ uint64_t wsum[kScanThreads / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint64_t inc = warp_incl_scan_u64(v);
    if (lane == 31) wsum[w] = inc;
    __syncthreads();
    if (w == 0) {
        constexpr int NW = kScanThreads / 32;
        uint64_t s = (lane < NW) ? wsum[lane] : 0;
        uint64_t si = warp_incl_scan_u64(s);
        if (lane < NW) wsum[lane] = si - s;  // exclusive offset of each warp
        if (lane == NW - 1) *total = si;
    }
    __syncthreads();
    uint64_t r = inc - v + wsum[w];
    __syncthreads();
    return r;
}

__global__ void k_scan_reduce(CountDev f, size_t n, uint64_t *bsum)
{
    size_t base = (size_t)blockIdx.x * kScanTile;
    uint64_t s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        size_t i = base + (size_t)k * kScanThreads + threadIdx.x;
        if (i < n) s += f(i);
    }
    __shared__ uint64_t tot;
    uint64_t t;
    (void)block_excl_scan_u64(s, &tot);
    __syncthreads();
    t = tot;
    if (threadIdx.x == 0) bsum[blockIdx.x] = t;
}

// Exclusive scan of nb block sums in place, one block of 1024 threads; bsum[nb] = total.  Block b
// scans the b-th array of nb + 1 entries.
__global__ void k_scan_blocks(uint64_t *bsum, size_t nb)
{
    bsum += blockIdx.x * (nb + 1);
    __shared__ uint64_t wsum[32];
    __shared__ uint64_t carry;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (size_t base = 0; base < nb; base += blockDim.x) {
        size_t i = base + threadIdx.x;
        uint64_t v = (i < nb) ? bsum[i] : 0;
        uint64_t inc = warp_incl_scan_u64(v);
        if (lane == 31) wsum[w] = inc;
        __syncthreads();
        if (w == 0) {
            uint64_t s = wsum[lane];
            uint64_t si = warp_incl_scan_u64(s);
            wsum[lane] = si - s;
        }
        __syncthreads();
        uint64_t ex = inc - v + wsum[w] + carry;
        __syncthreads();
        if (i < nb) bsum[i] = ex;
        if (threadIdx.x == blockDim.x - 1) carry = ex + v;
        __syncthreads();
    }
    if (threadIdx.x == 0) bsum[nb] = carry;
}

__global__ void k_scan_down(CountDev f, size_t n, size_t nb, const uint64_t *bsum, uint64_t *out)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) out[n] = bsum[nb];
    size_t base = (size_t)blockIdx.x * kScanTile + (size_t)threadIdx.x * kScanItems;
    uint64_t v[kScanItems];
    uint64_t s = 0;
    // blocked arrangement: thread t owns items base + 0..7 (contiguous)
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        size_t i = base + k;
        v[k] = (i < n) ? f(i) : 0;
        s += v[k];
    }
    __shared__ uint64_t tot;
    uint64_t ex = block_excl_scan_u64(s, &tot) + bsum[blockIdx.x];
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        size_t i = base + k;
        if (i < n) out[i] = ex;
        ex += v[k];
    }
}

gs_status exclusive_scan(const CountSpec &spec, size_t n, uint64_t *out, uint64_t *total,
                         cudaStream_t s)
{
    const CountDev f{(int)spec.kind, spec.row, spec.arr, spec.a};
    size_t nb = (n + kScanTile - 1) / kScanTile;
    if (nb == 0) nb = 1;
    StreamBuf sums(s);
    GS_TRY(sums.alloc((nb + 1) * sizeof(uint64_t)));
    uint64_t *bsum = sums.as<uint64_t>();
    k_scan_reduce<<<(unsigned)nb, kScanThreads, 0, s>>>(f, n, bsum);
    k_scan_blocks<<<1, 1024, 0, s>>>(bsum, nb);
    k_scan_down<<<(unsigned)nb, kScanThreads, 0, s>>>(f, n, nb, bsum, out);
    GS_CHECK_LAUNCH();
    if (total) {
        GS_CUDA(cudaMemcpyAsync(total, out + n, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
        GS_CUDA(cudaStreamSynchronize(s));
    }
    return GS_OK;
}

// ------------------------------------------------------------------ K1 layout
// Both prefix sums a K1 layout needs in one pass over its chunks' steps: slots (32 per step) and
// work units (pieces of kK1Split steps, at least one).
__device__ __forceinline__ uint64_t k1_units_of(uint32_t m)
{
    return m <= kK1Split ? 1u : ((uint64_t)m + kK1Split - 1u) / kK1Split;
}

__global__ void k_layout_reduce(const uint32_t *nmc, size_t n, size_t nb, uint64_t *bsum)
{
    const size_t base = (size_t)blockIdx.x * kScanTile;
    uint64_t slots = 0, units = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        const size_t i = base + (size_t)k * kScanThreads + threadIdx.x;
        if (i < n) {
            const uint32_t m = nmc[i];
            slots += 32ull * m;
            units += k1_units_of(m);
        }
    }
    __shared__ uint64_t ts, tu;
    (void)block_excl_scan_u64(slots, &ts);
    (void)block_excl_scan_u64(units, &tu);
    if (threadIdx.x == 0) {
        bsum[blockIdx.x] = ts;
        bsum[nb + 1 + blockIdx.x] = tu;
    }
}

// total: slots, units, 1 + the last unit of a cut chunk (0: no chunk is cut; cleared beforehand)
__global__ void k_layout_down(const uint32_t *nmc, size_t n, size_t nb, const uint64_t *bsum,
                              uint32_t *chp, uint32_t *unit_base, unsigned long long *total)
{
    const size_t base = (size_t)blockIdx.x * kScanTile + (size_t)threadIdx.x * kScanItems;
    uint32_t m[kScanItems];
    uint64_t slots = 0, units = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        m[k] = base + k < n ? nmc[base + k] : 0u;
        slots += 32ull * m[k];
        if (base + k < n) units += k1_units_of(m[k]);
    }
    __shared__ uint64_t ts, tu;
    uint64_t es = block_excl_scan_u64(slots, &ts) + bsum[blockIdx.x];
    uint64_t eu = block_excl_scan_u64(units, &tu) + bsum[nb + 1 + blockIdx.x];
    unsigned long long cut = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        if (base + k < n) {
            chp[base + k] = (uint32_t)es;
            unit_base[base + k] = (uint32_t)eu;
            const uint64_t u = k1_units_of(m[k]);
            if (u > 1) cut = eu + u;
            es += 32ull * m[k];
            eu += u;
        }
    }
    if (cut) atomicMax(total + 2, cut);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        total[0] = bsum[nb];
        total[1] = bsum[2 * nb + 1];
        unit_base[n] = (uint32_t)bsum[2 * nb + 1];
    }
}

gs_status k1_layout_scan(const uint32_t *nmc, uint32_t n, uint32_t *chp, uint32_t *unit_base,
                         uint64_t total[3], cudaStream_t s)
{
    size_t nb = ((size_t)n + kScanTile - 1) / kScanTile;
    if (nb == 0) nb = 1;
    StreamBuf sums(s), tot(s);
    GS_TRY(sums.alloc(2 * (nb + 1) * sizeof(uint64_t)));
    GS_TRY(tot.alloc_zero(3 * sizeof(uint64_t)));
    uint64_t *bsum = sums.as<uint64_t>();
    k_layout_reduce<<<(unsigned)nb, kScanThreads, 0, s>>>(nmc, n, nb, bsum);
    k_scan_blocks<<<2, 1024, 0, s>>>(bsum, nb);
    k_layout_down<<<(unsigned)nb, kScanThreads, 0, s>>>(nmc, n, nb, bsum, chp, unit_base,
                                                        tot.as<unsigned long long>());
    GS_CHECK_LAUNCH();
    GS_CUDA(cudaMemcpyAsync(total, tot.p, 3 * sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
    GS_CUDA(cudaStreamSynchronize(s));
    return GS_OK;
}

// ------------------------------------------------------------------ stable radix sort
// LSD radix sort of (key, index) pairs, at most 8 bits a pass.  A pass is bound by the bytes it
// moves (8 in, 8 out per element; the first reads only the keys and makes the indices, the last
// writes only the indices), so the wider the digit the fewer the bytes: one bit a pass took 14
// passes for row lengths and 20 for a million columns.  A block ranks a tile of kRadixTile
// elements: warps rank their own 256 in order (ballots of equal digits, one counter per digit and
// warp), the warps' counts are summed per digit, and the tile is reordered in shared memory
// before it is written, so that a digit's elements leave as one run (64 bytes on average with
// 256 digits and 4096 elements).  Between blocks there is no waiting: the tiles' digit counts
// are made by a pass of their own and scanned by one block per digit.
// 4.2M elements, 20-bit keys: 20 passes of one bit 1310 us, 3 passes of 7 bits about 130 us
// (150 in blocks of 256 threads with 16 elements each, whose registers left 3 blocks on an SM).
constexpr int kRadixThreads = 512;
constexpr int kRadixWarps = kRadixThreads / 32;
constexpr int kRadixItems = 8;
constexpr uint32_t kRadixTile = kRadixThreads * kRadixItems;
constexpr int kRadixDigits = 256;

// The first pass of a descending sort turns the keys round: ascending in flip - key
template <bool FIRST>
__device__ __forceinline__ uint32_t radix_key(uint32_t k, uint32_t flip)
{
    return FIRST && flip ? flip - k : k;
}

// count[d * tiles + t] = elements of tile t with digit d
template <bool FIRST>
__global__ void __launch_bounds__(kRadixThreads) k_radix_count(
    const uint32_t *__restrict__ kin, uint32_t n, uint32_t flip, uint32_t shift,
    uint32_t mask, uint32_t tiles, uint32_t *__restrict__ count)
{
    __shared__ uint32_t h[kRadixDigits];
    if (threadIdx.x < kRadixDigits) h[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t t0 = blockIdx.x * kRadixTile;
#pragma unroll
    for (int i = 0; i < kRadixItems; i++) {
        const uint32_t o = (uint32_t)i * kRadixThreads + threadIdx.x;
        if (o < n - t0)
            atomicAdd(&h[(radix_key<FIRST>(kin[t0 + o], flip) >> shift) & mask], 1u);
    }
    __syncthreads();
    if (threadIdx.x <= mask) count[(size_t)threadIdx.x * tiles + blockIdx.x] = h[threadIdx.x];
}

// Exclusive prefix of one value per thread over the block; *total (shared) = the sum.
__device__ __forceinline__ uint32_t radix_block_scan(uint32_t v, uint32_t *wsum, uint32_t *total)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t inc = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += u;
    }
    if (lane == 31) wsum[w] = inc;
    __syncthreads();
    uint32_t before = 0, all = 0;
#pragma unroll
    for (int i = 0; i < kRadixWarps; i++) {
        if (i < w) before += wsum[i];
        all += wsum[i];
    }
    if (threadIdx.x == 0) *total = all;
    __syncthreads();
    return before + inc - v;
}

// Block d: exclusive prefix of digit d's tile counts in place, total[d] = their sum.
__global__ void __launch_bounds__(kRadixThreads) k_radix_scan(uint32_t *__restrict__ count,
                                                              uint32_t tiles,
                                                              uint32_t *__restrict__ total)
{
    __shared__ uint32_t wsum[kRadixWarps], sum;
    uint32_t *c = count + (size_t)blockIdx.x * tiles;
    uint32_t carry = 0;
    for (uint32_t b = 0; b < tiles; b += kRadixThreads) {
        const uint32_t i = b + threadIdx.x;
        const uint32_t v = i < tiles ? c[i] : 0u;
        const uint32_t e = radix_block_scan(v, wsum, &sum);
        if (i < tiles) c[i] = carry + e;
        carry += sum;
        __syncthreads();
    }
    if (threadIdx.x == 0) total[blockIdx.x] = carry;
}

template <bool FIRST>
__global__ void __launch_bounds__(kRadixThreads) k_radix_scatter(
    const uint32_t *__restrict__ kin, const uint32_t *__restrict__ iin, uint32_t n,
    uint32_t flip, uint32_t shift, uint32_t mask, uint32_t tiles,
    const uint32_t *__restrict__ before, const uint32_t *__restrict__ total,
    uint32_t *__restrict__ kout, uint32_t *__restrict__ iout)
{
    __shared__ uint16_t wcount[kRadixWarps][kRadixDigits];
    __shared__ uint32_t start[kRadixDigits];  // digit's first position in the sorted tile
    __shared__ uint32_t dest[kRadixDigits];   // output index of that position
    __shared__ uint32_t skey[kRadixTile], sidx[kRadixTile];
    __shared__ uint32_t wsum[kRadixWarps], sum;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t t0 = blockIdx.x * kRadixTile;
    const uint32_t cnt = min(kRadixTile, n - t0);
    for (int i = threadIdx.x; i < kRadixWarps * kRadixDigits / 2; i += kRadixThreads)
        reinterpret_cast<uint32_t *>(&wcount[0][0])[i] = 0;
    __syncthreads();
    uint32_t key[kRadixItems], idx[kRadixItems], rank[kRadixItems];
    const uint32_t o0 = (uint32_t)w * 32u * kRadixItems + (uint32_t)lane;
#pragma unroll
    for (int i = 0; i < kRadixItems; i++) {
        const uint32_t o = o0 + 32u * i;
        key[i] = o < cnt ? radix_key<FIRST>(kin[t0 + o], flip) : 0u;
        idx[i] = FIRST ? t0 + o : (o < cnt ? iin[t0 + o] : 0u);
    }
#pragma unroll
    for (int i = 0; i < kRadixItems; i++) {
        const bool in = o0 + 32u * i < cnt;
        const unsigned live = __ballot_sync(0xffffffffu, in);
        if (in) {
            const uint32_t d = (key[i] >> shift) & mask;
            unsigned peers = live;  // lanes of the same digit, bit by bit
#pragma unroll
            for (int b = 0; b < 8; b++) {
                if ((mask >> b) & 1u) {
                    const unsigned B = __ballot_sync(live, (d >> b) & 1u);
                    peers &= ((d >> b) & 1u) ? B : ~B;
                }
            }
            const uint32_t below = (uint32_t)__popc(peers & ((1u << lane) - 1u));
            rank[i] = wcount[w][d] + below;
            __syncwarp(live);
            if (below == 0) wcount[w][d] += (uint16_t)__popc(peers);
            __syncwarp(live);
        }
    }
    __syncthreads();
    {
        const uint32_t d = threadIdx.x;
        uint32_t run = 0;
        if (d < kRadixDigits) {
#pragma unroll
            for (int i = 0; i < kRadixWarps; i++) {
                const uint32_t c = wcount[i][d];
                wcount[i][d] = (uint16_t)run;
                run += c;
            }
        }
        const uint32_t e = radix_block_scan(run, wsum, &sum);
        const uint32_t g = radix_block_scan(d <= mask ? total[d] : 0u, wsum, &sum);
        if (d < kRadixDigits) {
            start[d] = e;
            dest[d] = d <= mask ? g + before[(size_t)d * tiles + blockIdx.x] : 0u;
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kRadixItems; i++) {
        if (o0 + 32u * i < cnt) {
            const uint32_t d = (key[i] >> shift) & mask;
            const uint32_t p = start[d] + wcount[w][d] + rank[i];
            skey[p] = key[i];
            sidx[p] = idx[i];
        }
    }
    __syncthreads();
    for (uint32_t p = threadIdx.x; p < cnt; p += kRadixThreads) {
        const uint32_t k = skey[p], d = (k >> shift) & mask;
        const uint32_t g = dest[d] + (p - start[d]);
        if (kout) kout[g] = k;
        iout[g] = sidx[p];
    }
}

// idx[i] = i, and keys that are all 0
__global__ void k_iota(uint32_t n, uint32_t *idx, uint32_t *key)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    idx[i] = i;
    if (key) key[i] = 0u;
}

// key_out (or nullptr): the keys in their new order (flip - key where flip is given)
static gs_status stable_sort(const uint32_t *key, uint32_t n, uint32_t max_key, uint32_t flip,
                             uint32_t *idx_out, uint32_t *key_out, cudaStream_t s)
{
    if (n == 0) return GS_OK;
    int bits = 0;
    while (bits < 32 && (max_key >> bits) != 0) bits++;
    if (bits == 0) {  // all keys are 0: the order they came in
        k_iota<<<(n - 1) / 256 + 1, 256, 0, s>>>(n, idx_out, key_out);
        GS_CHECK_LAUNCH();
        return GS_OK;
    }
    const int passes = (bits + 7) / 8;
    const uint32_t db = (uint32_t)((bits + passes - 1) / passes);  // bits per pass
    const uint32_t mask = (1u << db) - 1u, digits = mask + 1u;
    const uint32_t tiles = (n - 1) / kRadixTile + 1;
    StreamBuf ka(s), kb(s), ib(s), cnt(s);
    GS_TRY(cnt.alloc(((size_t)digits * tiles + digits) * 4));
    if (passes > 1) {
        GS_TRY(ka.alloc((size_t)n * 4));
        GS_TRY(ib.alloc((size_t)n * 4));
    }
    if (passes > 2) GS_TRY(kb.alloc((size_t)n * 4));
    uint32_t *c = cnt.as<uint32_t>(), *tot = c + (size_t)digits * tiles;
    uint32_t *kbuf[2] = {ka.as<uint32_t>(), kb.as<uint32_t>()};
    const uint32_t *kin = key, *iin = nullptr;
    for (int p = 0; p < passes; p++) {
        const bool first = p == 0, last = p == passes - 1;
        const uint32_t shift = db * (uint32_t)p;
        uint32_t *kout = last ? key_out : kbuf[p & 1];
        // the last pass writes idx_out
        uint32_t *iout = ((passes - 1 - p) & 1) ? ib.as<uint32_t>() : idx_out;
        auto count = first ? k_radix_count<true> : k_radix_count<false>;
        auto scatter = first ? k_radix_scatter<true> : k_radix_scatter<false>;
        count<<<tiles, kRadixThreads, 0, s>>>(kin, n, flip, shift, mask, tiles, c);
        k_radix_scan<<<digits, kRadixThreads, 0, s>>>(c, tiles, tot);
        scatter<<<tiles, kRadixThreads, 0, s>>>(kin, iin, n, flip, shift, mask, tiles, c, tot,
                                                kout, iout);
        GS_CHECK_LAUNCH();
        kin = kout;
        iin = iout;
    }
    return GS_OK;
}

gs_status stable_sort_desc(const uint32_t *key, uint32_t n, uint32_t max_key, uint32_t *idx_out,
                           cudaStream_t s)
{
    return stable_sort(key, n, max_key, max_key, idx_out, nullptr, s);
}

gs_status stable_sort_asc(const uint32_t *key, uint32_t n, uint32_t max_key, uint32_t *idx_out,
                          uint32_t *key_out, cudaStream_t s)
{
    return stable_sort(key, n, max_key, 0, idx_out, key_out, s);
}

// ------------------------------------------------------------------ row lengths
__global__ void k_row_lengths(uint32_t n, const uint32_t *row, uint32_t nnz, uint32_t *len,
                              uint32_t *out)
{
    uint32_t top = 0, bad = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t b = row[i], e = row[i + 1];
        bad |= (b > e || (i == 0 && b != 0) || (i == n - 1u && e != nnz)) ? 1u : 0u;
        if (len) len[i] = e - b;
        top = max(top, e - b);
    }
    top = __reduce_max_sync(0xffffffffu, top);
    bad = __reduce_or_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0) {
        if (bad) atomicOr(out, bad);
        if (top) atomicMax(out + 1, top);
    }
}

gs_status row_lengths(uint32_t n, const uint32_t *row, uint32_t nnz, uint32_t *len, uint32_t *out,
                      cudaStream_t s)
{
    if (!n) return GS_OK;
    const uint32_t blocks = (n - 1) / 256 + 1;
    k_row_lengths<<<blocks < 148u * 8u ? blocks : 148u * 8u, 256, 0, s>>>(n, row, nnz, len, out);
    GS_CHECK_LAUNCH();
    return GS_OK;
}

}  // namespace gs
