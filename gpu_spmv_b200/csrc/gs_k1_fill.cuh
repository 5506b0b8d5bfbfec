// gs_k1_fill.cuh -- CSR order -> K1 slot order: values and columns of a matrix being converted,
// new values of a prepared one, the element indices of its transpose.
//
// K1 interleaves 32 rows (slot = chunk start + 32 step + lane), CSR keeps a row together, so this
// is a transpose of 32 x steps tiles.  A warp takes one work unit (a kK1Split-step piece of a
// chunk), 16 steps at a time: groups of 16, 8, .. lanes read the rows' next elements (whole
// sectors, several rows per instruction), a tile of 16 x 32 goes through shared memory, and every
// slot of the piece is written in order, the padding of short rows with it, so that nothing is
// cleared beforehand.  Bound by HBM.  One lane per row, reading its own row element by element,
// asked for 32 lines an instruction: 16.8M FP64 elements with columns 219 us and 41 us of
// clearing, 96 us here; 16.8M new FP32 values through a map of the slots 72 us, 33 us here (64 with
// loads into registers, whose 96 a thread left too few warps).
#pragma once

#include "gs_internal.cuh"

namespace gs {
namespace k1fill {

constexpr int kWarps = 4;
constexpr int kSteps = 16;

struct Args {
    uint32_t n, units;                       // rows of the layout, work units
    const uint32_t *unit_chunk, *unit_base;  // plan
    const uint32_t *nmc, *chp;               // layout
    const uint32_t *start, *len;             // sorted row g: elements start[g] .. + len[g] - 1
    const void *val;                         // elements in row order
    const uint32_t *col;
    void *oval;
    uint32_t *ocol;
    bool blocked;                            // k1_slot's lane-blocked order (reduced types)
};

template <class VIN, class VOUT> struct Convert {
    __device__ __forceinline__ static VOUT run(VIN v) { return (VOUT)v; }
};
template <class VIN> struct Convert<VIN, __nv_bfloat16> {
    __device__ __forceinline__ static __nv_bfloat16 run(VIN v)
    {
        if constexpr (sizeof(VIN) == 8) return __double2bfloat16(v);
        else return __float2bfloat16_rn(v);
    }
};
template <> struct Convert<double, float> {
    __device__ __forceinline__ static float run(double v) { return __double2float_rn(v); }
};

template <int B> __device__ __forceinline__ void copy_async(uint32_t d, const void *g)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(g), "n"(B) : "memory");
}

// A tile's rows into shared memory, 1 << LG lanes per row: element b + e (e < left, e < ns) of the
// row that lane q holds -> t[33 e + q].  Asynchronous copies, one element each: a tile's loads are
// all in flight and hold no registers.
template <int LG, class VIN, bool COLS>
__device__ __forceinline__ void load_tile(const VIN *__restrict__ val,
                                          const uint32_t *__restrict__ col, uint32_t b,
                                          uint32_t left, uint32_t lane, VIN *tv, uint32_t *tc)
{
    const uint32_t e = lane & ((1u << LG) - 1u), q0 = lane >> LG;
    const uint32_t dv = (uint32_t)__cvta_generic_to_shared(tv + e * 33u + q0);
    const uint32_t dc = (uint32_t)__cvta_generic_to_shared(tc + (COLS ? e * 33u + q0 : 0u));
#pragma unroll
    for (int i = 0; i < (1 << LG); i++) {
        const int q = i * (32 >> LG) + (int)q0;
        const uint32_t p = __shfl_sync(0xffffffffu, b, q) + e;
        if (e < __shfl_sync(0xffffffffu, left, q)) {
            copy_async<sizeof(VIN)>(dv + (uint32_t)(i * (32 >> LG) * (int)sizeof(VIN)), val + p);
            if constexpr (COLS) copy_async<4>(dc + (uint32_t)(i * (32 >> LG) * 4), col + p);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// pad: the value of a padding slot
template <class VIN, class VOUT, bool COLS, bool BLOCKED>
__global__ void __launch_bounds__(kWarps * 32, COLS ? 7 : 9) k_k1_fill(const Args a, const VOUT pad)
{
    __shared__ VIN tval[kWarps][kSteps * 33];
    __shared__ uint32_t tcol[kWarps][COLS ? kSteps * 33 : 1];
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const uint32_t u = blockIdx.x * kWarps + wid;
    if (u >= a.units) return;
    const VIN *__restrict__ val = static_cast<const VIN *>(a.val);
    VIN *tv = tval[wid];
    uint32_t *tc = tcol[wid];
    // an uncut chunk c behind the cut ones is unit c + units - chunks: tried first, so that the
    // chunk's loads do not wait for the plan's
    const uint32_t extra = a.units - (a.n + 31u) / 32u;
    uint32_t c = u >= extra ? u - extra : 0u;
    uint32_t ub, m, cb, b, len;
    auto chunk = [&] {
        const uint32_t g = 32u * c + lane;
        ub = __ldg(a.unit_base + c), m = __ldg(a.nmc + c), cb = __ldg(a.chp + c);
        b = g < a.n ? __ldg(a.start + g) : 0u, len = g < a.n ? __ldg(a.len + g) : 0u;
    };
    chunk();
    if (ub != u) {  // the same for the whole warp
        c = __ldg(a.unit_chunk + u);
        chunk();
    }
    const uint32_t j0 = (u - ub) * kK1Split;
    const uint32_t jend = min(m, j0 + kK1Split);
    for (uint32_t s = j0; s < jend; s += kSteps) {
        const uint32_t ns = min((uint32_t)kSteps, jend - s);       // steps of this tile
        const uint32_t left = len > s ? min(len - s, ns) : 0u;     // of this lane's row
        if (ns > 8) load_tile<4, VIN, COLS>(val, a.col, b + s, left, lane, tv, tc);
        else if (ns > 4) load_tile<3, VIN, COLS>(val, a.col, b + s, left, lane, tv, tc);
        else if (ns > 2) load_tile<2, VIN, COLS>(val, a.col, b + s, left, lane, tv, tc);
        else if (ns > 1) load_tile<1, VIN, COLS>(val, a.col, b + s, left, lane, tv, tc);
        else load_tile<0, VIN, COLS>(val, a.col, b + s, left, lane, tv, tc);
        __syncwarp();
        VOUT *ov = static_cast<VOUT *>(a.oval) + cb + 32u * s + lane;
        uint32_t *oc = a.ocol + (COLS ? cb + 32u * s + lane : 0u);
        auto put = [&](uint32_t i, uint32_t st, uint32_t q, bool in) {
            __stcs(ov + 32u * i, in ? Convert<VIN, VOUT>::run(tv[st * 33u + q]) : pad);
            if constexpr (COLS) __stcs(oc + 32u * i, in ? tc[st * 33u + q] : 0u);
        };
        uint32_t i = 0;
        if constexpr (BLOCKED) {
            // whole groups of 8 steps: each lane's 8 steps together, 4 lanes to a 32-slot line
            for (; i < kSteps && s + i + 8u <= (m & ~7u); i += 8) {
#pragma unroll
                for (uint32_t k = 0; k < 8; k++) {
                    const uint32_t o = k * 32u + lane, q = o >> 3, st = i + (o & 7u);
                    put(i + k, st, q, st < __shfl_sync(0xffffffffu, left, (int)q));
                }
            }
        }
        if (ns == (uint32_t)kSteps && i == 0) {
#pragma unroll
            for (uint32_t k = 0; k < (uint32_t)kSteps; k++) put(k, k, lane, k < left);
        } else {
            for (; i < ns; i++) put(i, i, lane, i < left);
        }
        __syncwarp();
    }
}

template <class VIN, class VOUT, bool COLS>
gs_status fill(const Args &a, VOUT pad, cudaStream_t s)
{
    if (!a.units) return GS_OK;
    const uint32_t blocks = (a.units + kWarps - 1) / kWarps;
    if constexpr (COLS && sizeof(VOUT) < 8) {
        if (a.blocked) {
            k_k1_fill<VIN, VOUT, COLS, true><<<blocks, kWarps * 32, 0, s>>>(a, pad);
            GS_CHECK_LAUNCH();
            return GS_OK;
        }
    }
    k_k1_fill<VIN, VOUT, COLS, false><<<blocks, kWarps * 32, 0, s>>>(a, pad);
    GS_CHECK_LAUNCH();
    return GS_OK;
}

}  // namespace k1fill
}  // namespace gs
