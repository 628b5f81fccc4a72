// BC backward pass shared by the single-query kernel and the batched one.
//
// Dependency accumulation of Brandes' algorithm over the forward level stack,
// deepest level first, one barrier per phase (StageTwoDD{,CTA}Fused,
// samples/hybrid_bc/hybrid_bc.cu:134-225; host form hybrid_bc_host.cpp:66-80):
//   delta[v] = sum over out-edges v->w with level[w] == level[v]+1 of
//              sigma[v]/sigma[w] * (1 + delta[w])
// With q(w) = (1 + delta[w]) / sigma[w], fixed once per vertex when its level is
// finished, that is delta[v] = sigma[v] * sum of q(w): an edge costs one 8-byte
// gather of w's (level, q) record instead of its level, then its path count and
// dependency, and a double division.
// Each vertex is owned by one thread (small out-degree) or one warp; vertices
// above kBcBigDegree out-edges are split into chunks whose partial sums are
// added atomically and finished after a barrier.  The source (depth 0) keeps
// delta 0, and the result is delta * 0.5 (hybrid_bc.cu:374-376).  Bound by the
// record gathers (one L1 lookup per edge).  Symmetric
// RMAT-22, forward and backward: 3.81 -> 3.50 ms.
#pragma once
#include <cstdint>

#include "sg_device.cuh"

namespace sepgraph {
namespace bc {

constexpr uint32_t kBcBigDegree = 256;
constexpr uint32_t kBcChunk = 256;

struct BCBackArgs {
    const uint32_t *row, *col;
    const uint32_t *level;
    const unsigned long long *sigma;
    float *delta;  // zero on entry
    uint2 *rec;    // (level, bits of q) of every vertex, scratch
    float *bc_out;  // delta * 0.5
    const uint32_t *stack, *ends;
    uint32_t nlevels, max_depth, nv;
    uint4 *chunks;  // (v, begin, len, 1 for a vertex's first), the levels one after the other
    uint32_t chunk_cap;
    uint32_t *chunk_count;  // chunks of each level [max_depth + 1], zero on entry
    uint32_t *bar;          // count, gen (single-query kernel)
    uint32_t *err;
    unsigned long long timeout_ns;
};

__device__ __forceinline__ float bc_q(unsigned long long sigma, float delta) {
    return (float)((1.0 + (double)delta) / (double)sigma);
}

// Sum of q over the out-edges [k, end) taken `step` apart that lead to `depth`,
// four records in flight.
__device__ __forceinline__ float bc_sum(const BCBackArgs &a, uint32_t k, uint32_t end, uint32_t step, uint32_t depth) {
    float s = 0.f;
    for (; k < end; k += 4 * step) {
        uint2 r[4];
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
            const uint32_t e = k + j * step;
            r[j] = make_uint2(0xffffffffu, 0u);
            if (e < end) r[j] = __ldcg(a.rec + __ldg(a.col + e));
        }
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) s += r[j].x == depth ? __uint_as_float(r[j].y) : 0.f;
    }
    return s;
}

// Dependency of v (sigma paths) from its sum, and its record for the level above.
__device__ __forceinline__ void bc_finish(const BCBackArgs &a, uint32_t v, unsigned long long sigma, float sum,
                                          uint32_t depth) {
    const float d = (float)((double)sigma * (double)sum);
    a.delta[v] = d;
    a.rec[v] = make_uint2(depth, __float_as_uint(bc_q(sigma, d)));
}

// The whole backward pass for one query, run by `nt` threads numbered from
// `gt` (warps gw of nw); `sync()` is a barrier over exactly those threads and
// returns false when a bounded wait gave up.
template <typename Sync>
__device__ bool backward(const BCBackArgs &a, uint32_t gt, uint32_t nt, Sync &&sync) {
    const uint32_t lane = dev::lane_id();
    const uint32_t gw = gt >> 5, nw = nt >> 5;
    uint32_t chunk0 = 0;  // first chunk of the level at hand
    // chunks of the split vertices of depth d, after `base` earlier ones; from
    // the last thread down, so that on a level smaller than the team other warps
    // sum meanwhile
    auto list_chunks = [&](uint32_t d, uint32_t base) {
        const uint32_t b = __ldcg(a.ends + d - 1), e = __ldcg(a.ends + d);
        for (uint32_t i = b + (nt - 1 - gt); i < e; i += nt) {
            const uint32_t v = __ldcg(a.stack + i);
            const uint32_t beg = __ldg(a.row + v), deg = __ldg(a.row + v + 1) - beg;
            if (deg <= kBcBigDegree) continue;
            const uint32_t nch = (deg + kBcChunk - 1) / kBcChunk;
            const uint32_t c0 = base + atomicAdd(a.chunk_count + d, nch);
            for (uint32_t c = 0; c < nch; ++c) {
                if (c0 + c < a.chunk_cap)
                    a.chunks[c0 + c] = make_uint4(v, beg + c * kBcChunk, min(kBcChunk, deg - c * kBcChunk), c == 0);
                else
                    atomicOr(a.err, dev::kErrChunkCapacity);
            }
        }
    };
    if (a.max_depth >= 1) {
        // vertices below max_depth have no successors: delta 0, q = 1 / sigma
        for (uint32_t v = gt; v < a.nv; v += nt) {
            const uint32_t lv = __ldcg(a.level + v);
            a.rec[v] = make_uint2(lv, lv != 0xffffffffu && lv > a.max_depth ? __float_as_uint(bc_q(__ldcg(a.sigma + v), 0.f)) : 0u);
        }
        list_chunks(a.max_depth, 0);
        if (!sync()) return false;
    }
    for (uint32_t d = a.max_depth; d >= 1; --d) {
        const uint32_t b = __ldcg(a.ends + d - 1), e = __ldcg(a.ends + d);
        const uint32_t end = min(chunk0 + __ldcg(a.chunk_count + d), a.chunk_cap);
        for (uint32_t c = chunk0 + gw; c < end; c += nw) {
            const uint4 ch = __ldcg(a.chunks + c);
            const float s = dev::warp_sum(bc_sum(a, ch.y + lane, ch.y + ch.z, 32, d + 1));
            if (lane == 0) atomicAdd(a.delta + ch.x, s);
        }
        for (uint32_t base = b + gw * 32; base < e; base += nw * 32) {
            const uint32_t i = base + lane;
            const bool valid = i < e;
            uint32_t v = 0, beg = 0, deg = 0;
            unsigned long long sigma = 0;  // in flight with the row: a trip less at the end of the chain
            if (valid) {
                v = __ldcg(a.stack + i);
                beg = __ldg(a.row + v);
                deg = __ldg(a.row + v + 1) - beg;
                sigma = __ldcg(a.sigma + v);
            }
            const bool mid = valid && deg <= kBcBigDegree && deg > 32;
            if (valid && deg <= 32) bc_finish(a, v, sigma, bc_sum(a, beg, beg + deg, 1, d + 1), d);
            uint32_t m = __ballot_sync(dev::kFullMask, mid);
            while (m) {
                const uint32_t j = __ffs(m) - 1;
                m &= m - 1;
                const uint32_t vj = __shfl_sync(dev::kFullMask, v, j);
                const uint32_t bj = __shfl_sync(dev::kFullMask, beg, j);
                const uint32_t dj = __shfl_sync(dev::kFullMask, deg, j);
                const unsigned long long sj = __shfl_sync(dev::kFullMask, sigma, j);
                const float s = dev::warp_sum(bc_sum(a, bj + lane, bj + dj, 32, d + 1));
                if (lane == 0) bc_finish(a, vj, sj, s, d);
            }
        }
        if (d > 1) list_chunks(d - 1, end);
        if (!sync()) return false;
        if (end > chunk0) {  // the same in every thread
            for (uint32_t c = chunk0 + gt; c < end; c += nt) {
                const uint4 ch = __ldcg(a.chunks + c);
                if (ch.w) bc_finish(a, ch.x, __ldcg(a.sigma + ch.x), __ldcg(a.delta + ch.x), d);
            }
            if (!sync()) return false;
            chunk0 = end;
        }
    }
    for (uint32_t v = gt; v < a.nv; v += nt) a.bc_out[v] = __ldcg(a.delta + v) * 0.5f;
    return true;
}

}  // namespace bc
}  // namespace sepgraph
