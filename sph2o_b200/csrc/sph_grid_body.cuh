/*
 * Per-particle bodies of the neighbour search (sph_grid.cu): the counting
 * sort's count, scan, scatter and rank + gather steps, kept apart from their kernels (one thread or
 * warp per index) so that other kernels can run the same steps on their own
 * index ranges, and the GatherSet the sort moves state with.
 */
#ifndef SPH2O_GRID_BODY_CUH
#define SPH2O_GRID_BODY_CUH

#include "sph_device.cuh"

namespace sph {

/* Arrays moved by the rank/gather step of the sort (NULL entries skipped).
   n_dev (may be NULL): device count of the particles to sort, read by the
   kernels in place of n (the fluid's active count when emitters add to it). */
struct GatherSet {
    const unsigned* n_dev;
    unsigned* orig_out;
    unsigned* cell_out;
    const float4* v4_in[4];
    float4* v4_out[4];
    const float* f_in[2];
    float* f_out[2];
};

/* Particle i (where `on`) in cell c: its cell, its arrival slot there, and the
   population of c's chunk of 4096 cells, added once per warp where its lanes
   share a chunk (neighbouring particles nearly always do). The whole warp
   calls. */
__device__ __forceinline__ void ns_count_at(bool on, unsigned c, int i, unsigned* __restrict__ cell_count,
                                            unsigned* __restrict__ chunk_sums, unsigned* __restrict__ cell_of,
                                            unsigned* __restrict__ slot)
{
    if (on) {
        cell_of[i] = c;
        slot[i] = atomicAdd(&cell_count[c], 1u);
    }
    const unsigned active = __ballot_sync(0xffffffffu, on);
    if (active == 0u) return;
    const int first = __ffs((int)active) - 1;
    const unsigned chunk = c >> 12, chunk0 = __shfl_sync(0xffffffffu, chunk, first);
    const unsigned same = __ballot_sync(0xffffffffu, on && chunk == chunk0);
    if ((int)(threadIdx.x & 31u) == first) atomicAdd(&chunk_sums[chunk0], (unsigned)__popc(same));
    else if (on && chunk != chunk0) atomicAdd(&chunk_sums[chunk], 1u);
}

/* Exclusive scan of chunk b's 4096 populations by 256 threads (16 per thread,
   four 16-byte loads in flight), offset by the totals of the chunks before it;
   the last chunk writes the grand total. ZERO: the populations are zeroed
   (count and start may be one array without it). */
template <bool ZERO>
__device__ __forceinline__ void scan_chunk_at(int b, unsigned* count, unsigned* start, const unsigned* chunk_sums,
                                              int nchunks, unsigned* total_out)
{
    __shared__ unsigned warp_tot[8], warp_off[8];
    const size_t base = (size_t)b * 4096 + (size_t)threadIdx.x * 16;
    uint4 c[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) c[k] = *reinterpret_cast<const uint4*>(count + base + 4 * k);
    unsigned before = 0;
    for (int k = (int)threadIdx.x; k < b; k += 256) before += chunk_sums[k];
    if (ZERO) {
#pragma unroll
        for (int k = 0; k < 4; ++k) *reinterpret_cast<uint4*>(count + base + 4 * k) = make_uint4(0, 0, 0, 0);
    }
    unsigned t = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) t += (c[k].x + c[k].y) + (c[k].z + c[k].w);
    unsigned incl = t;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    if (lane == 31) {
        warp_tot[wid] = incl;
        warp_off[wid] = before;
    }
    __syncthreads();
    unsigned run = incl - t;
#pragma unroll
    for (int w = 0; w < 8; ++w) run += warp_off[w] + (w < wid ? warp_tot[w] : 0u);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        uint4 o;
        o.x = run; run += c[k].x;
        o.y = run; run += c[k].y;
        o.z = run; run += c[k].z;
        o.w = run; run += c[k].w;
        *reinterpret_cast<uint4*>(start + base + 4 * k) = o;
    }
    if (b == nchunks - 1 && threadIdx.x == 255) *total_out = run;
}

/* (orig id, source index) of particle i into its cell segment */
__device__ __forceinline__ void ns_scatter_at(int i, const unsigned* __restrict__ cell_of,
                                              const unsigned* __restrict__ slot, const unsigned* __restrict__ cell_start,
                                              const unsigned* __restrict__ orig, unsigned* __restrict__ tmp_key,
                                              unsigned* __restrict__ tmp_src)
{
    const unsigned p = cell_start[cell_of[i]] + slot[i];
    tmp_key[p] = orig[i];
    tmp_src[p] = (unsigned)i;
}

/* Rank of segment entry p inside its cell by caller-order id (the
   reference's insertion order), then the carried state moved there. */
__device__ __forceinline__ void ns_rank_gather_at(int p, const unsigned* __restrict__ cell_of,
                                                  const unsigned* __restrict__ cell_start,
                                                  const unsigned* __restrict__ tmp_key,
                                                  const unsigned* __restrict__ tmp_src, const GatherSet& g)
{
    const unsigned src = tmp_src[p];
    /* the carried position and velocity are loaded before the cell lookup
       and the rank loop, so their latency overlaps that chain */
    const float4 v0 = g.v4_in[0] ? g.v4_in[0][src] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float4 v1 = g.v4_in[1] ? g.v4_in[1][src] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const unsigned c = cell_of[src];
    const unsigned key = tmp_key[p];
    const unsigned s = cell_start[c], e = cell_start[c + 1];
    unsigned rank = 0;
    for (unsigned q = s; q < e; ++q) rank += tmp_key[q] < key ? 1u : 0u;
    const unsigned dst = s + rank;
    g.orig_out[dst] = key;
    if (g.cell_out) g.cell_out[dst] = c;
    if (g.v4_in[0]) g.v4_out[0][dst] = v0;
    if (g.v4_in[1]) g.v4_out[1][dst] = v1;
    if (g.v4_in[2]) g.v4_out[2][dst] = g.v4_in[2][src];
    if (g.v4_in[3]) g.v4_out[3][dst] = g.v4_in[3][src];
    if (g.f_in[0]) g.f_out[0][dst] = g.f_in[0][src];
    if (g.f_in[1]) g.f_out[1][dst] = g.f_in[1][src];
}

/* Whether x's cell has boundary particles among its 27 cells (near: see
   k_mark_near). */
__device__ __forceinline__ bool boundary_near(const SimParams& P, const unsigned char* __restrict__ near, float4 x,
                                              const Grid& g)
{
    return P.nb > 0 && near[cell_index(x, P.h, g)] != 0;
}

} // namespace sph

#endif
