/*
 * Neighbour search on the GPU: the B200 replacement of SPH2O's spatial hash
 * (HashTable::insertFluidParticle / neighborhoodSearch, src/SPH2O/HashTable.cpp:3-86;
 * SPHSolver::insertFluidParticles / neighborhoodSearch, src/SPH2O/SPHSolver/SPHSolver.cpp:170-219).
 *
 * Per step:
 *   1. ns_count        cell key floor(x / h) -> cell index in brick order,
 *                      per-cell population by atomicAdd (slot = old count),
 *                      totals of chunks of 4096 cells
 *   2. scan            exclusive scan of the populations -> cellStart[ncells+1]
 *                      (the scan zeroes the populations for the next step)
 *   3. ns_scatter      (orig id, source index) into its cell segment
 *   4. ns_rank_gather  rank inside the cell by orig id (deterministic, equal
 *                      to the reference's insertion order: ascending index),
 *                      then gather the carried state into sorted order
 *   5. search          for each particle, the 27 cells in the reference's
 *                      offset order (x outermost, HashTable.cpp:59-65), keep
 *                      candidates with |xi - xj| <= h (exact IEEE test), in
 *                      neighbour lists by tiles of 32 particles; densities and
 *                      pressures of smaller scenes from the same candidates
 *                      (optionally one block per cell brick with the brick's
 *                      halo staged in shared memory: same lists)
 * The static boundary is sorted once at init with steps 1-4 into its own
 * cellStart table, and AkinciBoundaryObject::computeVolume
 * (src/SPH2O/BoundaryObject/AkinciBoundaryObject.cpp:10-34) runs on it.
 */
#include "sph_device.cuh"
#include "sph_grid_body.cuh"
#include "sph_internal.h"

namespace sph {

__global__ void __launch_bounds__(256) k_ns_count(SimParams P, SceneRef S, int n, const unsigned* n_dev,
                                                  const float4* __restrict__ pos, unsigned* __restrict__ cell_count,
                                                  unsigned* __restrict__ chunk_sums, unsigned* __restrict__ cell_of,
                                                  unsigned* __restrict__ slot)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool on = i < (n_dev ? (int)*n_dev : n);
    ns_count_at(on, on ? cell_index(pos[i], P.h, grid_for(P, S, (unsigned)i)) : 0u, i, cell_count, chunk_sums, cell_of,
                slot);
}

/* Exclusive scan of the populations in one launch: each 256-thread block scans
   4096 of them (scan_chunk_at) on top of the totals of the chunks before it,
   which the count step has summed, and zeroes the populations for the next
   search. A second launch that added the chunk offsets cost ~3 us per search. */
__global__ void __launch_bounds__(256) k_scan(unsigned* __restrict__ count, unsigned* __restrict__ start,
                                              const unsigned* __restrict__ chunk_sums, int nchunks,
                                              unsigned* __restrict__ total_out)
{
    scan_chunk_at<true>((int)blockIdx.x, count, start, chunk_sums, nchunks, total_out);
}

__global__ void __launch_bounds__(256) k_ns_scatter(int n, const unsigned* n_dev, const unsigned* __restrict__ cell_of,
                                                    const unsigned* __restrict__ slot,
                                                    const unsigned* __restrict__ cell_start,
                                                    const unsigned* __restrict__ orig,
                                                    unsigned* __restrict__ tmp_key, unsigned* __restrict__ tmp_src,
                                                    unsigned* __restrict__ chunk_sums, int nchunks)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    /* the scan is done with the chunk totals: zero for the next search */
    for (int k = i; k < nchunks; k += (int)(gridDim.x * blockDim.x)) chunk_sums[k] = 0u;
    if (i >= (n_dev ? (int)*n_dev : n)) return;
    ns_scatter_at(i, cell_of, slot, cell_start, orig, tmp_key, tmp_src);
}

/* Rank inside the cell by caller-order id, then move the carried state. */
__global__ void __launch_bounds__(256) k_ns_rank_gather(int n, const unsigned* __restrict__ cell_of,
                                                        const unsigned* __restrict__ cell_start,
                                                        const unsigned* __restrict__ tmp_key,
                                                        const unsigned* __restrict__ tmp_src, GatherSet g)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= (g.n_dev ? (int)*g.n_dev : n)) return;
    ns_rank_gather_at(p, cell_of, cell_start, tmp_key, tmp_src, g);
}

/* The n list entries out[32 k] (one thread wrote them): their density terms
   added to rho in list order. Four are evaluated at a time, all lanes of the
   warp together; past the end W is 0 and leaves the sum as it is. */
template <bool BOUNDARY>
__device__ __forceinline__ float add_density(const SimParams& P, float4 xi, const float4* __restrict__ xs,
                                             const unsigned* out, unsigned n, float rho)
{
    for (unsigned k = 0; k < n; k += 4) {
        unsigned q[4];
        float4 x[4];
        float w[4];
#pragma unroll
        for (unsigned u = 0; u < 4; ++u) q[u] = out[min(k + u, n - 1u) * 32u];
#pragma unroll
        for (unsigned u = 0; u < 4; ++u) x[u] = xs[q[u]];
#pragma unroll
        for (unsigned u = 0; u < 4; ++u)
            w[u] = __fmul_rn(BOUNDARY ? x[u].w : P.mass,
                             cs_W_exact(k + u < n ? dist2_exact(xi, x[u]) : 4.0f * P.h2, P));
#pragma unroll
        for (unsigned u = 0; u < 4; ++u) rho = __fadd_rn(rho, w[u]);
    }
    return rho;
}

/* Arrays of a search. */
struct SearchArrays {
    const float4* __restrict__ pos;
    const unsigned* __restrict__ cell_start;
    const float4* __restrict__ bpos;
    const unsigned* __restrict__ bcell_start;
    const unsigned char* __restrict__ near;
    unsigned *nbr_f, *cnt_f, *nbr_b, *cnt_b;
    float *rho, *press;
    const float4* __restrict__ vel;
    float4* rec;
    DevState* st;
};

/* What a search computes beside the lists: nothing, or the densities, the Tait
   pressures (EOS) and the records that the force pass reads. */
template <int MODE>
__device__ __forceinline__ void store_density(const SimParams& P, const SearchArrays& A, int i, float4 xi, float rho)
{
    if (MODE == SEARCH_LISTS) return;
    A.rho[i] = rho;
    float dp = 0.0f;
    if (MODE == SEARCH_EOS) {
        const float p = tait_pressure(rho, P, P.kr_g);
        A.press[i] = p;
        dp = p / (rho * rho);
    }
    store_rec(A.rec, i, xi, rho, A.vel[i], dp);
}

__device__ __forceinline__ void store_counts(const SimParams& P, const SearchArrays& A, int i, unsigned nF, unsigned nB)
{
    A.cnt_f[i] = min(nF, P.capF);
    A.cnt_b[i] = min(nB, P.capB);
    if (nF > P.capF || nB > P.capB) {
        atomicAdd(&A.st->overflow, 1u);
        atomicOr(&A.st->err, ERRBIT_OVERFLOW);
    }
}

/* Neighbour lists of particle i in the reference's candidate order, filtered
   at |r| <= h, and its density (MODE), by one thread. */
template <int MODE, typename Off>
__device__ __forceinline__ void search_at(const SimParams& P, const SceneRef& S, int i, const SearchArrays& A)
{
    const float4 xi = A.pos[i];
    /* |r| <= h as the reference rounds it, without the square root */
    const float s2max = P.h2_exact;
    const Grid g = grid_for(P, S, (unsigned)i);
    const auto list = [&](const unsigned* starts, const float4* xs, unsigned* out, unsigned cap) {
        unsigned m = 0, n = 0; /* accepted candidates of the stretch, of all */
        for_stretches27<Off>(
            xi, xi, P.h, g, starts, xs,
            [&](unsigned k, const float (&d)[4], unsigned) {
                const unsigned t = (d[0] <= s2max ? 1u : 0u) | (d[1] <= s2max ? 2u : 0u) | (d[2] <= s2max ? 4u : 0u) |
                                   (d[3] <= s2max ? 8u : 0u);
                m |= t << k;
            },
            [&](auto slot) {
                for (; m; m &= m - 1u) {
                    if (n < cap) __stcs(out + n * 32u, slot((unsigned)__ffs((int)m) - 1u));
                    ++n;
                }
            });
        return n;
    };
    unsigned* out_f = A.nbr_f + list_index(0, P.capF, i);
    unsigned* out_b = A.nbr_b + list_index(0, P.capB, i);
    const unsigned nF = list(A.cell_start, A.pos, out_f, P.capF);
    const unsigned nB = boundary_near(P, A.near, xi, g) ? list(A.bcell_start, A.bpos, out_b, P.capB) : 0u;
    store_counts(P, A, i, nF, nB);
    if (MODE == SEARCH_LISTS) return;
    float rho = add_density<false>(P, xi, A.pos, out_f, min(nF, P.capF), 0.0f);
    rho = add_density<true>(P, xi, A.bpos, out_b, min(nB, P.capB), rho);
    store_density<MODE>(P, A, i, xi, rho);
}

template <int MODE, typename Off>
__global__ void __launch_bounds__(128) k_search(SimParams P, SceneRef S, SearchArrays A)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= active_n(P, A.st)) return;
    search_at<MODE, Off>(P, S, i, A);
}

/* The same search for small scenes, one warp per particle: lane k < 27 loads the
   range of the particle's k-th cell (the reference's offset order), a warp scan
   lays the 27 ranges end to end, and the warp then tests the concatenated
   candidates 32 at a time; a ballot ranks each round's accepted candidates, so
   entries are written in candidate order. The accepted squared distances (and
   boundary weights) are collected in shared memory in that order, the kernel
   terms evaluated by all lanes, and added one after the other. */
constexpr int kSearchWarps = 4, kWarpBatch = 96;

template <int MODE>
__global__ void __launch_bounds__(kSearchWarps * 32) k_search_warp(SimParams P, SceneRef S, SearchArrays A)
{
    constexpr bool DENSITY = MODE != SEARCH_LISTS;
    __shared__ float s_w[kSearchWarps][DENSITY ? kWarpBatch : 1], s_psi[kSearchWarps][DENSITY ? kWarpBatch : 1];
    const int i = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    /* the whole warp shares i and leaves together */
    if (i >= active_n(P, A.st)) return;
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const float4 xi = A.pos[i];
    const Grid g = grid_for(P, S, (unsigned)i);
    const bool with_boundary = boundary_near(P, A.near, xi, g);
    unsigned s = 0, e = 0, bs = 0, be = 0;
    if (lane < 27) {
        const int xx = cell_coord(xi.x, P.h, g.cminx, g.dimx) + (int)lane / 9 - 1;
        const int yy = cell_coord(xi.y, P.h, g.cminy, g.dimy) + ((int)lane / 3) % 3 - 1;
        const int zz = cell_coord(xi.z, P.h, g.cminz, g.dimz) + (int)lane % 3 - 1;
        if (xx >= 0 && xx < g.dimx && yy >= 0 && yy < g.dimy && zz >= 0 && zz < g.dimz) {
            const unsigned c = cell_at(xx, yy, zz, g);
            s = A.cell_start[c];
            e = A.cell_start[c + 1];
            if (with_boundary) {
                bs = A.bcell_start[c];
                be = A.bcell_start[c + 1];
            }
        }
    }
    float rho = 0.0f;
    unsigned pending = 0; /* collected terms not yet in rho */
    const auto add_terms = [&](bool boundary) {
        __syncwarp();
        for (unsigned k = lane; k < pending; k += 32u)
            s_w[warp][k] = __fmul_rn(boundary ? s_psi[warp][k] : P.mass, cs_W_exact(s_w[warp][k], P));
        __syncwarp();
#pragma unroll 4
        for (unsigned k = 0; k < pending; ++k) rho = __fadd_rn(rho, s_w[warp][k]);
        __syncwarp();
        pending = 0;
    };
    const auto walk = [&](const float4* xs, unsigned begin, unsigned end, unsigned* out, unsigned cap, bool boundary) {
        const unsigned cnt = end - begin;
        unsigned incl = cnt, n = 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (unsigned)o) incl += v;
        }
        const unsigned total = __shfl_sync(0xffffffffu, incl, 31);
        const unsigned excl = incl - cnt;
        for (unsigned u0 = 0; u0 < total; u0 += 32) {
            const unsigned u = min(u0 + lane, total - 1u);
            /* cell of candidate u: the number of lanes whose ranges end at or before u */
            unsigned k = 0;
#pragma unroll
            for (unsigned step = 16; step >= 1; step >>= 1)
                if (__shfl_sync(0xffffffffu, incl, k + step - 1) <= u) k += step;
            const unsigned q = __shfl_sync(0xffffffffu, begin, k) + (u - __shfl_sync(0xffffffffu, excl, k));
            const float4 x = xs[q];
            const float d = dist2_exact(xi, x);
            const bool in = u0 + lane < total && d <= P.h2_exact;
            const unsigned bits = __ballot_sync(0xffffffffu, in);
            const unsigned rank = (unsigned)__popc(bits & ((1u << lane) - 1u));
            if (in && n + rank < cap) {
                __stcs(out + (n + rank) * 32u, q);
                if (DENSITY) {
                    s_w[warp][pending + rank] = d;
                    if (boundary) s_psi[warp][pending + rank] = x.w;
                }
            }
            const unsigned more = (unsigned)__popc(bits), kept = min(more, cap - min(n, cap));
            n += more;
            if (DENSITY) {
                pending += kept;
                if (pending > kWarpBatch - 32u) add_terms(boundary);
            }
        }
        if (DENSITY) add_terms(boundary);
        return n;
    };
    const unsigned nF = walk(A.pos, s, e, A.nbr_f + list_index(0, P.capF, (unsigned)i), P.capF, false);
    const unsigned nB = with_boundary ? walk(A.bpos, bs, be, A.nbr_b + list_index(0, P.capB, (unsigned)i), P.capB, true) : 0u;
    if (lane != 0) return;
    store_counts(P, A, i, nF, nB);
    store_density<MODE>(P, A, i, xi, rho);
}

/* The one-thread search, kept out of line: what the lane groups below fall
   back to. */
template <int MODE, typename Off>
__device__ __noinline__ void search_out_of_line(const SimParams& P, const SceneRef& S, int i, const SearchArrays& A)
{
    search_at<MODE, Off>(P, S, i, A);
}

/* The same search with four lanes per particle: the rows of cells are split
   3, 2, 2, 2 over the lanes in candidate order, each lane collects its accepted
   candidates and their squared distances in shared memory, the counts of the
   lanes before it place its list entries, and the kernel terms, evaluated by
   all four lanes, are added in list order. A particle with more than kLaneBatch
   accepted candidates in one lane is left to search_out_of_line. */
constexpr int kLanes = 4, kLaneBatch = 24, kLaneBlock = 128;

template <int MODE, typename Off>
__global__ void __launch_bounds__(kLaneBlock) k_search_lanes(SimParams P, SceneRef S, SearchArrays A)
{
    static_assert(MODE != SEARCH_LISTS, "a warp or one lane builds lists alone");
    __shared__ unsigned s_q[kLaneBatch][kLaneBlock];
    __shared__ float s_w[kLaneBatch + 1][kLaneBlock]; /* one spare row */
    const int i = (int)((blockIdx.x * blockDim.x + threadIdx.x) / kLanes);
    const unsigned tid = threadIdx.x, lane = tid & 31u, sub = lane % kLanes, first = lane - sub;
    const bool on = i < active_n(P, A.st);
    const float4 xi = on ? A.pos[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const Grid g = grid_for(P, S, on ? (unsigned)i : 0u);
    const float s2max = P.h2_exact;
    const int row0 = sub == 0 ? 0 : 2 * (int)sub + 1, row1 = 2 * (int)sub + 3;
    float rho = 0.0f;
    bool over = false;
    /* list (and density terms) of one particle set; its length */
    const auto set = [&](bool walk, const unsigned* starts, const float4* xs, unsigned* out, unsigned cap, bool boundary) {
        unsigned m = 0, nq = 0, nw = 0;
        if (walk)
            for_stretches27<Off>(
                xi, xi, P.h, g, starts, xs,
                [&](unsigned k, const float (&d)[4], unsigned) {
                    unsigned bits = 0;
#pragma unroll
                    for (unsigned u = 0; u < 4; ++u) {
                        const bool in = d[u] <= s2max;
                        bits |= in ? 1u << u : 0u;
                        s_w[min(nw, (unsigned)kLaneBatch)][tid] = d[u]; /* written over unless kept */
                        nw += in ? 1u : 0u;
                    }
                    m |= bits << k;
                },
                [&](auto slot) {
                    for (; m; m &= m - 1u, ++nq) s_q[min(nq, kLaneBatch - 1u)][tid] = slot((unsigned)__ffs((int)m) - 1u);
                },
                row0, row1);
        over |= ((__ballot_sync(0xffffffffu, nq > kLaneBatch) >> first) & ((1u << kLanes) - 1u)) != 0u;
        const unsigned own = min(nq, (unsigned)kLaneBatch);
        unsigned before = 0, total = 0;
#pragma unroll
        for (unsigned l = 0; l < kLanes; ++l) {
            const unsigned c = __shfl_sync(0xffffffffu, nq, first + l);
            before += l < sub ? c : 0u;
            total += c;
        }
        for (unsigned k = 0; k < own; ++k) {
            const unsigned q = s_q[k][tid];
            if (!over && before + k < cap) __stcs(out + (before + k) * 32u, q);
            s_w[k][tid] = __fmul_rn(boundary ? xs[q].w : P.mass, cs_W_exact(s_w[k][tid], P));
        }
        __syncwarp();
        unsigned left = cap;
        for (unsigned l = 0; l < kLanes; ++l) {
            const unsigned c = min(__shfl_sync(0xffffffffu, own, first + l), left);
            left -= c;
            for (unsigned k = 0; k < c; ++k) rho = __fadd_rn(rho, s_w[k][tid - sub + l]);
        }
        __syncwarp();
        return total;
    };
    const unsigned nF = set(on, A.cell_start, A.pos, A.nbr_f + list_index(0, P.capF, (unsigned)i), P.capF, false);
    const bool near = on && boundary_near(P, A.near, xi, g);
    unsigned nB = 0;
    if (__any_sync(0xffffffffu, near))
        nB = set(near, A.bcell_start, A.bpos, A.nbr_b + list_index(0, P.capB, (unsigned)i), P.capB, true);
    __syncwarp(); /* the other lanes' list entries come before the fallback's */
    if (!on || sub != 0) return;
    if (over) {
        search_out_of_line<MODE, Off>(P, S, i, A);
        return;
    }
    store_counts(P, A, i, nF, nB);
    store_density<MODE>(P, A, i, xi, rho);
}

/* ---------------------------------------------------------------------- */
/* List build with each brick's halo staged in shared memory.               */

/* the global-memory walk of one particle of a single scene, kept out of line */
__device__ __noinline__ void build_lists_global(const SimParams& P, int i, const float4* __restrict__ pos,
                                                const unsigned* __restrict__ cell_start,
                                                const float4* __restrict__ bpos,
                                                const unsigned* __restrict__ bcell_start,
                                                const unsigned char* __restrict__ near,
                                                unsigned* __restrict__ nbr_f, unsigned* __restrict__ cnt_f,
                                                unsigned* __restrict__ nbr_b, unsigned* __restrict__ cnt_b,
                                                DevState* st)
{
    search_at<SEARCH_LISTS, unsigned long long>(P, SceneRef{}, i, SearchArrays{pos, cell_start, bpos, bcell_start, near, nbr_f, cnt_f, nbr_b,
                                                           cnt_b, nullptr, nullptr, nullptr, nullptr, st});
}

/* Fluid particles of one brick's 6 x 6 x 6-cell halo that fit in shared
   memory (45 KB of float4); a brick with more takes the cells from global
   memory instead. */
constexpr unsigned kHaloCap = 2816;
constexpr int kStagedBlock = 256;

/* One block per 4 x 4 x 4-cell brick (single scenes in brick order). The
   block lists the 216 cells around the brick with their fluid and boundary
   ranges, lays the fluid cells' positions end to end in shared memory (one
   warp per cell, coalesced), then every thread walks its particles' 27 cells
   in the reference's offset order over the staged copies: the same
   candidates in the same order, the same exact test, the same global slot
   ids written, so the lists equal k_search's entry for entry. */
__global__ void __launch_bounds__(kStagedBlock) k_ns_build_lists_staged(
    SimParams P, const float4* __restrict__ pos, const unsigned* __restrict__ cell_start,
    const float4* __restrict__ bpos, const unsigned* __restrict__ bcell_start, const unsigned char* __restrict__ near,
    unsigned* __restrict__ nbr_f, unsigned* __restrict__ cnt_f, unsigned* __restrict__ nbr_b, unsigned* __restrict__ cnt_b, DevState* st)
{
    __shared__ float4 s_pos[kHaloCap];
    __shared__ unsigned s_off[217]; /* staged offset of each halo cell; [216] = total */
    __shared__ unsigned s_gs[216];  /* global slot of each halo cell's first fluid particle */
    __shared__ unsigned s_bs[216], s_be[216];
    const Grid g = grid_single(P);
    const unsigned b = blockIdx.x;
    const unsigned c0 = b << 6;
    const unsigned ps = cell_start[c0], pe = cell_start[c0 + 64];
    if (ps == pe) return; /* the whole block leaves */
    const int bx = (int)(b % (unsigned)g.nbx), by = (int)((b / (unsigned)g.nbx) % (unsigned)g.nby);
    const int bz = (int)(b / ((unsigned)g.nbx * (unsigned)g.nby));
    const int lane = (int)(threadIdx.x & 31u), warp = (int)(threadIdx.x >> 5);
    for (int h = (int)threadIdx.x; h < 216; h += kStagedBlock) {
        const int cx = 4 * bx - 1 + h % 6, cy = 4 * by - 1 + (h / 6) % 6, cz = 4 * bz - 1 + h / 36;
        unsigned s = 0, e = 0, bs = 0, be = 0;
        if (cx >= 0 && cx < g.dimx && cy >= 0 && cy < g.dimy && cz >= 0 && cz < g.dimz) {
            const unsigned c = cell_at(cx, cy, cz, g);
            s = cell_start[c];
            e = cell_start[c + 1];
            if (P.nb > 0) {
                bs = bcell_start[c];
                be = bcell_start[c + 1];
            }
        }
        s_gs[h] = s;
        s_off[h] = e - s; /* the population until the scan below */
        s_bs[h] = bs;
        s_be[h] = be;
    }
    __syncthreads();
    if (warp == 0) {
        /* exclusive scan of the 216 populations: 7 consecutive cells per lane */
        unsigned v[7], t = 0;
#pragma unroll
        for (int k = 0; k < 7; ++k) {
            const int h = 7 * lane + k;
            v[k] = h < 216 ? s_off[h] : 0u;
            t += v[k];
        }
        unsigned incl = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        unsigned run = incl - t;
#pragma unroll
        for (int k = 0; k < 7; ++k) {
            const int h = 7 * lane + k;
            if (h <= 216) s_off[h] = run;
            run += v[k];
        }
    }
    __syncthreads();
    const bool staged = s_off[216] <= kHaloCap;
    if (staged)
        for (int h = warp; h < 216; h += kStagedBlock / 32) {
            const unsigned s = s_gs[h], o = s_off[h], n = s_off[h + 1] - o;
            for (unsigned k = (unsigned)lane; k < n; k += 32u) s_pos[o + k] = pos[s + k];
        }
    __syncthreads();
    const float s2max = P.h2_exact;
    for (unsigned i = ps + threadIdx.x; i < pe; i += kStagedBlock) {
        const float4 xi = pos[i];
        /* the particle's cell inside the brick (its sort cell) */
        const int lx = cell_coord(xi.x, P.h, g.cminx, g.dimx) - 4 * bx;
        const int ly = cell_coord(xi.y, P.h, g.cminy, g.dimy) - 4 * by;
        const int lz = cell_coord(xi.z, P.h, g.cminz, g.dimz) - 4 * bz;
        if ((unsigned)lx > 3u || (unsigned)ly > 3u || (unsigned)lz > 3u) {
            /* moved out of its sort cell's brick since the sort: walk the
               cells around its position in global memory */
            build_lists_global(P, (int)i, pos, cell_start, bpos, bcell_start, near, nbr_f, cnt_f, nbr_b, cnt_b, st);
            continue;
        }
        unsigned nF = 0, nB = 0;
        /* x outermost, z innermost (HashTable.cpp:59-65); cells outside the
           grid have empty ranges */
        for (int dx = 0; dx < 3; ++dx)
            for (int dy = 0; dy < 3; ++dy)
                for (int dz = 0; dz < 3; ++dz) {
                    const int h = (lz + dz) * 36 + (ly + dy) * 6 + (lx + dx);
                    const unsigned o = s_off[h], n = s_off[h + 1] - o, s = s_gs[h];
                    for (unsigned k = 0; k < n; ++k) {
                        const float4 xq = staged ? s_pos[o + k] : pos[s + k];
                        if (dist2_exact(xi, xq) <= s2max) {
                            if (nF < P.capF) __stcs(nbr_f + list_index(nF, P.capF, i), s + k);
                            ++nF;
                        }
                    }
                    for (unsigned q = s_bs[h]; q < s_be[h]; ++q) {
                        if (dist2_exact(xi, bpos[q]) <= s2max) {
                            if (nB < P.capB) __stcs(nbr_b + list_index(nB, P.capB, i), q);
                            ++nB;
                        }
                    }
                }
        cnt_f[i] = min(nF, P.capF);
        cnt_b[i] = min(nB, P.capB);
        if (nF > P.capF || nB > P.capB) {
            atomicAdd(&st->overflow, 1u);
            atomicOr(&st->err, ERRBIT_OVERFLOW);
        }
    }
}

/* Akinci boundary volume V_b = 1 / sum_b' W(x_b - x_b') over the 27 cells
   (AkinciBoundaryObject.cpp:10-34); k_boundary_psi then stores
   psi = rho0 V_b in bpos.w for the fluid kernels. */
__global__ void __launch_bounds__(128) k_boundary_volume(SimParams P, SceneRef S, const float4* __restrict__ bpos,
                                                         const unsigned* __restrict__ bcell_start,
                                                         float* __restrict__ bvol)
{
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= P.nb) return;
    const float4 xb = bpos[b];
    float delta = 0.0f;
    for_candidates27(xb, P.h, grid_for(P, S, (unsigned)b), bcell_start, [&](unsigned q) {
        const float s2 = dist2_exact(xb, bpos[q]);
        if (s2 <= P.h2_guard) delta = __fadd_rn(delta, cs_W_exact(s2, P));
    });
    bvol[b] = __fdiv_rn(1.0f, delta);
}

__global__ void __launch_bounds__(256) k_boundary_psi(SimParams P, float4* __restrict__ bpos,
                                                      const float* __restrict__ bvol)
{
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b < P.nb) bpos[b].w = __fmul_rn(P.rho0, bvol[b]);
}

/* out[orig[i]] = in[i]: sorted order -> caller order */
__global__ void k_unsort_v4(int n, const unsigned* __restrict__ orig, const float4* __restrict__ in,
                            float* __restrict__ out3)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 v = in[i];
    const size_t o = (size_t)orig[i] * 3;
    out3[o] = v.x;
    out3[o + 1] = v.y;
    out3[o + 2] = v.z;
}

__global__ void k_unsort_f(int n, const unsigned* __restrict__ orig, const float* __restrict__ in,
                           float* __restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[orig[i]] = in[i];
}

/* caller order -> sorted slots (set_state between steps) */
__global__ void k_sort_v3(int n, const unsigned* __restrict__ orig, const float* __restrict__ in3,
                          float4* __restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const size_t o = (size_t)orig[i] * 3;
    out[i] = make_float4(in3[o], in3[o + 1], in3[o + 2], 0.0f);
}

__global__ void k_pack_v3(int n, const float* __restrict__ in3, float4* __restrict__ out, float w)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = make_float4(in3[3 * (size_t)i], in3[3 * (size_t)i + 1], in3[3 * (size_t)i + 2], w);
}

__global__ void k_iota(int n, unsigned* __restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (unsigned)i;
}

static inline int blocks_for(long long n, int bs) { return (int)((n + bs - 1) / bs); }

void launch_sort(const SimParams& P, const SceneRef& S, int n, const float4* pos_for_keys, unsigned* cell_count,
                 unsigned* cell_start,
                 unsigned* chunk_sums, unsigned* cell_of, unsigned* slot, unsigned* tmp_key, unsigned* tmp_src,
                 const unsigned* orig_in, const GatherSet& g, cudaStream_t s)
{
    if (n <= 0) {
        /* an empty set still needs an all-zero start table */
        cudaMemsetAsync(cell_start, 0, ((size_t)P.ncells + 1) * sizeof(unsigned), s);
        return;
    }
    const int nchunks = (int)(P.ncells / 4096);
    k_ns_count<<<blocks_for(n, 256), 256, 0, s>>>(P, S, n, g.n_dev, pos_for_keys, cell_count, chunk_sums, cell_of, slot);
    k_scan<<<nchunks, 256, 0, s>>>(cell_count, cell_start, chunk_sums, nchunks, cell_start + P.ncells);
    k_ns_scatter<<<blocks_for(n, 256), 256, 0, s>>>(n, g.n_dev, cell_of, slot, cell_start, orig_in, tmp_key, tmp_src,
                                                    chunk_sums, nchunks);
    k_ns_rank_gather<<<blocks_for(n, 256), 256, 0, s>>>(n, cell_of, cell_start, tmp_key, tmp_src, g);
}

/* Which search. A warp per particle in the smallest scenes, where one lane's
   walk over ~216 candidates is the critical path (1k WCSPH step 34.7 -> 26.8 us
   with the densities in it, 8k 40.2 -> 36.0); four lanes per particle up to
   where one lane each fills the GPU (33k WCSPH step 59.1 us, one lane 62.7, a
   warp 69.4); then one lane, whose instructions are the fewest (64k 80 us, four
   lanes 96, a warp 118). Lists alone (DFSPH): a warp up to the second line (33k
   DFSPH step 188 us, one lane 190, four lanes 199). */
constexpr int kSearchWarpMax = 1 << 14, kSearchLanesMax = 3 << 14;
/* Densities in the search kernel up to here: with more particles the lists and
   positions a thread has just walked have left the caches when it comes back
   for its density terms, and a second kernel is the faster one (125k 58 us
   against 42 + 27, 216k 86 against 61 + 29; 1M 333 against 209 + 85). */
constexpr int kSearchDensityMax = 1 << 18;

template <int MODE, typename Off>
static void search_by_lanes(const SimParams& P, const SceneRef& S, const SearchArrays& A, cudaStream_t s)
{
    if constexpr (MODE != SEARCH_LISTS)
        if (P.nf < kSearchLanesMax) {
            k_search_lanes<MODE, Off><<<blocks_for((long long)P.nf * kLanes, kLaneBlock), kLaneBlock, 0, s>>>(P, S, A);
            return;
        }
    k_search<MODE, Off><<<blocks_for(P.nf, 128), 128, 0, s>>>(P, S, A);
}

template <int MODE>
static void search_mode(const SimParams& P, const SceneRef& S, const SearchArrays& A, cudaStream_t s)
{
    if (P.nf < (MODE == SEARCH_LISTS ? kSearchLanesMax : kSearchWarpMax))
        k_search_warp<MODE><<<blocks_for(P.nf, kSearchWarps), kSearchWarps * 32, 0, s>>>(P, S, A);
    else if (narrow_slots((unsigned)P.nf, (unsigned)P.nb)) search_by_lanes<MODE, unsigned>(P, S, A, s);
    else search_by_lanes<MODE, unsigned long long>(P, S, A, s);
}

bool launch_search(const SimParams& P, const SceneRef& S, const DeviceArrays& D, int mode, cudaStream_t s, bool staged)
{
    if (P.nf <= 0) return true;
    const SearchArrays A{D.pos, D.cell_start, D.bpos, D.bcell_start, D.near, D.nbr_f, D.cnt_f, D.nbr_b,
                         D.cnt_b, D.rho, D.press, D.vel, D.rec, D.st};
    if (staged && !S.scenes && P.cell_order == 0 && P.nf >= (1 << 16)) {
        /* one block per brick; bricks without fluid leave at once */
        const int nbricks = P.nbx * P.nby * (P.dimz / 4);
        k_ns_build_lists_staged<<<nbricks, kStagedBlock, 0, s>>>(P, A.pos, A.cell_start, A.bpos, A.bcell_start, A.near,
                                                                  A.nbr_f, A.cnt_f, A.nbr_b, A.cnt_b, A.st);
        return false;
    }
    if (P.nf >= kSearchDensityMax) {
        search_mode<SEARCH_LISTS>(P, S, A, s);
        return mode == SEARCH_LISTS;
    }
    switch (mode) {
    case SEARCH_DENSITY: search_mode<SEARCH_DENSITY>(P, S, A, s); break;
    case SEARCH_EOS: search_mode<SEARCH_EOS>(P, S, A, s); break;
    default: search_mode<SEARCH_LISTS>(P, S, A, s); break;
    }
    return true;
}

/* near[c] = 1 for every cell c with a boundary particle in the 27 cells
   around it (near is zeroed by the caller): fluid particles of the other cells
   skip the boundary candidates. The boundary does not move, so this is done
   once per cell order. */
__global__ void __launch_bounds__(256) k_mark_near(SimParams P, SceneRef S, const float4* __restrict__ bpos,
                                                   unsigned char* __restrict__ near)
{
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= P.nb) return;
    const Grid g = grid_for(P, S, (unsigned)b);
    const float4 x = bpos[b];
    const int cx = cell_coord(x.x, P.h, g.cminx, g.dimx);
    const int cy = cell_coord(x.y, P.h, g.cminy, g.dimy);
    const int cz = cell_coord(x.z, P.h, g.cminz, g.dimz);
    for (int xx = max(cx - 1, 0); xx <= min(cx + 1, g.dimx - 1); ++xx)
        for (int yy = max(cy - 1, 0); yy <= min(cy + 1, g.dimy - 1); ++yy)
            for (int zz = max(cz - 1, 0); zz <= min(cz + 1, g.dimz - 1); ++zz) near[cell_at(xx, yy, zz, g)] = 1;
}

void launch_mark_near(const SimParams& P, const SceneRef& S, const float4* bpos, unsigned char* near, cudaStream_t s)
{
    if (P.nb > 0) k_mark_near<<<blocks_for(P.nb, 256), 256, 0, s>>>(P, S, bpos, near);
}

/* bad |= div_h(x) differs from x / h for a mantissa of x (sign and scale of x
   do not matter: every operation scales exactly). */
__global__ void __launch_bounds__(256) k_check_div_h(SimParams P, unsigned* bad)
{
    const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;
    P.h_div_exact = 1;
    const float x = __uint_as_float(0x3f800000u | m);
    if (div_h(x, P) != __fdiv_rn(x, P.h)) *bad = 1u;
}

void launch_check_div_h(const SimParams& P, unsigned* bad, cudaStream_t s)
{
    k_check_div_h<<<(1 << 23) / 256, 256, 0, s>>>(P, bad);
}

void launch_boundary_volume(const SimParams& P, const SceneRef& S, float4* bpos, const unsigned* bcell_start,
                            float* bvol, cudaStream_t s)
{
    if (P.nb <= 0) return;
    k_boundary_volume<<<blocks_for(P.nb, 128), 128, 0, s>>>(P, S, bpos, bcell_start, bvol);
    k_boundary_psi<<<blocks_for(P.nb, 256), 256, 0, s>>>(P, bpos, bvol);
}

void launch_unsort_v4(int n, const unsigned* orig, const float4* in, float* out3, cudaStream_t s)
{
    if (n > 0) k_unsort_v4<<<blocks_for(n, 256), 256, 0, s>>>(n, orig, in, out3);
}
void launch_unsort_f(int n, const unsigned* orig, const float* in, float* out, cudaStream_t s)
{
    if (n > 0) k_unsort_f<<<blocks_for(n, 256), 256, 0, s>>>(n, orig, in, out);
}
void launch_sort_v3(int n, const unsigned* orig, const float* in3, float4* out, cudaStream_t s)
{
    if (n > 0) k_sort_v3<<<blocks_for(n, 256), 256, 0, s>>>(n, orig, in3, out);
}
void launch_pack_v3(int n, const float* in3, float4* out, float w, cudaStream_t s)
{
    if (n > 0) k_pack_v3<<<blocks_for(n, 256), 256, 0, s>>>(n, in3, out, w);
}
void launch_iota(int n, unsigned* out, cudaStream_t s)
{
    if (n > 0) k_iota<<<blocks_for(n, 256), 256, 0, s>>>(n, out);
}

/* Cells of n particles listed by the search now completing: entry = the
   completed searches + 1 where still 0 (single-scene grids). */
__global__ void __launch_bounds__(256) k_mark_entries(SimParams P, const float4* __restrict__ pos, int n,
                                                      const unsigned* n_dev, unsigned* entry, const DevState* st)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (n_dev ? (int)*n_dev : n)) return;
    const unsigned c = cell_index(pos[i], P.h, grid_single(P));
    if (entry[c] == 0u) atomicCAS(&entry[c], 0u, st->ns_epoch + 1u);
}

__global__ void k_epoch_advance(DevState* st) { st->ns_epoch += 1u; }

void launch_mark_entries(const SimParams& P, const float4* pos, int n, const unsigned* n_dev, unsigned* entry,
                         DevState* st, bool advance, cudaStream_t s)
{
    if (n > 0) k_mark_entries<<<(n + 255) / 256, 256, 0, s>>>(P, pos, n, n_dev, entry, st);
    if (advance) k_epoch_advance<<<1, 1, 0, s>>>(st);
}

} // namespace sph
