/*
 * sph_density_noalloc: fluid densities for callers that cannot allocate GPU
 * memory.
 *
 * Who needs it: code that runs where cudaMalloc is off limits -- inside a
 * host callback or a custom allocator hook, in a process whose device memory
 * is owned and pooled by a framework, or on a real-time path that must not
 * take the allocator's locks or trigger an implicit synchronisation. Such a
 * caller owns its input and output buffers but no scratch.
 *
 * How: the neighbour-search scratch (cell table, sort buffers, sorted copies)
 * lives in one file-scope static __device__ array of fixed size, so this path
 * calls no cudaMalloc, cudaFree or allocating library routine. Every GPU that
 * loads the library holds the array (about 6 MiB) until the process exits.
 *
 * Rules for callers (also in include/sph2o_cuda.h):
 *   - sizes above SPH_NOALLOC_MAX_FLUID / _BOUNDARY / _CELLS are rejected
 *     with SPH_ERR_CAPACITY before anything is launched;
 *   - every call on a device uses the same array and leaves its contents
 *     behind; calls whose work overlaps on the GPU (different streams, or
 *     host threads calling concurrently) race on it and must be serialised
 *     by the caller;
 *   - the first call on each device looks up the array's device address with
 *     cudaGetSymbolAddress (once, with that device current); make that first
 *     call before any stream capture on the device. The address is cached per
 *     device ordinal and CUDA context id, so after cudaDeviceReset (a new
 *     primary context, the module possibly reloaded elsewhere) the next call
 *     looks it up again -- that call, too, belongs outside a stream capture.
 * The kernels reuse the bodies of the pipeline's sort (sph_grid_body.cuh) and evaluate each
 * density over the 27 cells in the same order and with the same exact
 * arithmetic as the context path, so for particles inside domain_min/max the
 * result equals sph_compute_phase(SPH_PHASE_DENSITY) bit for bit. A particle
 * outside the grid is clamped into an edge cell: it still finds every
 * neighbour, but visits them in another order, so its density can differ
 * from the context path's in the last bits.
 */
#include "../../include/sph2o_cuda.h"
#include "sph_internal.h"

#include <cuda.h> /* driver types only: the two driver calls are fetched at run time */

#include <climits>
#include <cmath>
#include <mutex>
#include <string>

namespace sph {
namespace {

constexpr size_t kMaxFluid = SPH_NOALLOC_MAX_FLUID;
constexpr size_t kMaxBoundary = SPH_NOALLOC_MAX_BOUNDARY;
constexpr size_t kMaxCells = SPH_NOALLOC_MAX_CELLS;  /* multiple of 4096 */

constexpr size_t align256(size_t b) { return (b + 255) / 256 * 256; }

/* byte offsets of the regions inside the scratch array: cell tables (counted
   and scanned in place) with their chunk totals, zeroed together at the start
   of a call; then the sort buffers and sorted copies */
constexpr size_t kOffStart = 0;
constexpr size_t kOffSums = kOffStart + align256((kMaxCells + 1) * 4);
constexpr size_t kOffBStart = kOffSums + align256(kMaxCells / 4096 * 4);
constexpr size_t kOffBSums = kOffBStart + align256((kMaxCells + 1) * 4);
constexpr size_t kOffCellOf = kOffBSums + align256(kMaxCells / 4096 * 4);
constexpr size_t kOffSlot = kOffCellOf + align256(kMaxFluid * 4);
constexpr size_t kOffSrc = kOffSlot + align256(kMaxFluid * 4);
constexpr size_t kOffOrig = kOffSrc + align256(kMaxFluid * 4);
constexpr size_t kOffBCellOf = kOffOrig + align256(kMaxFluid * 4);
constexpr size_t kOffBSlot = kOffBCellOf + align256(kMaxBoundary * 4);
constexpr size_t kOffBSrc = kOffBSlot + align256(kMaxBoundary * 4);
constexpr size_t kOffPos = kOffBSrc + align256(kMaxBoundary * 4);
constexpr size_t kOffBPos = kOffPos + align256(kMaxFluid * 16);
constexpr size_t kScratchBytes = kOffBPos + align256(kMaxBoundary * 16);

} // namespace

/* The scratch of sph_density_noalloc (see the file comment). */
static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

namespace {

std::mutex g_setup_mutex;

/* Device address of the scratch per device ordinal, valid for the CUDA
   context it was looked up in (ctx_id; 0 = unknown). */
struct ScratchAddr {
    unsigned long long ctx_id;
    unsigned char* ptr;
};
ScratchAddr g_scratch_dev[64] = {};

/* Unique id of the context current on this thread (cuCtxGetCurrent +
   cuCtxGetId, fetched through cudaGetDriverEntryPoint so the library does not
   link libcuda). Returns false when no context is current or the driver
   calls are unavailable. Called under g_setup_mutex. */
bool current_context_id(unsigned long long* id)
{
    using GetCurrent = CUresult (*)(CUcontext*);
    using GetId = CUresult (*)(CUcontext, unsigned long long*);
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    static bool resolved = false;
    if (!resolved) {
        cudaDriverEntryPointQueryResult q1{}, q2{};
        void* f1 = nullptr;
        void* f2 = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f1, cudaEnableDefault, &q1) == cudaSuccess &&
            cudaGetDriverEntryPoint("cuCtxGetId", &f2, cudaEnableDefault, &q2) == cudaSuccess &&
            q1 == cudaDriverEntryPointSuccess && q2 == cudaDriverEntryPointSuccess) {
            get_current = reinterpret_cast<GetCurrent>(f1);
            get_id = reinterpret_cast<GetId>(f2);
        }
        resolved = true;
    }
    if (!get_current || !get_id) return false;
    CUcontext ctx = nullptr;
    if (get_current(&ctx) != CUDA_SUCCESS || !ctx) return false;
    return get_id(ctx, id) == CUDA_SUCCESS;
}

/* One particle set (fluid or boundary) on its way through the counting sort.
   Fluid and boundary go through each step in one launch, the first blocks the
   fluid's: a call is six launches, where a sort of its own for each set, the
   packing and a scan in two steps made it fourteen (30,000 + 5,000 particles:
   123 us per call). */
struct NaSet {
    int n, blocks;           /* particles, blocks of 256 */
    const float* in;         /* the caller's array, `width` floats per particle */
    int width;
    unsigned *start, *sums;  /* cell table (populations, then starts) and its chunk totals */
    unsigned *cell_of, *slot, *src;
    unsigned* orig;          /* caller index of each sorted slot (fluid only, else NULL) */
    float4* out;             /* sorted copy */
};

__device__ __forceinline__ const NaSet& na_pick(const NaSet& f, const NaSet& b, int& i)
{
    const bool fluid = (int)blockIdx.x < f.blocks;
    i = (int)((blockIdx.x - (fluid ? 0u : (unsigned)f.blocks)) * blockDim.x + threadIdx.x);
    return fluid ? f : b;
}

__device__ __forceinline__ float4 na_load(const NaSet& s, int i)
{
    const float* p = s.in + (size_t)i * s.width;
    return make_float4(p[0], p[1], p[2], s.width == 4 ? p[3] : 0.0f);
}

__global__ void __launch_bounds__(256) k_na_zero(unsigned* start, unsigned* sums, unsigned* bstart, unsigned* bsums,
                                                 unsigned ncells)
{
    const unsigned k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < ncells) start[k] = bstart[k] = 0u;
    if (k < ncells / 4096u) sums[k] = bsums[k] = 0u;
    if (k == 0u) start[ncells] = bstart[ncells] = 0u; /* an empty set's total */
}

__global__ void __launch_bounds__(256) k_na_count(SimParams P, NaSet f, NaSet b)
{
    /* chunk totals per block first: the caller's order jumps between chunks of
       cells, and single additions to these few words queue up */
    __shared__ unsigned s_chunk[kMaxCells / 4096];
    for (unsigned k = threadIdx.x; k < kMaxCells / 4096; k += blockDim.x) s_chunk[k] = 0u;
    __syncthreads();
    int i;
    const NaSet& s = na_pick(f, b, i);
    if (i < s.n) {
        const unsigned c = cell_index(na_load(s, i), P.h, grid_single(P));
        s.cell_of[i] = c;
        s.slot[i] = atomicAdd(&s.start[c], 1u);
        atomicAdd(&s_chunk[c >> 12], 1u);
    }
    __syncthreads();
    for (unsigned k = threadIdx.x; k < kMaxCells / 4096; k += blockDim.x)
        if (s_chunk[k]) atomicAdd(&s.sums[k], s_chunk[k]);
}

__global__ void __launch_bounds__(256) k_na_scan(NaSet f, NaSet b, int nchunks)
{
    const bool fluid = (int)blockIdx.x < nchunks;
    const NaSet& s = fluid ? f : b;
    scan_chunk_at<false>((int)blockIdx.x - (fluid ? 0 : nchunks), s.start, s.start, s.sums, nchunks,
                         s.start + (size_t)nchunks * 4096);
}

__global__ void __launch_bounds__(256) k_na_scatter(NaSet f, NaSet b)
{
    int i;
    const NaSet& s = na_pick(f, b, i);
    if (i < s.n) s.src[s.start[s.cell_of[i]] + s.slot[i]] = (unsigned)i;
}

/* Rank inside the cell by caller index, then the sorted copy. */
__global__ void __launch_bounds__(256) k_na_rank_gather(NaSet f, NaSet b)
{
    int p;
    const NaSet& s = na_pick(f, b, p);
    if (p >= s.n) return;
    const unsigned i = s.src[p];
    const float4 x = na_load(s, (int)i);
    const unsigned c = s.cell_of[i], first = s.start[c], end = s.start[c + 1];
    unsigned dst = first;
    for (unsigned q = first; q < end; ++q) dst += s.src[q] < i ? 1u : 0u;
    s.out[dst] = x;
    if (s.orig) s.orig[dst] = i;
}

/* Density over the 27 cells by one thread: every fluid candidate first, then
   every boundary candidate, cells in the reference's offset order, exact W. */
__device__ __noinline__ float na_density_at(const SimParams& P, float4 xi, const float4* __restrict__ pos,
                                            const unsigned* __restrict__ cell_start, const float4* __restrict__ bpos,
                                            const unsigned* __restrict__ bcell_start)
{
    const Grid g = grid_single(P);
    float rho = 0.0f;
    for_candidates27(xi, P.h, g, cell_start, [&](unsigned q) {
        const float s2 = dist2_exact(xi, pos[q]);
        if (s2 <= P.h2_guard) rho = __fadd_rn(rho, __fmul_rn(P.mass, cs_W_exact(s2, P)));
    });
    if (P.nb > 0)
        for_candidates27(xi, P.h, g, bcell_start, [&](unsigned q) {
            const float4 xb = bpos[q];
            const float s2 = dist2_exact(xi, xb);
            if (s2 <= P.h2_guard) rho = __fadd_rn(rho, __fmul_rn(xb.w, cs_W_exact(s2, P)));
        });
    return rho;
}

/* The same sum with four lanes per particle (a call holds at most 65,536
   particles, too few to fill the GPU with one lane each): the rows of cells are
   split 3, 2, 2, 2 over the lanes in candidate order, each lane collects its
   accepted candidates in shared memory, the four evaluate the kernel terms, and
   the terms are added in candidate order. A particle with more than kNaBatch
   candidates in one lane is left to na_density_at. Written to the caller's order. */
constexpr int kNaBlock = 128, kNaLanes = 4, kNaBatch = 24;

__global__ void __launch_bounds__(kNaBlock) k_na_density(SimParams P, const float4* __restrict__ pos,
                                                         const unsigned* __restrict__ cell_start,
                                                         const unsigned* __restrict__ orig,
                                                         const float4* __restrict__ bpos,
                                                         const unsigned* __restrict__ bcell_start,
                                                         float* __restrict__ rho_out)
{
    __shared__ float s_w[kNaBatch + 1][kNaBlock]; /* one spare row */
    __shared__ unsigned s_q[kNaBatch][kNaBlock];
    const int i = (int)((blockIdx.x * blockDim.x + threadIdx.x) / kNaLanes);
    const unsigned tid = threadIdx.x, lane = tid & 31u, sub = lane % kNaLanes, first = lane - sub;
    const bool on = i < P.nf;
    const float4 xi = on ? pos[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const Grid g = grid_single(P);
    const int row0 = sub == 0 ? 0 : 2 * (int)sub + 1, row1 = 2 * (int)sub + 3;
    float rho = 0.0f;
    bool over = false;
    const auto set = [&](const unsigned* starts, const float4* xs, bool boundary) {
        unsigned m = 0, nq = 0, nw = 0;
        if (on)
            for_stretches27(
                xi, xi, P.h, g, starts, xs,
                [&](unsigned k, const float (&d)[4], unsigned) {
#pragma unroll
                    for (unsigned u = 0; u < 4; ++u) {
                        const bool in = d[u] <= P.h2_guard;
                        m |= (in ? 1u << u : 0u) << k;
                        s_w[min(nw, (unsigned)kNaBatch)][tid] = d[u]; /* written over unless kept */
                        nw += in ? 1u : 0u;
                    }
                },
                [&](auto slot) {
                    if (boundary)
                        for (; m; m &= m - 1u, ++nq)
                            s_q[min(nq, kNaBatch - 1u)][tid] = slot((unsigned)__ffs((int)m) - 1u);
                    m = 0;
                },
                row0, row1);
        over |= ((__ballot_sync(0xffffffffu, nw > kNaBatch) >> first) & ((1u << kNaLanes) - 1u)) != 0u;
        const unsigned own = min(nw, (unsigned)kNaBatch);
        for (unsigned k = 0; k < own; ++k)
            s_w[k][tid] = __fmul_rn(boundary ? xs[s_q[k][tid]].w : P.mass, cs_W_exact(s_w[k][tid], P));
        __syncwarp();
        for (unsigned l = 0; l < kNaLanes; ++l) {
            const unsigned c = __shfl_sync(0xffffffffu, own, first + l);
            for (unsigned k = 0; k < c; ++k) rho = __fadd_rn(rho, s_w[k][tid - sub + l]);
        }
        __syncwarp();
    };
    set(cell_start, pos, false);
    if (P.nb > 0) set(bcell_start, bpos, true);
    if (!on || sub != 0) return;
    if (over) rho = na_density_at(P, xi, pos, cell_start, bpos, bcell_start);
    rho_out[orig[i]] = rho;
}

thread_local std::string g_noalloc_error;

int na_fail(int code, const std::string& msg)
{
    g_noalloc_error = msg;
    return code;
}

} // namespace
} // namespace sph

using namespace sph;

extern "C" int sph_density_noalloc(float particle_radius, float density0, const float* xyz, unsigned nf,
                                   const float* bxyzpsi, unsigned nb, const float domain_min[3],
                                   const float domain_max[3], float* rho_out, void* stream)
{
    if (!(particle_radius > 0.0f) || !(density0 > 0.0f) || !domain_min || !domain_max)
        return na_fail(SPH_ERR_ARG, "particle_radius, density0 and the domain bounds are required");
    if (nf > 0 && (!xyz || !rho_out)) return na_fail(SPH_ERR_ARG, "null fluid input or output");
    if (nb > 0 && !bxyzpsi) return na_fail(SPH_ERR_ARG, "null boundary input");
    if (nf > kMaxFluid)
        return na_fail(SPH_ERR_CAPACITY, "sph_density_noalloc: " + std::to_string(nf) + " fluid particles exceed "
                                         "SPH_NOALLOC_MAX_FLUID = " + std::to_string(kMaxFluid));
    if (nb > kMaxBoundary)
        return na_fail(SPH_ERR_CAPACITY, "sph_density_noalloc: " + std::to_string(nb) + " boundary particles "
                                         "exceed SPH_NOALLOC_MAX_BOUNDARY = " + std::to_string(kMaxBoundary));

    /* grid over the caller's domain (+1 cell), brick-padded; particles outside
       it are clamped into the edge cells: still found, in another order */
    SimParams P{};
    P.r = particle_radius;
    P.h = 4.0f * particle_radius;
    P.h2 = P.h * P.h;
    P.h2_guard = (float)((double)P.h * (double)P.h * (1.0 + 1.0e-5));
    P.h2_exact = sqrt_le_bound(P.h);
    P.inv_h = 1.0f / P.h;
    P.rho0 = density0;
    const float diameter = 2.0f * particle_radius;
    P.mass = density0 * (float)std::pow((double)diameter, 3.0);
    const float h3 = P.h * P.h * P.h;
    P.cs_k = 8.0f / ((float)M_PI * h3);
    P.cs_k2 = 2.0 * (double)P.cs_k;
    P.nf = (int)nf;
    P.nb = (int)nb;
    int cmin[3], dim[3];
    for (int k = 0; k < 3; ++k) {
        if (!std::isfinite(domain_min[k]) || !std::isfinite(domain_max[k]))
            return na_fail(SPH_ERR_ARG, "sph_density_noalloc: domain bounds must be finite");
        if (!(domain_max[k] >= domain_min[k])) return na_fail(SPH_ERR_ARG, "domain_max < domain_min");
        const double a = std::floor((double)domain_min[k] / P.h) - 1.0;
        const double b = std::floor((double)domain_max[k] / P.h) + 1.0;
        if (a < (double)(INT_MIN / 2) || b > (double)(INT_MAX / 2))
            return na_fail(SPH_ERR_ARG, "sph_density_noalloc: domain bounds too far from the origin for cell "
                                        "indices of edge 4r");
        if (b - a + 1.0 > (double)kMaxCells) return na_fail(SPH_ERR_CAPACITY, "sph_density_noalloc: domain too large");
        cmin[k] = (int)a;
        dim[k] = ((int)(b - a + 1.0) + 3) / 4 * 4;
    }
    const unsigned long long cells = (unsigned long long)dim[0] * dim[1] * dim[2];
    const unsigned long long padded = (cells + 4095) / 4096 * 4096;
    if (padded > kMaxCells)
        return na_fail(SPH_ERR_CAPACITY, "sph_density_noalloc: the domain needs " + std::to_string(cells) +
                                         " cells of size 4r, above SPH_NOALLOC_MAX_CELLS = " + std::to_string(kMaxCells));
    P.cminx = cmin[0]; P.cminy = cmin[1]; P.cminz = cmin[2];
    P.dimx = dim[0]; P.dimy = dim[1]; P.dimz = dim[2];
    P.nbx = dim[0] / 4; P.nby = dim[1] / 4;
    P.ncells = (unsigned)padded;

    /* once per device, with that device current: the array's device address */
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return na_fail(SPH_ERR_NO_DEVICE, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
    if (dev < 0 || dev >= 64) return na_fail(SPH_ERR_NO_DEVICE, "device ordinal out of range");
    unsigned char* base = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_setup_mutex);
        unsigned long long ctx = 0;
        const bool known = current_context_id(&ctx);
        ScratchAddr& slot = g_scratch_dev[dev];
        if (!slot.ptr || !known || slot.ctx_id != ctx) {
            /* first call on this device, or its context changed (cudaDeviceReset) */
            void* p = nullptr;
            e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
            if (e != cudaSuccess)
                return na_fail(SPH_ERR_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
            if (!current_context_id(&ctx)) ctx = 0;  /* the lookup made the primary context current */
            slot.ptr = static_cast<unsigned char*>(p);
            slot.ctx_id = ctx;
        }
        base = slot.ptr;
    }
    if (nf == 0) return SPH_OK;

    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const auto words = [base](size_t off) { return reinterpret_cast<unsigned*>(base + off); };
    NaSet f{}, b{};
    f.n = (int)nf;
    f.in = xyz;
    f.width = 3;
    f.start = words(kOffStart); f.sums = words(kOffSums);
    f.cell_of = words(kOffCellOf); f.slot = words(kOffSlot); f.src = words(kOffSrc);
    f.orig = words(kOffOrig);
    f.out = reinterpret_cast<float4*>(base + kOffPos);
    b.n = (int)nb;
    b.in = bxyzpsi;
    b.width = 4;
    b.start = words(kOffBStart); b.sums = words(kOffBSums);
    b.cell_of = words(kOffBCellOf); b.slot = words(kOffBSlot); b.src = words(kOffBSrc);
    b.out = reinterpret_cast<float4*>(base + kOffBPos);
    f.blocks = (f.n + 255) / 256;
    b.blocks = (b.n + 255) / 256;
    const int blocks = f.blocks + b.blocks, nchunks = (int)(P.ncells / 4096);
    k_na_zero<<<(P.ncells + 255) / 256, 256, 0, s>>>(f.start, f.sums, b.start, b.sums, P.ncells);
    k_na_count<<<blocks, 256, 0, s>>>(P, f, b);
    k_na_scan<<<(nb > 0 ? 2 : 1) * nchunks, 256, 0, s>>>(f, b, nchunks);
    k_na_scatter<<<blocks, 256, 0, s>>>(f, b);
    k_na_rank_gather<<<blocks, 256, 0, s>>>(f, b);
    k_na_density<<<(f.n * kNaLanes + kNaBlock - 1) / kNaBlock, kNaBlock, 0, s>>>(P, f.out, f.start, f.orig, b.out, b.start,
                                                                                    rho_out);
    e = cudaGetLastError();
    if (e != cudaSuccess) return na_fail(SPH_ERR_CUDA, std::string("launch: ") + cudaGetErrorString(e));
    return SPH_OK;
}

extern "C" const char* sph_noalloc_error(void) { return g_noalloc_error.c_str(); }
