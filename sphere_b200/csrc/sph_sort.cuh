// sph_sort.cuh -- the cell sort and the neighbour-list build, sphere by
// sphere: device functions shared by the kernels of the step's chain
// (sph_kernels.cu) and the one-launch rebuilds (k_resort, k_pair_resort).
#pragma once

#include <cstdint>

#include "sph_device.cuh"
#include "sph_internal.h"
#include "sph_step.cuh"
#include "sph_sync.cuh"

namespace sph {

// sorting.cuh:7-51 calcParticleCellID + device.cu:241-276 position checks
// for sphere i at x, by whole warps (valid: the lane holds a sphere).
__device__ __forceinline__ void hash_sphere(const StepArgs &A, const DevBox &B, uint32_t i,
                                            double4 x, bool valid)
{
    const double xv[3] = {x.x, x.y, x.z};
    uint32_t c[3];
    bool nonfinite = !isfinite(x.x) || !isfinite(x.y) || !isfinite(x.z);
    bool outside = false;
    for (int d = 0; d < 3; ++d) {
        double f = floor((xv[d] - B.origo[d]) / (B.L[d] / B.num[d]));
        if (!(f >= 0.0)) { outside = true; f = 0.0; }
        if (f >= (double)B.num[d]) { outside = true; f = (double)(B.num[d] - 1); }
        c[d] = (uint32_t)f;
    }
    if (valid) {
        if (nonfinite) raise_flag(A.err, SPH_ERR_NAN);
        else if (outside || x.x > B.L[0] || x.y > B.L[1] || x.z > B.L[2])
            raise_flag(A.err, SPH_ERR_OUT_OF_GRID);
    }
    const uint32_t cell = B.cell_base + (c[2] * B.num[1]) * B.num[0] + c[1] * B.num[0] + c[0];
    // lanes of the warp in the same cell take consecutive slots with one
    // atomic (the slot order within a cell is free: k_place orders by index)
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t peers = __match_any_sync(0xffffffffu, valid ? cell : 0xffffffffu);
    const int leader = __ffs(peers) - 1;
    uint32_t base = 0;
    if (valid && (int)lane == leader) base = atomicAdd(&A.cell_count[cell], (uint32_t)__popc(peers));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (!valid) return;
    A.cell_id[i] = cell;
    if (A.cellc) A.cellc[i] = pack_cell(c[0], c[1], c[2]);
    A.local_off[i] = base + (uint32_t)__popc(peers & ((1u << lane) - 1u));
}

// Exclusive scan of n uint32 (3 launches): per-block totals, a one-block
// scan of the totals, then per-block scans with the block offset.
constexpr int SCAN_THREADS = 1024;
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t *smem,
                                                         uint32_t *total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) smem[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < (int)(blockDim.x >> 5) ? smem[lane] : 0u;
        uint32_t wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += y;
        }
        smem[lane] = wi - w;
        if (lane == 31) smem[32] = wi;
    }
    __syncthreads();
    const uint32_t r = smem[warp] + incl - v;
    *total = smem[32];
    __syncthreads();
    return r;
}

// The stable sort by cell id and the sorted copies (sorting.cuh:118-130)
// in one pass over the particles in original order: particle i goes to
// cell_off[c] + (the number of particles of its cell with a smaller index),
// so each cell is ordered by original index.  rank = inverse of perm.
template <bool ALL>
__device__ __forceinline__ void place_sphere(const StepArgs &A, uint32_t i)
{
    const uint32_t c = A.cell_id[i];
    const uint32_t s = A.cell_off[c], e = A.cell_off[c + 1];
    uint32_t j = s;
    for (uint32_t k = s; k < e; ++k) j += A.unsorted[k] < i ? 1u : 0u;
    A.perm[j] = i;
    const double4 x = A.x[i];
    A.xs[j] = x;
    A.xf[j] = make_float4((float)x.x, (float)x.y, (float)x.z, (float)x.w);
    A.rank[i] = j;
    if (ALL) {
        A.vs[j] = A.vel[i];
        A.ws[j] = A.angvel[i];
    }
}

// --------------------------------------------------------- neighbour lists

// Neighbour lists for the contact search of contact models 2 and 3: for the
// sphere at sorted position a, the ids of all spheres within
// ra + rb + vskin among the +-vrange cells around it (FP32 test widened by
// the prefilter margin, so the list may hold a few more), ascending and
// without repeats.  A sphere that moves less than vskin / 2 (checked in the
// integration against xref) keeps every sphere it can touch in its list.
// Runs only when vflag[0] is set; a list that overflows vcap (<= VL_MAX) is
// marked VL_MAX + 1 and that sphere uses the cell search.  Entry k of
// sphere i goes to vlist[i * row_stride + k * k_stride] (rows of VL_MAX for
// the FP64 form's lists, entry-major for the list step's).  lst: VL_MAX
// entries of shared scratch at stride RS.  Returns whether the sphere has a
// list.
__device__ __forceinline__ bool vlist_build_one(const StepArgs &A, uint32_t a, uint32_t *lst,
                                                uint32_t *vlist, uint32_t *vcount, uint32_t cap,
                                                uint32_t row_stride, uint32_t k_stride, int RS)
{
    const uint32_t i = A.perm[a];
    const DevBox &B = A.boxes[A.box_of[i]];
    const float4 xaf = A.xf[a];
    A.xref[i] = xaf;
    const int R = B.vrange;
    const uint32_t cm = B.P.contactmodel;
    if (R < 1 || (cm != 2 && cm != 3)) {
        vcount[i] = VL_MAX + 1;
        return false;
    }
    int g0, g1, g2;
    unpack_cell(A.cellc[i], g0, g1, g2);
    const int nx = (int)B.num[0], ny = (int)B.num[1];
    const float reach = B.pre_margin + B.vskin;
    const float Lf0 = (float)B.L[0], Lf1 = (float)B.L[1];
    int n = 0;
    bool over = false;
    for (int dz = -R; dz <= R && !over; ++dz)
        for (int dy = -R; dy <= R && !over; ++dy)
            for (int dx = -R; dx <= R && !over; ++dx) {
                int tx = g0 + dx, ty = g1 + dy, sx, sy;
                const int tz = g2 + dz;
                if (!image_cell(B, tx, ty, tz, sx, sy)) continue;
                const float fsx = sx == 0 ? 0.f : (sx > 0 ? Lf0 : -Lf0);
                const float fsy = sy == 0 ? 0.f : (sy > 0 ? Lf1 : -Lf1);
                const uint32_t cell = B.cell_base + (uint32_t)(tx + ty * nx + (nx * ny) * tz);
                const uint32_t start = A.cell_off[cell], end = A.cell_off[cell + 1];
                for (uint32_t b = start; b < end; ++b) {
                    if (b == a) continue;
                    if (!maybe_touching(xaf, A.xf[b], fsx, fsy, reach)) continue;
                    const uint32_t bo = A.perm[b];
                    int q = n;
                    while (q > 0 && lst[(q - 1) * RS] > bo) --q;
                    if (q > 0 && lst[(q - 1) * RS] == bo) continue;   // another image
                    if (n == (int)cap) {
                        over = true;
                        break;
                    }
                    for (int k = n; k > q; --k) lst[k * RS] = lst[(k - 1) * RS];
                    lst[q * RS] = bo;
                    ++n;
                }
            }
    if (over) {
        vcount[i] = VL_MAX + 1;
        return false;
    }
    uint32_t *out = vlist + (size_t)i * row_stride;
    for (int k = 0; k < n; ++k) out[(size_t)k * k_stride] = lst[k * RS];
    vcount[i] = (uint32_t)n;
    return true;
}

// A rebuild whose barrier gave up: the steps return as they are from here
// on (StepArgs::vflag).
__device__ __forceinline__ void stop_steps(const StepArgs &A)
{
    if (threadIdx.x == 0) A.vflag[3] = 1u;
}

// The whole sort by one cooperative launch of RESORT_THREADS-thread blocks:
// cell ids and counts, the exclusive scan, the stable placement and the
// sorted copies, with a grid barrier between the passes (false: a barrier
// timed out; the caller returns).  x(i): the position of sphere i, stored to
// A.x when STORE_X.  s_scan: 33 words of shared memory.
constexpr int RESORT_THREADS = 256;
constexpr int RESORT_ITEMS = SCAN_TILE / RESORT_THREADS;

template <bool STORE_X, class X>
__device__ __forceinline__ bool sort_all(const StepArgs &A, const GridSync &G, uint32_t *s_scan, X x)
{
    const uint32_t nt = gridDim.x * RESORT_THREADS, t0 = blockIdx.x * RESORT_THREADS + threadIdx.x;
    for (uint64_t c = t0; c < A.ncells; c += nt) A.cell_count[c] = 0u;
    if (!grid_barrier(G, gridDim.x, A.err)) return false;
    for (uint32_t base = blockIdx.x * RESORT_THREADS; base < A.ntot; base += nt) {
        const uint32_t i0 = base + threadIdx.x;
        const bool valid = i0 < A.ntot;
        const uint32_t i = valid ? i0 : 0u;
        const double4 xi = x(i);
        if (STORE_X && valid) A.x[i] = xi;
        hash_sphere(A, A.boxes[box_index(A, i)], i, xi, valid);
    }
    if (!grid_barrier(G, gridDim.x, A.err)) return false;
    const uint32_t tiles = (uint32_t)((A.ncells + SCAN_TILE - 1) / SCAN_TILE);
    // per tile its sum; the tiles' offsets; per tile the scan
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const uint64_t base = (uint64_t)tile * SCAN_TILE + (uint64_t)threadIdx.x * RESORT_ITEMS;
        uint32_t s = 0, total;
        for (int k = 0; k < RESORT_ITEMS; ++k)
            if (base + k < A.ncells) s += A.cell_count[base + k];
        block_exclusive_scan(s, s_scan, &total);
        if (threadIdx.x == 0) A.scan_tmp[tile] = total;
    }
    if (!grid_barrier(G, gridDim.x, A.err)) return false;
    if (blockIdx.x == 0) {
        // at most SCAN_TILE tiles (ncells <= 4096^2, checked at sph_create)
        uint32_t v[RESORT_ITEMS], s = 0, total;
#pragma unroll
        for (int k = 0; k < RESORT_ITEMS; ++k) {
            const uint32_t idx = threadIdx.x * RESORT_ITEMS + k;
            v[k] = idx < tiles ? A.scan_tmp[idx] : 0u;
            s += v[k];
        }
        uint32_t off = block_exclusive_scan(s, s_scan, &total);
#pragma unroll
        for (int k = 0; k < RESORT_ITEMS; ++k) {
            const uint32_t idx = threadIdx.x * RESORT_ITEMS + k;
            if (idx < tiles) A.scan_tmp[idx] = off;
            off += v[k];
        }
        if (threadIdx.x == 0) A.cell_off[A.ncells] = total;
    }
    if (!grid_barrier(G, gridDim.x, A.err)) return false;
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const uint64_t base = (uint64_t)tile * SCAN_TILE + (uint64_t)threadIdx.x * RESORT_ITEMS;
        uint32_t v[RESORT_ITEMS], s = 0, total;
#pragma unroll
        for (int k = 0; k < RESORT_ITEMS; ++k) {
            v[k] = base + k < A.ncells ? A.cell_count[base + k] : 0u;
            s += v[k];
        }
        uint32_t off = block_exclusive_scan(s, s_scan, &total) + A.scan_tmp[tile];
#pragma unroll
        for (int k = 0; k < RESORT_ITEMS; ++k) {
            if (base + k < A.ncells) A.cell_off[base + k] = off;
            off += v[k];
        }
    }
    if (!grid_barrier(G, gridDim.x, A.err)) return false;
    for (uint32_t i = t0; i < A.ntot; i += nt)
        A.unsorted[A.cell_off[A.cell_id[i]] + A.local_off[i]] = i;
    if (!grid_barrier(G, gridDim.x, A.err)) return false;
    for (uint32_t i = t0; i < A.ntot; i += nt) place_sphere<false>(A, i);
    return grid_barrier(G, gridDim.x, A.err);
}

// Launch a RESORT_THREADS-thread cooperative kernel over n spheres with the
// list scratch in dynamic shared memory: as many blocks as can be resident,
// at most one per RESORT_THREADS spheres.  (The kernel is a template argument,
// so that what is asked once of the device is asked once per kernel.)
template <auto KERN, class... Arg>
inline void launch_resort(uint64_t n, cudaStream_t st, Arg... args)
{
    const size_t sm = sizeof(uint32_t) * ((size_t)VL_MAX * RESORT_THREADS + 64);
    // (per thread: the device's answers, asked for once)
    static thread_local int for_dev = -1, sms = 0, per_sm = 0;
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev != for_dev) {
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaFuncSetAttribute(KERN, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, KERN, RESORT_THREADS, sm);
        for_dev = dev;
    }
    const uint64_t need = (n + RESORT_THREADS - 1) / RESORT_THREADS;
    const uint64_t cap = (uint64_t)(per_sm > 0 ? per_sm : 1) * (uint64_t)sms;
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3((unsigned)(need < cap ? need : cap));
    c.blockDim = dim3(RESORT_THREADS);
    c.dynamicSmemBytes = sm;
    c.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    c.attrs = at;
    c.numAttrs = 1;
    cudaLaunchKernelEx(&c, KERN, args...);
}

inline GridSync resort_sync(const StepArgs &A, const StepConfig &cfg)
{
    GridSync G;
    G.count = A.sort_bar;
    G.gen = A.sort_bar + 1;
    G.limit_ns = cfg.rebuild_limit_ns;
    return G;
}

}  // namespace sph
