// sph_kernels.cu -- FP64 kernels of the B200 DEM step.
//
// Compiled with -fmad=false: together with the operand order kept in
// sph_device.cuh this makes the FP64 step reproduce the reference's
// arithmetic bit for bit.
//
// One step (see launch_step):
//   memset cell_count
//   k_hash          cell id + atomic slot within the cell  (sorting.cuh:7-51)
//   scan (3)        exclusive scan of cell counts -> cell_off
//   k_scatter       unsorted[cell_off[c] + slot] = i
//   k_place         perm: each cell ordered by original index, the stable
//                   order of thrust::sort_by_key (device.cu:1075); sorted
//                   copies of x (+ vel, angvel, rank)  (sorting.cuh:56-132)
//   k_bonds         bond forces into per-bond buffers       (cohesion.cuh:8-233)
//   k_interact      topology + interact + walls + bond gather + integrate
//                   (contactsearch.cuh:329-726, integration.cuh:14-305)
//   k_block_sums    per-256 partial sums of the wall force  (integration.cuh:309-341)
//   k_box_step      integrateWalls + time/grid/velocity-step state
//                   (integration.cuh:344-450, device.cu:1050, 2455-2462, 2536)
// Boxes with a shear-stress top wall (wmode 3) need a global sum of forces
// between interact and integrate (device.cu:2427-2452); they use the
// unfused kernels k_interact<FUSED=false>, k_shear_stress, k_block_sums,
// k_tau_final and k_integrate.
#include <cstdint>
#include <cstdio>

#include "sph_device.cuh"
#include "sph_internal.h"
#include "sph_sort.cuh"
#include "sph_step.cuh"

namespace sph {

static inline unsigned blocks_for(uint64_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

// ------------------------------------------------------------------ sorting

__global__ void k_hash(StepArgs A)
{
    const uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i0 < A.ntot;
    const uint32_t i = valid ? i0 : 0u;
    const DevBox &B = A.boxes[A.nboxes == 1 ? 0u : A.box_of[i]];
    hash_sphere(A, B, i, A.x[i], valid);
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_reduce(const uint32_t *in, uint64_t n,
                                                              uint32_t *bsum)
{
    grid_dependency_wait();
    __shared__ uint32_t smem[33];
    const uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE + (uint64_t)threadIdx.x * SCAN_ITEMS;
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k)
        if (base + k < n) s += in[base + k];
    uint32_t total;
    block_exclusive_scan(s, smem, &total);
    if (threadIdx.x == 0) bsum[blockIdx.x] = total;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_top(uint32_t *bsum, uint32_t nb)
{
    grid_dependency_wait();
    __shared__ uint32_t smem[33];
    uint32_t v[SCAN_ITEMS];
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const uint32_t idx = threadIdx.x * SCAN_ITEMS + k;
        v[k] = idx < nb ? bsum[idx] : 0u;
        s += v[k];
    }
    uint32_t total;
    uint32_t off = block_exclusive_scan(s, smem, &total);
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const uint32_t idx = threadIdx.x * SCAN_ITEMS + k;
        if (idx < nb) bsum[idx] = off;
        off += v[k];
    }
    if (threadIdx.x == 0) bsum[nb] = total;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_down(const uint32_t *in, uint64_t n,
                                                            const uint32_t *bsum, uint32_t nb,
                                                            uint32_t *out)
{
    grid_dependency_wait();
    __shared__ uint32_t smem[33];
    const uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE + (uint64_t)threadIdx.x * SCAN_ITEMS;
    uint32_t v[SCAN_ITEMS];
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        v[k] = base + k < n ? in[base + k] : 0u;
        s += v[k];
    }
    uint32_t total;
    uint32_t off = block_exclusive_scan(s, smem, &total) + bsum[blockIdx.x];
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        if (base + k < n) out[base + k] = off;
        off += v[k];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) out[n] = bsum[nb];
}

__global__ void k_scatter(StepArgs A)
{
    grid_dependency_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.ntot) return;
    A.unsorted[A.cell_off[A.cell_id[i]] + A.local_off[i]] = i;
}

// place_sphere for every sphere; ALL: the sorted velocities too (the fused
// kernels; the split step reads velocities and partners in original order).
template <bool ALL>
__global__ void k_place(StepArgs A)
{
    grid_dependency_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < A.ntot) place_sphere<ALL>(A, i);
}

// --------------------------------------------------------- neighbour lists

// A grid of a few blocks per SM that strides over the spheres, so that the
// launch costs little on the steps that build nothing.
constexpr int VLIST_THREADS = 128;
constexpr unsigned VLIST_BLOCKS = 148u * 8u;

__global__ void __launch_bounds__(VLIST_THREADS) k_vlist_build(StepArgs A)
{
    grid_dependency_wait();
    if (A.vflag[0] == 0u) return;
    __shared__ uint32_t s_list[VL_MAX * VLIST_THREADS];
    for (uint32_t a = blockIdx.x * blockDim.x + threadIdx.x; a < A.ntot;
         a += gridDim.x * blockDim.x)
        vlist_build_one(A, a, s_list + threadIdx.x, A.vlist, A.vcount, A.vcap, VL_MAX, 1u,
                        VLIST_THREADS);
}

// The sort and the list build of the split step, when they are needed: the
// step's other kernels read the sorted order and the lists only, and those
// hold until a sphere has moved half the skin (vflag[0], raised by the
// integration) -- unless some sphere has no list (vflag[2]) and goes
// through the cells at every step, which takes this step's sort.  Most
// steps find neither and end at once: one launch of 1-2 us in the place of
// the chain k_hash .. k_vlist_done of eight, which took 57 us of a step at
// 1e6 spheres and 16 us of 33 at 1e4.
__global__ void __launch_bounds__(RESORT_THREADS) k_resort(StepArgs A, GridSync G)
{
    extern __shared__ uint32_t s_mem[];
    uint32_t *s_scan = s_mem + VL_MAX * RESORT_THREADS;
    const uint4 flags = *reinterpret_cast<const uint4 *>(A.vflag);
    const uint32_t rebuild = flags.x;
    if ((rebuild | flags.z | flags.w) == 0u) return;
    if (flags.w != 0u) {
        if (blockIdx.x == 0 && threadIdx.x == 0) raise_flag(A.err, SPH_ERR_TIMEOUT);
        return;
    }
    // (sort_all's barriers lie between these reads and the writes below)
    if (!sort_all<false>(A, G, s_scan, [&](uint32_t i) { return A.x[i]; })) return stop_steps(A);
    if (rebuild == 0u) return;
    uint32_t none = 0;
    for (uint32_t a = blockIdx.x * RESORT_THREADS + threadIdx.x; a < A.ntot;
         a += gridDim.x * RESORT_THREADS)
    {
        if (!vlist_build_one(A, a, s_mem + threadIdx.x, A.vlist, A.vcount, A.vcap, VL_MAX, 1u,
                             RESORT_THREADS))
            none = 1u;
        A.lmask[A.perm[a]] = 0ull;   // new lists: k_touch goes through the row
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) A.vflag[2] = 0u;
    if (!grid_barrier(G, gridDim.x, A.err)) return stop_steps(A);
    if (none) A.vflag[2] = 1u;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        A.vflag[0] = 0u;
        A.vflag[1] += 1u;
    }
}

// After the (possible) build: clear the request, count builds.
__global__ void k_vlist_done(StepArgs A)
{
    grid_dependency_wait();
    if (A.vflag[0] != 0u) {
        A.vflag[0] = 0u;
        A.vflag[1] += 1u;
    }
}

// -------------------------------------------------------------------- bonds

// cohesion.cuh:8-233 bondsLinear.  Forces go to per-bond buffers (w = 1
// when applied this step) and are added to the particles in ascending bond
// order by k_interact, instead of the reference's racing scatter-add.  A
// bond broken during the run stays broken (the reference re-activates it
// when nb0 < np, cohesion.cuh:30 and :205).
template <int LM>
__global__ void k_bonds(StepArgs A)
{
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= A.nbonds) return;
    const uint32_t stop = A.lazy_sort ? A.vflag[3] : 0u;   // a rebuild gave up
    const DevBox &B = A.boxes[A.bond_box[k]];
    const SphParams &P = B.P;
    const double dt = B.dt;
    const uint2 bd = A.bonds[k];
    A.bf[k] = make_double4(0.0, 0.0, 0.0, 0.0);
    if (!(bd.x < B.np) || A.bbroken[k]) return;
    if (!(bd.y < B.np)) { raise_flag(A.err, SPH_ERR_INPUT); return; }
    const uint32_t gi = B.p_base + bd.x, gj = B.p_base + bd.y;
    const double4 d4 = A.bdelta[k], o4 = A.bomega[k];
    d3 delta0_t = xyz(d4);
    const double delta0_n = d4.w;
    d3 omega0_t = xyz(o4);
    const double omega0_n = o4.w;
    const double4 x_i = A.x[gi], x_j = A.x[gj];
    const d3 vel_i = xyz(A.vel[gi]), vel_j = xyz(A.vel[gj]);
    const d3 angvel_i = xyz(A.angvel[gi]), angvel_j = xyz(A.angvel[gj]);
    const double R_bar = P.lambda_bar * fmin(x_i.w, x_j.w);
    const double Ar = PI * R_bar * R_bar;
    const double I = 0.25 * PI * R_bar * R_bar * R_bar * R_bar;
    const double J = I * 2.0;
    const d3 x = mk(x_i.x - x_j.x, x_i.y - x_j.y, x_i.z - x_j.z);
    const double x_length = vlen<LM>(x);
    const double overlap = fmin(0.0, x_length - (x_i.w + x_j.w));
    const d3 n = divs(x, x_length);
    delta0_t = vsub(delta0_t, muls(n, dot(n, delta0_t)));
    const d3 ddelta = muls(vadd(vadd(vsub(vel_i, vel_j), smul(x_i.w + overlap / 2.0, cross(n, angvel_i))),
                                smul(x_j.w + overlap / 2.0, cross(n, angvel_j))),
                           dt);
    const double ddelta_n = -dot(ddelta, n);
    const double delta_n = delta0_n + ddelta_n;
    const d3 ddelta_t = vsub(ddelta, muls(n, dot(n, ddelta)));
    const d3 delta_t = vadd(delta0_t, ddelta_t);
    const d3 f_n = smul(P.k_n * Ar * delta_n + P.gamma_n * ddelta_n / dt, n);
    const d3 f_t = vsub(smul(-P.k_t * Ar, delta_t), divs(smul(P.gamma_t, ddelta_t), dt));
    const d3 f = vadd(f_n, f_t);
    const d3 nn = vneg(n);
    omega0_t = vsub(omega0_t, muls(nn, dot(omega0_t, nn)));
    const d3 domega = muls(vsub(angvel_j, angvel_i), dt);
    const double domega_n = dot(domega, nn);
    const double omega_n = omega0_n + domega_n;
    const d3 domega_t = vsub(domega, smul(domega_n, nn));
    const d3 omega_t = vadd(omega0_t, domega_t);
    const d3 t_n = smul(-P.k_t * J * omega_n, nn);
    const d3 t_t = smul(-P.k_n * I, omega_t);
    const d3 t_j = vadd(t_n, t_t);
    const double sigma_max = vlen<LM>(f_n) / Ar + vlen<LM>(t_t) * R_bar / I;
    const double tau_max = vlen<LM>(f_t) / Ar + vlen<LM>(t_n) * R_bar / J;
    if (stop) return;   // the bond keeps its state
    if (sigma_max >= P.sigma_b || tau_max >= P.tau_b) {
        A.bonds[k].x = B.nb0;
        A.bbroken[k] = 1;
        return;
    }
    A.bdelta[k] = make_double4(delta_t.x, delta_t.y, delta_t.z, delta_n);
    A.bomega[k] = make_double4(omega_t.x, omega_t.y, omega_t.z, omega_n);
    A.bf[k] = make_double4(f.x, f.y, f.z, 1.0);
    A.bt[k] = make_double4(t_j.x, t_j.y, t_j.z, 0.0);
}

// Unfused integrate (boxes with a shear-stress wall).
__global__ void k_integrate(StepArgs A)
{
    const uint32_t a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= A.ntot) return;
    const uint32_t i = A.perm[a];
    const DevBox &B = A.boxes[A.box_of[i]];
    const double4 f = A.force[i], t = A.torque[i];
    integrate_particle(A, B, B, i, load_own(A, i), A.xs[a], A.vs[a], A.ws[a], xyz(f), xyz(t));
}

// integration.cuh:457-484 findShearStressOnFixedMovingParticles
__global__ void k_shear_stress(StepArgs A)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.ntot) return;
    const DevBox &B = A.boxes[A.box_of[i]];
    if (!(B.nw > 0 && B.wmode[0] == 3)) return;
    const double z = A.x[i].z;
    const double fixvel = A.vel[i].w;
    const double force_x = A.force[i].x;
    double f_x = 0.0;
    if (fixvel > 0.0 && z > B.L[2] * 0.5) f_x = force_x;
    A.tau_pp[i] = f_x / (B.L[0] * B.L[1]);
}

// integration.cuh:309-341 summation: one 256-thread block per partial, the
// same shared-memory tree as the reference.
__global__ void __launch_bounds__(256) k_block_sums(StepArgs A, const double *in, double *out,
                                                    int only_wmode3)
{
    __shared__ double cache[256];
    const uint32_t part = blockIdx.x;
    const DevBox &B = A.boxes[A.part_owner[part]];
    const bool active = B.nw > 0 && (!only_wmode3 || B.wmode[0] == 3);
    const uint32_t local = (part - B.part_base) * 256u + threadIdx.x;
    double temp = 0.0;
    if (active && local < B.np) temp += in[B.p_base + local];
    cache[threadIdx.x] = temp;
    __syncthreads();
    for (unsigned s = 128; s != 0; s /= 2) {
        if (threadIdx.x < s) cache[threadIdx.x] += cache[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[part] = cache[0];
}

// Per-box kernels: one block per box, partials staged in BOX_STAGE chunks.
constexpr int BOX_THREADS = 256;
constexpr int BOX_STAGE = 2048;

// In-order sum of cnt doubles staged in shared memory, by one thread, its
// loads issued eight at a time ahead of the additions.
__device__ __forceinline__ double ordered_sum(const double *v_s, uint32_t cnt, double acc)
{
    uint32_t k = 0;
    for (; k + 8 <= cnt; k += 8) {
        double v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = v_s[k + q];
#pragma unroll
        for (int q = 0; q < 8; ++q) acc += v[q];
    }
    for (; k < cnt; ++k) acc += v_s[k];
    return acc;
}

// Sum of the shear-stress partials per box (integration.cuh:65-68), once
// per box instead of once per particle: one block per box stages the
// partials in shared memory with coalesced loads and thread 0 adds them in
// block order, the reference's order.
__global__ void __launch_bounds__(BOX_THREADS) k_tau_final(StepArgs A)
{
    __shared__ double s_part[BOX_STAGE];
    const uint32_t b = blockIdx.x;
    if (b >= A.nboxes) return;
    DevBox &B = A.boxes[b];
    double tau = 0.0;
    if (B.nw > 0 && B.wmode[0] == 3) {
        for (uint32_t base = 0; base < B.nblocks; base += BOX_STAGE) {
            const uint32_t cnt = min((uint32_t)BOX_STAGE, B.nblocks - base);
            __syncthreads();
            for (uint32_t k = threadIdx.x; k < cnt; k += blockDim.x)
                s_part[k] = A.tau_partial[B.part_base + base + k];
            __syncthreads();
            if (threadIdx.x == 0) tau = ordered_sum(s_part, cnt, tau);
        }
    }
    if (threadIdx.x == 0) B.tau_eff_x = tau;
}

// integration.cuh:344-450 integrateWalls, then the loop bookkeeping of
// device.cu:2536-2538, the adaptive grid of device.cu:1050 and the
// velocity-step state of device.cu:2455-2462 for the next step.
// One block per box.  The wall-force total is the sequential sum of the
// per-block partials in block order (as the reference's integrateWalls
// loop); the block stages the partials in shared memory with coalesced
// loads and thread 0 adds them in order.
__global__ void __launch_bounds__(BOX_THREADS) k_box_step(StepArgs A)
{
    __shared__ double s_part[BOX_STAGE];
    const uint32_t b = blockIdx.x;
    if (b >= A.nboxes) return;
    __shared__ DevBox B;
    stage_box(B, A.boxes[b]);
    if (A.lazy_sort && B.halt) return;
    bool any = false;
    for (uint32_t w = 0; w < B.nw; ++w) any = any || B.wmode[w] != 0;
    double fsum = 0.0;
    if (B.np > 0 && any) {
        for (uint32_t base = 0; base < B.nblocks; base += BOX_STAGE) {
            const uint32_t cnt = min((uint32_t)BOX_STAGE, B.nblocks - base);
            __syncthreads();
            for (uint32_t k = threadIdx.x; k < cnt; k += blockDim.x)
                s_part[k] = A.wall_partial[B.part_base + base + k];
            __syncthreads();
            // the sequential sum of integrateWalls
            if (threadIdx.x == 0) fsum = ordered_sum(s_part, cnt, fsum);
        }
    }
    if (threadIdx.x == 0) advance_box(B, fsum);
    unstage_box(A.boxes[b], B);
}

// ------------------------------------------------------------- scene packing

// One Jacobi sweep of overlap removal (scene preparation, not part of the
// step): every overlapping pair pushes both spheres apart along the centre
// line by `alpha` times half the overlap; the floor (z = origo) and the
// ceiling z_top push spheres back inside; periodic images count as
// neighbours.  Partners are read from the sorted copies, so the sphere's
// new position goes straight to A.x; with `next` the sphere is also put
// into its cell for the next sweep's sort (cell_count, zeroed before: the
// candidate loop reads cell_off only).  The largest overlap seen is max-ed
// into *max_ov (as the bit pattern of a non-negative double), one atomic
// per block.
//
// Bound by the candidates' loads and tests: in a pack with a spread of radii
// the 27 cells around a sphere hold about 200 candidates, of which six
// overlap.  Each is tested in FP32 on the 16-byte copy (as maybe_touching:
// never negative for an overlapping pair), RELAX_BATCH loads in flight, and
// those that pass are noted in shared memory; the FP64 test, square root and
// division then run over the noted ones, all lanes of a warp at work, where
// in the candidate loop one lane of nine was (a sweep of 1e6 spheres: 1.26
// ms with the FP64 test on every candidate, 0.70 with it on those that pass,
// 0.62 with the notes, 0.47 with the tests of a batch as the sign bits of d^2 -
// r^2 instead of a branch each).  The notes keep the cells' visit order, so the
// sums are those of the plain loop.  The cells of a row (dx = -1, 0, 1) are
// neighbours in the cell order, so away from the grid's x edges a row is
// one range of candidates.
constexpr int RELAX_THREADS = 128;
constexpr int RELAX_BATCH = 8;
constexpr int RELAX_NOTES = 24;

__global__ void __launch_bounds__(RELAX_THREADS, 5) k_relax(StepArgs A, double alpha, double z_top,
                                                            unsigned long long *max_ov, bool next)
{
    __shared__ unsigned long long s_max[RELAX_THREADS / 32];
    __shared__ uint32_t s_note[RELAX_NOTES][RELAX_THREADS];   // sorted position | image code
    const uint32_t a0 = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = a0 < A.ntot;
    const uint32_t a = valid ? a0 : 0u;
    const uint32_t i = A.perm[a];
    const DevBox &B = A.boxes[A.box_of[i]];
    const double4 xa = A.xs[a];
    const float4 xaf = A.xf[a];
    const int nx = (int)B.num[0], ny = (int)B.num[1];
    const float Lf0 = (float)B.L[0], Lf1 = (float)B.L[1];
    const float margin = B.pre_margin;
    double dx = 0.0, dy = 0.0, dz = 0.0, worst = 0.0;
    // the noted candidates, in order
    uint32_t noted = 0;
    auto push_apart = [&]() {
        for (uint32_t k = 0; k < noted; ++k) {
            const uint32_t w = s_note[k][threadIdx.x];
            int sx, sy;
            decode_shift(w >> CODE_SHIFT, sx, sy);
            if ((w & ID_MASK) == a) continue;   // the sphere itself
            const d3 dm = shift_vec(B, sx, sy);
            const double4 xb = A.xs[w & ID_MASK];
            const double rx = xa.x - xb.x + dm.x, ry = xa.y - xb.y + dm.y, rz = xa.z - xb.z + dm.z;
            const double len = sqrt(rx * rx + ry * ry + rz * rz);
            const double ov = xa.w + xb.w - len;
            if (ov > 0.0 && len > 0.0) {
                const double s = 0.5 * alpha * ov / len;
                dx += s * rx;
                dy += s * ry;
                dz += s * rz;
                worst = fmax(worst, ov);
            }
        }
        noted = 0;
    };
    // the candidates [b0, b1) under image (sx, sy): maybe_touching as the sign
    // of d^2 - r^2, RELAX_BATCH bits at a time (A.xf has room for a batch past
    // its end)
    auto range = [&](uint32_t b0, uint32_t b1, int sx, int sy) {
        const uint32_t code = shift_code(sx, sy) << CODE_SHIFT;
        const float ax = xaf.x + (sx == 0 ? 0.f : (sx > 0 ? Lf0 : -Lf0));
        const float ay = xaf.y + (sy == 0 ? 0.f : (sy > 0 ? Lf1 : -Lf1));
        const float aw = xaf.w + margin;
        for (uint32_t b = b0; b < b1; b += RELAX_BATCH) {
            const float4 *p = A.xf + b;
            float4 xf[RELAX_BATCH];
#pragma unroll
            for (int j = 0; j < RELAX_BATCH; ++j) xf[j] = p[j];
            uint32_t m = 0;
#pragma unroll
            for (int j = 0; j < RELAX_BATCH; ++j) {
                const float cx = ax - xf[j].x, cy = ay - xf[j].y, cz = xaf.z - xf[j].z;
                const float rr = aw + xf[j].w;
                const float d2 = __fmaf_rn(cz, cz, __fmaf_rn(cy, cy, cx * cx));
                m |= (__float_as_uint(__fmaf_rn(-rr, rr, d2)) >> 31) << j;
            }
            m &= (1u << min(b1 - b, (uint32_t)RELAX_BATCH)) - 1u;
            if (noted + (uint32_t)__popc(m) > RELAX_NOTES) push_apart();
            for (; m; m &= m - 1u) s_note[noted++][threadIdx.x] = (b + (uint32_t)(__ffs(m) - 1)) | code;
        }
    };
    if (valid) {
        int g[3];
        g[0] = (int)floor((xa.x - B.origo[0]) / (B.L[0] / B.num[0]));
        g[1] = (int)floor((xa.y - B.origo[1]) / (B.L[1] / B.num[1]));
        g[2] = (int)floor((xa.z - B.origo[2]) / (B.L[2] / B.num[2]));
        const bool inner = g[0] >= 1 && g[0] < nx - 1;
        for (int oz = -1; oz < 2; ++oz)
            for (int oy = -1; oy < 2; ++oy)
                for (int ox = inner ? 0 : -1; ox < (inner ? 1 : 2); ++ox) {
                    int tx = g[0] + ox, ty = g[1] + oy, sx, sy;
                    if (!image_cell(B, tx, ty, g[2] + oz, sx, sy)) continue;
                    const uint32_t cell = B.cell_base + (uint32_t)(tx + ty * nx + (nx * ny) * (g[2] + oz));
                    // inner: the row's three cells at once
                    range(A.cell_off[inner ? cell - 1u : cell], A.cell_off[cell + (inner ? 2u : 1u)], sx, sy);
                }
        push_apart();
        const double below = (B.origo[2] + xa.w) - xa.z;
        if (below > 0.0) { dz += below; worst = fmax(worst, below); }
        const double above = xa.z + xa.w - z_top;
        if (above > 0.0) { dz -= above; worst = fmax(worst, above); }
        if (B.periodic == 0) {   // side walls along x
            const double lo = (B.origo[0] + xa.w) - xa.x, hi = xa.x + xa.w - B.L[0];
            if (lo > 0.0) { dx += lo; worst = fmax(worst, lo); }
            if (hi > 0.0) { dx -= hi; worst = fmax(worst, hi); }
        }
        if (B.periodic != 1) {   // side walls along y
            const double lo = (B.origo[1] + xa.w) - xa.y, hi = xa.y + xa.w - B.L[1];
            if (lo > 0.0) { dy += lo; worst = fmax(worst, lo); }
            if (hi > 0.0) { dy -= hi; worst = fmax(worst, hi); }
        }
    }
    double4 x = xa;
    x.x += dx;
    x.y += dy;
    x.z += dz;
    if (B.periodic == 1 || B.periodic == 2) {
        if (x.x < B.origo[0]) x.x += B.L[0] - B.origo[0];
        if (x.x >= B.L[0]) x.x -= B.L[0] - B.origo[0];
    }
    if (B.periodic == 1) {
        if (x.y < B.origo[1]) x.y += B.L[1] - B.origo[1];
        if (x.y >= B.L[1]) x.y -= B.L[1] - B.origo[1];
    }
    x.x = fmin(fmax(x.x, B.origo[0]), B.L[0] * (1.0 - 1e-12));
    x.y = fmin(fmax(x.y, B.origo[1]), B.L[1] * (1.0 - 1e-12));
    x.z = fmin(fmax(x.z, B.origo[2]), B.L[2] * (1.0 - 1e-12));
    if (valid) A.x[i] = x;
    // the block's largest overlap (the patterns of non-negative doubles
    // order as the values)
    unsigned long long w = (unsigned long long)__double_as_longlong(worst);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long v = __shfl_xor_sync(0xffffffffu, w, o);
        w = v > w ? v : w;
    }
    if ((threadIdx.x & 31u) == 0) s_max[threadIdx.x >> 5] = w;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < RELAX_THREADS / 32; ++k) w = s_max[k] > w ? s_max[k] : w;
        if (w) atomicMax(max_ov, w);
    }
    if (next) hash_sphere(A, B, i, x, valid);
}

// `sweeps` sweeps on st: the first sort's cells from the positions, the
// others' from the sweep before.
int relax_sweeps(const StepArgs &A, cudaStream_t st, uint32_t sweeps, double alpha, double z_top,
                 unsigned long long *d_max, uint64_t *launches)
{
    const uint32_t nb = blocks_for(A.ncells, SCAN_TILE);
    for (uint32_t k = 0; k < sweeps; ++k) {
        const bool next = k + 1 < sweeps;
        if (k == 0) {
            cudaMemsetAsync(A.cell_count, 0, sizeof(uint32_t) * A.ncells, st);
            k_hash<<<blocks_for(A.ntot, 256), 256, 0, st>>>(A);
        }
        k_scan_reduce<<<nb, SCAN_THREADS, 0, st>>>(A.cell_count, A.ncells, A.scan_tmp);
        k_scan_top<<<1, SCAN_THREADS, 0, st>>>(A.scan_tmp, nb);
        k_scan_down<<<nb, SCAN_THREADS, 0, st>>>(A.cell_count, A.ncells, A.scan_tmp, nb, A.cell_off);
        k_scatter<<<blocks_for(A.ntot, 256), 256, 0, st>>>(A);
        k_place<false><<<blocks_for(A.ntot, 256), 256, 0, st>>>(A);
        cudaMemsetAsync(d_max, 0, sizeof(unsigned long long), st);
        if (next) cudaMemsetAsync(A.cell_count, 0, sizeof(uint32_t) * A.ncells, st);
        k_relax<<<blocks_for(A.ntot, RELAX_THREADS), RELAX_THREADS, 0, st>>>(A, alpha, z_top, d_max, next);
        if (launches) *launches += k == 0 ? 7 : 6;
    }
    return cudaGetLastError() == cudaSuccess ? SPH_OK : SPH_ERR_CUDA;
}

// ---------------------------------------------------------------- analysis

// src/sphere.cpp:487-606 DEM::porosity, one block per slab.  The slab's
// void volume is the reference's sequential subtraction over the spheres in
// index order (one or two subtractions per sphere that reaches into the
// slab, none otherwise, src/sphere.cpp:520-587), so that the profile is the
// reference's, operation for operation.  That chain of dependent
// subtractions is the bound, and nothing else should lie on it: the producer
// warps compute the terms of POR_TILE spheres at a time and pack them, in
// index order, into one half of a shared buffer while one thread of the
// consumer warp subtracts the other half from the sum.
constexpr int POR_PRODUCERS = 512;
constexpr int POR_TILE = 2 * POR_PRODUCERS;      // two consecutive spheres per producer
constexpr int POR_THREADS = POR_PRODUCERS + 32;

// The terms of a sphere at height zc with radius r in [z_low, z_high]; their
// number (0 to 2).
__device__ __forceinline__ int porosity_terms(double zc, double r, double z_low, double z_high,
                                              double &t0, double &t1)
{
    const double zl = zc - r, zh = zc + r;
    // every term below needs a bound of the slab in [zl, zh], or the sphere
    // between the bounds
    if (zh < z_low || zl > z_high) return 0;
    const double V_s = 4.0 / 3.0 * M_PI * r * r * r;
    if (z_low <= zl && zh <= z_high) {
        t0 = V_s;
        return 1;
    }
    int n = 0;
    if (z_low >= zc && z_low <= zh) {
        const double h = zh - z_low;
        t0 = M_PI * h * h / 3.0 * (3.0 * r - h);
        n = 1;
    } else if (z_low < zc && z_low > zl) {
        const double h = z_low - zl;
        t0 = V_s + M_PI * h * h / 3.0 * (3.0 * r - h);
        n = 1;
    }
    double tb = 0.0;
    bool hb = false;
    if (z_high <= zc && z_high >= zl) {
        const double h = z_high - zl;
        tb = M_PI * h * h / 3.0 * (3.0 * r - h);
        hb = true;
    } else if (z_high > zc && z_high < zh) {
        const double h = zh - z_high;
        tb = V_s + M_PI * h * h / 3.0 * (3.0 * r - h);
        hb = true;
    }
    if (hb) {
        if (n == 0) t0 = tb;
        else t1 = tb;
        ++n;
    }
    return n;
}

__global__ void __launch_bounds__(POR_THREADS) k_porosity(const double4 *x, uint32_t p0,
                                                          uint32_t np, double h_slice,
                                                          double V_slice, uint32_t nslices,
                                                          double *z_pos, double *por)
{
    __shared__ double s_t[2][2 * POR_TILE];
    __shared__ int s_n[2], s_warp[POR_PRODUCERS / 32];
    const uint32_t iz = blockIdx.x;
    const double z_low = (double)iz * h_slice;
    const double z_high = z_low + h_slice;
    const uint32_t tiles = (np + POR_TILE - 1) / POR_TILE;
    const bool producer = threadIdx.x < POR_PRODUCERS;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    double V_void = V_slice;
    // height and radius of the producer's two spheres of the next tile,
    // loaded one tile ahead
    double2 q[2];
    auto load = [&](uint32_t tile) {
        const uint32_t i = tile * POR_TILE + 2u * threadIdx.x;
#pragma unroll
        for (int j = 0; j < 2; ++j)
            q[j] = i + j < np ? reinterpret_cast<const double2 *>(x + p0 + i + j)[1] : make_double2(0.0, 0.0);
    };
    if (producer && tiles) load(0);
    for (uint32_t tile = 0; tile <= tiles; ++tile) {
        if (producer && tile < tiles) {
            const uint32_t i = tile * POR_TILE + 2u * threadIdx.x;
            double t[4];
            int n0 = 0, n1 = 0;
            if (i < np) n0 = porosity_terms(q[0].x, q[0].y, z_low, z_high, t[0], t[1]);
            if (i + 1 < np) n1 = porosity_terms(q[1].x, q[1].y, z_low, z_high, t[2], t[3]);
            if (tile + 1 < tiles) load(tile + 1);
            int incl = n0 + n1;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= (uint32_t)o) incl += v;
            }
            if (lane == 31) s_warp[warp] = incl;
            asm volatile("bar.sync 1, %0;" ::"n"(POR_PRODUCERS) : "memory");
            int at = incl - n0 - n1, total = 0;
#pragma unroll
            for (int w = 0; w < POR_PRODUCERS / 32; ++w) {
                const int v = s_warp[w];
                if (w < (int)warp) at += v;
                total += v;
            }
            double *out = s_t[tile & 1u];
            if (n0 > 0) out[at++] = t[0];
            if (n0 > 1) out[at++] = t[1];
            if (n1 > 0) out[at++] = t[2];
            if (n1 > 1) out[at++] = t[3];
            if (threadIdx.x == 0) s_n[tile & 1u] = total;
        }
        if (threadIdx.x == POR_PRODUCERS && tile > 0) {
            const double *in = s_t[(tile - 1) & 1u];
            const int n = s_n[(tile - 1) & 1u];
            int k = 0;
            for (; k + 16 <= n; k += 16) {
                double v[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = in[k + j];
#pragma unroll
                for (int j = 0; j < 16; ++j) V_void -= v[j];
            }
            for (; k < n; ++k) V_void -= in[k];
        }
        __syncthreads();
    }
    if (threadIdx.x == POR_PRODUCERS && iz < nslices) {
        z_pos[iz] = z_low + 0.5 * h_slice;
        por[iz] = V_void / V_slice;
    }
}

int porosity_profile(const double4 *x, uint32_t p0, uint32_t np, double h_slice, double V_slice,
                     uint32_t nslices, double *z_pos, double *por, cudaStream_t st)
{
    k_porosity<<<nslices, POR_THREADS, 0, st>>>(x, p0, np, h_slice, V_slice, nslices, z_pos, por);
    return cudaGetLastError() == cudaSuccess ? SPH_OK : SPH_ERR_CUDA;
}

// src/sphere.cpp:677-725 DEM::findOverlaps on the device: the box's spheres
// binned into its own grid (clamped cells), each sphere i testing the
// spheres j > i in the cells within +-R (no periodic images), first
// counting, then writing its pairs in ascending j after an exclusive scan
// of the counts, so that the list is the reference's, in its order.

__device__ __forceinline__ void ov_cell(const OverlapArgs &O, double4 p, int c[3])
{
    const double v[3] = {p.x, p.y, p.z};
    for (int d = 0; d < 3; ++d) {
        double f = floor((v[d] - O.origo[d]) / O.cw[d]);
        if (!(f >= 0.0)) f = 0.0;
        if (f > (double)(O.num[d] - 1)) f = (double)(O.num[d] - 1);
        c[d] = (int)f;
    }
}

__global__ void k_ov_bin(OverlapArgs O)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= O.np) return;
    int c[3];
    ov_cell(O, O.x[O.p0 + i], c);
    const uint32_t cell = (uint32_t)((c[2] * O.num[1] + c[1]) * O.num[0] + c[0]);
    O.cell_of[i] = cell;
    O.slot[i] = atomicAdd(&O.count[cell], 1u);
}

__global__ void k_ov_scatter(OverlapArgs O)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= O.np) return;
    const uint32_t q = O.coff[O.cell_of[i]] + O.slot[i];
    O.items[q] = i;
    O.xs[q] = O.x[O.p0 + i];
}

// One thread per sphere in cell order (its candidates are then its warp's
// too); WRITE = false: count the pairs of sphere i; true: write them sorted
// by j.  The cells of a row are neighbours in the cell order, so each row of
// the search block is one range.  Most candidates are far apart: the squared
// distance against a bound just above (ri + rj)^2 drops those before the
// square root, and never drops an overlapping pair (the root and the sum
// each round by less than 2^-52).
template <bool WRITE>
__global__ void k_ov_pairs(OverlapArgs O)
{
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= O.np) return;
    const uint32_t i = O.items[p];
    const double4 xi = O.xs[p];
    const uint32_t cnt = WRITE ? O.npair[i] : 0u;
    if (WRITE && cnt == 0u) return;
    const bool free_i = O.vel[O.p0 + i].w == 0.0;
    int c[3];
    ov_cell(O, xi, c);
    uint32_t n = 0;
    const uint32_t base = WRITE ? O.poff[i] : 0u;
    const int x0 = max(c[0] - O.R, 0), x1 = min(c[0] + O.R, O.num[0] - 1);
    for (int dz = -O.R; dz <= O.R && free_i; ++dz)
        for (int dy = -O.R; dy <= O.R; ++dy) {
            const int ty = c[1] + dy, tz = c[2] + dz;
            if (ty < 0 || tz < 0 || ty >= O.num[1] || tz >= O.num[2]) continue;
            const uint32_t row = (uint32_t)((tz * O.num[1] + ty) * O.num[0]);
            const uint32_t q1 = O.coff[row + (uint32_t)x1 + 1u];
            for (uint32_t q = O.coff[row + (uint32_t)x0]; q < q1; ++q) {
                const double4 xj = O.xs[q];
                const double ddx = xj.x - xi.x, ddy = xj.y - xi.y, ddz = xj.z - xi.z;
                const double d2 = ddx * ddx + ddy * ddy + ddz * ddz, rr = xi.w + xj.w;
                if (d2 > rr * rr * (1.0 + 1e-12)) continue;
                const uint32_t j = O.items[q];
                if (j <= i) continue;
                const double len = sqrt(d2);
                const double d = len - rr;
                if (!(d < 0.0 && O.vel[O.p0 + j].w == 0.0)) continue;
                if (WRITE && n < cnt) {
                    // insertion by j into this sphere's part of the list
                    uint32_t k = n;
                    while (k > 0 && O.pairs[2 * (size_t)(base + k - 1) + 1] > j) {
                        O.pairs[2 * (size_t)(base + k)] = O.pairs[2 * (size_t)(base + k - 1)];
                        O.pairs[2 * (size_t)(base + k) + 1] = O.pairs[2 * (size_t)(base + k - 1) + 1];
                        O.delta[base + k] = O.delta[base + k - 1];
                        --k;
                    }
                    O.pairs[2 * (size_t)(base + k)] = i;
                    O.pairs[2 * (size_t)(base + k) + 1] = j;
                    O.delta[base + k] = d;
                }
                ++n;
            }
        }
    if (!WRITE) O.npair[i] = n;
}

int find_overlaps(OverlapArgs O, uint32_t ncells, uint32_t *scan_tmp, cudaStream_t st,
                  int stage)
{
    const unsigned gb = blocks_for(O.np, 256);
    if (stage == 0) {
        cudaMemsetAsync(O.count, 0, sizeof(uint32_t) * ncells, st);
        k_ov_bin<<<gb, 256, 0, st>>>(O);
        const uint32_t nb = blocks_for(ncells, SCAN_TILE);
        k_scan_reduce<<<nb, SCAN_THREADS, 0, st>>>(O.count, ncells, scan_tmp);
        k_scan_top<<<1, SCAN_THREADS, 0, st>>>(scan_tmp, nb);
        k_scan_down<<<nb, SCAN_THREADS, 0, st>>>(O.count, ncells, scan_tmp, nb, O.coff);
        k_ov_scatter<<<gb, 256, 0, st>>>(O);
        k_ov_pairs<false><<<gb, 256, 0, st>>>(O);
        const uint32_t np_b = blocks_for(O.np, SCAN_TILE);
        k_scan_reduce<<<np_b, SCAN_THREADS, 0, st>>>(O.npair, O.np, scan_tmp);
        k_scan_top<<<1, SCAN_THREADS, 0, st>>>(scan_tmp, np_b);
        k_scan_down<<<np_b, SCAN_THREADS, 0, st>>>(O.npair, O.np, scan_tmp, np_b, O.poff);
    } else {
        k_ov_pairs<true><<<gb, 256, 0, st>>>(O);
    }
    return cudaGetLastError() == cudaSuccess ? SPH_OK : SPH_ERR_CUDA;
}

// Live directed contacts (non-empty slots), for the roofline byte count.
__global__ void k_count_live(const uint32_t *slots, uint64_t nslots, unsigned long long *count)
{
    unsigned long long c = 0;
    for (uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; q < nslots;
         q += (uint64_t)gridDim.x * blockDim.x)
        c += slots[q] != EMPTY;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, c);
}

int count_live_slots(const StepArgs &A, cudaStream_t st, unsigned long long *d_count,
                     uint64_t *launches)
{
    cudaMemsetAsync(d_count, 0, sizeof(unsigned long long), st);
    k_count_live<<<4 * 148, 256, 0, st>>>(A.slots, (uint64_t)A.ntot * NC, d_count);
    if (launches) *launches += 1;
    return cudaGetLastError() == cudaSuccess ? SPH_OK : SPH_ERR_CUDA;
}

// ------------------------------------------------------------------ launch

// Record a profiling event on st.  Under stream capture the record must be
// external, or it only orders the capture and is never timed.
static inline void record(cudaEvent_t ev, cudaStream_t st)
{
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(st, &cs);
    if (cs == cudaStreamCaptureStatusActive) cudaEventRecordWithFlags(ev, st, cudaEventRecordExternal);
    else cudaEventRecord(ev, st);
}

static inline void mark(Prof *prof, cudaStream_t st, const char *name)
{
    if (!prof || prof->n >= Prof::MAX) return;
    prof->name[prof->n] = name;
    record(prof->ev[prof->n + 1], st);
    prof->n++;
}

// FP64 interact launcher (bit-exact form).
static void interact_fp64(const StepArgs &A, cudaStream_t st, unsigned grid, bool fused, int lm,
                          int variant)
{
    launch_interact<false>(A, st, grid, fused, lm, variant);
}

static void contacts_fp64(const StepArgs &A, const StepConfig &cfg, cudaStream_t st, unsigned grid,
                          bool pdl)
{
    launch_contacts<false>(A, cfg, st, grid, pdl);
}

// The cell counts and each sphere's place in its cell from the cell ids.
__global__ void k_recount(StepArgs A)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < A.ntot) A.local_off[i] = atomicAdd(&A.cell_count[A.cell_id[i]], 1u);
}

void scan_counts(const uint32_t *in, uint64_t n, uint32_t *tmp, uint32_t *off, cudaStream_t st)
{
    const uint32_t nb = blocks_for(n, SCAN_TILE);
    k_scan_reduce<<<nb, SCAN_THREADS, 0, st>>>(in, n, tmp);
    k_scan_top<<<1, SCAN_THREADS, 0, st>>>(tmp, nb);
    k_scan_down<<<nb, SCAN_THREADS, 0, st>>>(in, n, tmp, nb, off);
}

// The sorted order (cell_off, perm, rank) of the cell ids in A.cell_id; the
// sorted copies get the current positions.
int sort_from_ids(const StepArgs &A, cudaStream_t st)
{
    cudaMemsetAsync(A.cell_count, 0, sizeof(uint32_t) * A.ncells, st);
    k_recount<<<blocks_for(A.ntot, 256), 256, 0, st>>>(A);
    scan_counts(A.cell_count, A.ncells, A.scan_tmp, A.cell_off, st);
    k_scatter<<<blocks_for(A.ntot, 256), 256, 0, st>>>(A);
    k_place<false><<<blocks_for(A.ntot, 256), 256, 0, st>>>(A);
    return cudaGetLastError() == cudaSuccess ? SPH_OK : SPH_ERR_CUDA;
}

int launch_step(const StepArgs &A, const StepConfig &cfg, cudaStream_t st, uint64_t *launches,
                Prof *prof)
{
    return launch_step_with(A, cfg, st, launches, prof, interact_fp64, contacts_fp64);
}

int launch_step_with(const StepArgs &args, const StepConfig &cfg, cudaStream_t st,
                     uint64_t *launches, Prof *prof, InteractLauncher interact,
                     ContactLauncher contact)
{
    StepArgs A = args;
    A.lazy_sort = cfg.lazy_sort && split_active(A, cfg) ? 1u : 0u;
    A.touch = A.lazy_sort && cfg.touch ? 1u : 0u;
    uint64_t nl = 0;
    // programmatic dependent launches along the step's chain of kernels,
    // except where events are recorded between them (profiling)
    const bool pdl = prof == nullptr;
    if (prof) {
        prof->n = 0;
        record(prof->ev[0], st);
    }
    // the wall stage: wall-force partial sums and integrateWalls, time and
    // box state (integration.cuh:309-450, device.cu:2504-2537)
    auto wall_stage = [&](cudaStream_t s) {
        if (A.ntot > 0 && cfg.any_walls) {
            k_block_sums<<<A.npartials, 256, 0, s>>>(A, A.wf_pp, A.wall_partial, 0);
            mark(prof, s, "k_block_sums");
            nl += 1;
        }
        k_box_step<<<A.nboxes, BOX_THREADS, 0, s>>>(A);
        mark(prof, s, "k_box_step");
        nl += 1;
    };
    if (cfg.phase == STEP_TAIL) {
        wall_stage(st);
        if (launches) *launches += nl;
        return cudaGetLastError() == cudaSuccess ? SPH_OK : SPH_ERR_CUDA;
    }
    const bool overlap = cfg.phase == STEP_OVERLAP;
    if (overlap) {
        cudaEventRecord(cfg.fork, st);
        cudaStreamWaitEvent(cfg.side, cfg.fork, 0);
        wall_stage(cfg.side);
        cudaEventRecord(cfg.join, cfg.side);
    }
    if (A.ntot > 0) {
        const bool split = split_active(A, cfg);
        if (A.lazy_sort) {
            launch_resort<k_resort>(A.ntot, st, A, resort_sync(A, cfg));
            mark(prof, st, "k_resort");
            nl += 1;
        } else {
            cudaMemsetAsync(A.cell_count, 0, sizeof(uint32_t) * A.ncells, st);
            k_hash<<<blocks_for(A.ntot, 256), 256, 0, st>>>(A);
            mark(prof, st, "k_hash");
            const uint32_t nb = blocks_for(A.ncells, SCAN_TILE);
            launch_k(pdl, k_scan_reduce, nb, SCAN_THREADS, st, (const uint32_t *)A.cell_count,
                     A.ncells, A.scan_tmp);
            launch_k(pdl, k_scan_top, 1, SCAN_THREADS, st, A.scan_tmp, nb);
            launch_k(pdl, k_scan_down, nb, SCAN_THREADS, st, (const uint32_t *)A.cell_count, A.ncells,
                     (const uint32_t *)A.scan_tmp, nb, A.cell_off);
            mark(prof, st, "k_scan(3)");
            launch_k(pdl, k_scatter, blocks_for(A.ntot, 256), 256, st, A);
            mark(prof, st, "k_scatter");
            if (split) launch_k(pdl, k_place<false>, blocks_for(A.ntot, 256), 256, st, A);
            else launch_k(pdl, k_place<true>, blocks_for(A.ntot, 256), 256, st, A);
            mark(prof, st, "k_place");
            nl += 7;
            if (A.vlist) {
                const unsigned gv = blocks_for(A.ntot, VLIST_THREADS);
                launch_k(pdl, k_vlist_build, gv < VLIST_BLOCKS ? gv : VLIST_BLOCKS, VLIST_THREADS, st, A);
                launch_k(pdl, k_vlist_done, 1, 1, st, A);
                mark(prof, st, "k_vlist");
                nl += 2;
            }
        }
        if (A.nbonds) {
            if (cfg.lenmode == SPH_LEN_FP64) k_bonds<SPH_LEN_FP64><<<blocks_for(A.nbonds, 128), 128, 0, st>>>(A);
            else k_bonds<SPH_LEN_REFERENCE><<<blocks_for(A.nbonds, 128), 128, 0, st>>>(A);
            mark(prof, st, "k_bonds");
            nl += 1;
        }
        const unsigned gi = blocks_for(A.ntot, INTERACT_THREADS);
        if (split) {
            const unsigned gs = blocks_for(A.ntot, SEARCH_THREADS);
            // after k_bonds (when there are bonds) an ordinary launch
            const bool pdl_s = pdl && !A.nbonds;
            if (!A.touch) {
                if (cfg.lenmode == SPH_LEN_FP64)
                    launch_k(pdl_s, k_search<SPH_LEN_FP64>, gs, SEARCH_THREADS, st, A);
                else
                    launch_k(pdl_s, k_search<SPH_LEN_REFERENCE>, gs, SEARCH_THREADS, st, A);
                mark(prof, st, "k_search");
                nl += 1;
            }
            contact(A, cfg, st, blocks_for(A.ntot, CONTACT_THREADS), A.touch ? pdl_s : pdl);
            mark(prof, st, A.touch ? "k_touch" : "k_contacts");
            if (overlap) cudaStreamWaitEvent(st, cfg.join, 0);
            const unsigned gf = blocks_for(A.ntot, FINISH_THREADS);
            const bool lm64 = cfg.lenmode == SPH_LEN_FP64;
            if (cfg.box0) {
                const BoxConst C = box_const(*cfg.box0);
                if (lm64) k_finish1<SPH_LEN_FP64><<<gf, FINISH_THREADS, 0, st>>>(A, C);
                else k_finish1<SPH_LEN_REFERENCE><<<gf, FINISH_THREADS, 0, st>>>(A, C);
            } else {
                if (lm64) k_finish<SPH_LEN_FP64><<<gf, FINISH_THREADS, 0, st>>>(A);
                else k_finish<SPH_LEN_REFERENCE><<<gf, FINISH_THREADS, 0, st>>>(A);
            }
            mark(prof, st, "k_finish");
            nl += 2;
        } else if (!cfg.unfused) {
            if (overlap) cudaStreamWaitEvent(st, cfg.join, 0);
            interact(A, st, gi, true, cfg.lenmode,
                     cfg.variant == SPLIT_VARIANT ? 1 : cfg.variant);
            mark(prof, st, "k_interact");
            nl += 1;
        } else {
            if (overlap) cudaStreamWaitEvent(st, cfg.join, 0);
            interact(A, st, gi, false, cfg.lenmode,
                     cfg.variant == SPLIT_VARIANT ? 1 : cfg.variant);
            mark(prof, st, "k_interact");
            if (cfg.darcy) {
                // device.cu:1891-2419, between interact and integrate
                const int ds = launch_darcy(A, *cfg.darcy, cfg, st, &nl, prof);
                if (ds != SPH_OK) return ds;
            }
            k_shear_stress<<<blocks_for(A.ntot, 256), 256, 0, st>>>(A);
            k_block_sums<<<A.npartials, 256, 0, st>>>(A, A.tau_pp, A.tau_partial, 1);
            k_tau_final<<<A.nboxes, BOX_THREADS, 0, st>>>(A);
            mark(prof, st, "k_shear_stress+sums");
            k_integrate<<<blocks_for(A.ntot, 256), 256, 0, st>>>(A);
            mark(prof, st, "k_integrate");
            nl += 5;
        }
    } else if (overlap) {
        cudaStreamWaitEvent(st, cfg.join, 0);
    }
    if (A.ntot == 0 && cfg.darcy) {
        // a fluid without spheres (the reference's pure-fluid runs)
        const int ds = launch_darcy(A, *cfg.darcy, cfg, st, &nl, prof);
        if (ds != SPH_OK) return ds;
    }
    if (cfg.phase == STEP_WHOLE) wall_stage(st);
    if (cfg.darcy) {
        launch_darcy_tick(A, *cfg.darcy, st);
        nl += 1;
    }
    if (launches) *launches += nl;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        fprintf(stderr, "sphere_b200: kernel launch failed: %s\n", cudaGetErrorString(e));
        return SPH_ERR_CUDA;
    }
    return SPH_OK;
}

}  // namespace sph
