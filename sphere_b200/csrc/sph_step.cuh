// sph_step.cuh -- the fused per-sphere step kernel (topology, interact,
// walls, bond forces, TY3 integration) shared by the FP64 step
// (sph_kernels.cu, no FMA contraction) and the FP32-mixed step
// (sph_mixed.cu).
#pragma once

#include <cstdint>

#include "sph_device.cuh"
#include "sph_internal.h"
#include "sph_mixed_laws.cuh"

namespace sph {

// Conservative FP32 candidate test: false only when the pair certainly does
// not satisfy the exact FP64 test `length - (ra + rb) < extra` (extra = 0
// for contacts, db for capillary bonds).  B.pre_margin bounds the rounding
// of the FP32 copies, differences, periodic shifts and of the reference's
// FP32-rounded lengths (set per box by the host: 2^-19 (max L + 2 r_max)).
__device__ __forceinline__ bool maybe_touching(float4 xa, float4 xb, float sx, float sy,
                                               float margin_plus_extra)
{
    const float dx = (xa.x - xb.x) + sx, dy = (xa.y - xb.y) + sy, dz = xa.z - xb.z;
    const float rr = xa.w + xb.w + margin_plus_extra;
    return dx * dx + dy * dy + dz * dz < rr * rr;
}

// Box of sphere i; a single box needs no lookup (one dependent load fewer
// on the way to the box's parameters).
__device__ __forceinline__ uint32_t box_index(const StepArgs &A, uint32_t i)
{
    return A.nboxes == 1 ? 0u : A.box_of[i];
}

// floor((x - o) / (L / num)), the cell coordinate of sorting.cuh:7-20,
// from a product with num / L: that differs from the quotient by a few units
// in the last place, so away from an integer (by 1e-6, with |t| < 1e9) the
// floors are equal; else (and for NaN) the quotient itself.
__device__ __forceinline__ double cell_rate(const DevBox &B, int d) { return (double)B.num[d] / B.L[d]; }
__device__ __forceinline__ double cell_rate(const BoxConst &C, int d) { return C.cell_rate[d]; }

template <class BX>
__device__ __forceinline__ double cell_floor(const BX &B, double x, int k)
{
    const double d = x - B.origo[k];
    const double t = d * cell_rate(B, k);
    const double f = floor(t);
    if (fabs(t) < 1e9 && fabs((t - f) - 0.5) < 0.5 - 1e-6) return f;
    return floor(d / (B.L[k] / B.num[k]));
}

// Clamped cell coordinates of a position, as the sort stores them, from its
// cell_floor values; false when some coordinate lies outside the grid.
template <class BX>
__device__ __forceinline__ bool clamp_cell(const BX &B, const double f[3], uint32_t c[3])
{
    bool inside = true;
    for (int d = 0; d < 3; ++d) {
        double v = f[d];
        if (!(v >= 0.0)) { inside = false; v = 0.0; }
        if (v >= (double)B.num[d]) { inside = false; v = (double)(B.num[d] - 1); }
        c[d] = (uint32_t)v;
    }
    return inside;
}

// ---------------------------------------------------------------- integrate

// Keeps a load where it stands: a value that is used only behind a branch is
// else loaded behind it, one memory latency after the branch's own condition.
__device__ __forceinline__ void loaded(const double4 &v)
{
    asm volatile("" ::"d"(v.x), "d"(v.y), "d"(v.z), "d"(v.w));
}

// What the end of a step reads of the sphere's own state.  Loaded in one go
// before the first store of the sphere's results: a load after a store waits
// for the loads before it, since the compiler cannot tell the arrays apart.
struct OwnState {
    double4 angpos, xyzsum, acc, angacc;
    float4 xref;
    double es, ev;
};
__device__ __forceinline__ OwnState load_own(const StepArgs &A, uint32_t i)
{
    OwnState o;
    o.angpos = A.angpos[i];
    o.xyzsum = A.xyzsum[i];
    o.acc = A.acc[i];
    o.angacc = A.angacc[i];
    o.xref = A.xref ? A.xref[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    o.es = A.es[i];
    o.ev = A.ev[i];
    return o;
}

// integration.cuh:14-305 integrate (TY3) for one particle.
// (C: the box's constants, the box itself or BoxConst.)
template <class BX>
__device__ __forceinline__ void integrate_particle(const StepArgs &A, const DevBox &B, const BX &C,
                                                   uint32_t i, const OwnState &own, double4 x,
                                                   double4 vel, double4 angvel, d3 F, d3 T)
{
    const SphParams &P = C.P;
    const double dt = C.dt;
    const double4 angpos = own.angpos;
    double4 xyzsum = own.xyzsum;
    int wall0mode = 0;
    double wall0mass = 0.0;
    if (C.nw > 0) {
        wall0mode = B.wmode[0];
        wall0mass = B.wmvfd[0][0];
    }
    double4 acc0 = make_double4(0.0, 0.0, 0.0, 0.0), angacc0 = acc0;
    if (B.iter != 0) {
        acc0 = own.acc;
        angacc0 = own.angacc;
    }
    const double radius = x.w;
    const double m = 4.0 / 3.0 * PI * radius * radius * radius * P.rho;
    double acc[3], angacc[3];
    // (twelve quotients by three divisors)
    const Divisor by_m(m), by_i(2.0 / 5.0 * m * radius * radius), by_dt = divisor_dt(C);
    acc[0] = by_m.div(F.x) + P.g[0];
    acc[1] = by_m.div(F.y) + P.g[1];
    acc[2] = by_m.div(F.z) + P.g[2];
    angacc[0] = by_i.div(T.x * 1.0);
    angacc[1] = by_i.div(T.y * 1.0);
    angacc[2] = by_i.div(T.z * 1.0);
    double angacc_w = 0.0;
    if (wall0mode == 3 && vel.w > 0.0001 && x.z > B.L[2] * 0.5) {
        const double f_tau_x = (B.tau_x + B.tau_eff_x) * C.L[0] * C.L[1];
        acc[0] = f_tau_x / wall0mass;
        acc[1] = 0.0;
        acc[2] -= P.g[2];
        angacc[0] = angacc[1] = angacc[2] = 0.0;
        angacc_w = 0.0;
    } else if (vel.w > 0.0001 && vel.w < 10.0) {
        acc[0] = 0.0;
        acc[1] = 0.0;
        acc[2] -= P.g[2];
        angacc[0] = angacc[1] = angacc[2] = 0.0;
    }
    if (vel.w >= 10.0) {
        acc[1] = 0.0;
        angacc[0] = 0.0;
        angacc[2] = 0.0;
    }
    if (vel.w < -0.0001) {
        acc[0] = acc[1] = acc[2] = 0.0;
        angacc[0] = angacc[1] = angacc[2] = 0.0;
    }
    const double a0[3] = {acc0.x, acc0.y, acc0.z};
    const double w0[3] = {angacc0.x, angacc0.y, angacc0.z};
    const double xv[3] = {x.x, x.y, x.z};
    const double vv[3] = {vel.x, vel.y, vel.z};
    const double pv[3] = {angpos.x, angpos.y, angpos.z};
    const double wv[3] = {angvel.x, angvel.y, angvel.z};
    double sv[3] = {xyzsum.x, xyzsum.y, xyzsum.z};
    double xn[3], vn[3], pn[3], wn[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double dacc = by_dt.div(acc[d] - a0[d]);
        const double dangacc = by_dt.div(angacc[d] - w0[d]);
        xn[d] = xv[d] + vv[d] * dt + 0.5 * acc[d] * dt * dt + 1.0 / 6.0 * dacc * dt * dt * dt;
        vn[d] = vv[d] + acc[d] * dt + 0.5 * dacc * dt * dt;
        pn[d] = pv[d] + wv[d] * dt + 0.5 * angacc[d] * dt * dt + 1.0 / 6.0 * dangacc * dt * dt * dt;
        wn[d] = wv[d] + angacc[d] * dt + 0.5 * dangacc * dt * dt;
        sv[d] += vv[d] * dt + 0.5 * acc[d] * dt * dt + 1.0 / 6.0 * dacc * dt * dt * dt;
    }
    if (C.periodic == 1) {
        if (xn[0] < C.origo[0]) xn[0] += C.L[0];
        if (xn[0] > C.L[0]) xn[0] -= C.L[0];
        if (xn[1] < C.origo[1]) xn[1] += C.L[1];
        if (xn[1] > C.L[1]) xn[1] -= C.L[1];
    } else if (C.periodic == 2) {
        if (xn[0] < C.origo[0]) xn[0] += C.L[0];
        if (xn[0] > C.L[0]) xn[0] -= C.L[0];
    }
    if (A.xref) {
        // neighbour-list validity: displacement since the list build
        // (nearest periodic image), FP32
        const float4 r = own.xref;
        float ex = (float)xn[0] - r.x, ey = (float)xn[1] - r.y;
        const float ez = (float)xn[2] - r.z;
        if (C.periodic == 1 || C.periodic == 2) {
            const float lx = (float)C.L[0];
            if (ex > 0.5f * lx) ex -= lx;
            else if (ex < -0.5f * lx) ex += lx;
        }
        if (C.periodic == 1) {
            const float ly = (float)C.L[1];
            if (ey > 0.5f * ly) ey -= ly;
            else if (ey < -0.5f * ly) ey += ly;
        }
        if (!(ex * ex + ey * ey + ez * ez <= B.vdisp2)) A.vflag[0] = 1u;
    }
    if (A.lazy_sort) {
        // the next step's contact search reads the spheres' cells
        double f[3];
        uint32_t c[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) f[d] = cell_floor(C, xn[d], d);
        (void)clamp_cell(C, f, c);
        A.cellc[i] = pack_cell(c[0], c[1], c[2]);
    }
    if (vel.w > 5.0 && vel.w < 10.0) {
        if (B.change_velocity_state == 1) vn[0] *= 10.0;
        else if (B.change_velocity_state == -1) vn[0] /= 10.0;
    }
    xyzsum.x = sv[0];
    xyzsum.y = sv[1];
    xyzsum.z = sv[2];
    A.xyzsum[i] = xyzsum;
    A.acc[i] = make_double4(acc[0], acc[1], acc[2], 0.0);
    A.angacc[i] = make_double4(angacc[0], angacc[1], angacc[2], angacc_w);
    A.angvel[i] = make_double4(wn[0], wn[1], wn[2], angvel.w);
    A.vel[i] = make_double4(vn[0], vn[1], vn[2], vel.w);
    A.angpos[i] = make_double4(pn[0], pn[1], pn[2], angpos.w);
    A.x[i] = make_double4(xn[0], xn[1], xn[2], x.w);
}

// A box copied to shared memory by the block and back: the one thread that
// advances it reads and writes some twenty fields, and in memory each of
// those reads waits for the write before it (k_box_step 4.5 us at 500
// spheres, 3.3 with the copy).
__device__ __forceinline__ void stage_box(DevBox &s, const DevBox &g)
{
    static_assert(sizeof(DevBox) % 8 == 0, "copied in 8-byte words");
    unsigned long long *d = reinterpret_cast<unsigned long long *>(&s);
    const unsigned long long *q = reinterpret_cast<const unsigned long long *>(&g);
    for (uint32_t k = threadIdx.x; k < sizeof(DevBox) / 8; k += blockDim.x) d[k] = q[k];
    __syncthreads();
}
__device__ __forceinline__ void unstage_box(DevBox &g, const DevBox &s)
{
    __syncthreads();
    unsigned long long *d = reinterpret_cast<unsigned long long *>(&g);
    const unsigned long long *q = reinterpret_cast<const unsigned long long *>(&s);
    for (uint32_t k = threadIdx.x; k < sizeof(DevBox) / 8; k += blockDim.x) d[k] = q[k];
}

// integration.cuh:344-450 integrateWalls with the wall-force total fsum,
// then the loop bookkeeping of device.cu:2536-2538, the adaptive grid of
// device.cu:1050 and the velocity-step state of device.cu:2455-2462 for
// the next step.  One thread per box.
__device__ __forceinline__ void advance_box(DevBox &B, double fsum)
{
    const double dt = B.dt;
    if (B.np > 0) {
        for (uint32_t w = 0; w < B.nw; ++w) {
            const int wmode = B.wmode[w];
            if (wmode == 0) continue;
            const double acc0 = B.iter == 0 ? 0.0 : B.wacc[w];
            B.wmvfd[w][2] = fsum;
            // (without modulation the product is a zero, whatever the sine)
            const double mod =
                B.P.sigma0_A == 0.0 ? 0.0 : B.P.sigma0_A * sin(2.0 * PI * B.P.sigma0_f * B.t_current);
            const double sigma_0 = B.wmvfd[w][3] + mod;
            const double N = -sigma_0 * B.L[0] * B.L[1];
            double acc = (B.wmvfd[w][2] + N) / B.wmvfd[w][0];
            if (wmode == 2) acc = 0.0;
            const double dacc_dt = (acc - acc0) / dt;
            B.wnx[w][3] += B.wmvfd[w][1] * dt + 0.5 * acc * dt * dt + 1.0 / 6.0 * dacc_dt * dt * dt * dt;
            B.wmvfd[w][1] += acc * dt + 0.5 * dacc_dt * dt * dt;
            B.wacc[w] = acc;
        }
    }
    B.t_current += dt;
    B.iter += 1;
    B.L2_out = B.L[2];
    if (B.adaptive == 1 && B.nw > 0) B.L[2] = B.wnx[0][3];
    int change = 0;
    if (B.t_current >= 10.0 && B.t_current < 15.0 && B.velocity_state == 1) {
        change = 1;
        B.velocity_state = 2;
    } else if (B.t_current >= 15.0 && B.velocity_state == 2) {
        change = -1;
        B.velocity_state = 1;
    }
    B.change_velocity_state = change;
}

// ------------------------------------------------------------------ interact

// Neighbour-list entry k of sphere a (partner id bo): the cell search visits
// the partner's cell at ordinal (dz, dy, dx) of the 27-cell loop under image
// (sx, sy), and the exact FP64 test says the pair touches.  Returns the
// insertion key (ordinal << 10 | image code << 6 | k), or NO_KEY.
constexpr uint16_t NO_KEY = 0xffffu;

template <int LM>
__device__ __forceinline__ uint16_t list_key(const StepArgs &A, const DevBox &B, double4 xa,
                                             const int g[3], uint32_t bo, uint32_t k)
{
    int bx, by, bz, dx, dy, dz, sx, sy;
    unpack_cell(A.cellc[bo], bx, by, bz);
    if (!relative_cell(B, g, bx, by, bz, dx, dy, dz, sx, sy)) return NO_KEY;
    const double4 xb = A.xs[A.rank[bo]];
    const d3 dm = shift_vec(B, sx, sy);
    d3 x_ab = mk(xa.x - xb.x, xa.y - xb.y, xa.z - xb.z);
    x_ab = vadd(x_ab, dm);
    const double len = len_rn<LM>(x_ab);
    if (!(len - (xa.w + xb.w) < 0.0)) return NO_KEY;
    const int ord = ((dz + 1) * 3 + (dy + 1)) * 3 + (dx + 1);
    return (uint16_t)((ord << 10) | (shift_code(sx, sy) << 6) | (int)k);
}

// list_key for entries k0 .. k0 + KB - 1 (those below vc), their loads
// issued together so that KB gathers are in flight at once.  For the split
// step only: the partner's position is read in original order (A.x), which
// holds the step's start positions until k_finish, one gather fewer than
// the sorted copy through rank.
constexpr int KB = 4;   // (the overflow path of k_search spells out KB entries)

// FILTER: entries whose partner already holds a slot of the row (srow[j] >=
// 0) are not tested: only their image code is brought up to date (in place,
// *dirty set when it changes); the caller uses this when the row cannot
// overflow, where such entries do not change where the new ones go.
template <int LM, bool FILTER>
__device__ __forceinline__ void list_keys_batch(const StepArgs &A, const DevBox &B, double4 xa,
                                                const int g[3], const uint32_t bo[KB], uint32_t k0,
                                                uint32_t vc, uint16_t out[KB], const int srow[KB],
                                                uint32_t *row, int RS, bool *dirty)
{
    uint64_t cc[KB];
    double4 xb[KB];
#pragma unroll
    for (int j = 0; j < KB; ++j) {
        const bool test = k0 + j < vc && (!FILTER || srow[j] < 0);
        cc[j] = k0 + j < vc ? A.cellc[bo[j]] : 0ull;
        xb[j] = test ? A.x[bo[j]] : make_double4(0.0, 0.0, 0.0, 0.0);
    }
#pragma unroll
    for (int j = 0; j < KB; ++j) {
        out[j] = NO_KEY;
        if (k0 + j >= vc) continue;
        int bx, by, bz, dx, dy, dz, sx, sy;
        unpack_cell(cc[j], bx, by, bz);
        if (!relative_cell(B, g, bx, by, bz, dx, dy, dz, sx, sy)) continue;
        if (FILTER && srow[j] >= 0) {
            const uint32_t v = bo[j] | (shift_code(sx, sy) << CODE_SHIFT);
            if (row[srow[j] * RS] != v) {
                row[srow[j] * RS] = v;
                *dirty = true;
            }
            continue;
        }
        const d3 dm = shift_vec(B, sx, sy);
        d3 x_ab = mk(xa.x - xb[j].x, xa.y - xb[j].y, xa.z - xb[j].z);
        x_ab = vadd(x_ab, dm);
        const double len = len_rn<LM>(x_ab);
        if (!(len - (xa.w + xb[j].w) < 0.0)) continue;
        const int ord = ((dz + 1) * 3 + (dy + 1)) * 3 + (dx + 1);
        out[j] = (uint16_t)((ord << 10) | (shift_code(sx, sy) << 6) | (int)(k0 + j));
    }
}

// Insert the touching list entries, keys sorted ascending (keys[q * KS]),
// into the slot row with the reference's rule: an existing contact keeps
// its slot, a new one takes the last free slot (slot nc when none is free);
// more than NC contacts raise SPH_ERR_NC_OVERFLOW and skip the rest of that
// cell, as the cell search does.  occ: bit s set when slot s is in use
// (updated).  Returns whether the row changed.
__device__ __forceinline__ bool insert_keys(const StepArgs &A, const uint16_t *keys, int nk, int KS,
                                            const uint32_t *lst, uint32_t *row, int RS,
                                            uint32_t &occ)
{
    bool dirty = false;
    int nc = 0, cur_ord = -1;
    bool full = false;
    for (int q = 0; q < nk; ++q) {
        const uint32_t key = keys[q * KS];
        const int ord = (int)(key >> 10);
        if (ord != cur_ord) {
            cur_ord = ord;
            full = false;
        }
        if (full) continue;
        const uint32_t b_orig = lst[key & 63u];
        // the partner's slot if it is in the row, else the highest free slot
        int cpos = -1;
        for (uint32_t m = occ; m; m &= m - 1u) {
            const int s = __ffs(m) - 1;
            if ((row[s * RS] & ID_MASK) == b_orig) {
                cpos = s;
                break;
            }
        }
        if (cpos < 0) cpos = ~occ ? 31 - __clz(~occ) : nc;
        if (cpos < NC) {
            // the row goes back to memory only if an entry changed
            const uint32_t v = b_orig | (((key >> 6) & 15u) << CODE_SHIFT);
            if (row[cpos * RS] != v) {
                row[cpos * RS] = v;
                dirty = true;
            }
            occ |= 1u << cpos;
        } else {
            raise_flag(A.err, SPH_ERR_NC_OVERFLOW);
        }
        ++nc;
        if (nc > NC) {
            raise_flag(A.err, SPH_ERR_NC_OVERFLOW);
            full = true;
        }
    }
    return dirty;
}

__device__ __forceinline__ uint32_t occupancy(const uint32_t *row, int RS)
{
    uint32_t occ = 0;
#pragma unroll
    for (int s = 0; s < NC; ++s) occ |= (row[s * RS] != EMPTY ? 1u : 0u) << s;
    return occ;
}

// The 27-cell contact search (contactsearch.cuh:329-371 and :194-322) on
// the slot row, for spheres without a usable neighbour list.
template <int LM>
__device__ __forceinline__ bool search_cells(const StepArgs &A, const DevBox &B, uint32_t a,
                                             double4 xa, const int g[3], float4 xaf,
                                             uint32_t *row, int RS)
{
    const double radius_a = xa.w;
    const int nx = (int)B.num[0], ny = (int)B.num[1];
    const float Lf0 = (float)B.L[0], Lf1 = (float)B.L[1];
    const float margin = B.pre_margin;
    bool dirty = false;
    int nc = 0;
    for (int dz = -1; dz < 2; ++dz)
        for (int dy = -1; dy < 2; ++dy)
            for (int dx = -1; dx < 2; ++dx) {
                int tx = g[0] + dx, ty = g[1] + dy, sx, sy;
                const int tz = g[2] + dz;
                if (!image_cell(B, tx, ty, tz, sx, sy)) continue;
                const d3 dm = shift_vec(B, sx, sy);
                const float fsx = sx == 0 ? 0.f : (sx > 0 ? Lf0 : -Lf0);
                const float fsy = sy == 0 ? 0.f : (sy > 0 ? Lf1 : -Lf1);
                const uint32_t cell = B.cell_base + (uint32_t)(tx + ty * nx + (nx * ny) * tz);
                const uint32_t start = A.cell_off[cell], end = A.cell_off[cell + 1];
                for (uint32_t b = start; b < end; ++b) {
                    if (b == a) continue;
                    if (!maybe_touching(xaf, A.xf[b], fsx, fsy, margin)) continue;
                    const double4 xb = A.xs[b];
                    d3 x_ab = mk(xa.x - xb.x, xa.y - xb.y, xa.z - xb.z);
                    x_ab = vadd(x_ab, dm);
                    const double len = len_rn<LM>(x_ab);
                    const double delta = len - (radius_a + xb.w);
                    if (delta < 0.0) {
                        const uint32_t b_orig = A.perm[b];
                        int cpos = nc;
                        for (int s = 0; s < NC; ++s) {
                            const uint32_t w = row[s * RS];
                            if (w == EMPTY) cpos = s;
                            else if ((w & ID_MASK) == b_orig) { cpos = s; break; }
                        }
                        if (cpos < NC) {
                            const uint32_t v = b_orig | (shift_code(sx, sy) << CODE_SHIFT);
                            if (row[cpos * RS] != v) {
                                row[cpos * RS] = v;
                                dirty = true;
                            }
                        } else {
                            raise_flag(A.err, SPH_ERR_NC_OVERFLOW);
                        }
                        ++nc;
                        if (nc > NC) {
                            raise_flag(A.err, SPH_ERR_NC_OVERFLOW);
                            break;
                        }
                    }
                }
            }
    return dirty;
}

// The contact search of one sphere (contact models 2 and 3) on its slot row
// staged in shared memory (row[s * RS]), one thread: from the neighbour list
// when the sphere has one (the touching entries keyed and inserted in the
// order the cell search would find them), else the 27-cell search.  keys:
// shared scratch of VL_MAX entries at stride RS.  Returns whether the row
// changed.
template <int LM>
__device__ __forceinline__ bool search_contacts(const StepArgs &A, const DevBox &B, uint32_t a,
                                                uint32_t i, double4 xa, const int g[3],
                                                float4 xaf, uint32_t *row, uint16_t *keys,
                                                int RS)
{
    const uint32_t vc = A.vlist ? A.vcount[i] : (uint32_t)VL_MAX + 1u;
    if (vc > (uint32_t)VL_MAX) return search_cells<LM>(A, B, a, xa, g, xaf, row, RS);
    const uint32_t *lst = A.vlist + (size_t)i * VL_MAX;
    int nk = 0;
    for (uint32_t k = 0; k < vc; ++k) {
        const uint16_t key = list_key<LM>(A, B, xa, g, lst[k], k);
        if (key == NO_KEY) continue;
        int q = nk;
        while (q > 0 && keys[(q - 1) * RS] > key) {
            keys[q * RS] = keys[(q - 1) * RS];
            --q;
        }
        keys[q * RS] = key;
        ++nk;
    }
    uint32_t occ = occupancy(row, RS);
    return insert_keys(A, keys, nk, RS, lst, row, RS, occ);
}

// Static and dynamic walls (contactsearch.cuh:428-465 and :602-701) and the
// bond forces in ascending bond order (cohesion.cuh:220-226), added to acc
// after the contacts.  Returns the normal force on wall 0.
template <int LM, class BX>
__device__ __forceinline__ double walls_and_bonds(const StepArgs &A, const DevBox &B, const BX &C,
                                                  uint32_t i,
                                                  double4 xa, d3 vel_a, d3 angvel_a, Acc &acc)
{
    const SphParams &P = C.P;
    const double dt = C.dt;
    const double radius_a = xa.w;
    // wall w is the box's wall w when w < nw, else the default plane (top at
    // L[2], sides at 0 and L); read where it is used
    const uint32_t nw = C.nw;
    auto plane = [&](uint32_t w, double dx, double dy, double dz, double dpos, d3 &n, double &pos,
                     double &vel) {
        if (w < nw) {
            n = mk(B.wnx[w][0], B.wnx[w][1], B.wnx[w][2]);
            pos = B.wnx[w][3];
            vel = B.wmvfd[w][1];
        } else {
            n = mk(dx, dy, dz);
            pos = dpos;
            vel = 0.0;
        }
    };
    double w0_force = 0.0;
    {
        d3 n;
        double pos, wv;
        plane(0, 0.0, 0.0, -1.0, B.L[2], n, pos, wv);
        double delta_w = pos - (xa.z + radius_a);
        if (delta_w < 0.0)
            w0_force = contact_linear_wall<LM>(P, dt, acc, vel_a, angvel_a, radius_a, n, delta_w, wv);
        delta_w = xa.z - radius_a - C.origo[2];
        if (delta_w < 0.0)
            (void)contact_linear_wall<LM>(P, dt, acc, vel_a, angvel_a, radius_a, mk(0.0, 0.0, 1.0),
                                          delta_w, 0.0);
        if (C.periodic == 0) {
            plane(1, -1.0, 0.0, 0.0, C.L[0], n, pos, wv);
            delta_w = pos - (xa.x + radius_a);
            if (delta_w < 0.0)
                (void)contact_linear_wall<LM>(P, dt, acc, vel_a, angvel_a, radius_a, n, delta_w, wv);
            plane(2, 1.0, 0.0, 0.0, 0.0, n, pos, wv);
            delta_w = xa.x - radius_a - pos;
            if (delta_w < 0.0)
                (void)contact_linear_wall<LM>(P, dt, acc, vel_a, angvel_a, radius_a, n, delta_w, wv);
        }
        if (C.periodic == 0 || C.periodic == 2) {
            plane(3, 0.0, -1.0, 0.0, C.L[1], n, pos, wv);
            delta_w = pos - (xa.y + radius_a);
            if (delta_w < 0.0)
                (void)contact_linear_wall<LM>(P, dt, acc, vel_a, angvel_a, radius_a, n, delta_w, wv);
            plane(4, 0.0, 1.0, 0.0, 0.0, n, pos, wv);
            delta_w = xa.y - radius_a - pos;
            if (delta_w < 0.0)
                (void)contact_linear_wall<LM>(P, dt, acc, vel_a, angvel_a, radius_a, n, delta_w, wv);
        }
    }

    // ---- bond forces in ascending bond order: cohesion.cuh:220-226
    if (A.nbonds) {
        const uint32_t e0 = A.bcsr_off[i], e1 = A.bcsr_off[i + 1];
        for (uint32_t e = e0; e < e1; ++e) {
            const uint32_t ent = A.bcsr_ent[e];
            const uint32_t k = ent >> 1;
            const double4 f = A.bf[k];
            if (f.w == 0.0) continue;
            const double4 t = A.bt[k];
            if ((ent & 1u) == 0) {
                acc.F = vadd(acc.F, xyz(f));
                acc.T = vsub(acc.T, xyz(t));
            } else {
                acc.F = vsub(acc.F, xyz(f));
                acc.T = vadd(acc.T, xyz(t));
            }
        }
    }

    return w0_force;
}

// The per-sphere sums of the step (contactsearch.cuh:707-724).
template <class BX>
__device__ __forceinline__ void store_sums(const StepArgs &A, const BX &B, uint32_t i,
                                           const OwnState &own, const Acc &acc, double w0_force)
{
    const double dt = B.dt;
    A.force[i] = make_double4(acc.F.x, acc.F.y, acc.F.z, 0.0);
    A.torque[i] = make_double4(acc.T.x, acc.T.y, acc.T.z, 0.0);
    A.es_dot[i] = acc.es_dot;
    A.ev_dot[i] = acc.ev_dot;
    A.es[i] = own.es + acc.es_dot * dt;
    A.ev[i] = own.ev + acc.ev_dot * dt;
    A.p[i] = acc.p;
    if (B.nw > 0) A.wf_pp[i] = w0_force;

}

constexpr int INTERACT_THREADS = 128;

// Fused topology + interact + walls + bond gather (+ integrate when FUSED)
// for the particle at sorted position a.  Neighbour data is read from the
// sorted copies only, so writing the particle's new state in place is safe.
// The particle's contact row is staged in shared memory (slot-major, one
// column per thread); only live slots are processed, empty slots keep a
// zero tangential history by construction.
template <int LM, bool FUSED, bool MIXED, int MINB>
__global__ void __launch_bounds__(INTERACT_THREADS, MINB) k_interact(StepArgs A)
{
    __shared__ uint32_t s_row[NC * INTERACT_THREADS];
    __shared__ uint16_t s_keys[VL_MAX * INTERACT_THREADS];
    const uint32_t a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= A.ntot) return;
    uint32_t *row = s_row + threadIdx.x;
    const int RS = INTERACT_THREADS;
    const uint32_t i = A.perm[a];
    const DevBox &B = A.boxes[box_index(A, i)];
    const SphParams &P = B.P;
    const double dt = B.dt;
    const double4 xa = A.xs[a];
    const double radius_a = xa.w;
    const double4 va4 = A.vs[a];
    const double4 wa4 = A.ws[a];
    const d3 vel_a = xyz(va4);
    const d3 angvel_a = xyz(wa4);
    const uint32_t cm = P.contactmodel;

    const uint4 *grow = reinterpret_cast<const uint4 *>(A.slots + (size_t)i * NC);
#pragma unroll
    for (int q = 0; q < NC / 4; ++q) {
        const uint4 w = grow[q];
        row[(4 * q + 0) * RS] = w.x;
        row[(4 * q + 1) * RS] = w.y;
        row[(4 * q + 2) * RS] = w.z;
        row[(4 * q + 3) * RS] = w.w;
    }
    bool dirty = false;
    if (A.tape_rows_pre) {
        uint4 *t = reinterpret_cast<uint4 *>(A.tape_rows_pre + (size_t)i * NC);
#pragma unroll
        for (int q = 0; q < NC / 4; ++q) t[q] = grow[q];
    }

    Acc acc;
    acc.F = mk(0.0, 0.0, 0.0);
    acc.T = mk(0.0, 0.0, 0.0);
    acc.es_dot = 0.0;
    acc.ev_dot = 0.0;
    acc.p = 0.0;

    const int nx = (int)B.num[0], ny = (int)B.num[1];
    int g[3];
    if (cm != 0) {
        g[0] = (int)floor((xa.x - B.origo[0]) / (B.L[0] / B.num[0]));
        g[1] = (int)floor((xa.y - B.origo[1]) / (B.L[1] / B.num[1]));
        g[2] = (int)floor((xa.z - B.origo[2]) / (B.L[2] / B.num[2]));
    }

    const float4 xaf = A.xf[a];
    const float Lf0 = (float)B.L[0], Lf1 = (float)B.L[1];
    if (cm == 2 || cm == 3) {
        // ---- topology: contactsearch.cuh:329-371 and :194-322
        if (search_contacts<LM>(A, B, a, i, xa, g, xaf, row, s_keys + threadIdx.x, RS)) dirty = true;

        // ---- interact over the contact row: contactsearch.cuh:484-559
        double4 *hist = A.hist + (size_t)i * NC;
        if (A.tape_rows_post) {
            for (int s = 0; s < NC; ++s) {
                const uint32_t w = row[s * RS];
                A.tape_rows_post[(size_t)i * NC + s] = w;
                if (w != EMPTY) A.tape_hist[(size_t)i * NC + s] = hist[s];
            }
        }
        // live slots in ascending order, so that the threads of a warp work
        // on their q-th contact together (the forces still add up in slot
        // order)
        uint16_t *live = s_keys + threadIdx.x;
        int nlive = 0;
        for (int s = 0; s < NC; ++s)
            if (row[s * RS] != EMPTY) live[(nlive++) * RS] = (uint16_t)s;
        for (int q = 0; q < nlive; ++q) {
            const int s = live[q * RS];
            const uint32_t w = row[s * RS];
            const uint32_t b_orig = w & ID_MASK;
            int sx, sy;
            decode_shift(w >> CODE_SHIFT, sx, sy);
            const d3 dm = shift_vec(B, sx, sy);
            const uint32_t bs = A.rank[b_orig];
            const double4 xb = A.xs[bs];
            const d3 x_ab = mk(xa.x - xb.x + dm.x, xa.y - xb.y + dm.y, xa.z - xb.z + dm.z);
            const double x_ab_length = vlen<LM>(x_ab);
            const double delta_n = x_ab_length - (radius_a + xb.w);
            if (delta_n < 0.0) {
                const d3 vel_b = xyz(A.vs[bs]);
                const d3 h0 = xyz(hist[s]);
                d3 nd;
                if (MIXED) {
                    const MixedPair q = mixed_pair(x_ab, x_ab_length, delta_n, vel_a, vel_b,
                                                   tof(angvel_a), xyzf(A.ws[bs]), radius_a, xb.w);
                    if (cm == 2) nd = contact_linear_mixed(P, dt, acc, q, h0);
                    else nd = contact_hertz_mixed(P, dt, acc, q, h0);
                } else {
                    const d3 angvel_b = xyz(A.ws[bs]);
                    if (cm == 2)
                        nd = contact_linear<LM>(P, dt, acc, vel_a, vel_b, angvel_a, angvel_b,
                                                radius_a, xb.w, x_ab, x_ab_length, delta_n, h0);
                    else
                        nd = contact_hertz<LM>(P, dt, acc, vel_a, vel_b, angvel_a, angvel_b,
                                               radius_a, xb.w, x_ab, x_ab_length, delta_n, h0);
                }
                hist[s] = make_double4(nd.x, nd.y, nd.z, 0.0);
            } else {
                row[s * RS] = EMPTY;
                dirty = true;
                hist[s] = make_double4(0.0, 0.0, 0.0, 0.0);
            }
        }
    } else if (cm == 1) {
        // ---- contact model 1: contactsearch.cuh:564-598 and :91-186
        const float reach = B.pre_margin + (float)fmax(P.db, 0.0) * 1.0001f;
        for (int dz = -1; dz < 2; ++dz)
            for (int dy = -1; dy < 2; ++dy)
                for (int dx = -1; dx < 2; ++dx) {
                    int tx = g[0] + dx, ty = g[1] + dy, sx, sy;
                    const int tz = g[2] + dz;
                    if (!image_cell(B, tx, ty, tz, sx, sy)) continue;
                    const d3 dm = shift_vec(B, sx, sy);
                    const float fsx = sx == 0 ? 0.f : (sx > 0 ? Lf0 : -Lf0);
                    const float fsy = sy == 0 ? 0.f : (sy > 0 ? Lf1 : -Lf1);
                    const uint32_t cell = B.cell_base + (uint32_t)(tx + ty * nx + (nx * ny) * tz);
                    const uint32_t start = A.cell_off[cell], end = A.cell_off[cell + 1];
                    for (uint32_t b = start; b < end; ++b) {
                        if (b == a) continue;
                        if (!maybe_touching(xaf, A.xf[b], fsx, fsy, reach)) continue;
                        const double4 xb = A.xs[b];
                        const double kappa = P.kappa;
                        d3 x_ab = mk(xa.x - xb.x, xa.y - xb.y, xa.z - xb.z);
                        x_ab = vadd(x_ab, dm);
                        const double x_ab_length = vlen<LM>(x_ab);
                        const double delta_ab = x_ab_length - (radius_a + xb.w);
                        if (delta_ab < 0.0) {
                            if (MIXED)
                                contact_linear_viscous_mixed(
                                    P, acc,
                                    mixed_pair(x_ab, x_ab_length, delta_ab, vel_a, xyz(A.vs[b]),
                                               tof(angvel_a), xyzf(A.ws[b]), radius_a, xb.w),
                                    (float)kappa);
                            else
                                contact_linear_viscous<LM>(P, acc, vel_a, xyz(A.vs[b]), angvel_a,
                                                           xyz(A.ws[b]), radius_a, xb.w, x_ab,
                                                           x_ab_length, delta_ab, kappa);
                        } else if (delta_ab < P.db) {
                            capillary_cohesion_exp(P, acc, radius_a, xb.w, delta_ab, x_ab,
                                                   x_ab_length, kappa);
                        }
                    }
                }
    }

    const double w0_force = walls_and_bonds<LM>(A, B, B, i, xa, vel_a, angvel_a, acc);

    if (dirty) {
        uint4 *wrow = reinterpret_cast<uint4 *>(A.slots + (size_t)i * NC);
#pragma unroll
        for (int q = 0; q < NC / 4; ++q)
            wrow[q] = make_uint4(row[(4 * q) * RS], row[(4 * q + 1) * RS], row[(4 * q + 2) * RS],
                                 row[(4 * q + 3) * RS]);
    }

    const OwnState own = load_own(A, i);
    store_sums(A, B, i, own, acc, w0_force);

    if (FUSED) integrate_particle(A, B, B, i, own, xa, va4, wa4, acc.F, acc.T);
}

// ------------------------------------------------------------ split step
//
// The step of k_interact for contact models 2 and 3 with fused integration,
// in three launches that keep more memory requests in flight (two where
// k_touch takes the place of the first two):
//   k_search   one thread per sphere: contact search on the slot row (kept
//              with a bitmask of the slots in use), the list of live slots
//              (ascending);
//   k_contacts one warp per 32 spheres, the warp's live contacts dealt to
//              its lanes 32 at a time: the contact law with its additions
//              recorded (ContactRec), the new history written, ended
//              contacts removed from the row; the records go through shared
//              memory to the lane of their sphere, which adds them in slot
//              order and stores the sums;
//   k_finish   one thread per sphere, original order: walls, bonds, sums,
//              integration.
// Each contact's arithmetic and the order of every sum are those of
// k_interact, so the results are bit-identical.
constexpr int SEARCH_THREADS = 128;
constexpr int CONTACT_THREADS = 128;
constexpr int FINISH_THREADS = 128;

// In a step without k_hash: its checks of the sphere's position and its cell
// id.
template <class BX>
__device__ __forceinline__ void position_check(const StepArgs &A, const BX &B, uint32_t i,
                                               double4 x)
{
    const double f[3] = {cell_floor(B, x.x, 0),
                         cell_floor(B, x.y, 1),
                         cell_floor(B, x.z, 2)};
    uint32_t c[3];
    const bool inside = clamp_cell(B, f, c);
    if (!isfinite(x.x) || !isfinite(x.y) || !isfinite(x.z)) raise_flag(A.err, SPH_ERR_NAN);
    else if (!inside || x.x > B.L[0] || x.y > B.L[1] || x.z > B.L[2])
        raise_flag(A.err, SPH_ERR_OUT_OF_GRID);
    A.cell_id[i] = B.cell_base + (c[2] * B.num[1]) * B.num[0] + c[1] * B.num[0] + c[0];
}

// The image shift that brings b nearest to a along the periodic axes.
template <class BX>
__device__ __forceinline__ void nearest_image(const BX &B, const double4 &xa, const double4 &xb,
                                              int &sx, int &sy)
{
    sx = sy = 0;
    if (B.periodic == 1 || B.periodic == 2) {
        const double d = xa.x - xb.x;
        sx = d > 0.5 * B.L[0] ? -1 : (d < -0.5 * B.L[0] ? 1 : 0);
    }
    if (B.periodic == 1) {
        const double d = xa.y - xb.y;
        sy = d > 0.5 * B.L[1] ? -1 : (d < -0.5 * B.L[1] ? 1 : 0);
    }
}

// Contact search of sphere i (original index: its row, list and state are
// read without a permutation lookup) on its slot row, staged in shared
// memory (row[s * RS]), or, IN_PLACE, in the row itself; returns the bitmask
// of occupied slots.
template <int LM, bool IN_PLACE>
__device__ __forceinline__ uint32_t search_sphere(const StepArgs &A, uint32_t i, uint32_t *row,
                                                  uint16_t *keys, int RS)
{
    const DevBox &B = A.boxes[box_index(A, i)];
    const double4 xa = A.x[i];
    const uint4 *grow = reinterpret_cast<const uint4 *>(A.slots + (size_t)i * NC);
    uint32_t occ = 0;
#pragma unroll
    for (int q = 0; q < NC / 4; ++q) {
        const uint4 w = grow[q];
        if (!IN_PLACE) {
            row[(4 * q + 0) * RS] = w.x;
            row[(4 * q + 1) * RS] = w.y;
            row[(4 * q + 2) * RS] = w.z;
            row[(4 * q + 3) * RS] = w.w;
        }
        occ |= (w.x != EMPTY ? 1u : 0u) << (4 * q);
        occ |= (w.y != EMPTY ? 1u : 0u) << (4 * q + 1);
        occ |= (w.z != EMPTY ? 1u : 0u) << (4 * q + 2);
        occ |= (w.w != EMPTY ? 1u : 0u) << (4 * q + 3);
    }
    if (A.tape_rows_pre) {
        uint4 *tp = reinterpret_cast<uint4 *>(A.tape_rows_pre + (size_t)i * NC);
#pragma unroll
        for (int q = 0; q < NC / 4; ++q) tp[q] = grow[q];
    }
    double gf[3];
    gf[0] = cell_floor(B, xa.x, 0);
    gf[1] = cell_floor(B, xa.y, 1);
    gf[2] = cell_floor(B, xa.z, 2);
    const int g[3] = {(int)gf[0], (int)gf[1], (int)gf[2]};
    if (!IN_PLACE && A.lazy_sort) position_check(A, B, i, xa);
    const uint32_t *lst = A.vlist ? A.vlist + (size_t)i * VL_MAX : nullptr;
    const uint32_t vc = lst ? A.vcount[i] : (uint32_t)VL_MAX + 1u;
    // the first entries are read together with the count (the list row
    // holds VL_MAX >= 2 KB entries; those at or past the count go unused)
    uint32_t nb[KB];
#pragma unroll
    for (int j = 0; j < KB; ++j) nb[j] = lst ? lst[j] : 0u;
    bool dirty = false;
    if (vc <= (uint32_t)VL_MAX) {
        // Partners already in the row keep their slots whatever the order,
        // so when the row cannot overflow only the other entries are
        // tested and inserted (in visit order, each into the highest free
        // slot); otherwise every entry goes through the reference's
        // counting of touching entries.
        const uint32_t occ0 = occ;
        int nk = 0;
        for (uint32_t k0 = 0; k0 < vc; k0 += KB) {
            uint32_t bo[KB];
            int srow[KB];
#pragma unroll
            for (int j = 0; j < KB; ++j) {
                bo[j] = nb[j];
                srow[j] = -1;
                if (k0 + j < vc)
                    for (uint32_t m = occ0; m; m &= m - 1u) {
                        const int sl = __ffs(m) - 1;
                        if ((row[sl * RS] & ID_MASK) == bo[j]) {
                            srow[j] = sl;
                            break;
                        }
                    }
            }
            if (k0 + KB < vc) {
#pragma unroll
                for (int j = 0; j < KB; ++j) nb[j] = lst[k0 + KB + j];
            }
            uint16_t kb[KB];
            list_keys_batch<LM, true>(A, B, xa, g, bo, k0, vc, kb, srow, row, RS, &dirty);
#pragma unroll
            for (int j = 0; j < KB; ++j) {
                const uint16_t key = kb[j];
                if (key == NO_KEY) continue;
                int q = nk;
                while (q > 0 && keys[(q - 1) * RS] > key) {
                    keys[q * RS] = keys[(q - 1) * RS];
                    --q;
                }
                keys[q * RS] = key;
                ++nk;
            }
        }
        if (__popc(occ0) + nk > NC) {
            // the row may overflow: all touching entries, counted in order
            nk = 0;
            const int none[KB] = {-1, -1, -1, -1};
            for (uint32_t k0 = 0; k0 < vc; k0 += KB) {
                uint32_t bo[KB];
#pragma unroll
                for (int j = 0; j < KB; ++j) bo[j] = k0 + j < vc ? lst[k0 + j] : 0u;
                uint16_t kb[KB];
                list_keys_batch<LM, false>(A, B, xa, g, bo, k0, vc, kb, none, row, RS, &dirty);
#pragma unroll
                for (int j = 0; j < KB; ++j) {
                    const uint16_t key = kb[j];
                    if (key == NO_KEY) continue;
                    int q = nk;
                    while (q > 0 && keys[(q - 1) * RS] > key) {
                        keys[q * RS] = keys[(q - 1) * RS];
                        --q;
                    }
                    keys[q * RS] = key;
                    ++nk;
                }
            }
        }
        if (insert_keys(A, keys, nk, RS, lst, row, RS, occ)) dirty = true;
    } else {
        const uint32_t a = A.rank[i];   // the cell search walks the sorted copies
        dirty = search_cells<LM>(A, B, a, xa, g, A.xf[a], row, RS);
        occ = occupancy(row, RS);
    }
    if (A.tape_rows_post) {
        const double4 *hist = A.hist + (size_t)i * NC;
        for (int s = 0; s < NC; ++s) {
            const uint32_t w = row[s * RS];
            A.tape_rows_post[(size_t)i * NC + s] = w;
            if (w != EMPTY) A.tape_hist[(size_t)i * NC + s] = hist[s];
        }
    }
    if (!IN_PLACE && dirty) {
        uint4 *wrow = reinterpret_cast<uint4 *>(A.slots + (size_t)i * NC);
#pragma unroll
        for (int q = 0; q < NC / 4; ++q)
            wrow[q] = make_uint4(row[(4 * q) * RS], row[(4 * q + 1) * RS], row[(4 * q + 2) * RS],
                                 row[(4 * q + 3) * RS]);
    }
    return occ;
}

template <int LM>
__global__ void __launch_bounds__(SEARCH_THREADS) k_search(StepArgs A)
{
    __shared__ uint32_t s_row[NC * SEARCH_THREADS];
    __shared__ uint16_t s_keys[VL_MAX * SEARCH_THREADS];
    grid_dependency_wait();
    if (A.lazy_sort && A.vflag[3] != 0u) return;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u;
    const int RS = SEARCH_THREADS;
    uint32_t *row = s_row + threadIdx.x;
    const uint32_t occ =
        i < A.ntot ? search_sphere<LM, false>(A, i, row, s_keys + threadIdx.x, RS) : 0u;
    // the warp's live contacts, sphere after sphere, each in slot order,
    // written contiguously from the start of the warp's region
    const uint32_t nl = __popc(occ);
    uint32_t incl = nl;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += v;
    }
    if (i >= A.ntot) return;
    uint2 *ent = A.lent + (size_t)(i - lane) * NC + (incl - nl);
    uint32_t q = 0;
    for (uint32_t m = occ; m; m &= m - 1u) {
        const int sl = __ffs(m) - 1;
        // slot word (partner's original id | image code), i | slot << 27
        ent[q++] = make_uint2(row[sl * RS], i | ((uint32_t)sl << 27));
    }
    A.nlive[i] = nl;
}

// One warp-round of contact records in shared memory, field by field
// (consecutive lanes hit consecutive words).
struct RecSlab {
    double f[10][CONTACT_THREADS];   // F.x F.y F.z T.x T.y T.z ev0 ev1 es p
    int32_t n[CONTACT_THREADS];      // (nev + 1) | nes << 4
};

__device__ __forceinline__ void put_rec(RecSlab &S, int t, const ContactRec &r)
{
    S.f[0][t] = r.F.x;
    S.f[1][t] = r.F.y;
    S.f[2][t] = r.F.z;
    S.f[3][t] = r.T.x;
    S.f[4][t] = r.T.y;
    S.f[5][t] = r.T.z;
    S.f[6][t] = r.ev0;
    S.f[7][t] = r.ev1;
    S.f[8][t] = r.es;
    S.f[9][t] = r.p;
    S.n[t] = (r.nev + 1) | (r.nes << 4);
}

__device__ __forceinline__ ContactRec get_rec(const RecSlab &S, int t)
{
    ContactRec r;
    r.F = mk(S.f[0][t], S.f[1][t], S.f[2][t]);
    r.T = mk(S.f[3][t], S.f[4][t], S.f[5][t]);
    r.ev0 = S.f[6][t];
    r.ev1 = S.f[7][t];
    r.es = S.f[8][t];
    r.p = S.f[9][t];
    const int32_t n = S.n[t];
    r.nev = (n & 15) - 1;
    r.nes = n >> 4;
    return r;
}

// The contact of slot s (word w) of sphere i: the law with its additions
// recorded in r and the new history written, or the slot freed when the
// pair no longer touches (r.nev < 0 then); returns whether it touches.
// NEAREST: the image is the nearest one (see k_touch) and the slot's code is
// brought up to date; else the slot's code says it.
// B, M: the box's constants and its contact parameters.
template <int LM, bool MIXED, bool NEAREST, class BX, class PT>
__device__ __forceinline__ bool slot_contact(const StepArgs &A, const BX &B, const PT &M, uint32_t i,
                                             int s, uint32_t w, ContactRec &r)
{
    const SphParams &P = B.P;
    const double dt = B.dt;
    const uint32_t cm = P.contactmodel;
    // the sphere's own data in original order (the step's start
    // state until k_finish), like its partner's
    const double4 xa = A.x[i];
    const double radius_a = xa.w;
    const d3 vel_a = xyz(A.vel[i]);
    const d3 angvel_a = xyz(A.angvel[i]);
    uint32_t *slots = A.slots + (size_t)i * NC;
    double4 *hist = A.hist + (size_t)i * NC;
    const uint32_t bo = w & ID_MASK;   // partner's original id
    // the partner's data (original order: A.x, A.vel, A.angvel hold
    // the step's start state until k_finish) and the history are
    // loaded together
    const double4 xb = A.x[bo];
    const double4 vb4 = A.vel[bo];
    const double4 wb4 = A.angvel[bo];
    const double4 h4 = hist[s];
    int sx, sy;
    if (NEAREST) nearest_image(B, xa, xb, sx, sy);
    else decode_shift(w >> CODE_SHIFT, sx, sy);
    const d3 dm = shift_vec(B, sx, sy);
    const d3 x_ab = mk(xa.x - xb.x + dm.x, xa.y - xb.y + dm.y, xa.z - xb.z + dm.z);
    const double x_ab_length = vlen<LM>(x_ab);
    const double delta_n = x_ab_length - (radius_a + xb.w);
    if (!(delta_n < 0.0)) {
        slots[s] = EMPTY;
        hist[s] = make_double4(0.0, 0.0, 0.0, 0.0);
        return false;
    }
    if (NEAREST) {
        const uint32_t v = bo | (shift_code(sx, sy) << CODE_SHIFT);
        if (v != w) {
            slots[s] = v;
            if (A.tape_rows_post) A.tape_rows_post[(size_t)i * NC + s] = v;
        }
    }
    r.nev = 0;
    const d3 vel_b = xyz(vb4);
    const d3 h0 = xyz(h4);
    d3 nd;
    if (MIXED) {
        const MixedPair mp = mixed_pair(x_ab, x_ab_length, delta_n, vel_a, vel_b,
                                        tof(angvel_a), xyzf(wb4), radius_a, xb.w);
        if (cm == 2) nd = contact_linear_mixed(M, dt, r, mp, h0);
        else nd = contact_hertz_mixed(M, dt, r, mp, h0);
    } else {
        const d3 angvel_b = xyz(wb4);
        if (cm == 2)
            nd = contact_linear<LM>(P, dt, r, vel_a, vel_b, angvel_a, angvel_b,
                                    radius_a, xb.w, x_ab, x_ab_length, delta_n, h0);
        else
            nd = contact_hertz<LM>(P, dt, r, vel_a, vel_b, angvel_a, angvel_b,
                                   radius_a, xb.w, x_ab, x_ab_length, delta_n, h0);
    }
    hist[s] = make_double4(nd.x, nd.y, nd.z, 0.0);
    return true;
}

__device__ __forceinline__ Acc zero_acc()
{
    Acc acc;
    acc.F = mk(0.0, 0.0, 0.0);
    acc.T = mk(0.0, 0.0, 0.0);
    acc.es_dot = 0.0;
    acc.ev_dot = 0.0;
    acc.p = 0.0;
    return acc;
}

__device__ __forceinline__ ContactRec no_rec()
{
    ContactRec r;
    r.F = mk(0.0, 0.0, 0.0);
    r.T = mk(0.0, 0.0, 0.0);
    r.ev0 = r.ev1 = r.es = r.p = 0.0;
    r.nev = -1;   // nothing to add unless a live contact is computed
    r.nes = 0;
    return r;
}

__device__ __forceinline__ uint32_t warp_inclusive(uint32_t v, uint32_t lane)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= (uint32_t)o) v += u;
    }
    return v;
}

// The records of one warp round (S, from the warp's word wbase) that belong
// to the lane's sphere -- contacts [excl, incl) of the warp -- added in slot
// order.
__device__ __forceinline__ void replay_round(Acc &acc, const RecSlab &S, int wbase, uint32_t base,
                                             uint32_t excl, uint32_t incl)
{
    const uint32_t lo = max(excl, base), hi = min(incl, base + 32u);
    for (uint32_t e = lo; e < hi; ++e) {
        const ContactRec o = get_rec(S, wbase + (int)(e - base));
        if (o.nev >= 0) replay(acc, o);
    }
}

// One warp per 32 consecutive spheres (original indexes), its lanes dealt
// the warp's live contacts in order: round r computes contacts 32r .. 32r +
// 31 of the warp's list (the spheres' live lists one after the other), so a
// lane is idle only in the last round.  Each lane then adds, in slot order,
// the round's records of its own sphere.
template <int LM, bool MIXED>
__global__ void __launch_bounds__(CONTACT_THREADS, 6) k_contacts(StepArgs A)
{
    __shared__ RecSlab S;
    grid_dependency_wait();
    if (A.lazy_sort && A.vflag[3] != 0u) return;
    const uint32_t lane = threadIdx.x & 31u;
    const int wbase = (int)(threadIdx.x & ~31u);
    const uint32_t i_own = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t i0 = i_own - lane;
    const bool valid = i_own < A.ntot;
    const uint32_t nl_own = valid ? A.nlive[i_own] : 0u;
    const uint32_t incl = warp_inclusive(nl_own, lane);
    const uint32_t excl = incl - nl_own;
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    Acc acc = zero_acc();
    const uint2 *ent = A.lent + (size_t)i0 * NC;
    for (uint32_t base = 0; base < total; base += 32) {
        const uint32_t f = base + lane;
        ContactRec r = no_rec();
        if (f < total) {
            const uint2 e = ent[f];
            const uint32_t i = e.y & SPLIT_ID_MASK;
            const DevBox &B = A.boxes[box_index(A, i)];
            (void)slot_contact<LM, MIXED, false>(A, B, B.P, i, (int)(e.y >> 27), e.x, r);
        }
        put_rec(S, (int)threadIdx.x, r);
        __syncwarp();
        replay_round(acc, S, wbase, base, excl, incl);
        __syncwarp();
    }
    if (valid) A.csum[i_own] = acc;
}

// Search and contacts in one kernel, for the lazily sorted split step on
// grids whose cells are wider than the largest diameter (cfg.touch).
//
// The search's work hardly changes from step to step: the row keeps its
// contacts, and an entry of the neighbour list that is not in the row seldom
// starts to touch.  So the entries that are in the row are remembered (a bit
// per list entry, A.lmask, with LMASK_VALID while it holds; the occupied
// slots in A.occ), and a step tests only the others.  One that touches takes
// the highest free slot, as the reference's rule has it; only when several
// do, or the lists are new, does the sphere go through search_sphere, on its
// row in memory.  At 1e6 spheres in contact with 4.3
// others of 5.7 listed that leaves 1.4 position gathers per sphere of the
// row, the list and 5.7 cell gathers.
//
// The image of a pair is the nearest one.  A touching pair's centres are
// less than a cell apart along each axis, so their cells are neighbours, and
// with at least three cells along a periodic axis the image under which the
// cell search visits the partner is the nearest; a pair that touches under
// neither is no contact under both.
//
// Contacts are then dealt to the warp's lanes as in k_contacts, contact f of
// the warp found from the lanes' counts and occupied slots.
constexpr unsigned long long LMASK_VALID = 1ull << 63;
// Resident blocks per SM, which sets the registers: 4 (128 a thread) for the
// FP64 laws, 5 (96) for the mixed ones.  us of k_touch with 6 / 5 / 4 blocks:
// FP64, 1e6 spheres 508 / 451 / 436, 60,013 spheres 50 / 42 / 36 (60 values
// spilled with 6, 13 with 5, none with 4); mixed, 200,000 bonded spheres 80 /
// 78 / 84.
constexpr int touch_blocks(bool mixed) { return mixed ? 5 : 4; }

// Where touch_warp finds the constants of sphere i's box and its contact
// parameters.
struct TableBoxes {
    const StepArgs &A;
    __device__ __forceinline__ const DevBox &box(uint32_t i) const { return A.boxes[box_index(A, i)]; }
    __device__ __forceinline__ const SphParams &params(uint32_t i) const { return box(i).P; }
};
struct OneBox {
    const BoxConst &C;
    const MixedParams &M;
    __device__ __forceinline__ const BoxConst &box(uint32_t) const { return C; }
    __device__ __forceinline__ const MixedParams &params(uint32_t) const { return M; }
};

// The search of sphere i on its row in memory; which entries of its list are
// in the row is found anew.  (Rare: not inlined, for the registers.)
template <int LM>
__device__ __noinline__ uint32_t touch_row(const StepArgs &A, uint32_t i)
{
    uint32_t *row = A.slots + (size_t)i * NC;
    const uint32_t *lst = A.vlist + (size_t)i * VL_MAX;
    const uint32_t vc = A.vcount[i];
    uint16_t keys[VL_MAX];
    const uint32_t occ = search_sphere<LM, true>(A, i, row, keys, 1);
    A.occ[i] = occ;
    // the list entries that are in the row
    unsigned long long in = 0ull;
    if (vc <= (uint32_t)VL_MAX) {
        for (uint32_t m2 = occ; m2; m2 &= m2 - 1u) {
            const uint32_t b = row[__ffs(m2) - 1] & ID_MASK;
            for (uint32_t k = 0; k < vc; ++k)
                if (lst[k] == b) in |= 1ull << k;
        }
        in |= LMASK_VALID;
    }
    A.lmask[i] = in;
    return occ;
}

template <int LM, class BX>
__device__ __forceinline__ uint32_t touch_search(const StepArgs &A, const BX &B, uint32_t i)
{
    const unsigned long long m = A.lmask[i];
    const uint32_t vc = A.vcount[i];
    uint32_t occ = A.occ[i];
    const uint32_t stop = A.vflag[3];   // a rebuild gave up
    const uint32_t *lst = A.vlist + (size_t)i * VL_MAX;
    const double4 xa = A.x[i];
    position_check(A, B, i, xa);
    if (A.tape_state) {
        A.tape_state[i] = xa;
        A.tape_state[A.ntot + i] = A.vel[i];
        A.tape_state[2 * (size_t)A.ntot + i] = A.angvel[i];
    }
    if (vc > (uint32_t)VL_MAX || !(m & LMASK_VALID)) return stop ? 0u : touch_row<LM>(A, i);
    // the first entry that is not in the row and touches, and its slot word
    uint32_t found = 0, kf = 0, wf = 0;
    for (unsigned long long todo = ((1ull << vc) - 1ull) & ~m; todo;) {
        // the next KB entries' gathers in flight together
        uint32_t bo[KB], ke[KB];
        double4 xb[KB];
        int nb = 0;
#pragma unroll
        for (int j = 0; j < KB; ++j) {
            if (todo) {
                ke[j] = (uint32_t)(__ffsll((long long)todo) - 1);
                bo[j] = lst[ke[j]];
                todo &= todo - 1ull;
                ++nb;
            }
        }
#pragma unroll
        for (int j = 0; j < KB; ++j)
            if (j < nb) xb[j] = A.x[bo[j]];
#pragma unroll
        for (int j = 0; j < KB; ++j) {
            if (j >= nb) continue;
            int sx, sy;
            nearest_image(B, xa, xb[j], sx, sy);
            const d3 dm = shift_vec(B, sx, sy);
            d3 x_ab = mk(xa.x - xb[j].x, xa.y - xb[j].y, xa.z - xb[j].z);
            x_ab = vadd(x_ab, dm);
            if (len_rn<LM>(x_ab) - (xa.w + xb[j].w) < 0.0) {
                if (found++ == 0u) {
                    kf = ke[j];
                    wf = bo[j] | (shift_code(sx, sy) << CODE_SHIFT);
                }
            }
        }
    }
    // Stopped: no contacts, and no row is written.  (Here and not ahead of the
    // loads, where every thread waited for the word first, 1 to 5 % of the
    // kernel; what the search read is there, each list with its own length.)
    if (stop) return 0u;
    // several new contacts take their slots in the cells' visit order
    if (found > 1u || (found == 1u && occ == 0xffffffffu)) return touch_row<LM>(A, i);
    uint32_t *row = A.slots + (size_t)i * NC;
    const uint4 *row4 = reinterpret_cast<const uint4 *>(row);
    if (A.tape_rows_pre) {
        uint4 *t = reinterpret_cast<uint4 *>(A.tape_rows_pre + (size_t)i * NC);
#pragma unroll
        for (int q = 0; q < NC / 4; ++q) t[q] = row4[q];
    }
    if (found) {
        // one: the highest free slot
        const int s = 31 - __clz((int)~occ);
        row[s] = wf;
        occ |= 1u << s;
        A.occ[i] = occ;
        A.lmask[i] = m | (1ull << kf);
    }
    if (A.tape_rows_post) {
        uint4 *t = reinterpret_cast<uint4 *>(A.tape_rows_post + (size_t)i * NC);
#pragma unroll
        for (int q = 0; q < NC / 4; ++q) t[q] = row4[q];
        for (uint32_t m2 = occ; m2; m2 &= m2 - 1u) {
            const size_t q = (size_t)i * NC + (size_t)(__ffs(m2) - 1);
            A.tape_hist[q] = A.hist[q];
        }
    }
    return occ;
}

// SPW: spheres of a warp (see launch_contacts_lm).
template <int LM, bool MIXED, int SPW, class Boxes>
__device__ __forceinline__ void touch_warp(const StepArgs &A, RecSlab &S, const Boxes &at)
{
    const uint32_t lane = threadIdx.x & 31u;
    const int wbase = (int)(threadIdx.x & ~31u);
    const uint32_t i0 = (blockIdx.x * blockDim.x + threadIdx.x) / 32u * SPW;
    const uint32_t i_own = i0 + lane;
    const bool valid = lane < (uint32_t)SPW && i_own < A.ntot;
    const uint32_t occ_own = valid ? touch_search<LM>(A, at.box(i_own), i_own) : 0u;
    const uint32_t nl_own = (uint32_t)__popc(occ_own);
    const uint32_t incl = warp_inclusive(nl_own, lane);
    const uint32_t excl = incl - nl_own;
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    Acc acc = zero_acc();
    __syncwarp();   // the rows and tape rows written above are read and patched below
    for (uint32_t base = 0; base < total; base += 32) {
        const uint32_t f = base + lane;
        // the sphere of contact f: the first lane whose inclusive count
        // exceeds f
        uint32_t o = 0;
#pragma unroll
        for (int st = 16; st > 0; st >>= 1) {
            const uint32_t v = __shfl_sync(0xffffffffu, incl, (int)(o + (uint32_t)st - 1u));
            if (v <= f) o += (uint32_t)st;
        }
        o = min(o, 31u);
        uint32_t m = __shfl_sync(0xffffffffu, occ_own, (int)o);
        const uint32_t e0 = __shfl_sync(0xffffffffu, excl, (int)o);
        ContactRec r = no_rec();
        if (f < total) {
            for (uint32_t q = f - e0; q; --q) m &= m - 1u;
            const int s = __ffs(m) - 1;
            const uint32_t i = i0 + o;
            const uint32_t w = A.slots[(size_t)i * NC + s];
            if (!slot_contact<LM, MIXED, true>(A, at.box(i), at.params(i), i, s, w, r)) {
                // the contact ended: its entry is no longer in the row
                const uint32_t *lst = A.vlist + (size_t)i * VL_MAX;
                const uint32_t vc = A.vcount[i];
                uint32_t k = 0;
                if (vc <= (uint32_t)VL_MAX)
                    while (k < vc && lst[k] != (w & ID_MASK)) ++k;
                if (k < vc && vc <= (uint32_t)VL_MAX) atomicAnd(&A.lmask[i], ~(1ull << k));
                atomicAnd(&A.occ[i], ~(1u << s));
            }
        }
        put_rec(S, (int)threadIdx.x, r);
        __syncwarp();
        replay_round(acc, S, wbase, base, excl, incl);
        __syncwarp();
    }
    if (valid) A.csum[i_own] = acc;
}

template <int LM, bool MIXED, int SPW>
__global__ void __launch_bounds__(CONTACT_THREADS, touch_blocks(MIXED)) k_touch(const __grid_constant__ StepArgs A)
{
    __shared__ RecSlab S;
    grid_dependency_wait();
    touch_warp<LM, MIXED, SPW>(A, S, TableBoxes{A});
}

// k_touch of a one-box handle: the box's constants from the arguments.
template <int LM, bool MIXED, int SPW>
__global__ void __launch_bounds__(CONTACT_THREADS, touch_blocks(MIXED)) k_touch1(const __grid_constant__ StepArgs A,
                                                                          const __grid_constant__ BoxConst C,
                                                                          const __grid_constant__ MixedParams M)
{
    __shared__ RecSlab S;
    grid_dependency_wait();
    touch_warp<LM, MIXED, SPW>(A, S, OneBox{C, M});
}

// Original order: every access is to the sphere's own entries, so they are
// all coalesced (x, vel, angvel still hold the state at the start of the
// step: only this thread rewrites them).
template <int LM, class BX>
__device__ __forceinline__ void finish_one(const StepArgs &A, const DevBox &B, const BX &C, uint32_t i)
{
    const double4 xa = A.x[i];
    const double4 va4 = A.vel[i];
    const double4 wa4 = A.angvel[i];
    Acc acc = A.csum[i];   // the contacts' sums, added in slot order
    const OwnState own = load_own(A, i);
    const uint32_t stop = A.lazy_sort ? A.vflag[3] : 0u;
    loaded(own.angpos);
    loaded(own.xyzsum);
    loaded(own.acc);
    loaded(own.angacc);
    asm volatile("" ::"d"(own.es), "d"(own.ev), "f"(own.xref.x), "r"(stop));
    const double w0_force = walls_and_bonds<LM>(A, B, C, i, xa, xyz(va4), xyz(wa4), acc);
    if (stop) {   // (here, where every load ahead of the first store is under way)
        for (uint32_t b = i; b < A.nboxes; b += A.ntot) A.boxes[b].halt = 1u;
        return;
    }
    store_sums(A, C, i, own, acc, w0_force);
    integrate_particle(A, B, C, i, own, xa, va4, wa4, acc.F, acc.T);
}

template <int LM>
__global__ void __launch_bounds__(FINISH_THREADS, 4) k_finish(const __grid_constant__ StepArgs A)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.ntot) return;
    const DevBox &B = A.boxes[box_index(A, i)];
    finish_one<LM>(A, B, B, i);
}

// k_finish of a one-box handle: the box's constants from the arguments.
template <int LM>
__global__ void __launch_bounds__(FINISH_THREADS, 4) k_finish1(const __grid_constant__ StepArgs A,
                                                               const __grid_constant__ BoxConst C)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < A.ntot) finish_one<LM>(A, A.boxes[0], C, i);
}

// Launch variants of k_interact (INTERACT_VARIANTS): the minimum resident
// blocks per SM given to the compiler (register budget 255, 128 and 80 per
// thread), chosen per handle by sph_autotune.  The arithmetic is the same
// in every variant.

template <bool MIXED, int LM, bool FUSED>
inline void launch_interact_lm(const StepArgs &A, cudaStream_t st, unsigned grid, int variant)
{
    if (variant == 0) k_interact<LM, FUSED, MIXED, 1><<<grid, INTERACT_THREADS, 0, st>>>(A);
    else if (variant == 2) k_interact<LM, FUSED, MIXED, 6><<<grid, INTERACT_THREADS, 0, st>>>(A);
    else k_interact<LM, FUSED, MIXED, 4><<<grid, INTERACT_THREADS, 0, st>>>(A);
}

template <bool MIXED, int LM, int SPW>
inline void launch_touch(const StepArgs &A, const DevBox *box0, cudaStream_t st, bool pdl)
{
    const unsigned per_block = CONTACT_THREADS / 32 * SPW;
    const unsigned grid = (A.ntot + per_block - 1) / per_block;
    if (box0)
        launch_k(pdl, k_touch1<LM, MIXED, SPW>, grid, CONTACT_THREADS, st, A, box_const(*box0),
                 mixed_params(box0->P));
    else
        launch_k(pdl, k_touch<LM, MIXED, SPW>, grid, CONTACT_THREADS, st, A);
}

template <bool MIXED, int LM>
inline void launch_contacts_lm(const StepArgs &A, const DevBox *box0, cudaStream_t st, unsigned grid,
                               bool pdl)
{
    // Fewer spheres to a warp while all warps fit on the chip at once
    // (touch_blocks on each of 148 SMs): their contacts then take fewer
    // rounds, the warps run side by side.  us of k_touch with 32 / 16 / 8 / 4
    // spheres a warp (at five blocks per SM): 500 spheres (FP64) 21.0 / 14.5 / 10.9 / 9.4; 60,013: 42.2 /
    // 43.9 / 46.9 / 55; 1e6: 451 / 559 / 729 / 951.
    constexpr uint32_t WARPS = 148u * touch_blocks(MIXED) * (CONTACT_THREADS / 32);
    if (!A.touch) launch_k(pdl, k_contacts<LM, MIXED>, grid, CONTACT_THREADS, st, A);
    else if (A.ntot <= 4u * WARPS) launch_touch<MIXED, LM, 4>(A, box0, st, pdl);
    else if (A.ntot <= 8u * WARPS) launch_touch<MIXED, LM, 8>(A, box0, st, pdl);
    else if (A.ntot <= 16u * WARPS) launch_touch<MIXED, LM, 16>(A, box0, st, pdl);
    else launch_touch<MIXED, LM, 32>(A, box0, st, pdl);
}

template <bool MIXED>
inline void launch_contacts(const StepArgs &A, const StepConfig &cfg, cudaStream_t st, unsigned grid,
                            bool pdl)
{
    if (cfg.lenmode == SPH_LEN_FP64) launch_contacts_lm<MIXED, SPH_LEN_FP64>(A, cfg.box0, st, grid, pdl);
    else launch_contacts_lm<MIXED, SPH_LEN_REFERENCE>(A, cfg.box0, st, grid, pdl);
}

template <bool MIXED>
inline void launch_interact(const StepArgs &A, cudaStream_t st, unsigned grid, bool fused, int lm,
                            int variant)
{
    if (fused) {
        if (lm == SPH_LEN_FP64) launch_interact_lm<MIXED, SPH_LEN_FP64, true>(A, st, grid, variant);
        else launch_interact_lm<MIXED, SPH_LEN_REFERENCE, true>(A, st, grid, variant);
    } else {
        if (lm == SPH_LEN_FP64) launch_interact_lm<MIXED, SPH_LEN_FP64, false>(A, st, grid, variant);
        else launch_interact_lm<MIXED, SPH_LEN_REFERENCE, false>(A, st, grid, variant);
    }
}

}  // namespace sph
