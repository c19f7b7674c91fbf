// D3Q19 mesoscale step (the L1 grid of the mod): two-relaxation-time
// hydrodynamic and thermal double distributions relaxed toward targets built
// from a 25-channel forcing, pull streaming with bounce-back off solid cells
// and the ground, equilibrium inflow with a two-cell blend at the sides and
// top, macro export (native/src/aero_lbm_mesoscale.cpp:146-738).
//
// A call from the host is three launches: `meso_derive_kernel` (what the step
// reads of the forcing and the pull classification),
// `meso_collide_kernel` (targets + TRT, one thread per cell; writes post-collision f and g and the next surface /
// deep-ground temperatures) and `meso_stream_kernel` (pull + boundaries +
// macro export; writes the new f and g, the ambient field and the output
// state). The collision needs the neighbours' previous temperatures
// (laplacians) and the pull needs the neighbours' post-collision populations,
// so the step has two grid-wide dependencies and cannot be one launch. Within
// a window of resident steps the pull moves into the next collision, and the
// pass between two collisions (`meso_ambient_kernel`) forms the streamed
// temperature alone. Populations are structure-of-arrays f[q][cell] (the
// reference stores f[cell*19+q]; the layout is internal to both).
//
// This file is built with --fmad=false and every expression keeps the
// reference's operation order (products by the integer lattice components
// included), so the step is bit-identical to the reference CPU step. The
// options the reference does not have (periodic x/z sides, a free-slip lid, a
// uniform Guo body force, a fixed hydrodynamic tau, Smagorinsky on the even
// rate, no edge blend) follow the oracle's restatement and are off by default.
#include <cuda_fp16.h>

#include "d3q27_kernels.cuh"
#include "lattice.cuh"
#include "meso.cuh"
#include "meso_lattice.cuh"
#include "pdl.cuh"

namespace aero {
namespace meso {

__device__ __forceinline__ float fx_(int q) { return (float)mcx(q); }
__device__ __forceinline__ float fy_(int q) { return (float)mcy(q); }
__device__ __forceinline__ float fz_(int q) { return (float)mcz(q); }

// std::max / std::min / std::clamp
__device__ __forceinline__ float smax(float a, float b) { return (a < b) ? b : a; }
__device__ __forceinline__ float smin(float a, float b) { return (b < a) ? b : a; }
__device__ __forceinline__ float sclamp(float v, float lo, float hi) { return (v < lo) ? lo : ((hi < v) ? hi : v); }
__device__ __forceinline__ float clamp_speed(float u) { return sclamp(u, -0.35f, 0.35f); }

// hydro_feq_3d / thermal_feq_3d (native/src/aero_lbm_mesoscale.cpp:254-263)
__device__ __forceinline__ float hfeq(int q, float r, float ux, float uy, float uz) {
    const float cu = 3.0f * (fx_(q) * ux + fy_(q) * uy + fz_(q) * uz);
    const float uu = ux * ux + uy * uy + uz * uz;
    return mw(q) * r * (1.0f + cu + 0.5f * cu * cu - 1.5f * uu);
}
__device__ __forceinline__ float tfeq(int q, float t, float ux, float uy, float uz) {
    const float cu = 3.0f * (fx_(q) * ux + fy_(q) * uy + fz_(q) * uz);
    return mw(q) * t * (1.0f + cu);
}

__device__ __forceinline__ float ch(const float* __restrict__ F, long long cell, int c) {
    return __ldg(F + cell * kMesoForcingChannels + c);
}
__device__ __forceinline__ bool solid_at(const float* __restrict__ F, long long cell) { return ch(F, cell, kChSolidMask) > 0.5f; }
__device__ __forceinline__ float wall_temp(const float* __restrict__ F, long long cell) {
    return ch(F, cell, kChSurfaceTarget) + ch(F, cell, kChNestedSurfaceDelta);
}

template <class Args>
__device__ __forceinline__ long long midx(const Args& A, int x, int y, int z) {
    return ((long long)x * A.ny + y) * A.nz + z;
}
// horizontal (x, z) and vertical (y) laplacians with clamped neighbours
// (native/src/aero_lbm_mesoscale.cpp:335-373)
__device__ __forceinline__ float hlap(const MesoArgs& A, const float* a, int x, int y, int z) {
    const float c = a[midx(A, x, y, z)];
    const float xp = a[midx(A, min(A.nx - 1, x + 1), y, z)], xm = a[midx(A, max(0, x - 1), y, z)];
    const float zp = a[midx(A, x, y, min(A.nz - 1, z + 1))], zm = a[midx(A, x, y, max(0, z - 1))];
    return xp + xm + zp + zm - 4.0f * c;
}
__device__ __forceinline__ float vlap(const MesoArgs& A, const float* a, int x, int y, int z) {
    if (A.ny <= 1) return 0.0f;
    const float c = a[midx(A, x, y, z)];
    const float yp = a[midx(A, x, min(A.ny - 1, y + 1), z)], ym = a[midx(A, x, max(0, y - 1), z)];
    return yp + ym - 2.0f * c;
}

__device__ __forceinline__ float dv(const MesoArgs& A, int k, long long i) {
    return A.derived[k * ((long long)A.nx * A.ny * A.nz) + i];
}

// Directions whose component along an axis is +1 / -1, as a bit set.
__host__ __device__ constexpr uint32_t mdirs(int axis, int sign) {
    uint32_t m = 0;
    for (int q = 0; q < 19; ++q)
        if ((axis == 0 ? mcx(q) : (axis == 1 ? mcy(q) : mcz(q))) == sign) m |= 1u << q;
    return m;
}

// Pull classification of a fluid cell (see meso_hydro_flags): solid(n) of the
// 19 sources is read whatever the cell's place (an open side's from the
// wrapped cell, the ground's and the lid's from the cell's own row), so the
// loads do not wait for one another.
template <class Args, class Solid>
__device__ __forceinline__ uint32_t pull_class(const Args& A, int x, int y, int z, Solid solid) {
    const int nx = A.nx, ny = A.ny, nz = A.nz;
    long long X[3], Y[3], Z[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int sx = x + k - 1, sy = y + k - 1, sz = z + k - 1;
        X[k] = (long long)(sx < 0 ? sx + nx : (sx >= nx ? sx - nx : sx)) * ny * nz;
        Y[k] = (long long)min(max(sy, 0), ny - 1) * nz;
        Z[k] = sz < 0 ? sz + nz : (sz >= nz ? sz - nz : sz);
    }
    uint32_t hit = 0;
#pragma unroll
    for (int q = 0; q < 19; ++q)
        hit |= solid(X[1 - mcx(q)] + Y[1 - mcy(q)] + Z[1 - mcz(q)]) ? 1u << q : 0u;
    uint32_t side = 0;
    if (!A.periodic_sides)
        side = (x == 0 ? mdirs(0, 1) : 0u) | (x == nx - 1 ? mdirs(0, -1) : 0u) | (z == 0 ? mdirs(2, 1) : 0u) |
               (z == nz - 1 ? mdirs(2, -1) : 0u);
    const uint32_t ground = y == 0 ? mdirs(1, 1) : 0u, lid = y == ny - 1 ? mdirs(1, -1) : 0u;
    // inside the grid (or reflected at a free-slip lid): off the solid cell
    // there; the ground always; an open side or lid never
    const uint32_t open = (side | (A.free_slip_top ? 0u : lid)) & ~ground;
    const uint32_t w = (hit & ~open) | ground;
    int edge = min(min(x, z), min(nx - 1 - x, nz - 1 - z));
    int top = ny - 1 - y;
    if (A.periodic_sides) edge = 1 << 20;
    if (A.free_slip_top) top = 1 << 20;
    const bool slow = (A.edge_blend && min(edge, top) < 2) || ((side | lid) & ~ground) != 0;
    return w | (slow ? kHydroSlow : 0u);
}

// The forcing terms of compute_cell_targets and of the open boundaries that
// do not depend on the state (native/src/aero_lbm_mesoscale.cpp:393-530,
// 620-734), each expression as the reference has it.
__global__ void __launch_bounds__(128) meso_derive_kernel(MesoArgs A) {
    pdl_trigger();
    const long long cells = (long long)A.nx * A.ny * A.nz;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cells) return;
    int x, y, z;
    cell_xyz32(i, A.ny, A.nz, x, y, z);
    const float* F = A.forcing;
    const float conv_m = ch(F, i, kChConvectiveMoistening), tor_m = ch(F, i, kChTornadoMoistening);
    const float conv_x = ch(F, i, kChConvectiveInflowX), conv_z = ch(F, i, kChConvectiveInflowZ);
    const float tor_x = ch(F, i, kChTornadoWindX), tor_z = ch(F, i, kChTornadoWindZ);
    const float tor_up = ch(F, i, kChTornadoUpdraft), nest_up = ch(F, i, kChNestedUpdraft);
    const float bx = ch(F, i, kChBackgroundWindX) + ch(F, i, kChNestedWindXDelta) + conv_x + tor_x;
    const float bz = ch(F, i, kChBackgroundWindZ) + ch(F, i, kChNestedWindZDelta) + conv_z + tor_z;
    const float by = nest_up + tor_up;
    const float den = smax(1.0e-6f, A.velocity_scale);
    const int xp = min(A.nx - 1, x + 1), xm = max(0, x - 1), zp = min(A.nz - 1, z + 1), zm = max(0, z - 1);
    float v[kDCount];
    v[kDLatticeX] = clamp_speed(bx / den);
    v[kDLatticeY] = clamp_speed(by / den);
    v[kDLatticeZ] = clamp_speed(bz / den);
    v[kDSlopeX] = 0.5f * (ch(F, midx(A, xp, y, z), kChTerrainHeight) - ch(F, midx(A, xm, y, z), kChTerrainHeight));
    v[kDSlopeZ] = 0.5f * (ch(F, midx(A, x, y, zp), kChTerrainHeight) - ch(F, midx(A, x, y, zm), kChTerrainHeight));
    const float rough = smax(0.0f, ch(F, i, kChRoughness));
    v[kDDrag] = sclamp(rough * 0.02f, 0.0f, 0.25f);
    v[kDHumidity] = sclamp(ch(F, i, kChHumidity) + conv_m + tor_m, 0.0f, 1.0f);
    v[kDAmbient] = ch(F, i, kChAmbientTarget) + ch(F, i, kChNestedAmbientDelta);
    v[kDDeep] = ch(F, i, kChDeepGroundTarget);
    v[kDSurface] = wall_temp(F, i);
    v[kDConvHeat] = ch(F, i, kChConvectiveHeating);
    v[kDTornadoHeat] = ch(F, i, kChTornadoHeating);
    v[kDTornadoUp] = tor_up;
    v[kDNestedUp] = nest_up;
    const bool solid = solid_at(F, i);
    A.flags[i] = solid ? kHydroSelfSolid : pull_class(A, x, y, z, [&](long long n) { return solid_at(F, n); });
#pragma unroll
    for (int k = 0; k < kDCount; ++k) A.derived[k * cells + i] = v[k];
}

struct Targets {
    float rho, ux, uy, uz, teq, nsurf, ndeep;
};

// compute_cell_targets (native/src/aero_lbm_mesoscale.cpp:393-530); D: the
// cell's derived forcing terms
__device__ __forceinline__ Targets cell_targets(const MesoArgs& A, const float (&f)[19], const float (&g)[19], long long i,
                                                int x, int y, int z, bool solid, const float (&D)[kDCount]) {
    const float dt = smax(1.0e-3f, A.dt_s);
    const float amb_relax = sclamp(dt / 600.0f, 0.0f, 1.0f);
    const float deep_relax = sclamp(dt / 2400.0f, 0.0f, 1.0f);
    const float surf_relax = sclamp(dt / 300.0f, 0.0f, 1.0f);
    const float wind_relax = sclamp(dt / 60.0f, 0.0f, 1.0f);
    const float deep_t = D[kDDeep], surf_t = D[kDSurface];
    if (solid) return Targets{1.0f, 0.0f, 0.0f, 0.0f, surf_t, surf_t, deep_t};
    float r = 0.0f, ux = 0.0f, uy = 0.0f, uz = 0.0f, amb = 0.0f;
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        r += f[q];
        ux += f[q] * fx_(q);
        uy += f[q] * fy_(q);
        uz += f[q] * fz_(q);
        amb += g[q];
    }
    r = smax(1.0e-6f, r);
    ux /= r;
    uy /= r;
    uz /= r;
    const float amb_t = D[kDAmbient];
    const float conv_h = D[kDConvHeat], tor_h = D[kDTornadoHeat];
    const float tor_up = D[kDTornadoUp], nest_up = D[kDNestedUp];
    const float hum = D[kDHumidity];
    const float sx = D[kDSlopeX], sz = D[kDSlopeZ];
    const float s_hl = hlap(A, A.surface, x, y, z), s_vl = vlap(A, A.surface, x, y, z);
    const float d_vl = vlap(A, A.deep, x, y, z);
    const float a_hl = hlap(A, A.ambient, x, y, z), a_vl = vlap(A, A.ambient, x, y, z);
    const float deep_i = A.deep[i], surf_i = A.surface[i];
    const float ndeep = deep_i + deep_relax * (deep_t - deep_i) + 0.01f * d_vl;
    const float damp = 1.0f - 0.12f * hum;
    const float nsurf = surf_i + surf_relax * damp * (surf_t - surf_i) + 0.10f * (ndeep - surf_i) + 0.04f * conv_h +
                        0.08f * tor_h + 0.05f * s_hl + 0.025f * s_vl;
    const float lx = D[kDLatticeX], ly = D[kDLatticeY], lz = D[kDLatticeZ];
    const float push = 0.0008f * (nsurf - amb);
    const float nsw = 1.0f - (float)y / smax(1.0f, (float)(A.ny - 1));
    const float lift = 0.0015f * (lx * sx + lz * sz) * nsw;
    const float blift = 0.0009f * (nsurf - amb) * nsw;
    const float steer_x = -0.005f * sx * lz;
    const float steer_z = 0.005f * sz * lx;
    const float drag = D[kDDrag];
    const float tux = clamp_speed(lx + steer_x + push * sx - drag * ux);
    const float tuz = clamp_speed(lz + steer_z + push * sz - drag * uz);
    const float tuy = clamp_speed(ly + lift + blift - drag * uy);
    const float rux = clamp_speed((1.0f - wind_relax) * ux + wind_relax * tux);
    const float ruy = clamp_speed((1.0f - wind_relax) * uy + wind_relax * tuy);
    const float ruz = clamp_speed((1.0f - wind_relax) * uz + wind_relax * tuz);
    const float src = amb_relax * (amb_t - amb) + (0.018f + 0.004f * hum) * (nsurf - amb) + 0.01f * (ndeep - amb) +
                      0.08f * conv_h * (0.5f + 0.5f * hum) + 0.10f * tor_h * (0.45f + 0.55f * hum) + 0.06f * tor_up +
                      0.06f * nest_up + 0.01f * a_hl + 0.02f * a_vl;
    return Targets{r, rux, ruy, ruz, amb + src, nsurf, ndeep};
}

// TRT on the hydrodynamic distribution toward feq(rho, u + F / 2 rho) with
// the Guo source and Smagorinsky on the even rate when enabled
// (native/src/aero_lbm_mesoscale.cpp:573-606 plus the restatement's options).
__device__ __forceinline__ void trt_hydro(const HydroRates& H, const float (&f)[19], float rho, float ux, float uy,
                                          float uz, bool solid, float (&pf)[19]) {
    float om_even = H.omega_even;
    const float om_odd = H.omega_odd;
    float tux = ux, tuy = uy, tuz = uz;
    const bool forced = H.forced && !solid;
    if (forced) {
        tux += 0.5f * H.fx / rho;
        tuy += 0.5f * H.fy / rho;
        tuz += 0.5f * H.fz / rho;
    }
    if (H.enable_sgs && !solid) {
        float pxx = 0.0f, pyy = 0.0f, pzz = 0.0f, pxy = 0.0f, pxz = 0.0f, pyz = 0.0f;
#pragma unroll
        for (int q = 0; q < 19; ++q) {
            const float ne = f[q] - hfeq(q, rho, tux, tuy, tuz);
            pxx += ne * (float)(mcx(q) * mcx(q));
            pyy += ne * (float)(mcy(q) * mcy(q));
            pzz += ne * (float)(mcz(q) * mcz(q));
            pxy += ne * (float)(mcx(q) * mcy(q));
            pxz += ne * (float)(mcx(q) * mcz(q));
            pyz += ne * (float)(mcy(q) * mcz(q));
        }
        const float qn = sqrtf(pxx * pxx + pyy * pyy + pzz * pzz + 2.0f * (pxy * pxy + pxz * pxz + pyz * pyz));
        const float nu0 = (H.tau_h - 0.5f) / 3.0f;
        const float cs2 = H.smagorinsky_c * H.smagorinsky_c;
        const float nut = smin(cs2 * qn / smax(1e-6f, 2.0f * rho * nu0), 5.0f * nu0);
        om_even = 1.0f / (0.5f + 3.0f * (nu0 + nut));
    }
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        const int qo = mopp(q);
        if (q > qo) continue;
        float sq = 0.0f, sqo = 0.0f;
        if (forced) {
            const float pref = 1.0f - 0.5f * om_even;
            const float cu = fx_(q) * tux + fy_(q) * tuy + fz_(q) * tuz;
            const float cf = fx_(q) * H.fx + fy_(q) * H.fy + fz_(q) * H.fz;
            const float uf = tux * H.fx + tuy * H.fy + tuz * H.fz;
            sq = pref * mw(q) * (3.0f * (cf - uf) + 9.0f * cu * cf);
            sqo = pref * mw(q) * (3.0f * (-cf - uf) + 9.0f * cu * cf);
        }
        if (q == qo) {
            const float fe = hfeq(q, rho, tux, tuy, tuz);
            pf[q] = f[q] - om_even * (f[q] - fe) + sq;
            continue;
        }
        const float fe = hfeq(q, rho, tux, tuy, tuz), feo = hfeq(qo, rho, tux, tuy, tuz);
        const float fev = 0.5f * (f[q] + f[qo]), fod = 0.5f * (f[q] - f[qo]);
        const float feev = 0.5f * (fe + feo), feod = 0.5f * (fe - feo);
        const float fep = fev - om_even * (fev - feev);
        const float fop = fod - om_odd * (fod - feod);
        pf[q] = fep + fop + sq;
        pf[qo] = fep - fop + sqo;
    }
}

// Streamed populations of cell i from the post-collision ones (pull
// streaming, native/src/aero_lbm_mesoscale.cpp:620-734). Every population is
// one load at an address formed by selects, the same for interior and
// boundary cells (half of the warps hold cells of an open side: as separate
// paths each of their 38 loads waited twice); cells that pull through an open
// side or the lid, or are blended, then replace or blend the values.
// kHydro false: the thermal populations only. I: unsigned where 19 x cells
// fits 32 bits.
template <bool kHydro, class I>
__device__ __forceinline__ void pull_model(const MesoArgs& A, long long i, int x, int y, int z, uint32_t w, float (&fn)[19],
                                           float (&gn)[19]) {
    const int nx = A.nx, ny = A.ny, nz = A.nz;
    const I cells = (I)nx * (I)ny * (I)nz, own = (I)i;
    const float *pf = A.src_f, *pg = A.src_g, *wall = A.derived + kDSurface * (long long)cells;
    if (w & kHydroSelfSolid) {
        const float wt = wall[i];
#pragma unroll
        for (int q = 0; q < 19; ++q) {
            if (kHydro) fn[q] = hfeq(q, 1.0f, 0.0f, 0.0f, 0.0f);
            gn[q] = tfeq(q, wt, 0.0f, 0.0f, 0.0f);
        }
        return;
    }
    // neighbour terms per axis: wrapped sides (a pull through an open side
    // loads an unused value there), the grid's own row at the ground and the lid
    I X[3], Y[3], Z[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int sx = x + k - 1, sy = y + k - 1, sz = z + k - 1;
        X[k] = (I)(sx < 0 ? sx + nx : (sx >= nx ? sx - nx : sx)) * ((I)ny * (I)nz);
        Y[k] = (I)min(max(sy, 0), ny - 1) * (I)nz;
        Z[k] = (I)(sz < 0 ? sz + nz : (sz >= nz ? sz - nz : sz));
    }
    const uint32_t ground = y == 0 ? mdirs(1, 1) : 0u, lid = (A.free_slip_top && y == ny - 1) ? mdirs(1, -1) : 0u;
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        const bool bounced = (w >> q) & 1u;
        const I src = ((ground >> q) & 1u) ? own : X[1 - mcx(q)] + Y[1 - mcy(q)] + Z[1 - mcz(q)];
        // specular reflection at the lid: the mirrored population of the same row
        const I from = (mcy(q) == -1 && (lid >> q) & 1u) ? (I)mmirror(q) * cells + src : (I)q * cells + src;
        if (kHydro) fn[q] = pf[bounced ? (I)mopp(q) * cells + own : from];
        gn[q] = *(bounced ? wall + src : pg + from);
    }
#pragma unroll
    for (int q = 0; q < 19; ++q)
        if ((w >> q) & 1u) gn[q] = tfeq(q, gn[q], 0.0f, 0.0f, 0.0f);
    if (!(w & kHydroSlow)) return;
    uint32_t away = 0;
    if (!A.periodic_sides)
        away = (x == 0 ? mdirs(0, 1) : 0u) | (x == nx - 1 ? mdirs(0, -1) : 0u) | (z == 0 ? mdirs(2, 1) : 0u) |
               (z == nz - 1 ? mdirs(2, -1) : 0u);
    if (!A.free_slip_top && y == ny - 1) away |= mdirs(1, -1);
    away &= ~ground;
    int edge = min(min(x, z), min(nx - 1 - x, nz - 1 - z));
    int top = ny - 1 - y;
    if (A.periodic_sides) edge = 1 << 20;
    if (A.free_slip_top) top = 1 << 20;
    const int sponge = min(edge, top);
    float alpha = sponge <= 0 ? 1.0f : (sponge < 2 ? 0.5f : 0.0f);
    if (!A.edge_blend) alpha = 0.0f;
    const float bx = dv(A, kDLatticeX, i), by = dv(A, kDLatticeY, i), bz = dv(A, kDLatticeZ, i), btemp = dv(A, kDAmbient, i);
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        if (((w >> q) & 1u) && !((away >> q) & 1u)) continue;
        const float fb = kHydro ? hfeq(q, 1.0f, bx, by, bz) : 0.0f, gb = tfeq(q, btemp, bx, by, bz);
        if ((away >> q) & 1u) {
            if (kHydro) fn[q] = fb;
            gn[q] = gb;
        }
        if (alpha > 0.0f) {
            if (kHydro) fn[q] = (1.0f - alpha) * fn[q] + alpha * fb;
            gn[q] = (1.0f - alpha) * gn[q] + alpha * gb;
        }
    }
}

// The same for the hydrodynamic distribution alone, in any storage, with the
// wind from the forcing itself.
template <class S, class I>
__device__ __forceinline__ void pull_hydro(const HydroArgs& A, const typename S::T* __restrict__ src, long long i, uint32_t w,
                                           float (&f)[19]) {
    if (w & kHydroSelfSolid) {
#pragma unroll
        for (int q = 0; q < 19; ++q) f[q] = hfeq(q, 1.0f, 0.0f, 0.0f, 0.0f);
        return;
    }
    const int nx = A.nx, ny = A.ny, nz = A.nz;
    const I cells = (I)nx * (I)ny * (I)nz, own = (I)i;
    int x, y, z;
    cell_xyz32(i, ny, nz, x, y, z);
    I X[3], Y[3], Z[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int sx = x + k - 1, sy = y + k - 1, sz = z + k - 1;
        X[k] = (I)(sx < 0 ? sx + nx : (sx >= nx ? sx - nx : sx)) * ((I)ny * (I)nz);
        Y[k] = (I)min(max(sy, 0), ny - 1) * (I)nz;
        Z[k] = (I)(sz < 0 ? sz + nz : (sz >= nz ? sz - nz : sz));
    }
    const uint32_t ground = y == 0 ? mdirs(1, 1) : 0u;
    const bool lid = A.free_slip_top && y == ny - 1;
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        const I from = X[1 - mcx(q)] + Y[1 - mcy(q)] + Z[1 - mcz(q)] + (mcy(q) == -1 && lid ? (I)mmirror(q) : (I)q) * cells;
        f[q] = S::load(src + (((w >> q) & 1u) ? (I)mopp(q) * cells + own : from), q, A.inv_scale);
    }
    if (!(w & kHydroSlow)) return;
    uint32_t away = 0;
    if (!A.periodic_sides)
        away = (x == 0 ? mdirs(0, 1) : 0u) | (x == nx - 1 ? mdirs(0, -1) : 0u) | (z == 0 ? mdirs(2, 1) : 0u) |
               (z == nz - 1 ? mdirs(2, -1) : 0u);
    if (!A.free_slip_top && y == ny - 1) away |= mdirs(1, -1);
    away &= ~ground;
    int edge = min(min(x, z), min(nx - 1 - x, nz - 1 - z));
    int top = ny - 1 - y;
    if (A.periodic_sides) edge = 1 << 20;
    if (A.free_slip_top) top = 1 << 20;
    const int sponge = min(edge, top);
    float alpha = sponge <= 0 ? 1.0f : (sponge < 2 ? 0.5f : 0.0f);
    if (!A.edge_blend) alpha = 0.0f;
    // the inflow wind is read only where a pull leaves the grid through an
    // open side or the open top, or where the edge blend acts
    if (away == 0 && alpha <= 0.0f) return;
    const float* F = A.forcing_prev;
    const float den = smax(1.0e-6f, A.velocity_scale);
    const float bx = clamp_speed((ch(F, i, kChBackgroundWindX) + ch(F, i, kChNestedWindXDelta) + ch(F, i, kChConvectiveInflowX) +
                                  ch(F, i, kChTornadoWindX)) / den);
    const float bz = clamp_speed((ch(F, i, kChBackgroundWindZ) + ch(F, i, kChNestedWindZDelta) + ch(F, i, kChConvectiveInflowZ) +
                                  ch(F, i, kChTornadoWindZ)) / den);
    const float by = clamp_speed((ch(F, i, kChNestedUpdraft) + ch(F, i, kChTornadoUpdraft)) / den);
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        if (((w >> q) & 1u) && !((away >> q) & 1u)) continue;
        const float fb = hfeq(q, 1.0f, bx, by, bz);
        if ((away >> q) & 1u) f[q] = fb;
        if (alpha > 0.0f) f[q] = (1.0f - alpha) * f[q] + alpha * fb;
    }
}

// Targets + TRT of both distributions (native/src/aero_lbm_mesoscale.cpp:573-618).
// kPull: the last step's streaming on the way in, so that a window of steps
// reads and writes the populations once per step instead of twice
// (128 x 24 x 128, 30 steps and the state: 1,975 us; 2,161 launched one after
// the other, 3,714 as collide + stream over the forcing records).
template <bool kPull, class I>
__global__ void __launch_bounds__(128) meso_collide_kernel(MesoArgs A) {
    pdl_trigger();
    pdl_wait();
    const long long cells = (long long)A.nx * A.ny * A.nz;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cells) return;
    int x, y, z;
    cell_xyz32(i, A.ny, A.nz, x, y, z);
    const uint32_t w = A.flags[i];
    // the derived terms first: ordinary loads (pdl.cuh) that no branch or store
    // of the pull holds back (128 x 24 x 128, 30 steps: 1,963 us against 2,081
    // where cell_targets loads them)
    float D[kDCount];
#pragma unroll
    for (int k = 0; k < kDCount; ++k) D[k] = dv(A, k, i);
    float f[19], g[19];
    if (kPull) {
        pull_model<true, I>(A, i, x, y, z, w, f, g);
    } else {
#pragma unroll
        for (int q = 0; q < 19; ++q) {
            f[q] = A.src_f[q * cells + i];
            g[q] = A.src_g[q * cells + i];
        }
    }
    const bool solid = (w & kHydroSelfSolid) != 0;
    const Targets t = cell_targets(A, f, g, i, x, y, z, solid, D);
    A.next_deep[i] = t.ndeep;
    A.next_surface[i] = t.nsurf;
    float pf[19];
    trt_hydro(A.h, f, t.rho, t.ux, t.uy, t.uz, solid, pf);
    const float om_t_even = A.omega_t_even, om_t_odd = A.omega_t_odd;
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        A.dst_f[q * cells + i] = pf[q];
        const int qo = mopp(q);
        if (q > qo) continue;
        if (q == qo) {
            const float ge = tfeq(q, t.teq, t.ux, t.uy, t.uz);
            A.dst_g[q * cells + i] = g[q] - om_t_even * (g[q] - ge);
            continue;
        }
        const float ge = tfeq(q, t.teq, t.ux, t.uy, t.uz), geo = tfeq(qo, t.teq, t.ux, t.uy, t.uz);
        const float gev = 0.5f * (g[q] + g[qo]), god = 0.5f * (g[q] - g[qo]);
        const float geev = 0.5f * (ge + geo), geod = 0.5f * (ge - geo);
        const float gep = gev - om_t_even * (gev - geev);
        const float gop = god - om_t_odd * (god - geod);
        A.dst_g[q * cells + i] = gep + gop;
        A.dst_g[qo * cells + i] = gep - gop;
    }
}

template <class I>
__global__ void __launch_bounds__(128) meso_ambient_kernel(MesoArgs A) {
    pdl_trigger();
    pdl_wait();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)A.nx * A.ny * A.nz) return;
    int x, y, z;
    cell_xyz32(i, A.ny, A.nz, x, y, z);
    const uint32_t w = A.flags[i];
    if (w & kHydroSelfSolid) {
        A.ambient[i] = dv(A, kDSurface, i);
        return;
    }
    float f[19], g[19];
    pull_model<false, I>(A, i, x, y, z, w, f, g);
    float amb = 0.0f;
#pragma unroll
    for (int q = 0; q < 19; ++q) amb += g[q];
    A.ambient[i] = amb;
}

// Pull streaming and macro export (native/src/aero_lbm_mesoscale.cpp:620-734).
template <class I>
__global__ void __launch_bounds__(128) meso_stream_kernel(MesoArgs A) {
    pdl_trigger();
    pdl_wait();
    const long long cells = (long long)A.nx * A.ny * A.nz;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cells) return;
    int x, y, z;
    cell_xyz32(i, A.ny, A.nz, x, y, z);
    const uint32_t w = A.flags[i];
    float* out = A.out_state ? A.out_state + i * kMesoStateChannels : nullptr;
    float fn[19], gn[19];
    pull_model<true, I>(A, i, x, y, z, w, fn, gn);
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        A.dst_f[q * cells + i] = fn[q];
        A.dst_g[q * cells + i] = gn[q];
    }
    if (w & kHydroSelfSolid) {
        const float wt = dv(A, kDSurface, i);
        A.ambient[i] = wt;
        if (out) {
            out[0] = wt;
            out[1] = A.deep[i];
            out[2] = A.surface[i];
            out[3] = 0.0f;
            out[4] = 0.0f;
            out[5] = 0.0f;
        }
        return;
    }
    float r = 0.0f, ux = 0.0f, uy = 0.0f, uz = 0.0f, amb = 0.0f;
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        r += fn[q];
        ux += fn[q] * fx_(q);
        uy += fn[q] * fy_(q);
        uz += fn[q] * fz_(q);
        amb += gn[q];
    }
    r = smax(1.0e-6f, r);
    ux /= r;
    uy /= r;
    uz /= r;
    A.ambient[i] = amb;
    if (out) {
        const float ms = A.max_speed;
        out[0] = amb;
        out[1] = A.deep[i];
        out[2] = A.surface[i];
        out[3] = sclamp(ux * A.velocity_scale, -ms, ms);
        out[4] = sclamp(uy * A.velocity_scale, -ms, ms);
        out[5] = sclamp(uz * A.velocity_scale, -ms, ms);
    }
}

// seed_mesoscale_state (native/src/aero_lbm_mesoscale.cpp:298-333)
__global__ void meso_seed_kernel(MesoArgs A) {
    const long long cells = (long long)A.nx * A.ny * A.nz;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cells) return;
    const float* F = A.forcing;
    const float amb_t = ch(F, i, kChAmbientTarget) + ch(F, i, kChNestedAmbientDelta);
    const float surf_t = ch(F, i, kChSurfaceTarget) + ch(F, i, kChNestedSurfaceDelta);
    const bool s = solid_at(F, i);
    const float bx = ch(F, i, kChBackgroundWindX) + ch(F, i, kChNestedWindXDelta);
    const float bz = ch(F, i, kChBackgroundWindZ) + ch(F, i, kChNestedWindZDelta);
    const float by = ch(F, i, kChNestedUpdraft) + ch(F, i, kChTornadoUpdraft);
    const float den = smax(1.0e-6f, A.velocity_scale);
    const float lx = clamp_speed((s ? 0.0f : bx) / den);
    const float ly = clamp_speed((s ? 0.0f : by) / den);
    const float lz = clamp_speed((s ? 0.0f : bz) / den);
    const float amb = s ? surf_t : amb_t;
    A.ambient[i] = amb;
    A.deep[i] = ch(F, i, kChDeepGroundTarget);
    A.surface[i] = surf_t;
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        A.dst_f[q * cells + i] = hfeq(q, 1.0f, lx, ly, lz);
        A.dst_g[q * cells + i] = tfeq(q, amb, lx, ly, lz);
    }
}


// ---------------------------------------------------------------------------
// Hydrodynamic-only step (the mesoscale hydrodynamic distribution without the
// thermal distribution and without target relaxation: the collision relaxes
// toward the cell's own rho and u). One fused launch per call: pull the
// previous call's post-collision populations with the previous call's mask
// and forcing (the reference streams at the end of each call with that call's
// inputs), then collide with this call's mask. The first call collides the
// seeded state; outputs stream the current post-collision state once more.
// Two population buffers; each holds post-collision values.
//
// Bound: issue (one scalar cell per thread in the reference's order). Every
// load has one selected 32-bit address (64-bit where 19 x cells needs it):
// 256 x 64 x 256, FP32 209 us a step, 16-bit fixed point 223, against 280 and
// 300 with a divergent second pull path and 64-bit addresses.
template <class S, int kMode, class I>
__global__ void __launch_bounds__(256) meso_hydro_kernel(HydroArgs A) {
    using T = typename S::T;
    const int nx = A.nx, ny = A.ny, nz = A.nz;
    const I cells = (I)nx * (I)ny * (I)nz;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)nx * ny * nz) return;
    const I own = (I)i;
    const T* __restrict__ src = static_cast<const T*>(A.src);
    float f[19];
    if (kMode == kHydroInit) {
#pragma unroll
        for (int q = 0; q < 19; ++q) f[q] = S::load(src + ((I)q * cells + own), q, A.inv_scale);
    } else {
        pull_hydro<S, I>(A, src, i, A.flags_prev[i], f);
    }
    if (kMode == kHydroOutput) {
        static_assert(kMesoStateChannels == 6, "three words of two floats");
        float2* o = reinterpret_cast<float2*>(A.out_state) + 3 * i;
        if (A.flags_prev[i] & kHydroSelfSolid) {
            o[0] = make_float2(1.0f, 0.0f);
            o[1] = o[2] = make_float2(0.0f, 0.0f);
            return;
        }
        float r = 0.0f, ux = 0.0f, uy = 0.0f, uz = 0.0f;
#pragma unroll
        for (int q = 0; q < 19; ++q) {
            r += f[q];
            ux += f[q] * fx_(q);
            uy += f[q] * fy_(q);
            uz += f[q] * fz_(q);
        }
        r = smax(1.0e-6f, r);
        ux /= r;
        uy /= r;
        uz /= r;
        const float ms = A.max_speed;
        o[0] = make_float2(r, 0.0f);
        o[1] = make_float2(0.0f, sclamp(ux * A.velocity_scale, -ms, ms));
        o[2] = make_float2(sclamp(uy * A.velocity_scale, -ms, ms), sclamp(uz * A.velocity_scale, -ms, ms));
        return;
    }
    const bool solid = A.solid_cur[i] != 0;
    float r = 1.0f, ux = 0.0f, uy = 0.0f, uz = 0.0f;
    if (!solid) {
        r = 0.0f;
#pragma unroll
        for (int q = 0; q < 19; ++q) {
            r += f[q];
            ux += f[q] * fx_(q);
            uy += f[q] * fy_(q);
            uz += f[q] * fz_(q);
        }
        r = smax(1.0e-6f, r);
        ux /= r;
        uy /= r;
        uz /= r;
    }
    float pf[19];
    trt_hydro(A.h, f, r, ux, uy, uz, solid, pf);
    T* __restrict__ dst = static_cast<T*>(A.dst);
#pragma unroll
    for (int q = 0; q < 19; ++q) S::store(dst + ((I)q * cells + own), q, pf[q], A.scale);
}

// Seed of the hydrodynamic-only state: seed_mesoscale_state's populations
// (native/src/aero_lbm_mesoscale.cpp:298-333) and the solid mask.
template <class S>
__global__ void meso_hydro_seed_kernel(const float* __restrict__ F, int nx, int ny, int nz, float velocity_scale,
                                       float scale, typename S::T* __restrict__ dst, uint8_t* __restrict__ solid) {
    const long long cells = (long long)nx * ny * nz;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cells) return;
    const bool s = solid_at(F, i);
    const float bx = ch(F, i, kChBackgroundWindX) + ch(F, i, kChNestedWindXDelta);
    const float bz = ch(F, i, kChBackgroundWindZ) + ch(F, i, kChNestedWindZDelta);
    const float by = ch(F, i, kChNestedUpdraft) + ch(F, i, kChTornadoUpdraft);
    const float den = smax(1.0e-6f, velocity_scale);
    const float lx = clamp_speed((s ? 0.0f : bx) / den);
    const float ly = clamp_speed((s ? 0.0f : by) / den);
    const float lz = clamp_speed((s ? 0.0f : bz) / den);
    solid[i] = s ? 1 : 0;
#pragma unroll
    for (int q = 0; q < 19; ++q) S::store(dst + q * cells + i, q, hfeq(q, 1.0f, lx, ly, lz), scale);
}

__global__ void meso_hydro_flags_kernel(HydroArgs A, const uint8_t* __restrict__ solid, uint32_t* __restrict__ flags) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)A.nx * A.ny * A.nz) return;
    int x, y, z;
    cell_xyz32(i, A.ny, A.nz, x, y, z);
    flags[i] = solid[i] ? kHydroSelfSolid : pull_class(A, x, y, z, [&](long long n) { return __ldg(solid + n) != 0; });
}

__global__ void meso_mask_kernel(const float* __restrict__ F, long long cells, uint8_t* __restrict__ solid) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < cells) solid[i] = solid_at(F, i) ? 1 : 0;
}

}  // namespace meso

cudaError_t meso_launch_seed(const meso::MesoArgs& a, cudaStream_t s) {
    const long long cells = (long long)a.nx * a.ny * a.nz;
    meso::meso_seed_kernel<<<(unsigned)((cells + 127) / 128), 128, 0, s>>>(a);
    count_launch();
    return cudaGetLastError();
}

static unsigned model_blocks(const meso::MesoArgs& a) { return (unsigned)(((long long)a.nx * a.ny * a.nz + 127) / 128); }

cudaError_t meso_launch_derive(const meso::MesoArgs& a, cudaStream_t s) {
    meso::meso_derive_kernel<<<model_blocks(a), 128, 0, s>>>(a);
    count_launch();
    return cudaGetLastError();
}

// 32-bit population indices where they fit.
static bool model_narrow(const meso::MesoArgs& a) { return 19LL * a.nx * a.ny * a.nz < (1LL << 32); }

// The kernels of a step follow one another through programmatic launches:
// each waits for its predecessor before it reads anything, so only the launch
// gaps overlap (8 x 4 x 8 host-driven step 43.8 us against
// 46.1 us one after the other, 42.0 with the classification in the derive
// kernel; 128 x 24 x 128, 30 resident steps 2,081 against 2,161).
template <class K>
static cudaError_t model_launch(K kernel, const meso::MesoArgs& a, cudaStream_t s) {
    count_launch();
    return launch_pdl(kernel, dim3(model_blocks(a)), dim3(128), 0, s, a);
}

cudaError_t meso_launch_collide(const meso::MesoArgs& a, bool pull, cudaStream_t s) {
    using Wide = unsigned long long;
    if (!pull) return model_launch(meso::meso_collide_kernel<false, Wide>, a, s);
    return model_narrow(a) ? model_launch(meso::meso_collide_kernel<true, unsigned>, a, s)
                           : model_launch(meso::meso_collide_kernel<true, Wide>, a, s);
}

cudaError_t meso_launch_ambient(const meso::MesoArgs& a, cudaStream_t s) {
    return model_narrow(a) ? model_launch(meso::meso_ambient_kernel<unsigned>, a, s)
                           : model_launch(meso::meso_ambient_kernel<unsigned long long>, a, s);
}

cudaError_t meso_launch_stream(const meso::MesoArgs& a, cudaStream_t s) {
    return model_narrow(a) ? model_launch(meso::meso_stream_kernel<unsigned>, a, s)
                           : model_launch(meso::meso_stream_kernel<unsigned long long>, a, s);
}

cudaError_t meso_hydro_seed(const float* forcing, int nx, int ny, int nz, float velocity_scale, int storage, float scale,
                            void* dst, uint8_t* solid, cudaStream_t s) {
    const long long cells = (long long)nx * ny * nz;
    const unsigned blocks = (unsigned)((cells + 255) / 256);
    if (storage == kMesoStoreF16)
        meso::meso_hydro_seed_kernel<meso::MesoF16><<<blocks, 256, 0, s>>>(forcing, nx, ny, nz, velocity_scale, scale,
                                                                           static_cast<__half*>(dst), solid);
    else if (storage == kMesoStoreI16)
        meso::meso_hydro_seed_kernel<meso::MesoI16><<<blocks, 256, 0, s>>>(forcing, nx, ny, nz, velocity_scale, scale,
                                                                           static_cast<short*>(dst), solid);
    else
        meso::meso_hydro_seed_kernel<meso::MesoF32><<<blocks, 256, 0, s>>>(forcing, nx, ny, nz, velocity_scale, scale,
                                                                           static_cast<float*>(dst), solid);
    count_launch();
    return cudaGetLastError();
}

cudaError_t meso_hydro_flags(const meso::HydroArgs& a, const uint8_t* solid, uint32_t* flags, cudaStream_t s) {
    const long long cells = (long long)a.nx * a.ny * a.nz;
    meso::meso_hydro_flags_kernel<<<(unsigned)((cells + 255) / 256), 256, 0, s>>>(a, solid, flags);
    count_launch();
    return cudaGetLastError();
}

cudaError_t meso_hydro_mask(const float* forcing, long long cells, uint8_t* solid, cudaStream_t s) {
    meso::meso_mask_kernel<<<(unsigned)((cells + 255) / 256), 256, 0, s>>>(forcing, cells, solid);
    count_launch();
    return cudaGetLastError();
}

template <class S, class I>
static void hydro_dispatch(const meso::HydroArgs& a, int mode, unsigned blocks, int threads, cudaStream_t s) {
    if (mode == kHydroInit)
        meso::meso_hydro_kernel<S, kHydroInit, I><<<blocks, threads, 0, s>>>(a);
    else if (mode == kHydroStep)
        meso::meso_hydro_kernel<S, kHydroStep, I><<<blocks, threads, 0, s>>>(a);
    else
        meso::meso_hydro_kernel<S, kHydroOutput, I><<<blocks, threads, 0, s>>>(a);
}

template <class S>
static void hydro_dispatch(const meso::HydroArgs& a, int mode, unsigned blocks, int threads, cudaStream_t s) {
    // 32-bit element indices where 19 x cells fits them
    if (19LL * a.nx * a.ny * a.nz < (1LL << 32)) hydro_dispatch<S, unsigned>(a, mode, blocks, threads, s);
    else hydro_dispatch<S, long long>(a, mode, blocks, threads, s);
}

cudaError_t meso_hydro_launch(const meso::HydroArgs& a, int mode, int storage, int threads, cudaStream_t s) {
    if (threads != 64 && threads != 128 && threads != 256) return cudaErrorInvalidValue;
    const long long cells = (long long)a.nx * a.ny * a.nz;
    const unsigned blocks = (unsigned)((cells + threads - 1) / threads);
    if (storage == kMesoStoreF16)
        hydro_dispatch<meso::MesoF16>(a, mode, blocks, threads, s);
    else if (storage == kMesoStoreI16)
        hydro_dispatch<meso::MesoI16>(a, mode, blocks, threads, s);
    else
        hydro_dispatch<meso::MesoF32>(a, mode, blocks, threads, s);
    count_launch();
    return cudaGetLastError();
}

}  // namespace aero
