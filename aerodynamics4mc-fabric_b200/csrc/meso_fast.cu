// Packed D3Q19 hydrodynamic step: two z-adjacent cells per thread, the TRT
// collision (Smagorinsky on the even rate, Guo body force) in sm_100 packed
// FP32 (FFMA2 / FADD2 / FMUL2), built with multiply-add contraction.
//
// Same scheme and call semantics as meso_hydro_kernel<S, kHydroStep>
// (meso_exact.cu): pull the previous call's post-collision populations with
// the previous call's mask and forcing, collide with this call's mask. It
// differs in arithmetic only: sums skip the zero lattice components, the
// non-equilibrium second moment is the population second moment minus the
// equilibrium's rho (I/3 + u u), and the TRT works on the even / odd halves of
// each direction pair — agreement with the reference-order kernel is to FP32
// rounding, not bit for bit. Warps without a bounce or a wrap along z read
// their 19 slots at line-uniform offsets; the others select each slot's
// address; what an open side, an open lid or the edge blend put in its place
// is settled after the loads.
#include <cuda_fp16.h>

#include <type_traits>

#include "collide27_x2.cuh"
#include "d3q27_kernels.cuh"
#include "lattice.cuh"
#include "meso.cuh"
#include "meso_lattice.cuh"

namespace aero {
namespace meso {
namespace {

__device__ __forceinline__ float hfeq_f(int q, float r, float ux, float uy, float uz) {
    const float cu = 3.0f * ((float)mcx(q) * ux + (float)mcy(q) * uy + (float)mcz(q) * uz);
    const float uu = ux * ux + uy * uy + uz * uz;
    return mw(q) * r * (1.0f + cu + 0.5f * cu * cu - 1.5f * uu);
}
__device__ __forceinline__ float clamp_sp(float u) { return fminf(0.35f, fmaxf(-0.35f, u)); }

// Directions whose component along the axis is `sign`, as a bit set.
__host__ __device__ constexpr uint32_t hdirs(int axis, int sign) {
    uint32_t m = 0;
    for (int q = 0; q < 19; ++q)
        if ((axis == 0 ? mcx(q) : (axis == 1 ? mcy(q) : mcz(q))) == sign) m |= 1u << q;
    return m;
}

// What a solid cell, or a cell at an open side, an open lid or in the edge
// blend, takes instead of (or blended into) the loaded populations: the pull
// rules of meso_hydro_kernel. A rare lane (an edge of an open grid, a solid
// cell), after the loads that every lane makes.
__device__ __forceinline__ void settle_cell(const HydroArgs& A, long long i, int x, int y, int z, uint32_t w, float (&f)[19]) {
    const int nx = A.nx, ny = A.ny, nz = A.nz;
    if (w & kHydroSelfSolid) {
#pragma unroll
        for (int q = 0; q < 19; ++q) f[q] = mw(q);
        return;
    }
    if (!(w & kHydroSlow)) return;
    uint32_t away = 0;
    if (!A.periodic_sides)
        away = (x == 0 ? hdirs(0, 1) : 0u) | (x == nx - 1 ? hdirs(0, -1) : 0u) | (z == 0 ? hdirs(2, 1) : 0u) |
               (z == nz - 1 ? hdirs(2, -1) : 0u);
    if (!A.free_slip_top && y == ny - 1) away |= hdirs(1, -1);
    if (y == 0) away &= ~hdirs(1, 1);
    int edge = min(min(x, z), min(nx - 1 - x, nz - 1 - z));
    int top = ny - 1 - y;
    if (A.periodic_sides) edge = 1 << 20;
    if (A.free_slip_top) top = 1 << 20;
    const int sponge = min(edge, top);
    float alpha = sponge <= 0 ? 1.0f : (sponge < 2 ? 0.5f : 0.0f);
    if (!A.edge_blend) alpha = 0.0f;
    if (away == 0 && alpha <= 0.0f) return;
    const float* F = A.forcing_prev + i * kMesoForcingChannels;
    const float den = fmaxf(1.0e-6f, A.velocity_scale);
    const float bx = clamp_sp((F[kChBackgroundWindX] + F[kChNestedWindXDelta] + F[kChConvectiveInflowX] + F[kChTornadoWindX]) / den);
    const float bz = clamp_sp((F[kChBackgroundWindZ] + F[kChNestedWindZDelta] + F[kChConvectiveInflowZ] + F[kChTornadoWindZ]) / den);
    const float by = clamp_sp((F[kChNestedUpdraft] + F[kChTornadoUpdraft]) / den);
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        const bool gone = (away >> q) & 1u;
        if (((w >> q) & 1u) && !gone) continue;
        const float fb = hfeq_f(q, 1.0f, bx, by, bz);
        if (gone) f[q] = fb;
        if (alpha > 0.0f) f[q] = (1.0f - alpha) * f[q] + alpha * fb;
    }
}

// signed sum of the lanes' values over the non-zero components of c_q
template <int q>
__device__ __forceinline__ F2 cdot2(F2 x, F2 y, F2 z) {
    constexpr int cx = mcx(q), cy = mcy(q), cz = mcz(q);
    F2 s;
    bool any = false;
    if (cx != 0) { s = cx > 0 ? x : -x; any = true; }
    if (cy != 0) { s = any ? (cy > 0 ? s + y : s - y) : (cy > 0 ? y : -y); any = true; }
    if (cz != 0) { s = any ? (cz > 0 ? s + z : s - z) : (cz > 0 ? z : -z); any = true; }
    return s;
}

template <int q>
__device__ __forceinline__ float cdot1(float x, float y, float z) {
    return (float)mcx(q) * x + (float)mcy(q) * y + (float)mcz(q) * z;
}

// one direction pair (q, q + 1) of the TRT update; the results are twice the
// populations (the halves of the even and odd parts, exact powers of two, go
// into the store: its own product for 16-bit storage, one product for FP32)
template <int q>
__device__ __forceinline__ void trt_pair(F2 (&f)[19], const HydroRates& H, F2 rho2, F2 tux, F2 tuy, F2 tuz, F2 uu, F2 om_e,
                                         F2 pref2, F2 uf) {
    constexpr int qo = q + 1;
    const F2 w = f2(mw(q));
    const F2 cu = cdot2<q>(tux, tuy, tuz);
    const F2 wr = w * rho2;
    const F2 feq_even = wr * fma2(f2(4.5f) * cu, cu, fma2(f2(-1.5f), uu, f2(1.0f)));
    const F2 feq_odd = (f2(3.0f) * wr) * cu;
    const F2 fev = f[q] + f[qo];
    const F2 fod = f[q] - f[qo];
    const F2 fep = fev - om_e * (fev - feq_even);
    const F2 fop = fod - f2(H.omega_odd) * (fod - feq_odd);
    F2 A = f2(0.0f), B = f2(0.0f);
    if (H.forced) {
        const float cf = cdot1<q>(H.fx, H.fy, H.fz);
        const F2 pw = pref2 * w;
        A = pw * fma2(f2(9.0f * cf), cu, f2(-3.0f) * uf);
        B = pw * f2(3.0f * cf);
    }
    f[q] = (fep + fop) + (A + B);
    f[qo] = (fep - fop) + (A - B);
}

// Two adjacent populations of one direction: raw storage words (loaded
// first, decoded after every load of the cell pair has been issued) and the
// decoded values. Stores are one word: the pair's own index i0 is even (nz
// even) and so is every q * cells.
// Scalar loads: 2-element vector loads of the aligned pairs measured slower
// (256 x 64 x 256, FP16 168 us against 131).
template <class S>
struct MesoPair;
template <>
struct MesoPair<MesoF32> {
    using Raw = float2;
    __device__ __forceinline__ static Raw raw(const float* p0, const float* p1) { return make_float2(__ldg(p0), __ldg(p1)); }
    __device__ __forceinline__ static F2 decode(Raw r, int, float) { return F2{r}; }
    __device__ __forceinline__ static void store(float* p, int, F2 v, float, float by) {
        *reinterpret_cast<float2*>(p) = by == 1.0f ? v.v : (f2(by) * v).v;
    }
};
template <>
struct MesoPair<MesoF16> {
    using Raw = __half2;
    __device__ __forceinline__ static Raw raw(const __half* p0, const __half* p1) { return __halves2half2(__ldg(p0), __ldg(p1)); }
    __device__ __forceinline__ static F2 decode(Raw r, int q, float inv_scale) {
        const float w = mw(q), k = w * inv_scale;
        return F2{__ffma2_rn(__half22float2(r), make_float2(k, k), make_float2(w, w))};
    }
    __device__ __forceinline__ static void store(__half* p, int q, F2 v, float scale, float by) {
        const float k = scale * (1.0f / mw(q)) * by;
        const float2 h = __ffma2_rn(v.v, make_float2(k, k), make_float2(-scale, -scale));
        *reinterpret_cast<__half2*>(p) = __floats2half2_rn(h.x, h.y);
    }
};
template <>
struct MesoPair<MesoI16> {
    using Raw = short2;
    __device__ __forceinline__ static Raw raw(const short* p0, const short* p1) { return make_short2(__ldg(p0), __ldg(p1)); }
    __device__ __forceinline__ static F2 decode(Raw r, int q, float inv_scale) {
        const float w = mw(q), k = w * inv_scale;
        const unsigned bits = (unsigned)(unsigned short)r.x | ((unsigned)(unsigned short)r.y << 16);
        return F2{__ffma2_rn(s16x2_to_float2(bits), make_float2(k, k), make_float2(w, w))};
    }
    __device__ __forceinline__ static void store(short* p, int q, F2 v, float scale, float by) {
        const float k = scale * (1.0f / mw(q)) * by;
        const float2 h = __ffma2_rn(v.v, make_float2(k, k), make_float2(-scale, -scale));
        *reinterpret_cast<short2*>(p) = make_short2(sat_round_s16(h.x), sat_round_s16(h.y));
    }
};

// kWide: 64-bit slot offsets (grids of 19 x cells >= 2^31 elements); else
// the launch-uniform offsets of a direction are 32-bit and every slot address
// is the pair's own address plus one of them.
//
// Bound: issue and load latency, not memory (256 x 64 x 256: 340 MB a step in
// 16 bits, classification and mask included, 52 us at the measured copy rate). Every lane issues its 19 loads
// through one selected address each: no divergent slow pull, and the lid, the
// ground and open sides ride along, so a warp at the lid keeps the uniform
// path. Blocks per SM by storage: the 16-bit forms hold their raw words in
// half the registers, so 7 blocks (72 registers) beat 5 / 6 / 8 (16-bit fixed
// point 106.0 us against 111.0 / 108.8 / 119.0, FP16 100.6 against 104.9 /
// 100.7 / 107.0); FP32 wants 5 (96 registers: 122.6 us against 146.2 / 142.4
// / 157.2 at 6 / 7 / 8). With the two-path pull and 6 blocks for all it was
// 136.1 (16-bit), 131.6 (FP16) and 131.1 us (FP32).
template <class S>
constexpr int kHydroBlocks = sizeof(typename S::T) == 4 ? 5 : 7;
template <class S, bool kWide>
__global__ void __launch_bounds__(128, kHydroBlocks<S>) meso_hydro2_kernel(HydroArgs A) {
    using T = typename S::T;
    using Off = typename std::conditional<kWide, long long, int>::type;
    const int nx = A.nx, ny = A.ny, nz = A.nz;
    const int z0 = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
    if (z0 >= nz) return;
    const int y = blockIdx.y, x = blockIdx.z;
    const long long cells = (long long)nx * ny * nz;
    const long long i0 = ((long long)x * ny + y) * nz + z0;
    const T* __restrict__ src = static_cast<const T*>(A.src);
    const uint32_t w0 = A.flags_prev[i0], w1 = A.flags_prev[i0 + 1];
    F2 f[19];
    {
        // Sources leave the grid along x for the whole line (both cells alike), along z for the first
        // cell of the line's first pair and the second cell of its last pair
        // only: they wrap around (periodic sides; an open side's value is
        // replaced below). At the lid a pull stays in the row, with the
        // mirrored direction when the lid reflects.
        const T* __restrict__ own = src + i0;
        const Off plane = (Off)cells;
        const bool xlo = x == 0, xhi = x == nx - 1, zlo = z0 == 0, zhi = z0 + 2 == nz, floor = y == 0, lid = y == ny - 1;
        typename MesoPair<S>::Raw raw[19];
        auto normal = [&](int q) {  // line-uniform
            Off n = (Off)q * plane - (((Off)mcx(q) * ny + mcy(q)) * nz + mcz(q));
            if (mcx(q) == 1 && xlo) n += plane;
            if (mcx(q) == -1 && xhi) n -= plane;
            if (mcy(q) == -1 && lid) n += (Off)((A.free_slip_top ? mmirror(q) : q) - q) * plane - (Off)nz;
            return n;
        };
        // a warp none of whose lanes bounces back or leaves along z reads
        // every slot at its line-uniform offset
        if (__all_sync(__activemask(), ((w0 | w1) & ((1u << 19) - 1u)) == 0u && !zlo && !zhi) && !floor) {
#pragma unroll
            for (int q = 0; q < 19; ++q) raw[q] = MesoPair<S>::raw(own + normal(q), own + normal(q) + 1);
        } else {
#pragma unroll
            for (int q = 0; q < 19; ++q) {
                const Off n0 = normal(q);
                const Off na = n0 + ((mcz(q) == 1 && zlo) ? (Off)nz : (Off)0);
                const Off nb = n0 - ((mcz(q) == -1 && zhi) ? (Off)nz : (Off)0);
                const Off b0 = (Off)mopp(q) * plane;
                const bool under = mcy(q) == 1 && floor;  // also of solid cells, which set no bits
                const bool bb0 = under || ((w0 >> q) & 1u), bb1 = under || ((w1 >> q) & 1u);
                raw[q] = MesoPair<S>::raw(own + (bb0 ? b0 : na), own + (bb1 ? b0 : nb) + 1);
            }
        }
#pragma unroll
        for (int q = 0; q < 19; ++q) f[q] = MesoPair<S>::decode(raw[q], q, A.inv_scale);
    }
    if ((w0 | w1) & (kHydroSelfSolid | kHydroSlow)) {
        float a[19], b[19];
#pragma unroll
        for (int q = 0; q < 19; ++q) {
            a[q] = f[q].v.x;
            b[q] = f[q].v.y;
        }
        settle_cell(A, i0, x, y, z0, w0, a);
        settle_cell(A, i0 + 1, x, y, z0 + 1, w1, b);
#pragma unroll
        for (int q = 0; q < 19; ++q) f[q] = f2(a[q], b[q]);
    }

    // moments
    const F2 rsum = ((((f[0] + f[1]) + (f[2] + f[3])) + ((f[4] + f[5]) + (f[6] + f[7]))) +
                     (((f[8] + f[9]) + (f[10] + f[11])) + ((f[12] + f[13]) + (f[14] + f[15])))) + ((f[16] + f[17]) + f[18]);
    const F2 jx = ((f[1] - f[2]) + (f[7] - f[8])) + ((f[9] - f[10]) + ((f[11] - f[12]) + (f[13] - f[14])));
    const F2 jy = ((f[3] - f[4]) + (f[7] - f[8])) + ((f[10] - f[9]) + ((f[15] - f[16]) + (f[17] - f[18])));
    const F2 jz = ((f[5] - f[6]) + (f[11] - f[12])) + ((f[14] - f[13]) + ((f[15] - f[16]) + (f[18] - f[17])));
    const bool s0 = A.solid_cur[i0] != 0, s1 = A.solid_cur[i0 + 1] != 0;
    const F2 rr = fmax2(rsum, 1.0e-6f);
    const F2 ir = rcp2(rr);
    const F2 live = f2(s0 ? 0.0f : 1.0f, s1 ? 0.0f : 1.0f);
    // solid lanes relax toward rest: rho 1, u 0
    const F2 rho = f2(s0 ? 1.0f : rr.v.x, s1 ? 1.0f : rr.v.y);
    const F2 ux = live * (jx * ir), uy = live * (jy * ir), uz = live * (jz * ir);
    const HydroRates& H = A.h;
    F2 tux = ux, tuy = uy, tuz = uz;
    if (H.forced) {
        const F2 hi = live * (f2(0.5f) * ir);
        tux = fma2(f2(H.fx), hi, tux);
        tuy = fma2(f2(H.fy), hi, tuy);
        tuz = fma2(f2(H.fz), hi, tuz);
    }
    F2 om_e = f2(H.omega_even);
    if (H.enable_sgs && !(s0 && s1)) {
        const F2 sxx = (f[1] + f[2]) + ((f[7] + f[8]) + (f[9] + f[10])) + ((f[11] + f[12]) + (f[13] + f[14]));
        const F2 syy = (f[3] + f[4]) + ((f[7] + f[8]) + (f[9] + f[10])) + ((f[15] + f[16]) + (f[17] + f[18]));
        const F2 szz = (f[5] + f[6]) + ((f[11] + f[12]) + (f[13] + f[14])) + ((f[15] + f[16]) + (f[17] + f[18]));
        const F2 sxy = (f[7] + f[8]) - (f[9] + f[10]);
        const F2 sxz = (f[11] + f[12]) - (f[13] + f[14]);
        const F2 syz = (f[15] + f[16]) - (f[17] + f[18]);
        const F2 third = f2(1.0f / 3.0f);
        const F2 pxx = sxx - rho * fma2(tux, tux, third), pyy = syy - rho * fma2(tuy, tuy, third);
        const F2 pzz = szz - rho * fma2(tuz, tuz, third);
        const F2 pxy = sxy - rho * (tux * tuy), pxz = sxz - rho * (tux * tuz), pyz = syz - rho * (tuy * tuz);
        const F2 qn2 = fma2(pxx, pxx, fma2(pyy, pyy, pzz * pzz)) + f2(2.0f) * fma2(pxy, pxy, fma2(pxz, pxz, pyz * pyz));
        const F2 qn = sqrt2(fmax2(qn2, 0.0f));
        const float nu0 = (H.tau_h - 0.5f) / 3.0f;
        const F2 nut = fmin2(div2(f2(H.smagorinsky_c * H.smagorinsky_c) * qn, fmax2(f2(2.0f * nu0) * rho, 1e-6f)), 5.0f * nu0);
        const F2 om_sgs = rcp2(fma2(f2(3.0f), f2(nu0) + nut, f2(0.5f)));
        om_e = f2(s0 ? H.omega_even : om_sgs.v.x, s1 ? H.omega_even : om_sgs.v.y);
    }
    const F2 uu = fma2(tux, tux, fma2(tuy, tuy, tuz * tuz));
    F2 pref = f2(0.0f), uf = f2(0.0f);
    if (H.forced) {
        pref = live * fma2(f2(-0.5f), om_e, f2(1.0f));
        uf = fma2(tux, f2(H.fx), fma2(tuy, f2(H.fy), tuz * f2(H.fz)));
    }
    {
        const F2 w0r = f2(mw(0)) * rho;
        const F2 feq0 = w0r * fma2(f2(-1.5f), uu, f2(1.0f));
        f[0] = (f[0] - om_e * (f[0] - feq0)) + (pref * f2(mw(0))) * (f2(-3.0f) * uf);
    }
    const F2 rho2 = f2(2.0f) * rho, pref2 = f2(2.0f) * pref;
    trt_pair<1>(f, H, rho2, tux, tuy, tuz, uu, om_e, pref2, uf);
    trt_pair<3>(f, H, rho2, tux, tuy, tuz, uu, om_e, pref2, uf);
    trt_pair<5>(f, H, rho2, tux, tuy, tuz, uu, om_e, pref2, uf);
    trt_pair<7>(f, H, rho2, tux, tuy, tuz, uu, om_e, pref2, uf);
    trt_pair<9>(f, H, rho2, tux, tuy, tuz, uu, om_e, pref2, uf);
    trt_pair<11>(f, H, rho2, tux, tuy, tuz, uu, om_e, pref2, uf);
    trt_pair<13>(f, H, rho2, tux, tuy, tuz, uu, om_e, pref2, uf);
    trt_pair<15>(f, H, rho2, tux, tuy, tuz, uu, om_e, pref2, uf);
    trt_pair<17>(f, H, rho2, tux, tuy, tuz, uu, om_e, pref2, uf);
    T* __restrict__ dst = static_cast<T*>(A.dst) + i0;
#pragma unroll
    for (int q = 0; q < 19; ++q) MesoPair<S>::store(dst + (Off)q * (Off)cells, q, f[q], A.scale, q == 0 ? 1.0f : 0.5f);
}

}  // namespace
}  // namespace meso

cudaError_t meso_hydro_fast_step(const meso::HydroArgs& a, int storage, cudaStream_t s) {
    if (a.nz % 2) return cudaErrorInvalidValue;
    const int pairs = a.nz / 2;
    const int block = pairs >= 128 ? 128 : ((pairs + 31) / 32) * 32;
    const dim3 grid((unsigned)((pairs + block - 1) / block), (unsigned)a.ny, (unsigned)a.nx);
    const bool wide = 19LL * a.nx * a.ny * a.nz >= (1LL << 31);
    if (storage == kMesoStoreF16) {
        if (wide) meso::meso_hydro2_kernel<meso::MesoF16, true><<<grid, block, 0, s>>>(a);
        else meso::meso_hydro2_kernel<meso::MesoF16, false><<<grid, block, 0, s>>>(a);
    } else if (storage == kMesoStoreI16) {
        if (wide) meso::meso_hydro2_kernel<meso::MesoI16, true><<<grid, block, 0, s>>>(a);
        else meso::meso_hydro2_kernel<meso::MesoI16, false><<<grid, block, 0, s>>>(a);
    } else {
        if (wide) meso::meso_hydro2_kernel<meso::MesoF32, true><<<grid, block, 0, s>>>(a);
        else meso::meso_hydro2_kernel<meso::MesoF32, false><<<grid, block, 0, s>>>(a);
    }
    count_launch();
    return cudaGetLastError();
}

}  // namespace aero
