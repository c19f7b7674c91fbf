// Per-cell D3Q27 cumulant collision in the reference's exact operation order.
//
// Every floating-point operation of the reference CPU collide
// (native/src/aero_lbm_jni.cpp:2209-2413, with compute_raw_moments 1335-1357,
// compute_central_moments 1359-1382, cumulant_relax_closure 1384-1430,
// central_to_raw 1432-1455, raw_to_populations 1457-1473, feq
// native/src/aero_lbm_hydro_core.cpp:48-52, guo_force_source jni.cpp:1270-1281)
// is performed here in the same order with the same rounding, so the result is
// bit-identical to the reference on IEEE hardware. Rules that keep it so:
//   * this header is compiled only in translation units built with
//     --fmad=false (no multiply-add contraction), except where a product is
//     exact (a power-of-two coefficient), where fmaf gives the same rounding;
//   * terms whose coefficient is zero (c = 0 in a moment, a zero post-collision
//     central moment) are skipped: adding +-0 to a finite non-zero partial sum
//     is the identity, so the sums are unchanged;
//   * only the moments the collision reads are formed (the reference computes
//     all 27 pre-collision central moments but uses the second-order six).
// The operations left are about a quarter of the reference dense loops; the
// collision is still ALU-heavier than the factorised form (collide27.cuh).
#pragma once

#include "collide27.cuh"

namespace aero {
namespace exact {

// std::max / std::min semantics (argument order matters for NaN and zeros).
__device__ __forceinline__ float rmax(float a, float b) { return (a < b) ? b : a; }
__device__ __forceinline__ float rmin(float a, float b) { return (b < a) ? b : a; }
__device__ __forceinline__ float rclamp(float v, float lo, float hi) { return rmin(hi, rmax(lo, v)); }

__host__ __device__ constexpr int binom2(int n, int k) { return (k < 0 || k > n) ? 0 : ((n <= 1 || k == 0 || k == n) ? 1 : 2); }

// Signed sum over q (in q order) of f[q] * cx^a cy^b cz^c, terms with a zero
// coefficient skipped: the reference's raw moment / momentum sums.
template <int A, int B, int C>
__device__ __forceinline__ float qsum(const float (&f)[27]) {
    float s = 0.0f;
#pragma unroll
    for (int q = 0; q < 27; ++q) {
        const int cx = q_cx(q), cy = q_cy(q), cz = q_cz(q);
        const int px = A == 0 ? 1 : (A == 1 ? cx : cx * cx);
        const int py = B == 0 ? 1 : (B == 1 ? cy : cy * cy);
        const int pz = C == 0 ? 1 : (C == 2 ? cz * cz : (C == 1 ? cz : 1));
        const int coef = px * py * pz;
        if (coef == 0) continue;
        s = coef > 0 ? s + f[q] : s - f[q];
    }
    return s;
}

// ---- the part after the cumulant relaxation, over one cell (V = float) or
// two (V = X2 of collide27_exact_x2.cuh). It performs the reference's roundings
// and drops what rounds nothing:
//   * opposite directions share their products: c.u and c.F only change sign,
//     and every rounding commutes with a change of sign;
//   * the products of velocity powers are formed once, without the binomial
//     coefficient (1, 2, 4, 8), which goes into the sum's fused multiply-add
//     (an exact product);
//   * the 1-D inverse rows {0,-1/2,1/2}, {1,0,-1}, {0,1/2,1/2} run as plain
//     sums: populations are carried as 2^k(q) f_q (k(q): non-zero components
//     of c_q; those with c_x = -1 negated as well, so that c_x = -1 and +1
//     share the sum over R[1]) until a fused multiply-add takes them up.
// The 128^3 step (FP32 in-place, two cells per thread, B200) went from 204.8 to
// 188.7 us, its stream-collide launch from 174.9 to 160.3, without spills.
struct PlainMul {
    __device__ __forceinline__ float operator()(float a, float b) const { return a * b; }
};
template <class V>
__device__ __forceinline__ V splat(float a);
template <>
__device__ __forceinline__ float splat<float>(float a) { return a; }
// c * x + s for a power of two c: the reference's product and sum
__device__ __forceinline__ float fma_pow2(float c, float x, float s) { return fmaf(c, x, s); }
__device__ __forceinline__ float mul_pow2(float c, float x) { return c * x; }

// 2^k(q), and the sign the carried population has
__host__ __device__ constexpr float carried(int q) {
    return (q_cx(q) < 0 ? -1.0f : 1.0f) * (q_cx(q) != 0 ? 2.0f : 1.0f) * (q_cy(q) != 0 ? 2.0f : 1.0f) * (q_cz(q) != 0 ? 2.0f : 1.0f);
}

// c_q . (x, y, z) for q > 13 (the first non-zero component is +1)
template <class V>
__device__ __forceinline__ V cdot_pos(int q, V x, V y, V z) {
    const int cx = q_cx(q), cy = q_cy(q), cz = q_cz(q);
    V s = cx ? x : (cy ? y : z);
    if (cx && cy) s = cy > 0 ? s + y : s - y;
    if ((cx || cy) && cz) s = cz > 0 ? s + z : s - z;
    return s;
}

// Signed sum over q (in q order) of the carried populations' true values
// times c_A (A: 0 none, 1 x, 2 y, 3 z).
template <int A, class V>
__device__ __forceinline__ V carried_sum(const V (&fc)[27]) {
    V s;
    bool first = true;
#pragma unroll
    for (int q = 0; q < 27; ++q) {
        const int c = A == 0 ? 1 : (A == 1 ? q_cx(q) : (A == 2 ? q_cy(q) : q_cz(q)));
        if (c == 0) continue;
        const float k = (float)c / carried(q);
        s = first ? mul_pow2(k, fc[q]) : fma_pow2(k, fc[q], s);
        first = false;
    }
    return s;
}

// Carried populations fc from the post-collision central moments K
// (central_to_raw, raw_to_populations).
template <class V, class M>
__device__ __forceinline__ void central_to_populations(const M& mul, const V (&K)[3][3][3], V ux, V uy, V uz, V (&fc)[27]) {
    const V px[3] = {ux, ux, mul(ux, ux)}, py[3] = {uy, uy, mul(uy, uy)}, pz[3] = {uz, uz, mul(uz, uz)};
    // entry R[a][b][c] = sum over (p, q, r) <= (a, b, c), p + q + r even, of
    // binomials * ((ux^(a-p) uy^(b-q)) uz^(c-r)) * K[p][q][r]
    V R[3][3][3];
    auto raw = [&](int a, int b, int c) {
        V sum;
        bool first = true;
#pragma unroll
        for (int p = 0; p <= a; ++p)
#pragma unroll
            for (int qq = 0; qq <= b; ++qq)
#pragma unroll
                for (int r = 0; r <= c; ++r) {
                    if (((p + qq + r) & 1) != 0) continue;  // odd-order post-collision moments are zero
                    const int i = a - p, j = b - qq, k = c - r;
                    V t = K[p][qq][r];
                    if (i && j && k) t = mul(mul(mul(px[i], py[j]), pz[k]), t);
                    else if (i && j) t = mul(mul(px[i], py[j]), t);
                    else if (i && k) t = mul(mul(px[i], pz[k]), t);
                    else if (j && k) t = mul(mul(py[j], pz[k]), t);
                    else if (i) t = mul(px[i], t);
                    else if (j) t = mul(py[j], t);
                    else if (k) t = mul(pz[k], t);
                    const int coef = binom2(a, p) * binom2(b, qq) * binom2(c, r);
                    sum = first ? t : (coef == 1 ? sum + t : fma_pow2((float)coef, t, sum));
                    first = false;
                }
        R[a][b][c] = sum;
    };
    // signs of the two non-zero entries of inverse row i (times 2 for i != 1)
    constexpr int lo[3] = {1, 0, 1}, s_lo[3] = {-1, 1, 1}, s_hi[3] = {1, -1, 1};
    // sum + / - the entries of raw slab a for the (iy, iz) population, in (b, c)
    // order; sign: of the slab
    auto slab = [&](int a, int iy, int iz, int sign, bool start, V s) {
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int sg = sign * (b ? s_hi[iy] : s_lo[iy]) * (c ? s_hi[iz] : s_lo[iz]);
                const V r = R[a][b ? 2 : lo[iy]][c ? 2 : lo[iz]];
                if (start && b == 0 && c == 0) s = sg > 0 ? r : -r;
                else s = sg > 0 ? s + r : s - r;
            }
        return s;
    };
    // c_x = 0 reads only R[0] and R[2], the others only R[1] and R[2]: R[0] and
    // R[1] are never live together
#pragma unroll
    for (int b = 0; b < 3; ++b)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            raw(0, b, c);
            raw(2, b, c);
        }
#pragma unroll
    for (int iy = 0; iy < 3; ++iy)
#pragma unroll
        for (int iz = 0; iz < 3; ++iz) fc[9 + iy * 3 + iz] = slab(2, iy, iz, -1, false, slab(0, iy, iz, 1, true, R[0][0][0]));
#pragma unroll
    for (int b = 0; b < 3; ++b)
#pragma unroll
        for (int c = 0; c < 3; ++c) raw(1, b, c);
#pragma unroll
    for (int iy = 0; iy < 3; ++iy)
#pragma unroll
        for (int iz = 0; iz < 3; ++iz) {
            const V s = slab(1, iy, iz, 1, true, R[1][0][0]);
            fc[iy * 3 + iz] = slab(2, iy, iz, -1, false, s);       // negated
            fc[18 + iy * 3 + iz] = slab(2, iy, iz, 1, false, s);
        }
}

// feq(q) / w and feq(26 - q) / w, q > 13: rho (1 + cu + 0.5 cu^2 - 1.5 u.u), cu = 3 c.u
template <class V, class M>
__device__ __forceinline__ void feq_pair(const M& mul, int q, V wr, V ux, V uy, V uz, V uu15, V& e, V& eo) {
    const V cu = mul(splat<V>(3.0f), cdot_pos(q, ux, uy, uz));
    const V t = mul(mul(splat<V>(0.5f), cu), cu), one = splat<V>(1.0f);
    e = mul(wr, ((one + cu) + t) - uu15);
    eo = mul(wr, ((one - cu) + t) - uu15);
}

// w_q classes by the number of non-zero components: 0, 1, 2, 3
__host__ __device__ constexpr int w_class(int q) { return (q_cx(q) != 0) + (q_cy(q) != 0) + (q_cz(q) != 0); }
__host__ __device__ constexpr int w_member(int k) { return k == 0 ? 13 : (k == 1 ? 14 : (k == 2 ? 17 : 26)); }

// fc (carried) -> f: the conservation fix-up.
template <class V, class M>
__device__ __forceinline__ void conserve(const M& mul, const V (&fc)[27], V rho, V ux, V uy, V uz, V rho_c, V uxc, V uyc, V uzc,
                                         V (&f)[27]) {
    const V uu15 = mul(splat<V>(1.5f), (mul(ux, ux) + mul(uy, uy)) + mul(uz, uz));
    const V uuc15 = mul(splat<V>(1.5f), (mul(uxc, uxc) + mul(uyc, uyc)) + mul(uzc, uzc));
    V wr[4], wc[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        wr[k] = mul(splat<V>(q_w(w_member(k))), rho);
        wc[k] = mul(splat<V>(q_w(w_member(k))), rho_c);
    }
    const V one = splat<V>(1.0f);
    f[13] = fc[13] + (mul(wr[0], one - uu15) - mul(wc[0], one - uuc15));
#pragma unroll
    for (int q = 14; q < 27; ++q) {
        V e, eo, g, go;
        feq_pair(mul, q, wr[w_class(q)], ux, uy, uz, uu15, e, eo);
        feq_pair(mul, q, wc[w_class(q)], uxc, uyc, uzc, uuc15, g, go);
        f[q] = fma_pow2(1.0f / carried(q), fc[q], e - g);
        f[26 - q] = fma_pow2(1.0f / carried(26 - q), fc[26 - q], eo - go);
    }
}

// f += Guo source, pref w ((c.F - u.F) / cs2 + (c.u)(c.F) / cs4)
template <class V, class M, class Put>
__device__ __forceinline__ void guo(const M& mul, V pref, V ux, V uy, V uz, V fx, V fy, V fz, const V (&f)[27], Put put) {
    const float inv_cs2 = 1.0f / kCs2f;
    const float inv_cs4 = inv_cs2 * inv_cs2;
    const V uf = (mul(ux, fx) + mul(uy, fy)) + mul(uz, fz);
    V pw[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) pw[k] = mul(pref, splat<V>(q_w(w_member(k))));
    put(13, f[13] - mul(pw[0], mul(uf, splat<V>(inv_cs2))));
#pragma unroll
    for (int q = 14; q < 27; ++q) {
        const V cf = cdot_pos(q, fx, fy, fz);
        const V d = mul(mul(cdot_pos(q, ux, uy, uz), cf), splat<V>(inv_cs4));
        const V w = pw[w_class(q)];
        put(q, f[q] + mul(w, mul(cf - uf, splat<V>(inv_cs2)) + d));
        put(26 - q, f[26 - q] + mul(w, d - mul(cf + uf, splat<V>(inv_cs2))));
    }
}

// Collide one fluid cell in place (benchmark-mode reference collide: no fan
// forcing, no edge nudge, no sponge). Returns false, with f untouched, when
// the input is not finite; the caller reseeds the cell.
__device__ __forceinline__ bool collide27_exact(float (&f)[27], const CollideParams& P, const float* temperature,
                                                float cfx, float cfy, float cfz, CollideOut& out,
                                                const CellExtras* ex = nullptr) {
    bool bad = false;
#pragma unroll
    for (int q = 0; q < 27; ++q) bad |= !isfinite(f[q]);
    const float rho = qsum<0, 0, 0>(f);
    const float mom_x = qsum<1, 0, 0>(f);
    const float mom_y = qsum<0, 1, 0>(f);
    const float mom_z = qsum<0, 0, 1>(f);
    if (bad || !isfinite(rho) || !isfinite(mom_x) || !isfinite(mom_y) || !isfinite(mom_z)) return false;
    const float rho_safe = rmax(1e-6f, rho);
    const float inv_rho = 1.0f / rho_safe;
    float ux = mom_x * inv_rho;
    float uy = mom_y * inv_rho;
    float uz = mom_z * inv_rho;
    if (!isfinite(rho_safe) || !isfinite(inv_rho) || !isfinite(ux) || !isfinite(uy) || !isfinite(uz)) return false;
    float fx = 0.0f, fy = 0.0f, fz = 0.0f;
    if (ex && P.fan_beta > 0.0f && ex->fan_mask > 0.0f) fan_force(*ex, P, rho_safe, ux, uy, uz, fx, fy, fz);
    if (P.enable_buoyancy) {
        const float buoy = rclamp(P.buoy_beta * *temperature, -P.buoy_fmax, P.buoy_fmax);
        const float add = rho_safe * buoy;
        if (P.gravity_axis == 0) fx += add;
        else if (P.gravity_axis == 1) fy += add;
        else fz += add;
    }
    // Body force (absent from the reference; zero keeps it bit-identical).
    if (P.body_force[0] != 0.0f || P.body_force[1] != 0.0f || P.body_force[2] != 0.0f) {
        fx += P.body_force[0]; fy += P.body_force[1]; fz += P.body_force[2];
    }
    if (cfx != 0.0f || cfy != 0.0f || cfz != 0.0f) {
        fx += cfx; fy += cfy; fz += cfz;
    }
    const bool forced = (fx != 0.0f) | (fy != 0.0f) | (fz != 0.0f);
    if (forced) {
        ux += 0.5f * (fx * inv_rho);
        uy += 0.5f * (fy * inv_rho);
        uz += 0.5f * (fz * inv_rho);
        if (!isfinite(ux) || !isfinite(uy) || !isfinite(uz)) return false;
    }
    if (ex && P.state_nudge > 0.0f) {
        // runtime-mode state nudge (jni.cpp:2314-2322)
        const float sn = ex->nudge;
        ux = (1.0f - sn) * ux + sn * ex->ref_x;
        uy = (1.0f - sn) * uy + sn * ex->ref_y;
        uz = (1.0f - sn) * uz + sn * ex->ref_z;
        if (!isfinite(ux) || !isfinite(uy) || !isfinite(uz)) return false;
    }
    const float speed2 = ux * ux + uy * uy + uz * uz;
    if (!isfinite(speed2)) return false;
    if (speed2 > P.max_speed * P.max_speed) {
        const float scale = P.max_speed / sqrtf(speed2);
        ux *= scale; uy *= scale; uz *= scale;
    }
    out.rho = rho; out.ux = ux; out.uy = uy; out.uz = uz; out.reseeded = false;

    // Raw moments read by the second-order central moments (raw000 = rho and
    // raw100/010/001 = momentum are the same sums in the same order).
    const float r200 = qsum<2, 0, 0>(f), r020 = qsum<0, 2, 0>(f), r002 = qsum<0, 0, 2>(f);
    const float r110 = qsum<1, 1, 0>(f), r101 = qsum<1, 0, 1>(f), r011 = qsum<0, 1, 1>(f);

    // Second-order central moments: binomial shift with s = (1, -u, u*u), terms
    // in (p, q, r) loop order, products left to right.
    const float sx1 = -ux, sy1 = -uy, sz1 = -uz;
    const float sx2 = ux * ux, sy2 = uy * uy, sz2 = uz * uz;
    const float c200 = (sx2 * rho + (2.0f * sx1) * mom_x) + r200;
    const float c020 = (sy2 * rho + (2.0f * sy1) * mom_y) + r020;
    const float c002 = (sz2 * rho + (2.0f * sz1) * mom_z) + r002;
    const float c110 = (((sx1 * sy1) * rho + sx1 * mom_y) + sy1 * mom_x) + r110;
    const float c101 = (((sx1 * sz1) * rho + sx1 * mom_z) + sz1 * mom_x) + r101;
    const float c011 = (((sy1 * sz1) * rho + sy1 * mom_z) + sz1 * mom_y) + r011;

    const float tau_s_base = P.tau_shear_base, tau_n_base = P.tau_normal_base;
    float tau_s = tau_s_base, tau_n = tau_n_base;
    if (P.enable_sgs) {
        const float nu0 = P.nu0;
        const float nxx = c200 - rho_safe * kCs2f;
        const float nyy = c020 - rho_safe * kCs2f;
        const float nzz = c002 - rho_safe * kCs2f;
        const float q_norm2 = nxx * nxx + nyy * nyy + nzz * nzz + 2.0f * (c110 * c110 + c101 * c101 + c011 * c011);
        const float q_mag = sqrtf(rmax(0.0f, q_norm2));
        const float s_mag = q_mag / rmax(1e-6f, 2.0f * rho_safe * nu0);
        float nu_t = P.sgs_c2 * s_mag;
        nu_t = rmin(nu_t, P.sgs_nut_cap);
        tau_s = rclamp(0.5f + 3.0f * rclamp(nu0 + nu_t, kNuShearMin, kNuShearMax), kTauMin, kTauMax);
        tau_n = rclamp(tau_n_base + (tau_s - tau_s_base) * P.sgs_bulk, kTauMin, kTauMax);
    }
    const float omega_diag = 1.0f / tau_n;
    const float omega_off = 1.0f / tau_s;

    // cumulant_relax_closure with rho = rho_safe.
    float K[3][3][3];
    const float eq_second = rho_safe * kCs2f;
    const float s_diag = rclamp(omega_diag, 0.0f, 1.95f);
    const float s_off = rclamp(omega_off, 0.0f, 1.95f);
    K[0][0][0] = rho_safe;
    K[2][0][0] = c200 + s_diag * (eq_second - c200);
    K[0][2][0] = c020 + s_diag * (eq_second - c020);
    K[0][0][2] = c002 + s_diag * (eq_second - c002);
    K[1][1][0] = (1.0f - s_off) * c110;
    K[1][0][1] = (1.0f - s_off) * c101;
    K[0][1][1] = (1.0f - s_off) * c011;
    {
        const float k200 = K[2][0][0], k020 = K[0][2][0], k002 = K[0][0][2];
        const float k110 = K[1][1][0], k101 = K[1][0][1], k011 = K[0][1][1];
        const float ir = 1.0f / rmax(1e-6f, rho_safe);
        K[2][2][0] = k200 * k020 * ir + 2.0f * k110 * k110 * ir;
        K[2][0][2] = k200 * k002 * ir + 2.0f * k101 * k101 * ir;
        K[0][2][2] = k020 * k002 * ir + 2.0f * k011 * k011 * ir;
        K[2][1][1] = (k200 * k011 + 2.0f * k110 * k101) * ir;
        K[1][2][1] = (k020 * k101 + 2.0f * k110 * k011) * ir;
        K[1][1][2] = (k002 * k110 + 2.0f * k101 * k011) * ir;
        K[2][2][2] = (k200 * k020 * k002 + 2.0f * k110 * k110 * k002 + 2.0f * k101 * k101 * k020 +
                      2.0f * k011 * k011 * k200 + 8.0f * k110 * k101 * k011) * ir * ir;
    }

    const PlainMul mul;
    float fc[27];
    central_to_populations(mul, K, ux, uy, uz, fc);
    const float rho_cs = rmax(1e-6f, carried_sum<0>(fc));
    const float uxc = carried_sum<1>(fc) / rho_cs, uyc = carried_sum<2>(fc) / rho_cs, uzc = carried_sum<3>(fc) / rho_cs;
    conserve(mul, fc, rho_safe, ux, uy, uz, rho_cs, uxc, uyc, uzc, f);
    if (forced) {
        const float pref = rmax(0.0f, 1.0f - 0.5f * rclamp(omega_off, 0.0f, 1.999f));
        guo(mul, pref, ux, uy, uz, fx, fy, fz, f, [&](int q, float v) { f[q] = v; });
    }
    return true;
}

// write_output / extract macro readout in the reference's order
// (jni.cpp:2535-2581): sums in q order, clamped rho, true division.
__device__ __forceinline__ void macro_out_exact(const float (&f)[27], bool solid, float scale, float* o) {
    if (solid) { o[0] = o[1] = o[2] = o[3] = 0.0f; return; }
    bool bad = false;
#pragma unroll
    for (int q = 0; q < 27; ++q) bad |= !isfinite(f[q]);
    float rho = qsum<0, 0, 0>(f);
    float ux = qsum<1, 0, 0>(f), uy = qsum<0, 1, 0>(f), uz = qsum<0, 0, 1>(f);
    if (bad || !isfinite(rho) || !isfinite(ux) || !isfinite(uy) || !isfinite(uz)) {
        o[0] = o[1] = o[2] = o[3] = 0.0f;
        return;
    }
    rho = rclamp(rho, 0.97f, 1.03f);
    ux /= rho; uy /= rho; uz /= rho;
    if (!isfinite(ux) || !isfinite(uy) || !isfinite(uz)) ux = uy = uz = 0.0f;
    if (fabsf(rho - 1.0f) < 1e-6f) rho = 1.0f;
    if (fabsf(ux) < 1e-7f) ux = 0.0f;
    if (fabsf(uy) < 1e-7f) uy = 0.0f;
    if (fabsf(uz) < 1e-7f) uz = 0.0f;
    o[0] = ux * scale;
    o[1] = uy * scale;
    o[2] = uz * scale;
    o[3] = rclamp(rho - 1.0f, -0.03f, 0.03f);
}

}  // namespace exact
}  // namespace aero
