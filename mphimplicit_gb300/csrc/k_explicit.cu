// k_explicit.cu - explicit particle physics and output-step fields.
//
//   k_density       : calculateDensityA + calculateGravityCenter +
//                     calculateDensityP (main.cpp:1737, 1767, 1903) in one
//                     neighbour pass, in the list's order
//   k_pressure_a_*  : calculatePressureA (main.cpp:1801)
//   k_diffuse       : calculateDiffuseInterface (main.cpp:1851)
//   k_accelerate    : calculatePhysicalCoefficients' mass (main.cpp:1710),
//                     calculateGravity and calculateAcceleration
//                     (main.cpp:2065, 2076)
//   k_div_pressure, k_output_forces : calculateDivergenceP,
//                     calculatePressureP, calculateViscosityV and
//                     calculateVirialStressAtParticle (main.cpp:1932-2063,
//                     4494-4738), output steps only
// When every surface-tension coefficient CofA is zero the pressure-A and
// diffuse-interface forces are exact zeros and their passes are skipped.
#include "mph_device.cuh"

namespace mph {

// sqrt(v) of v >= 0 from the reciprocal square root: v y and one residual
// correction (P. Markstein, "Computation of elementary functions on the IBM
// RISC System/6000", 1990), within a hair of half a unit in the last place
__device__ __forceinline__ double sqrt_by_rsqrt(double v)
{
    if (__double_as_longlong(v) == 0) return 0.0;
    const double y = rsqrt(v), r = v * y;
    return __fma_rn(__fma_rn(-r, r, v), 0.5 * y, r);
}

// The density pass is bound by the FP64 pipe (about 180 neighbours a particle
// in 3-D, all of them inside the radii).  The weights' constants stand before
// the sums, w_a = kf t (1 - t)^2 and w = kf (1 - t)^2 with t = r / RadiusA
// (RadiusG is RadiusA, main.cpp:236-307, 888), so a pair is one root, one
// 1 - t, two products for the density and a product and three multiply-adds
// for the gravity centre: some 37 FP64 operations where the reference's terms
// one by one took 80, with roundings left out accordingly.  The sums run in
// pieces of 32 neighbours, which keeps their own roundings below those of one
// long sum.  The radius tests compare bit patterns on the integer pipe.
// 326,592 particles: 6.42 -> 2.79 ms; 71,200: 1.84 -> 0.80.
constexpr int kDensityRun = 32;

template <int D>
__global__ void __launch_bounds__(128) k_density(DevParams P, const int* __restrict__ type, const double* __restrict__ pos,
                                                 const int* __restrict__ nc, const long long* __restrict__ nptr,
                                                 const int* __restrict__ nind, double* __restrict__ densA,
                                                 double* __restrict__ gcen, double* __restrict__ vsp)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    const int ti = type[i];
    double xi[3];
    load_vec<D>(pos, i, xi);
    const double rA2 = DMUL(P.rA, P.rA), rP2 = DMUL(P.rP, P.rP);
    double sa = 0.0, sp = 0.0, sg[3] = {0.0, 0.0, 0.0};
    const long long b = nptr[i];
    const int n = nc[i];
    for (int k0 = 0; k0 < n; k0 += kDensityRun) {
        double ra = 0.0, rp = 0.0, rg[3] = {0.0, 0.0, 0.0};
        for (int k = k0; k < min(n, k0 + kDensityRun); ++k) {
            const int j = nind[b + k];
            if (j == i) continue;
            double xj[3], q[3];
            load_vec<D>(pos, j, xj);
            sep_vec<D>(P, xj, xi, q);
            const double r2 = norm2_fma<D>(q);
            const bool inA = r2_within(r2, rA2), inP = r2_within(r2, rP2);
            if (!(inA || inP)) continue;
            const double r = sqrt_by_rsqrt(r2);
            if (inA) {
                const double ratio = P.ratio[ti][type[j]];
                const double oq = __fma_rn(-r, P.inv_ra_lo, __fma_rn(-r, P.inv_ra, 1.0)), w = ratio * (oq * oq);
                ra += r * w;
#pragma unroll
                for (int d = 0; d < D; ++d) rg[d] += w * q[d];
            }
            if (inP) {
                const double oq = __fma_rn(-r, P.inv_rp, 1.0);
                rp += oq * oq;
            }
        }
        sa += ra;
        sp += rp;
#pragma unroll
        for (int d = 0; d < D; ++d) sg[d] += rg[d];
    }
    densA[i] = sa * (P.kfa * P.inv_ra);
    const double cg = P.kfg * P.rG / P.R2g;
#pragma unroll
    for (int d = 0; d < D; ++d) sg[d] *= cg;
    store_vec<D>(gcen, i, sg);
    if (vsp) vsp[i] = __fma_rn(P.kfp, sp, -P.N0p);
}

__global__ void k_pressure_a(DevParams P, const int* __restrict__ type, const double* __restrict__ densA, double* __restrict__ presA)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    const double a = densA[i];
    presA[i] = (P.N0a <= a) ? 0.0 : DDIV(DMUL(P.cofA[type[i]], DSUB(a, P.N0a)), P.l0);
}

// Pressure-A and diffuse-interface forces (main.cpp:1801-1898).  Bound by the
// FP64 pipe: a pair's force is gathered into one factor of q = x_j - x_i and
// one of h = ratio_ji g_j - ratio_ij g_i, with one reciprocal square root and
// the constants' products formed once, about 60 FP64 operations a pair
// against some 30 divisions with the terms formed one by one.  4.82 -> 1.31
// ms on 71,200 particles.
template <int D>
__global__ void __launch_bounds__(128) k_surface_forces(DevParams P, const int* __restrict__ type, const double* __restrict__ pos,
                                                        const int* __restrict__ nc, const long long* __restrict__ nptr,
                                                        const int* __restrict__ nind, const double* __restrict__ presA,
                                                        const double* __restrict__ gcen, double* __restrict__ force)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    const int ti = type[i];
    double xi[3], gi[3];
    load_vec<D>(pos, i, xi);
    load_vec<D>(gcen, i, gi);
    const double rA2 = P.rA * P.rA;   // RadiusG = RadiusA (main.cpp:888)
    // both coefficients from i's type (main.cpp:1857, 1863)
    const double K = P.cofA[ti] * P.cofK * P.cofK * P.rG * (P.vol / P.l0) / P.R2g;
    const double pa_i = presA[i];
    const double ih = P.inv_ra;
    const double ca = P.kfa * ih * P.vol, cw = K * P.kfg, cd = cw * (-2.0 * ih);
    double f[3] = {0, 0, 0};
    const long long b = nptr[i];
    const int n = nc[i];
    for (int k = 0; k < n; ++k) {
        const int j = nind[b + k];
        if (j == i) continue;
        double xj[3], q[3], gj[3];
        load_vec<D>(pos, j, xj);
        sep_vec<D>(P, xj, xi, q);
        const double r2 = norm2_exact<D>(q);
        if (!r2_pos_below(r2, rA2)) continue;
        const int tj = type[j];
        const double rij = P.ratio[ti][tj], rji = P.ratio[tj][ti];
        const double inv = rsqrt(r2);
        const double t = (r2 * inv) * ih, oq = 1.0 - t;
        // pressure A: s q / |q| with s = (p_i ratio_ij + p_j ratio_ji) w_a'(|q|) vol
        const double s = (pa_i * rij + presA[j] * rji) * (ca * oq * (1.0 - 3.0 * t));
        load_vec<D>(gcen, j, gj);
        double h[3], hq = 0.0;
#pragma unroll
        for (int d = 0; d < D; ++d) {
            h[d] = rji * gj[d] - rij * gi[d];
            hq += h[d] * q[d];
        }
        // diffuse interface: - K (w h + w' (h . q) q / |q|)
        const double fq = inv * (s - cd * oq * hq), fh = cw * (oq * oq);
#pragma unroll
        for (int d = 0; d < D; ++d) f[d] += fq * q[d] - fh * h[d];
    }
    double f0[3];
    load_vec<D>(force, i, f0);
#pragma unroll
    for (int d = 0; d < D; ++d) f[d] = f0[d] + f[d];
    store_vec<D>(force, i, f);
}

template <int D>
__global__ void k_accelerate(DevParams P, int fB, int fE, const int* __restrict__ type, double* __restrict__ force,
                             double* __restrict__ vel)
{
    const int i = fB + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= fE) return;
    const double m = DMUL(P.density[type[i]], P.vol);
    double f[3], v[3];
    load_vec<D>(force, i, f);
    load_vec<D>(vel, i, v);
#pragma unroll
    for (int d = 0; d < D; ++d) {
        f[d] = DADD(f[d], DMUL(m, P.gravity[d]));
        v[d] = DADD(v[d], DMUL(DDIV(f[d], m), P.dt));
    }
    store_vec<D>(force, i, f);
    store_vec<D>(vel, i, v);
}

// ---- output-step fields ----------------------------------------------------
// DivergenceP and PressureP (main.cpp:1932-1990) over the P-list, which holds
// exactly the pairs with r^2 <= RadiusP^2 in the full list's order: about 19
// slots a particle in 3-D instead of 180.  5.79 -> 0.34 ms on 326,592
// particles.
template <int D>
__global__ void __launch_bounds__(128) k_div_pressure(DevParams P, const int* __restrict__ type, const double* __restrict__ pos,
                                                      const double* __restrict__ vel, const int* __restrict__ ncp,
                                                      const long long* __restrict__ nptrP, const int* __restrict__ nindP,
                                                      const double* __restrict__ vsp, double* __restrict__ divP,
                                                      double* __restrict__ presP)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    double xi[3], vi[3];
    load_vec<D>(pos, i, xi);
    load_vec<D>(vel, i, vi);
    double sum = 0.0;
    const long long b = nptrP[i];
    const int n = ncp[i];
    for (int k = 0; k < n; ++k) {
        const int j = nindP[b + k];
        if (j == i) continue;
        double xj[3], q[3], vj[3];
        load_vec<D>(pos, j, xj);
        sep_vec<D>(P, xj, xi, q);
        const double r2 = norm2_exact<D>(q);
        if (r2 == 0.0) continue;
        const double inv = rsqrt(r2);
        const double dw = P.kfp * (P.m2h_rp * (1.0 - (r2 * inv) * P.inv_rp));
        load_vec<D>(vel, j, vj);
        double ue = 0.0;
#pragma unroll
        for (int d = 0; d < D; ++d) ue += (vj[d] - vi[d]) * q[d];
        sum -= ue * inv * dw;
    }
    divP[i] = sum;
    const int t = type[i];
    const double kap = vsp[i] < 0.0 ? 0.0 : P.bulk[t];
    double p = -P.lambda[t] * sum;
    if (vsp[i] > 0.0) p += kap * vsp[i];
    presP[i] = p;
}

// The pressure-P and viscosity forces and the virial stress of a frame
// (main.cpp:1990-2063, 4494-4738) in one pass over the neighbours.  Bound by
// the FP64 pipe, so a pair costs one reciprocal square root and no division:
// every force but the diffuse interface's first term lies along q, so the
// pair's virial is one factor times q (x) q (six sums in 3-D), and that first
// term is g_i (x) sum w q (three sums).  The pairs within RadiusP are those of
// the P-list, so its virial needs no second walk.  SURF false: every CofA is
// zero, so the pressure-A and diffuse-interface terms are exact zeros and are
// not formed.  104.3 -> 4.64 ms on 326,592 particles (59 million pairs).
template <int D, bool SURF>
__global__ void __launch_bounds__(128) k_output_forces(DevParams P, const int* __restrict__ type, const double* __restrict__ pos,
                                                       const double* __restrict__ vel, const int* __restrict__ nc,
                                                       const long long* __restrict__ nptr, const int* __restrict__ nind,
                                                       const double* __restrict__ presP, const double* __restrict__ presA,
                                                       const double* __restrict__ gcen, double* __restrict__ force,
                                                       double* __restrict__ virS, double* __restrict__ virP)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    const int ti = type[i];
    double xi[3], vi[3], gi[3] = {0.0, 0.0, 0.0};
    load_vec<D>(pos, i, xi);
    load_vec<D>(vel, i, vi);
    const double pi = presP[i];
    double pa = 0.0, Kd = 0.0;
    if (SURF) {
        load_vec<D>(gcen, i, gi);
        pa = presA[i];
        Kd = P.cofA[ti] * P.cofK * P.cofK / P.R2g * P.rG / P.l0;
    }
    const double rA2 = P.rA * P.rA, rP2 = P.rP * P.rP, rV2 = P.rV * P.rV;
    const double cv = -P.kfv * P.m2h_rv * P.visc, cp = P.kfp * P.m2h_rp;
    const double ca = SURF ? pa * P.kfa * P.inv_ra : 0.0;
    double fq[3] = {0, 0, 0}, wq[3] = {0, 0, 0};
    double T[6] = {0, 0, 0, 0, 0, 0};   // xx xy xz yy yz zz
    const long long b = nptr[i];
    const int n = nc[i];
    for (int k = 0; k < n; ++k) {
        const int j = nind[b + k];
        if (j == i) continue;
        double xj[3], q[3];
        load_vec<D>(pos, j, xj);
        sep_vec<D>(P, xj, xi, q);
        const double r2 = norm2_exact<D>(q);
        if (r2 == 0.0) continue;
        const double inv = rsqrt(r2), r = r2 * inv;
        const int tj = type[j];
        double S = 0.0, F = 0.0;           // the pair's factors of q (x) q and, over vol, of q
        if (r2_pos_below(r2, rV2)) {       // viscosity: visc mu_ij (u . e) e w' / |q|
            double vj[3], ue = 0.0;
            load_vec<D>(vel, j, vj);
#pragma unroll
            for (int d = 0; d < D; ++d) ue += (vj[d] - vi[d]) * q[d];
            F = (P.muij[ti][tj] * cv) * (ue * (1.0 - r * P.inv_rv)) * (inv * inv * inv);
            S = 0.5 * F;
        }
        if (r2_pos_below(r2, rP2)) {       // pressure P
            const double dw = cp * (1.0 - r * P.inv_rp) * inv;
            F += (pi + presP[j]) * dw;
            S += pi * dw;
        }
        if (SURF && r2_pos_below(r2, rA2)) {   // pressure A and the diffuse interface (RadiusG = RadiusA)
            const double ratio = P.ratio[ti][tj];
            const double t = r * P.inv_ra, oq = 1.0 - t;
            double gq = 0.0;
#pragma unroll
            for (int d = 0; d < D; ++d) gq += gi[d] * q[d];
            const double w = ratio * P.kfg * oq;
            S += (ca * ratio * oq * (1.0 - 3.0 * t) + Kd * gq * w * (-2.0 * P.inv_ra)) * inv;
#pragma unroll
            for (int d = 0; d < D; ++d) wq[d] += (w * oq) * q[d];
        }
        double sq[3];
#pragma unroll
        for (int d = 0; d < D; ++d) {
            fq[d] += F * q[d];
            sq[d] = S * q[d];
        }
        T[0] += sq[0] * q[0];
        T[1] += sq[0] * q[1];
        T[3] += sq[1] * q[1];
        if (D == 3) {
            T[2] += sq[0] * q[2];
            T[4] += sq[1] * q[2];
            T[5] += sq[2] * q[2];
        }
    }
    double f[3];
    load_vec<D>(force, i, f);
#pragma unroll
    for (int d = 0; d < D; ++d) f[d] += fq[d] * P.vol;
    store_vec<D>(force, i, f);
    const double full[3][3] = {{T[0], T[1], T[2]}, {T[1], T[3], T[4]}, {T[2], T[4], T[5]}};
    double tr = 0.0;
#pragma unroll
    for (int aa = 0; aa < 3; ++aa)
#pragma unroll
        for (int bb = 0; bb < 3; ++bb) {
            double v = 0.0;
            if (aa < D && bb < D) v = full[aa][bb] + (SURF ? Kd * gi[aa] * wq[bb] : 0.0);
            virS[9 * (size_t)i + 3 * aa + bb] = v;
            if (aa == bb) tr += v;
        }
    virP[i] = -1.0 / (double)D * tr;
}

// calculateDensityP alone over the P-list.  The P-list holds exactly the
// pairs with r^2 <= RadiusP^2, in the full list's order (the sum differs from
// the full-list pass's by the rounding of its pieces).  As k_density: 37 FP64
// operations a pair became 28; 340 -> 243 us on 326,592 particles.
template <int D, int L>
__global__ void __launch_bounds__(128) k_density_p(DevParams P, const double* __restrict__ pos, const int* __restrict__ ncp,
                                                   const long long* __restrict__ nptrP, const int* __restrict__ nindP,
                                                   double* __restrict__ vsp)
{
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) / L, part = threadIdx.x % L;
    double xi[3] = {0.0, 0.0, 0.0};
    if (i < P.N) load_vec<D>(pos, i, xi);
    const double rP2 = DMUL(P.rP, P.rP);
    double sp = 0.0;
    const long long b = i < P.N ? nptrP[i] : 0;
    const int n = i < P.N ? ncp[i] : 0;
    for (int k = part; k < n; k += L) {
        const int j = nindP[b + k];
        if (j == i) continue;
        double xj[3], q[3];
        load_vec<D>(pos, j, xj);
        sep_vec<D>(P, xj, xi, q);
        const double r2 = norm2_fma<D>(q);
        if (r2_within(r2, rP2)) {   // w_quad
            const double oq = __fma_rn(-sqrt_by_rsqrt(r2), P.inv_rp, 1.0);
            sp += oq * oq;
        }
    }
    sp = row_sum<L>(sp);
    if (i < P.N && part == 0) vsp[i] = __fma_rn(P.kfp, sp, -P.N0p);
}

static void launch_density_p(mph_case* c)
{
    const DevParams& P = c->dp;
    const int L = plist_lanes(P.N);
    auto go = [&](auto kern) {
        kern<<<grid_for((long long)P.N * L, 128), 128, 0, c->stream>>>(P, c->d.pos, c->d.ncp, c->d.nptrP, c->d.nindP, c->d.vsp);
        MPH_COUNT_LAUNCH();
    };
    if (c->dim == 2) L == 4 ? go(k_density_p<2, 4>) : go(k_density_p<2, 1>);
    else L == 4 ? go(k_density_p<3, 4>) : go(k_density_p<3, 1>);
}

// The full density pass (DensityA, GravityCenter, and DensityP where CofA is
// not all zero) and PressureA.  Without surface tension VolStrainP is
// k_density_p's, always: its sums run in another order than this pass's, and a
// reader's request must not change what the step goes on with.
void launch_density_full(mph_case* c)
{
    const DevParams& P = c->dp;
    const unsigned g = grid_for(P.N, 128);
    double* vsp = P.surface ? c->d.vsp : nullptr;
    if (c->dim == 2)
        { k_density<2><<<g, 128, 0, c->stream>>>(P, c->d.type, c->d.pos, c->d.nc, c->d.nptr, c->d.nind, c->d.densA, c->d.gcen, vsp); MPH_COUNT_LAUNCH(); }
    else
        { k_density<3><<<g, 128, 0, c->stream>>>(P, c->d.type, c->d.pos, c->d.nc, c->d.nptr, c->d.nind, c->d.densA, c->d.gcen, vsp); MPH_COUNT_LAUNCH(); }
    { k_pressure_a<<<grid_for(P.N, 256), 256, 0, c->stream>>>(P, c->d.type, c->d.densA, c->d.presA); MPH_COUNT_LAUNCH(); }
    c->densa_valid = true;
}

// DensityA, GravityCenter and PressureA only act through the surface-tension
// coefficients CofA.  With every CofA zero they are dead in the step, so the
// step computes DensityP alone; they are computed from the same positions and
// lists when a reader (export, output fields) asks for them.
void ensure_density_a(mph_case* c)
{
    if (!c->densa_valid) launch_density_full(c);
}

void launch_explicit(mph_case* c)
{
    const DevParams& P = c->dp;
    const unsigned g = grid_for(P.N, 128);
    if (P.surface) {
        launch_density_full(c);
    } else {
        launch_density_p(c);
        c->densa_valid = false;
    }
    if (P.surface) {
        if (c->dim == 2)
            { k_surface_forces<2><<<g, 128, 0, c->stream>>>(P, c->d.type, c->d.pos, c->d.nc, c->d.nptr, c->d.nind, c->d.presA, c->d.gcen, c->d.force); MPH_COUNT_LAUNCH(); }
        else
            { k_surface_forces<3><<<g, 128, 0, c->stream>>>(P, c->d.type, c->d.pos, c->d.nc, c->d.nptr, c->d.nind, c->d.presA, c->d.gcen, c->d.force); MPH_COUNT_LAUNCH(); }
    }
    const int nf = c->fE - c->fB;
    if (nf > 0) {
        if (c->dim == 2)
            { k_accelerate<2><<<grid_for(nf, 256), 256, 0, c->stream>>>(P, c->fB, c->fE, c->d.type, c->d.force, c->d.vel); MPH_COUNT_LAUNCH(); }
        else
            { k_accelerate<3><<<grid_for(nf, 256), 256, 0, c->stream>>>(P, c->fB, c->fE, c->d.type, c->d.force, c->d.vel); MPH_COUNT_LAUNCH(); }
    }
}

// the density pass alone: the initial pass of main() (main.cpp:371-373)
void launch_explicit_density_only(mph_case* c)
{
    launch_density_full(c);
    if (!c->dp.surface) launch_density_p(c);
}

void launch_output_fields(mph_case* c)
{
    const DevParams& P = c->dp;
    const unsigned g = grid_for(P.N, 128);
    // with every CofA zero the frame needs VolStrainP alone of the density
    // pass (DensityA and the rest follow when a reader asks for them)
    if (P.surface) ensure_density_a(c);
    else launch_density_p(c);
    DeviceState& d = c->d;
    auto go = [&](auto dp, auto of) {
        dp<<<g, 128, 0, c->stream>>>(P, d.type, d.pos, d.vel, d.ncp, d.nptrP, d.nindP, d.vsp, d.divP, d.presP);
        MPH_COUNT_LAUNCH();
        of<<<g, 128, 0, c->stream>>>(P, d.type, d.pos, d.vel, d.nc, d.nptr, d.nind, d.presP, d.presA, d.gcen, d.force, d.virS, d.virP);
        MPH_COUNT_LAUNCH();
    };
    if (c->dim == 2) {
        if (P.surface) go(k_div_pressure<2>, k_output_forces<2, true>);
        else go(k_div_pressure<2>, k_output_forces<2, false>);
    } else {
        if (P.surface) go(k_div_pressure<3>, k_output_forces<3, true>);
        else go(k_div_pressure<3>, k_output_forces<3, false>);
    }
}

}  // namespace mph
