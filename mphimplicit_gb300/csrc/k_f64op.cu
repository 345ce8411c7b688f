// k_f64op.cu - the FP64 form's operator y = A s in three parts.
//
// A = inertia + V + C Lambda C^T (calculateMatrixA main.cpp:2251-2335,
// multiplyMatrixC main.cpp:2574-2642).  Stored as 3 x 3 blocks it takes 9
// FP64 multiply-adds and 72 bytes a neighbour (about 170 a row in 3-D), and
// the FP64 units bound it: 0.69 ms an application on 216,000 fluid particles for
// 2.7 GB of blocks.  In parts it takes 0.35:
//
//   t_k = lambda_k sum_{j in P(k)} C_jk . s_j,  (C Lambda C^T s)_i = sum_{k in P(i)} C_ik t_k   FP64, over P-lists of about 20
//   (V s)_i = sum_j g_ij (g_ij . (s_i - s_j)) + W_i s_i,   g = sqrt(f) q / |q|, W_i the wall slots' block
//
// the pairs carry 24 bytes and three-component products.  The pair part runs
// in two floats (about 47 bits), while FP32 issues at 64 times the FP64 rate
// here.  It is at most a tenth of the inertia where this operator is used, so
// its 2^-46 or less of itself is at most some 2^-49 of the inertia, below what
// FP64 leaves of the C Lambda C^T part of the row (up to 150 times the inertia,
// which the blocks' sums round as a whole).  Measured, error of b - A x against
// 128-bit sums over the inertia term's norm, parts and blocks:
// smooth velocities 0.7-1.7e-14 and 1.2-3.6e-14, white noise 6.4-12.1e-14 and
// 6.4-12.1e-14, on 800 to 29,000 fluid particles with viscosities from 0.01 to
// the admitted tenth, one fluid and two; with two particles 0.3 to 1e-6 of a
// spacing apart (f up to 600 times the inertia) 7.1e-14 and 7.2e-14.
// Everything in it is relative to the inertia and to the solve's scale, so
// that no unit system leaves FP32's range.  Measured at the kernels.
//
// The stored blocks are still assembled: the multigrid levels and the exports
// are made from them.
#include "mph_device.cuh"
#include "mph_solver.cuh"
#include "mph_twofloat.cuh"

namespace mph {

// The power of two that brings a solve's vectors (at most about
// |b| / inertia) to order one for the two-float records; rr0 = (b, b).
__device__ __forceinline__ double f64_scale(double rr0, double inert, bool inverse = false)
{
    const int e = ((__double2hiint(rr0) >> 20) & 0x7ff) - 1023, m = ((__double2hiint(inert) >> 20) & 0x7ff) - 1023;
    const int k = max(-900, min(900, m - (e >> 1)));
    return __hiloint2double((1023 + (inverse ? -k : k)) << 20, 0);
}

__device__ __forceinline__ void f64_split(double v, float& h, float& l)
{
    h = (float)v;
    l = (float)(v - (double)h);
}

// record of a row: float4 (hx, hy, hz, lx) and float2 (ly, lz)
__device__ __forceinline__ void f64_record(double v, int r, size_t i, float4* __restrict__ rec, float2* __restrict__ rec2)
{
    float h, l;
    f64_split(v, h, l);
    float* a = reinterpret_cast<float*>(rec + i);
    a[r] = h;
    if (r == 0) a[3] = l;
    else reinterpret_cast<float*>(rec2 + i)[r - 1] = l;
}

__global__ void __launch_bounds__(256) k_f64_pack(int n, const double* __restrict__ s, double inert, const double* __restrict__ scal,
                                                  float4* __restrict__ rec, float2* __restrict__ rec2)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const double sc = f64_scale(scal[kSRR0], inert);
    f64_record(s[k] * sc, k % 3, k / 3, rec, rec2);
}

// x += alpha p, r -= alpha q, s -= alpha u with s's records, (r, r) -> rr
// (k_update_xrs with the records written where s is in registers)
__global__ void __launch_bounds__(kReduceThreads) k_f64_update_xrs(int n, double* __restrict__ x, double* __restrict__ r, double* __restrict__ s,
                                                                   const double* __restrict__ p, const double* __restrict__ q,
                                                                   const double* __restrict__ u, double* __restrict__ scal,
                                                                   int* __restrict__ flags, double* __restrict__ partials,
                                                                   unsigned* __restrict__ counter, double inert,
                                                                   float4* __restrict__ rec, float2* __restrict__ rec2)
{
    if (flags[kFlagDone]) return;
    __shared__ double alpha_s;   // the quotient once a block
    if (threadIdx.x == 0) alpha_s = scal[cr_rho_slot(flags[kFlagIter])] / scal[kSQU];
    __syncthreads();
    const double alpha = alpha_s;
    const double sc = f64_scale(scal[kSRR0], inert);
    double acc = 0.0;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        x[k] += alpha * p[k];
        const double rk = r[k] - alpha * q[k], sk = s[k] - alpha * u[k];
        r[k] = rk;
        s[k] = sk;
        f64_record(sk * sc, k % 3, k / 3, rec, rec2);
        acc += rk * rk;
    }
    reduce_finalize_step(acc, partials, counter, scal + kSRR, flags + kFlagIter);
}

// two-float reciprocal square root: the FP32 one and a Newton step,
// y (3 - v y^2) / 2 written as y + y (1 - v y^2) / 2
__device__ __forceinline__ F2 f2_rsqrt(F2 v)
{
    const float y = rsqrtf(v.h);
    const F2 vy = f2_mul(v, F2{y, 0.f});
    const F2 e = f2_add(F2{1.f, 0.f}, f2_mul(F2{-vy.h, -vy.l}, F2{y, 0.f}));
    return f2_fast(y, __fmul_rn(0.5f * y, e.h));
}

// g of every fluid slot, in the blocks' slices (float4 (x, y, z, x's second
// float) and float2, a thread a row), and the wall slots' diagonal block in
// FP64 (6 of 8 doubles a row, rows with wall slots only).  With r in units of
// RadiusV, f / inertia = A (1/r - 1), A = visc mu_ij kf 2 / RadiusV^2 / inertia
// up to the sign (main.cpp:2261-2289), so g = sqrt(A (1/r - 1)) r_vec / r, from
// the FP64 separation on in two floats: in FP64 throughout the kernel took
// 3.6 ms on 216,000 fluid particles, once a solve; it takes 2.4.  type_out: the types at an
// address that stays from step to step (the particle arrays swap with their
// alternates; the iteration's graph is replayed).
__global__ void __launch_bounds__(128) k_f64_pairs(DevParams P, double inert, const int* __restrict__ type, const double* __restrict__ pos,
                                                   const int* __restrict__ nc, const int* __restrict__ nfc,
                                                   const long long* __restrict__ nptr, const int* __restrict__ nind,
                                                   const long long* __restrict__ sptr, const int* __restrict__ acol,
                                                   float2* __restrict__ g, long long gslots, double* __restrict__ sdiag64,
                                                   int* __restrict__ type_out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < P.N) type_out[i] = type[i];
    if (i >= P.Nf) return;
    const int lane = i & 31, ti = type[i], n = nc[i], nf = nfc[i];
    const long long base = sptr[i >> 5], nb = nptr[i];
    double xi[3];
    load_vec<3>(pos, i, xi);
    const double A = P.visc * (-P.kfv * P.m2h_rv) / inert * P.inv_rv;
    F2 a2[2];
    f64_split(A * P.muij[ti][0], a2[0].h, a2[0].l);
    f64_split(A * P.muij[ti][1], a2[1].h, a2[1].l);
    float4* gp = reinterpret_cast<float4*>(g) + base + lane;
    float2* gp2 = g + gslots * 2 + base + lane;
#pragma unroll 2
    for (int k = 0; k < nf; ++k) {
        const int j = acol[base + (long long)k * 32 + lane];
        double xj[3], q[3];
        load_vec<3>(pos, j, xj);
        sep_vec<3>(P, xj, xi, q);
        F2 u[3], v[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
#pragma unroll
        for (int d = 0; d < 3; ++d) f64_split(q[d] * P.inv_rv, u[d].h, u[d].l);
        const F2 r2 = f2_add(f2_add(f2_mul(u[0], u[0]), f2_mul(u[1], u[1])), f2_mul(u[2], u[2]));
        if (r2.h > 0.f) {
            const F2 inv = f2_rsqrt(r2);
            F2 f = f2_add(inv, F2{-1.f, 0.f});
            if (f.h > 0.f) {
                f = f2_mul(f, type[j] ? a2[1] : a2[0]);
                // the square root's second float: the residual f - s^2 over 2 s
                F2 s{sqrtf(f.h), 0.f};
                if (s.h > 0.f) s = f2_fast(s.h, __fdiv_rn(__fadd_rn(__fmaf_rn(-s.h, s.h, f.h), f.l), 2.f * s.h));
                s = f2_mul(s, inv);
#pragma unroll
                for (int d = 0; d < 3; ++d) v[d] = f2_mul(s, u[d]);
            }
        }
        gp[(long long)k * 32] = make_float4(v[0].h, v[1].h, v[2].h, v[0].l);
        gp2[(long long)k * 32] = make_float2(v[1].l, v[2].l);
    }
    if (n == nf) return;
    double w[6] = {0, 0, 0, 0, 0, 0};
    const double rV2 = P.rV * P.rV;
    for (int k = nf; k < n; ++k) {
        const int j = nind[nb + k];
        double xj[3], q[3];
        load_vec<3>(pos, j, xj);
        sep_vec<3>(P, xj, xi, q);
        const double r2 = norm2_exact<3>(q);
        if (!r2_pos_below(r2, rV2)) continue;
        const double inv = rsqrt(r2);
        const double wd = -P.kfv * (P.m2h_rv * (1.0 - (r2 * inv) * P.inv_rv));
        const double f = P.visc * P.muij[ti][type[j]] * wd * inv;
#pragma unroll
        for (int r = 0, m = 0; r < 3; ++r)
#pragma unroll
            for (int s = r; s < 3; ++s, ++m) w[m] += f * (q[r] * inv) * (q[s] * inv);
    }
#pragma unroll
    for (int m = 0; m < 6; ++m) sdiag64[(size_t)i * 8 + m] = w[m];
}

// One launch, two kinds of blocks: lambda t of every particle from its own
// P-list, four threads a row (C_jk = - C_kj, and C_kk for a fluid row
// itself), and the pairs' part of y, four threads (of four warps) a row.  A
// pair streams 28 bytes, gathers 24 (the neighbour's record, mostly from L1
// and L2) and takes about 90 FP32 instructions; the latency of column, then
// record, bounds it.  On 216,000 fluid particles 308 us with four threads a row
// and eight pairs in flight (a thread a row: 438 with two, 350 with eight;
// eight threads a row, 322; 288 with the stop test's quotient once a block),
// the stream of records alone some 160.
constexpr int kF64Lanes = 4;      // threads a row of t
constexpr int kPairSplit = 4;     // and of the pairs
constexpr int kPairUnroll = 8;
constexpr int kPartThreads = 128;

template <int MODE>
__global__ void __launch_bounds__(kPartThreads) k_f64_parts(DevParams P, int nbT, double inert, const int* __restrict__ type,
                                                   const int* __restrict__ nfc, const long long* __restrict__ sptr,
                                                   const int* __restrict__ acol, const float2* __restrict__ g, long long gslots,
                                                   const float4* __restrict__ rec, const float2* __restrict__ rec2,
                                                   double* __restrict__ vacc, const int* __restrict__ ncp,
                                                   const long long* __restrict__ nptrP, const int* __restrict__ nindP,
                                                   const double* __restrict__ cval, const double* __restrict__ x, double* __restrict__ t,
                                                   const double* __restrict__ scal, const int* __restrict__ flags, int cap, double tol2)
{
    if (MODE == 1 && cr_stop(scal, flags, cap, tol2)) return;
    if ((int)blockIdx.x < nbT) {
        const int k = (blockIdx.x * blockDim.x + threadIdx.x) / kF64Lanes, part = threadIdx.x % kF64Lanes;
        double s = 0.0;
        if (k < P.N) {
            const long long b = nptrP[k];
            const int n = ncp[k];
#pragma unroll 2
            for (int a = part; a < n; a += kF64Lanes) {
                const int j = nindP[b + a];
                if (j >= P.Nf) continue;
                double v = 0.0;
#pragma unroll
                for (int d = 0; d < 3; ++d) v += cval[(b + a) * 3 + d] * x[(size_t)j * 3 + d];
                s = j == k ? s + v : s - v;
            }
        }
#pragma unroll
        for (int o = kF64Lanes / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (k < P.N && part == 0) t[k] = P.lambda[type[k]] * s;
        return;
    }
    constexpr int rows = kPartThreads / kPairSplit;
    const int w = threadIdx.x / rows;
    const int i = (blockIdx.x - nbT) * rows + threadIdx.x % rows;
    const int lane = i & 31, n = i < P.Nf ? nfc[i] : 0;
    const long long base = i < P.Nf ? sptr[i >> 5] : 0;
    const int* cp = acol + base + lane;
    const float4* gp = reinterpret_cast<const float4*>(g) + base + lane;
    const float2* gp2 = g + gslots * 2 + base + lane;
    const float4 si = i < P.Nf ? rec[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float2 si2 = i < P.Nf ? rec2[i] : make_float2(0.f, 0.f);
    float yh[3] = {0.f, 0.f, 0.f}, yl[3] = {0.f, 0.f, 0.f};
#pragma unroll kPairUnroll
    for (int k = w; k < n; k += kPairSplit) {
        const int j = cp[(long long)k * 32];
        const float4 g4 = gp[(long long)k * 32];
        const float2 g2 = gp2[(long long)k * 32];
        const float2 gx = make_float2(g4.x, g4.w), gy = make_float2(g4.y, g2.x), gz = make_float2(g4.z, g2.y);
        const float4 sj = rec[j];
        const float2 sj2 = rec2[j];
        float ex, ey, ez;   // s_i - s_j
        const float dx = f2_two_sum(si.x, -sj.x, ex), dy = f2_two_sum(si.y, -sj.y, ey), dz = f2_two_sum(si.z, -sj.z, ez);
        ex = __fadd_rn(ex, __fadd_rn(si.w, -sj.w));
        ey = __fadd_rn(ey, __fadd_rn(si2.x, -sj2.x));
        ez = __fadd_rn(ez, __fadd_rn(si2.y, -sj2.y));
        // its product with g
        const float px = __fmul_rn(gx.x, dx), py = __fmul_rn(gy.x, dy), pz = __fmul_rn(gz.x, dz);
        float lo = __fmaf_rn(gx.x, ex, __fmul_rn(gx.y, dx));
        lo = __fmaf_rn(gy.x, ey, __fmaf_rn(gy.y, dy, lo));
        lo = __fmaf_rn(gz.x, ez, __fmaf_rn(gz.y, dz, lo));
        float e1, e2;
        const float th = f2_two_sum(f2_two_sum(px, py, e1), pz, e2);
        lo = __fadd_rn(lo, __fadd_rn(__fmaf_rn(gx.x, dx, -px), __fmaf_rn(gy.x, dy, -py)));
        lo = __fadd_rn(lo, __fadd_rn(__fmaf_rn(gz.x, dz, -pz), __fadd_rn(e1, e2)));
        const float2 gv[3] = {gx, gy, gz};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const float p = __fmul_rn(gv[d].x, th);
            float e;
            yh[d] = f2_two_sum(yh[d], p, e);
            const float m = __fmaf_rn(gv[d].y, th, __fmaf_rn(gv[d].x, lo, __fmaf_rn(gv[d].x, th, -p)));
            yl[d] = __fadd_rn(yl[d], __fadd_rn(e, m));
        }
    }
    __shared__ float2 part_s[3][kPartThreads];
#pragma unroll
    for (int d = 0; d < 3; ++d) part_s[d][threadIdx.x] = make_float2(yh[d], yl[d]);
    __syncthreads();
    if (w > 0 || i >= P.Nf) return;
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int v = 1; v < kPairSplit; ++v) {
            const float2 o = part_s[d][threadIdx.x + v * rows];
            float e;
            yh[d] = f2_two_sum(yh[d], o.x, e);
            yl[d] = __fadd_rn(yl[d], __fadd_rn(e, o.y));
        }
    const double back = inert * f64_scale(scal[kSRR0], inert, true);
#pragma unroll
    for (int d = 0; d < 3; ++d) vacc[(size_t)i * 3 + d] = back * ((double)yh[d] + (double)yl[d]);
}

// the rest of y, a thread a row (shuffled FP64 sums of several threads cost more
// than they hide: 87 us with four, 68 with one): MODE 0: r = b - A x with (r, r) -> out;
// MODE 1: y = A s with (s, y) -> the iteration's rho slot
template <int MODE>
__global__ void __launch_bounds__(128) k_f64_rows(DevParams P, const int* __restrict__ type, const int* __restrict__ nc,
                                                  const int* __restrict__ nfc, const int* __restrict__ ncp,
                                                  const long long* __restrict__ nptrP, const int* __restrict__ nindP,
                                                  const double* __restrict__ cval, const double* __restrict__ t,
                                                  const double* __restrict__ sdiag64, const double* __restrict__ vacc,
                                                  const double* __restrict__ x, const double* __restrict__ b, double* __restrict__ yout,
                                                  double* __restrict__ scal, int* __restrict__ flags, int cap, double tol2,
                                                  double* __restrict__ partials, unsigned* __restrict__ counter, double* __restrict__ out)
{
    if (MODE == 1) {
        const int stop = cr_stop(scal, flags, cap, tol2);
        if (stop) {
            if (stop > 1 && blockIdx.x == 0 && threadIdx.x == 0) {
                flags[kFlagDone] = 1;
                if (stop == 3) flags[kFlagBad] = 1;
            }
            return;
        }
        out = scal + cr_rho_slot(flags[kFlagIter]);
    }
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double y[3] = {0.0, 0.0, 0.0}, acc = 0.0;
    if (i < P.Nf) {
        const long long pb = nptrP[i];
        const int np = ncp[i];
#pragma unroll 2
        for (int a = 0; a < np; ++a) {
            const double lt = t[nindP[pb + a]];
#pragma unroll
            for (int d = 0; d < 3; ++d) y[d] += cval[(pb + a) * 3 + d] * lt;
        }
        double xi[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            xi[d] = x[(size_t)i * 3 + d];
            y[d] += vacc[(size_t)i * 3 + d];
        }
        if (nc[i] > nfc[i]) {   // (xx, xy, xz, yy, yz, zz)
            const double* w = sdiag64 + (size_t)i * 8;
            y[0] += w[0] * xi[0] + w[1] * xi[1] + w[2] * xi[2];
            y[1] += w[1] * xi[0] + w[3] * xi[1] + w[4] * xi[2];
            y[2] += w[2] * xi[0] + w[4] * xi[1] + w[5] * xi[2];
        }
        const double inert = P.inert64[type[i]];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const size_t k = (size_t)i * 3 + d;
            const double v = y[d] + inert * xi[d];
            if (MODE == 0) {
                const double rv = b[k] - v;
                yout[k] = rv;
                acc += rv * rv;
            } else {
                yout[k] = v;
                acc += xi[d] * v;
            }
        }
    }
    reduce_finalize(acc, partials, counter, out);
}

// ---- host side ---------------------------------------------------------------------
// Whether a step's FP64 solve runs on the operator in parts: 3-D (in 2-D a
// block is 32 bytes and the FP64 units do not bind), C couplings that all lie
// within the neighbour lists (the stored matrix has only those), pair
// coefficients of one sign and a viscous part of at most a tenth of the
// inertia (the two-float pairs).
bool f64_parts_apply(const mph_case* c)
{
    return c->dim == 3 && c->precision != MPH_PRECISION_MIXED && c->factored && 2.0 * c->dp.rP < c->dp.maxR && c->visc_nonneg &&
           c->visc_ratio < 0.1 && c->dp.Nf > 0;
}

// the inertia the pair part is relative to: the largest
static double f64_inert(const mph_case* c) { return std::max(c->dp.inert64[0], c->dp.inert64[1]); }

// The pair records of this solve.  *ok = false: no memory for them, the
// stored blocks are applied.
int f64_parts_build(mph_case* c, bool* ok)
{
    DeviceState& d = c->d;
    const DevParams& P = c->dp;
    *ok = false;
    // three float2 a slot: float4 for every slot the arrays have room for, then float2
    const size_t need = (size_t)c->nslots * 3;
    if ((long long)need > d.cap_f64g) {
        if (d.f64g) cudaFree(d.f64g);
        d.f64g = nullptr;
        d.cap_f64g = 0;
        const size_t want = (need + need / 8 + 1024) / 3 * 3;
        if (cudaMalloc((void**)&d.f64g, want * sizeof(float2)) != cudaSuccess) {
            cudaGetLastError();
            d.f64g = nullptr;
            return MPH_OK;
        }
        d.cap_f64g = (long long)want;
    }
    c->f64_slots = d.cap_f64g / 3;
    auto have = [](auto** p, size_t bytes) {
        if (!*p && cudaMalloc((void**)p, bytes) != cudaSuccess) {
            cudaGetLastError();
            *p = nullptr;
        }
        return *p != nullptr;
    };
    if (!have(&d.f64rec, (size_t)P.Nf * (sizeof(float4) + sizeof(float2))) || !have(&d.f64type, (size_t)P.N * sizeof(int)) ||
        !have(&d.vacc, (size_t)P.Nf * 3 * sizeof(double)) || !have(&d.tct, (size_t)(P.N + 1) * sizeof(double)) ||
        !have(&d.sdiag64, (size_t)P.Nf * 8 * sizeof(double)))
        return MPH_OK;
    { k_f64_pairs<<<grid_for(P.N, 128), 128, 0, c->stream>>>(P, f64_inert(c), d.type, d.pos, d.nc, d.nfc, d.nptr, d.nind, d.sptr, d.acol,
                                                              d.f64g, c->f64_slots, d.sdiag64, d.f64type); MPH_COUNT_LAUNCH(); }
    MPH_CUDA(cudaGetLastError());
    *ok = true;
    return MPH_OK;
}

static float2* f64_rec2(const mph_case* c) { return reinterpret_cast<float2*>(c->d.f64rec + c->dp.Nf); }

void launch_f64_pack(mph_case* c, const double* s)
{
    const int n = c->dp.Nf * 3;
    { k_f64_pack<<<grid_for(n, 256), 256, 0, c->stream>>>(n, s, f64_inert(c), c->d.scal, c->d.f64rec, f64_rec2(c)); MPH_COUNT_LAUNCH(); }
}

// mode 0: r = b - A x, (r, r) -> out; mode 1: y = A s, (s, y) -> the rho slot (records of the vector first)
void launch_f64_apply(mph_case* c, int mode, const double* x, double* y, int cap, double tol2, double* out)
{
    DeviceState& d = c->d;
    const DevParams& P = c->dp;
    cudaStream_t st = c->stream;
    unsigned* counter = (unsigned*)(d.flags + kFlagCounter);
    const int nbT = (int)grid_for((long long)P.N * kF64Lanes, kPartThreads);
    const unsigned gp = nbT + grid_for(P.Nf, kPartThreads / kPairSplit), gr = grid_for(P.Nf, 128);
    const double inert = f64_inert(c);
    if (mode == 0) {
        { k_f64_parts<0><<<gp, kPartThreads, 0, st>>>(P, nbT, inert, d.f64type, d.nfc, d.sptr, d.acol, d.f64g, c->f64_slots, d.f64rec, f64_rec2(c), d.vacc, d.ncp, d.nptrP,
                                             d.nindP, d.cval, x, d.tct, d.scal, d.flags, cap, tol2); MPH_COUNT_LAUNCH(); }
        { k_f64_rows<0><<<gr, 128, 0, st>>>(P, d.f64type, d.nc, d.nfc, d.ncp, d.nptrP, d.nindP, d.cval, d.tct, d.sdiag64, d.vacc, x, d.bvec, y,
                                            d.scal, d.flags, cap, tol2, d.partials, counter, out); MPH_COUNT_LAUNCH(); }
    } else {
        { k_f64_parts<1><<<gp, kPartThreads, 0, st>>>(P, nbT, inert, d.f64type, d.nfc, d.sptr, d.acol, d.f64g, c->f64_slots, d.f64rec, f64_rec2(c), d.vacc, d.ncp, d.nptrP,
                                             d.nindP, d.cval, x, d.tct, d.scal, d.flags, cap, tol2); MPH_COUNT_LAUNCH(); }
        { k_f64_rows<1><<<gr, 128, 0, st>>>(P, d.f64type, d.nc, d.nfc, d.ncp, d.nptrP, d.nindP, d.cval, d.tct, d.sdiag64, d.vacc, x, d.bvec, y,
                                            d.scal, d.flags, cap, tol2, d.partials, counter, out); MPH_COUNT_LAUNCH(); }
    }
}

void launch_f64_update_xrs(mph_case* c, int blocks)
{
    DeviceState& d = c->d;
    { k_f64_update_xrs<<<blocks, kReduceThreads, 0, c->stream>>>(c->dp.Nf * 3, d.x, d.r, d.s, d.p, d.q, d.u, d.scal, d.flags, d.partials,
                                                                 (unsigned*)(d.flags + kFlagCounter), f64_inert(c), d.f64rec, f64_rec2(c)); MPH_COUNT_LAUNCH(); }
}

}  // namespace mph
