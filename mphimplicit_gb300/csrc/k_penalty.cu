// k_penalty.cu - the inner CR iteration of the point-Jacobi mixed form.
//
// A = inertia + V + C Lambda C^T (calculateMatrixA main.cpp:2251-2335,
// multiplyMatrixC main.cpp:2574-2642).  The viscous part V is small against
// the inertia (the factored form is used up to 0.1 of it, host estimate; a few
// 1e-3 in the benchmark cases), while its pairs, about 180 a row in 3-D, took
// two thirds of an inner iteration.  The inner CR therefore solves with
//
//   M = m_i I + C Lambda C^T,   m_i = inertia + 0.6 of the lattice's viscous diagonal,
//
// and the FP64 outer residual b - A x, with all of V, carries the result: V's
// eigenvalues lie between 0 and about 1.3 of that diagonal, so a refinement
// phase leaves at most about 0.7 of diagonal / inertia of the residual (4e-4
// in the benchmark's tank, below the phase's own target of 1e-3, which is
// raised to that bound where the fluid is more viscous, and to what a close
// pair leaves, k_pen_system).
//
// C is not stored: C_ik = w(|q|) q / |q| with q = x_k - x_i and
// C_ii = sum_k C_ik, so with P-lists that are symmetric (k in P(i) <=> i in
// P(k), r^2 <= RadiusP^2 both ways)
//
//   t_k = sum_j C_jk . s_j = sum_{j in P(k)} C_kj . (s_k - s_j)     (s = 0 on walls)
//   y_i = m_i s_i + sum_{k in P(i)} C_ik (lambda_k t_k + lambda_i t_i)
//
// and both sums run over one list with a 2-byte index a slot (40 MB on
// 1.3 million particles, which stays in L2 from one iteration to the next)
// instead of two lists of 16-byte records (640 MB, read from HBM every time).
// Positions are fixed point, about MaxRadius / 2^30 a unit and modulo 2^32, so
// that their differences are exact minimum images (C_ik = -C_ki to the bit)
// and good to FP32's own rounding down to MaxRadius / 256 (k_fixed_positions).
//
// On 1,297,696 particles an application takes 93 us (k_pen_t 49, k_pen_y 44;
// the viscous pairs and stored records: 398) and the vectors 20 us in one
// kernel (43 in two), with 142 CR iterations where there were 140.
//
// A block of rows stages its distinct neighbours (position with s, or with
// lambda t) in shared memory; a block with too many of them gathers by the
// P-list's own columns.  Both evaluate pen_coef in the same order, so they
// give the same bits.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>

#include "mph_device.cuh"
#include "mph_pairs.cuh"
#include "mph_shapes.h"
#include "mph_solver.cuh"
#include "mph_twofloat.cuh"

namespace mph {

constexpr int kSIn0 = 16, kSIn = 17, kSTol2 = 23;         // as in k_mixed.cu
constexpr int kSAlpha = 25, kSQUPrev = 27;   // this iteration's alpha and beta (two floats), (q, D^-1 q) of the last one
constexpr int kSStop = 28;                   // the phase's target (r, r) in two floats
__device__ __forceinline__ int rho_slot32(int it) { return 20 + (it & 1); }

constexpr int kPlWords = 1 << 13;   // bitmap of a row block's columns: 2^18 particles, fluid and wall window together
constexpr int kMaxPenRows = 256;   // threads of a row block (rows times threads a row) of the per-iteration kernels
constexpr int kCrThreads = 512;    // of the resident iteration's blocks, two an SM
constexpr int kCrBlocks = 2 * 152;
// Rows a block at least.  A solve alone is fastest on many blocks (22,000
// particles in 3-D: 2.01, 1.89, 2.00 ms with 128, 192, 256; 12,000 in 2-D,
// where a row is a fifth of the work: 1.00, 1.04, 1.08 with 192, 256, 384),
// but the blocks of a solve hold their SMs until it ends: an ensemble of 64
// two-dimensional cases on their streams takes 52.9, 46.3, 37.9 and 37.5 ms
// with 192, 256, 384 and 512.
constexpr int kCrMinRows3 = 192, kCrMinRows2 = 384;
// Staged neighbours a thread loads while alpha and beta are formed: in blocks
// alone on their SM, and in two blocks an SM (in 3-D none there: its twelve
// registers would spill; a step of 89,000 particles 3.31 ms, 3.49 with one)
constexpr int kCrAhead = 3, kCrShared3 = 0, kCrShared2 = 1;
constexpr int kCrSmem = 100 * 1024;   // dynamic: two blocks an SM with their 7 KB of static shared memory
// Staged neighbours a block of `rows` rows has room for.  Blocks of a
// 3.5-spacing cell order have about 2.8 (256 rows) to 3.9 (64) times their
// rows of them, against some 20 slots a row; one with more (a solve of 211
// blocks of 599 on average: 9.12 ms staged, 9.34 gathered) gains little.
static constexpr int pen_ucap(int rows) { return 4 * rows + 128; }

// Fixed-point positions with the particle's type, of the penalty operator and
// of the viscous pairs.  An axis's unit is its domain width / (m 2^32), m the
// integer that brings it next to MaxRadius / 2^30, and the 32 bits are kept: a
// difference modulo 2^32 is the minimum image by itself, in domains of any
// width, and the lists' separations (at most MaxRadius, or half the width) fit
// it exactly.  A difference in units of RadiusP is its float times fix_c, with
// FP32's relative rounding down to distances of 2^24 units: the phases' true
// residual meets the directions' error enlarged by the depth of the fluid in
// spacings (a pair's share of the pressure against the net force).  Units of
// RadiusP / 2^22 over the whole domain took 480 iterations instead of 170 for
// a pair of particles 0.01 spacings apart in 504, and did not converge at
// 0.001.
template <int D>
__global__ void __launch_bounds__(256) k_fixed_positions(DevParams P, const int* __restrict__ type, const double* __restrict__ pos,
                                                         int4* __restrict__ ipos)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    double x[3];
    load_vec<D>(pos, i, x);
    int u[3] = {0, 0, 0};
#pragma unroll
    for (int d = 0; d < D; ++d) u[d] = (int)(unsigned)(unsigned long long)__double2ll_rn((x[d] - P.dmin[d]) * P.fix_scale[d]);
    ipos[i] = make_int4(u[0], u[1], u[2], type[i]);
}
// x_j - x_i of an axis, in units of RadiusP
__device__ __forceinline__ float fixed_sep(const DevParams& P, int d, int uj, int ui)
{
    return __fmul_rn(__int2float_rn((int)((unsigned)uj - (unsigned)ui)), P.fix_c[d]);
}

// The same in units of RadiusV with the unit in two floats, for the viscous
// pairs that the outer residual carries: their roundings are then at random,
// and no constant's own (the unit's, 1 / RadiusV, mu_00: exact or applied in
// FP64) goes through every pair.  A frame of 326,592 particles is 5.3e-11 from
// the 64-bit one, 6.6e-11 with the constants rounded.
__device__ __forceinline__ float fixed_sep_v(const DevParams& P, int d, int uj, int ui)
{
    const float v = __int2float_rn((int)((unsigned)uj - (unsigned)ui));
    return __fmaf_rn(v, P.fix_v[d], __fmul_rn(v, P.fix_vl[d]));
}

// The P-lists of a block of rows as 2-byte ranks among the block's distinct
// columns: uniq[block][0 .. U) the columns in ascending order, idx the rank of
// every slot, four slots of a row in one 8-byte word, a row's words 32 words
// apart (a warp reads 256 bytes); a row's last word is filled up with the
// row's own rank (its separation is zero, so it adds zero).  groups[slice]:
// words a row of the slice has.  The columns are found through a bitmap of
// two index windows, the fluid particles' and the walls' (walls follow the
// fluid in the order).  ucount[block] = U, or -1 where the windows or U are
// too large.
__global__ void __launch_bounds__(kCrThreads) k_plist_ranks(int N, int Nf, int pw4, int ucap, const int* __restrict__ ncp,
                                                             const long long* __restrict__ nptrP, const int* __restrict__ nindP,
                                                             uint2* __restrict__ idx, int* __restrict__ groups,
                                                             int* __restrict__ uniq, int* __restrict__ ucount,
                                                             const int* __restrict__ near)
{
    extern __shared__ unsigned pl_smem[];
    unsigned* bm = pl_smem;
    unsigned* rank = pl_smem + kPlWords;
    __shared__ int red[4][32];
    __shared__ unsigned wsum[32];
    const int tid = threadIdx.x, lane = tid & 31, wl = tid >> 5, nwl = blockDim.x >> 5;
    const int i = blockIdx.x * blockDim.x + tid;
    if (blockIdx.x == 0 && tid == 0) ucount[gridDim.x + 4] = *near;   // rides in the host's read
    const int n = i < N ? ncp[i] : 0;
    const int* col = nindP + (i < N ? nptrP[i] : 0);
    int lf = INT_MAX, hf = -1, lw = INT_MAX, hw = -1;
    for (int k = 0; k < n; ++k) {
        const int j = col[k];
        if (j < Nf) { lf = min(lf, j); hf = max(hf, j); }
        else { lw = min(lw, j); hw = max(hw, j); }
    }
    int nm = n;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lf = min(lf, __shfl_xor_sync(0xffffffffu, lf, o));
        hf = max(hf, __shfl_xor_sync(0xffffffffu, hf, o));
        lw = min(lw, __shfl_xor_sync(0xffffffffu, lw, o));
        hw = max(hw, __shfl_xor_sync(0xffffffffu, hw, o));
        nm = max(nm, __shfl_xor_sync(0xffffffffu, nm, o));
    }
    const int ng = (nm + 3) >> 2;
    if (lane == 0) {
        red[0][wl] = lf; red[1][wl] = hf; red[2][wl] = lw; red[3][wl] = hw;
        if (blockIdx.x * blockDim.x + wl * 32 < N) groups[(blockIdx.x * blockDim.x >> 5) + wl] = ng;
    }
    __syncthreads();
    lf = lw = INT_MAX;
    hf = hw = -1;
    for (int w = 0; w < nwl; ++w) {
        lf = min(lf, red[0][w]); hf = max(hf, red[1][w]);
        lw = min(lw, red[2][w]); hw = max(hw, red[3][w]);
    }
    const int nwf = hf < 0 ? 0 : ((hf - lf) >> 5) + 1, nww = hw < 0 ? 0 : ((hw - lw) >> 5) + 1;
    const int nw = nwf + nww;
    if (nw > kPlWords || nw == 0) {
        if (tid == 0) ucount[blockIdx.x] = nw == 0 ? 0 : -1;
        return;
    }
    auto bit = [&](int j) { return j < Nf ? j - lf : (nwf << 5) + (j - lw); };
    for (int w = tid; w < nw; w += blockDim.x) bm[w] = 0u;
    __syncthreads();
    for (int k = 0; k < n; ++k) {
        const int b = bit(col[k]);
        atomicOr(&bm[b >> 5], 1u << (b & 31));
    }
    __syncthreads();
    const int per = (nw + blockDim.x - 1) / blockDim.x;
    const int w0 = min(nw, tid * per), w1 = min(nw, w0 + per);
    unsigned cs = 0;
    for (int w = w0; w < w1; ++w) cs += __popc(bm[w]);
    unsigned inc = cs;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
    }
    if (lane == 31) wsum[wl] = inc;
    __syncthreads();
    unsigned woff = 0, total = 0;
    for (int w = 0; w < nwl; ++w) {
        if (w < wl) woff += wsum[w];
        total += wsum[w];
    }
    unsigned r = woff + inc - cs;
    for (int w = w0; w < w1; ++w) {
        rank[w] = r;
        r += __popc(bm[w]);
    }
    __syncthreads();
    const int U = (int)total;
    if (U > ucap) {
        if (tid == 0) ucount[blockIdx.x] = -1;
        return;
    }
    auto rank_of = [&](int j) {
        const int b = bit(j);
        return rank[b >> 5] + __popc(bm[b >> 5] & ((1u << (b & 31)) - 1u));
    };
    if (n > 0) {   // a row with neighbours has itself among them
        uint2* ip = idx + ((long long)(i >> 5) * pw4) * 32 + lane;
        const unsigned own = rank_of(i);
        for (int g = 0; g < ng; ++g) {
            unsigned v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = 4 * g + u < n ? rank_of(col[4 * g + u]) : own;
            ip[(long long)g * 32] = make_uint2(v[0] | (v[1] << 16), v[2] | (v[3] << 16));
        }
    }
    int* ul = uniq + (size_t)blockIdx.x * ucap;
    for (int w = w0; w < w1; ++w) {
        unsigned word = bm[w];
        unsigned rr = rank[w];
        while (word) {
            const int b = __ffs(word) - 1;
            ul[rr++] = w < nwf ? lf + w * 32 + b : lw + (w - nwf) * 32 + b;
            word &= word - 1u;
        }
    }
    if (tid == 0) {   // after the blocks: the largest count; the staged blocks and their columns, of all rows and of the fluid rows
        const int nb = gridDim.x;
        ucount[blockIdx.x] = U;
        atomicMax(ucount + nb, U);
        atomicAdd(ucount + nb + 1, 1);
        if ((int)(blockIdx.x * blockDim.x) < Nf) {
            atomicAdd(ucount + nb + 2, 1);
            atomicAdd((unsigned*)ucount + nb + 3, (unsigned)U);
        }
    }
}

// q = x_j - x_i in units of RadiusP and cf = 1 / |q| - 1 (0 beyond RadiusP),
// so that C_ij = kfp (2 / RadiusP) cf q.  |q| = 0 (the row itself, coincident
// particles) gives a finite cf, and zero with its q.
template <int D>
__device__ __forceinline__ float pen_coef(const DevParams& P, const int* ui, const int* uj, float* q)
{
#pragma unroll
    for (int d = 0; d < D; ++d) q[d] = fixed_sep(P, d, uj[d], ui[d]);
    float r2 = __fmul_rn(q[0], q[0]);
    r2 = __fmaf_rn(q[1], q[1], r2);
    if (D == 3) r2 = __fmaf_rn(q[2], q[2], r2);
    float inv;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(fmaxf(r2, 1e-18f)));
    return fmaxf(__fadd_rn(inv, -1.f), 0.f);
}

struct PenArgs {
    int N, Nf, pw4, ucap, umax, cap;
    const int4* ipos;
    const uint2* idx;
    const int *groups, *uniq, *ucount;      // ucount null: every block gathers by column
    const int *ncp, *nindP;
    const long long* nptrP;
    float *s, *y, *p, *q, *z, *t;
    const float* invD;
    double* scal;
    int* flags;
    double* partials;
    unsigned* counter;
};

// Sums over the grid of NC values a thread (256 threads a block): FP32 in a
// warp, two floats beyond, in one order.  Thread 0 of the last block to arrive
// gets them (true).  Two floats because an FP64 addition is some hundred
// clocks long here and the chains of these sums, and of the quotients made
// from them, stood at the end of two kernels an iteration (12 us of vectors
// took 4 to stream).
template <int NC>
__device__ __forceinline__ bool grid_sums(const float* v, const PenArgs& A, int lb, int nb, int tid, F2* out)
{
    constexpr int NW = 8;   // warps
    __shared__ float ws[NC][NW];
    __shared__ F2 wf[NC][NW];
    __shared__ bool last;
    const int lane = tid & 31, wid = tid >> 5;
    float2* parts = reinterpret_cast<float2*>(A.partials);
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        float x = v[c];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (lane == 0) ws[c][wid] = x;
    }
    __syncthreads();
    const int c = min(lane >> 3, NC - 1), w = lane & 7;   // eight lanes a value
    if (wid == 0) {
        const F2 x = f2_warp_sum(F2{ws[c][w], 0.f}, NW / 2);
        if (w == 0 && (lane >> 3) < NC) __stcg(parts + (size_t)NC * lb + c, make_float2(x.h, x.l));
        __syncwarp();
        if (lane == 0) {
            __threadfence();
            last = atomicAdd(A.counter, 1u) == (unsigned)nb - 1;
        }
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    constexpr int K = (kReduceBlocks + 255) / 256;
    float2 p[K][NC];
#pragma unroll
    for (int u = 0; u < K; ++u)
#pragma unroll
        for (int d = 0; d < NC; ++d) {
            const int k = tid + 256 * u;
            p[u][d] = k < nb ? __ldcg(parts + (size_t)NC * k + d) : make_float2(0.f, 0.f);
        }
#pragma unroll
    for (int d = 0; d < NC; ++d) {
        F2 x{p[0][d].x, p[0][d].y};
#pragma unroll
        for (int u = 1; u < K; ++u)
            if (256 * u < nb) x = f2_add(x, F2{p[u][d].x, p[u][d].y});
        x = f2_warp_sum(x, 16);
        if (lane == 0) wf[d][wid] = x;
    }
    __syncthreads();
    if (wid != 0) return false;
    const F2 x = f2_warp_sum(wf[c][w], NW / 2);
#pragma unroll
    for (int d = 0; d < NC; ++d)
        out[d] = F2{__shfl_sync(0xffffffffu, x.h, 8 * d), __shfl_sync(0xffffffffu, x.l, 8 * d)};
    if (lane == 0) *A.counter = 0u;
    return lane == 0;
}

// What a thread has in flight before its block's neighbours are staged: the
// first columns it stages and the first words of its row.  Their loads do not
// wait for the block's count or the row's length (both buffers have room for
// every index read here); what lies beyond is not used.  A block's time is
// this chain of loads, so nothing in it waits that need not.
// (Three columns and three words: a solve of three steps on 1.3 million particles
// 66.7 ms, of one on 326,592 7.78; with four words, whose registers k_pen_t
// spilled, 67.5 and 8.03, with two words 67.7, with two columns 70.2.)
constexpr int kPreCols = 3, kPreWords = 3;
struct PenPre {
    int col[kPreCols];
    uint2 word[kPreWords];
    int U, ng, n;
};

__device__ __forceinline__ void pen_prefetch(const PenArgs& A, int lb, int i, int rows_end, int tid, int nth, int w, int W, PenPre& R)
{
    R.U = -1;
    if (A.ucount) {
        R.U = A.ucount[lb];
        const int* ul = A.uniq + (size_t)lb * A.ucap;
#pragma unroll
        for (int u = 0; u < kPreCols; ++u) R.col[u] = tid + u * nth < A.ucap ? ul[tid + u * nth] : 0;
    }
    R.n = 0;
    R.ng = 0;
    if (i < rows_end) {
        R.n = A.ncp[i];
        if (A.ucount) {
            R.ng = A.groups[i >> 5];
            const uint2* ip = A.idx + ((long long)(i >> 5) * A.pw4) * 32 + (i & 31);
#pragma unroll
            for (int u = 0; u < kPreWords; ++u)
                R.word[u] = w + u * W < A.pw4 ? __ldg(ip + (long long)(w + u * W) * 32) : make_uint2(0u, 0u);
        }
    }
}

// stage(k, j): neighbour j becomes the block's record k
template <typename F>
__device__ __forceinline__ void pen_stage(const PenArgs& A, int lb, int tid, int nth, const PenPre& R, F&& stage)
{
#pragma unroll
    for (int u = 0; u < kPreCols; ++u)
        if (tid + u * nth < R.U) stage(tid + u * nth, R.col[u]);
    const int* ul = A.uniq + (size_t)lb * A.ucap;
    for (int k = tid + kPreCols * nth; k < R.U; k += nth) stage(k, ul[k]);
}

// The slots of row i, in the order of its words: this thread takes every W-th
// word from the w-th on.  term(k): a staged record, or term(j): a column.
template <typename F>
__device__ __forceinline__ void pen_row(const PenArgs& A, int i, int w, int W, const PenPre& R, F&& term)
{
    if (R.U >= 0) {
        auto four = [&](uint2 v) {
            term((int)(v.x & 0xffffu));
            term((int)(v.x >> 16));
            term((int)(v.y & 0xffffu));
            term((int)(v.y >> 16));
        };
#pragma unroll
        for (int u = 0; u < kPreWords; ++u)
            if (w + u * W < R.ng) four(R.word[u]);
        const uint2* ip = A.idx + ((long long)(i >> 5) * A.pw4) * 32 + (i & 31);
        for (int g = w + kPreWords * W; g < R.ng; g += W) four(__ldg(ip + (long long)g * 32));
    } else {
        const int* col = A.nindP + A.nptrP[i];
        for (int g = w; 4 * g < R.n; g += W)
            for (int k = 4 * g; k < min(R.n, 4 * g + 4); ++k) term(col[k]);
    }
}

// lambda_k t_k of every particle (the iteration's first kernel).  Bound by the
// shared-memory gathers (24 bytes a slot at random ranks, about 9 wavefronts a
// warp) and the load chain of a block, not by HBM.
template <int D>
__device__ __forceinline__ void pen_t_body(const DevParams& P, const PenArgs& A, int lb)
{
    extern __shared__ int4 pen_smem[];
    const int rows = blockDim.x, W = blockDim.y;
    const int tid = threadIdx.y * rows + threadIdx.x, nth = rows * W;
    const int i = lb * rows + threadIdx.x;
    const int done = A.flags[kFlagDone];
    PenPre R;
    pen_prefetch(A, lb, i, A.N, tid, nth, threadIdx.y, W, R);
    int4 pi = make_int4(0, 0, 0, 0);
    float si[3] = {0.f, 0.f, 0.f};
    if (i < A.N) pi = A.ipos[i];
    if (i < A.Nf) {
#pragma unroll
        for (int d = 0; d < D; ++d) si[d] = A.s[(size_t)i * D + d];
    }
    if (done) return;   // block-uniform: set before this launch
    int4* sa = pen_smem;
    float2* sb = reinterpret_cast<float2*>(pen_smem + A.umax);
    pen_stage(A, lb, tid, nth, R, [&](int k, int j) {
        int4 p = A.ipos[j];
        float v[3] = {0.f, 0.f, 0.f};
        if (j < A.Nf) {
#pragma unroll
            for (int d = 0; d < D; ++d) v[d] = A.s[(size_t)j * D + d];
        }
        if (D == 3) {
            p.w = __float_as_int(v[0]);
            sb[k] = make_float2(v[1], v[2]);
        } else {
            p.z = __float_as_int(v[0]);
            p.w = __float_as_int(v[1]);
        }
        sa[k] = p;
    });
    __syncthreads();
    float acc = 0.f;
    const int ui[3] = {pi.x, pi.y, pi.z};
    if (R.n > 0) {
        auto one = [&](const int* uj, const float* sj) {
            float q[3];
            const float cf = pen_coef<D>(P, ui, uj, q);
            float dot = __fmul_rn(q[0], __fadd_rn(si[0], -sj[0]));
            dot = __fmaf_rn(q[1], __fadd_rn(si[1], -sj[1]), dot);
            if (D == 3) dot = __fmaf_rn(q[2], __fadd_rn(si[2], -sj[2]), dot);
            acc = __fmaf_rn(cf, dot, acc);
        };
        if (R.U >= 0)
            pen_row(A, i, threadIdx.y, W, R, [&](int k) {
                const int4 p = sa[k];
                const int uj[3] = {p.x, p.y, p.z};
                if (D == 3) {
                    const float2 b = sb[k];
                    const float sj[3] = {__int_as_float(p.w), b.x, b.y};
                    one(uj, sj);
                } else {
                    const float sj[3] = {__int_as_float(p.z), __int_as_float(p.w), 0.f};
                    one(uj, sj);
                }
            });
        else
            pen_row(A, i, threadIdx.y, W, R, [&](int j) {
                const int4 p = A.ipos[j];
                const int uj[3] = {p.x, p.y, p.z};
                float sj[3] = {0.f, 0.f, 0.f};
                if (j < A.Nf) {
#pragma unroll
                    for (int d = 0; d < D; ++d) sj[d] = A.s[(size_t)j * D + d];
                }
                one(uj, sj);
            });
    }
    if (W > 1) {   // the row's partial sums in the order of w
        __shared__ float part[kMaxPenRows];
        part[threadIdx.y * rows + threadIdx.x] = acc;
        __syncthreads();
        if (threadIdx.y) return;
        for (int w = 1; w < W; ++w) acc += part[w * rows + threadIdx.x];
    }
    if (i < A.N) A.t[i] = R.n > 0 ? P.pen_lam32[pi.w] * acc : 0.f;
}

// y = M s, and the iteration's scalars: rho = (s, y), and with
// q <- y + beta q the product (q, D^-1 q) from (y, D^-1 y), (y, D^-1 q) and
// the last iteration's, so that one vector kernel can follow with alpha and
// beta both known.
// A block takes row blocks lb0, lb0 + nb, ... (nrb of them): the reduction's
// fence and ticket, once a block, would otherwise come every 256 rows and
// invalidate the L1 the other blocks of the SM gather through.
template <int D>
__device__ __forceinline__ void pen_y_body(const DevParams& P, const PenArgs& A, int lb0, int nb, int nrb)
{
    extern __shared__ int4 pen_smem[];
    const int rows = blockDim.x, W = blockDim.y;
    const int tid = threadIdx.y * rows + threadIdx.x, nth = rows * W;
    const int done = A.flags[kFlagDone], it = A.flags[kFlagIter];
    if (done) return;   // block-uniform: set before this launch
    int4* sa = pen_smem;
    float v[3] = {0.f, 0.f, 0.f};
    for (int lb = lb0; lb < nrb; lb += nb) {
        const int i = lb * rows + threadIdx.x;
        PenPre R;
        pen_prefetch(A, lb, i, A.Nf, tid, nth, threadIdx.y, W, R);
        int4 pi = make_int4(0, 0, 0, 0);
        float ti = 0.f, sv[3] = {0.f, 0.f, 0.f}, dv[3] = {0.f, 0.f, 0.f}, qv[3] = {0.f, 0.f, 0.f};
        if (i < A.Nf) {
            pi = A.ipos[i];
            ti = A.t[i];
            if (threadIdx.y == 0) {
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    sv[d] = A.s[(size_t)i * D + d];
                    dv[d] = A.invD[(size_t)i * D + d];
                    qv[d] = A.q[(size_t)i * D + d];
                }
            }
        }
        if (lb != lb0) __syncthreads();   // the last row block's records have been read
        pen_stage(A, lb, tid, nth, R, [&](int k, int j) {
            int4 p = A.ipos[j];
            const int t = __float_as_int(A.t[j]);
            if (D == 3) p.w = t;
            else p.z = t;
            sa[k] = p;
        });
        __syncthreads();
        float y[3] = {0.f, 0.f, 0.f};
        const int ui[3] = {pi.x, pi.y, pi.z};
        if (R.n > 0) {
            auto one = [&](const int* uj, float tj) {
                float q[3];
                const float c = __fmul_rn(pen_coef<D>(P, ui, uj, q), __fadd_rn(tj, ti));
#pragma unroll
                for (int d = 0; d < D; ++d) y[d] = __fmaf_rn(c, q[d], y[d]);
            };
            if (R.U >= 0)
                pen_row(A, i, threadIdx.y, W, R, [&](int k) {
                    const int4 p = sa[k];
                    const int uj[3] = {p.x, p.y, p.z};
                    one(uj, __int_as_float(D == 3 ? p.w : p.z));
                });
            else
                pen_row(A, i, threadIdx.y, W, R, [&](int j) {
                    const int4 p = A.ipos[j];
                    const int uj[3] = {p.x, p.y, p.z};
                    one(uj, A.t[j]);
                });
        }
        if (W > 1) {
            __shared__ float part[kMaxPenRows * D];
#pragma unroll
            for (int d = 0; d < D; ++d) part[(threadIdx.y * rows + threadIdx.x) * D + d] = y[d];
            __syncthreads();
            if (threadIdx.y == 0)
                for (int w = 1; w < W; ++w)
#pragma unroll
                    for (int d = 0; d < D; ++d) y[d] += part[(w * rows + threadIdx.x) * D + d];
        }
        if (threadIdx.y == 0 && i < A.Nf) {
            const float m = P.pen_diag32[pi.w];
#pragma unroll
            for (int d = 0; d < D; ++d) {
                const float yd = __fmaf_rn(m, sv[d], __fmul_rn(P.pen_w32, y[d])), u = dv[d] * yd;
                A.y[(size_t)i * D + d] = yd;
                v[0] += sv[d] * yd;
                v[1] += u * yd;
                if (it > 0) v[2] += u * qv[d];   // q of a first iteration is not set
            }
        }
    }
    F2 x[3];
    if (!grid_sums<3>(v, A, lb0, nb, tid, x)) return;
    float2* scal2 = reinterpret_cast<float2*>(A.scal);   // these slots hold two floats here
    F2 be{0.f, 0.f}, qu = x[1];
    if (it > 0) {
        const float2 rp = scal2[rho_slot32(it - 1)], qp = scal2[kSQUPrev];
        be = f2_div(x[0], F2{rp.x, rp.y});
        qu = f2_add(qu, f2_mul(be, f2_add(F2{2.f * x[2].h, 2.f * x[2].l}, f2_mul(be, F2{qp.x, qp.y}))));
    }
    scal2[rho_slot32(it)] = make_float2(x[0].h, x[0].l);
    scal2[kSQUPrev] = make_float2(qu.h, qu.l);
    scal2[kSAlpha] = make_float2(f2_div(x[0], qu).h, be.h);
}

// p = s + beta p, q = y + beta q, z += alpha p, s -= alpha D^-1 q, and (r, r)
// of r = D s -> kSIn; the last block advances the iteration and applies the
// next one's stop test (in the device-driven solve also to its loop's
// condition).  r itself and u = D^-1 q are not stored: ten vector streams an
// iteration instead of seventeen in two kernels.
template <bool COND>
__device__ __forceinline__ void pen_vec_body(const PenArgs& A, int lb, int nb, int n, int use_cond, cudaGraphConditionalHandle cond)
{
    __shared__ int it_s;
    __shared__ float ab[2];
    if (threadIdx.x == 0) {
        it_s = A.flags[kFlagDone] ? -1 : A.flags[kFlagIter];
        const float2 v = reinterpret_cast<const float2*>(A.scal)[kSAlpha];
        ab[0] = v.x;
        ab[1] = v.y;
    }
    __syncthreads();
    const int it = it_s;
    if (it < 0) {   // block-uniform
        if constexpr (COND)
            if (use_cond && lb == 0 && threadIdx.x == 0) cudaGraphSetConditional(cond, 0u);
        return;
    }
    const float alpha = ab[0], beta = ab[1];
    float acc = 0.f;
    auto one = [&](float& s, float y, float d, float& p, float& q, float& z) {
        p = it == 0 ? s : beta * p + s;
        q = it == 0 ? y : beta * q + y;
        z += alpha * p;
        s = s - alpha * (d * q);
        const float r = d != 0.f ? __fdividef(s, d) : 0.f;
        acc += r * r;
    };
    // four components a thread (the vectors are 16-byte aligned), the last n mod 4 one by one
    for (int k = lb * blockDim.x + threadIdx.x; k < (n >> 2); k += nb * blockDim.x) {
        float4 s = reinterpret_cast<float4*>(A.s)[k], z = reinterpret_cast<float4*>(A.z)[k];
        const float4 y = reinterpret_cast<const float4*>(A.y)[k], d = reinterpret_cast<const float4*>(A.invD)[k];
        float4 p = make_float4(0.f, 0.f, 0.f, 0.f), q = p;
        if (it > 0) {
            p = reinterpret_cast<float4*>(A.p)[k];
            q = reinterpret_cast<float4*>(A.q)[k];
        }
        one(s.x, y.x, d.x, p.x, q.x, z.x);
        one(s.y, y.y, d.y, p.y, q.y, z.y);
        one(s.z, y.z, d.z, p.z, q.z, z.z);
        one(s.w, y.w, d.w, p.w, q.w, z.w);
        reinterpret_cast<float4*>(A.s)[k] = s;
        reinterpret_cast<float4*>(A.z)[k] = z;
        reinterpret_cast<float4*>(A.p)[k] = p;
        reinterpret_cast<float4*>(A.q)[k] = q;
    }
    if (lb == 0 && (int)threadIdx.x < (n & 3)) {
        const int k = (n & ~3) + threadIdx.x;
        float s = A.s[k], z = A.z[k], p = it > 0 ? A.p[k] : 0.f, q = it > 0 ? A.q[k] : 0.f;
        one(s, A.y[k], A.invD[k], p, q, z);
        A.s[k] = s;
        A.z[k] = z;
        A.p[k] = p;
        A.q[k] = q;
    }
    F2 rr;
    if (grid_sums<1>(&acc, A, lb, nb, threadIdx.x, &rr)) {
        const float2 t = reinterpret_cast<const float2*>(A.scal)[kSStop];
        const bool bad = !(rr.h == rr.h);
        const bool below = __fadd_rn(__fadd_rn(rr.h, -t.x), __fadd_rn(rr.l, -t.y)) < 0.f;
        const bool stop = it + 1 >= A.cap || below || bad;
        A.flags[kFlagIter] = it + 1;   // every block has read it (they all took their tickets)
        if (stop) {
            A.flags[kFlagDone] = 1;
            if (bad) A.flags[kFlagBad] = 1;
        }
        A.scal[kSIn] = (double)rr.h + (double)rr.l;
        if constexpr (COND)
            if (use_cond) cudaGraphSetConditional(cond, stop ? 0u : 1u);
    }
}

// blocks resident on an SM: k_pen_y's 64 registers allow four (a solve on 1.3
// million particles: 25.8 ms a step with 4, 26.2 with 3, 27.4 with 5, 29.5 with 6)
constexpr int kPenResident = 4;
template <int D>
__global__ void __launch_bounds__(kMaxPenRows, kPenResident + 1) k_pen_t(DevParams P, PenArgs A) { pen_t_body<D>(P, A, (int)blockIdx.x); }
template <int D>
__global__ void __launch_bounds__(kMaxPenRows, kPenResident) k_pen_y(DevParams P, PenArgs A, int nrb) { pen_y_body<D>(P, A, (int)blockIdx.x, (int)gridDim.x, nrb); }
template <bool COND>
__global__ void __launch_bounds__(kReduceThreads) k_pen_vec(PenArgs A, int n, int use_cond, cudaGraphConditionalHandle cond)
{
    pen_vec_body<COND>(A, (int)blockIdx.x, (int)gridDim.x, n, use_cond, cond);
}

// ---- the resident iteration -----------------------------------------------------------
// All CR iterations of a refinement phase in one cooperative kernel, for the
// cases whose rows fit the chip at once (up to 155,648 particles).  Such a
// case's iteration is not bound by anything a kernel does but by three
// launches, their load chains and their last-block reductions (19 us on 22,000
// particles, 33 on 155,000; resident 8.1 and 18.4).  Here a block keeps its
// rows' neighbours' positions and ranks in shared memory and its vectors in
// registers for the whole phase, and an iteration crosses the grid's barrier
// twice:
//
//   after t    lambda t of every particle, and (r, r) of the vectors it came from
//   after y    s, D^-1 y and D^-1 q of every row, and the dot products
//
// With alpha and beta known (every block adds the blocks' sums in the same
// order) a block forms the new s of its own rows and of its staged neighbours
// alike, s - alpha (D^-1 y + beta D^-1 q), so the new s needs no barrier of
// its own.
//
// The sums across warps and blocks are in two floats (48 bits): an FP64
// addition takes this part some hundred clocks, and the chain of them took 4
// us an iteration; a warp's own terms are summed in FP32 as elsewhere.
//
// All blocks are resident (cooperative launch), so a wait ends; it is bounded
// all the same (option wait_polls), and a block whose wait runs out raises
// kFlagStall and leaves, as the others then do.  A launch runs at most
// mph_case::cr_iters iterations (option launch_iterations).

struct PenCr {
    float4* rec;                   // per row 3 records: s, a = D^-1 y, b = D^-1 q
    float *v3, *v1;                // the blocks' (s, y), (y, a), (y, b) in two floats each; (r, r)
    unsigned* count;               // arrivals of this launch's crossings
    // the phase's end: x += scale z, z as records for the residual, the
    // velocity array
    double scale;
    int iters, polls;              // iterations of a launch, polls of a wait at most
    double *x, *vel;
    float4* z4;
};

// The grid's crossing number `epoch`: this block's nv values (mine, shared
// memory) are out, and whatever the block's threads wrote before it can be
// read (through L2) by every block after it.  The arrivals are counted (the
// count only grows during a launch) and one thread a block waits for them; a
// word per block and value that every block polls instead was slower (nb^2
// polls).
__device__ __forceinline__ bool cr_cross(unsigned* count, float* vals, const float* mine, int nv, unsigned epoch, int lb, int nb, int tid,
                                         int* flags, int polls)
{
    __shared__ int ok_s;
    __syncthreads();
    if (tid < 32) {
        if (tid < nv) vals[(size_t)lb * nv + tid] = mine[tid];
        __syncwarp();
        if (tid == 0) {
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
            const unsigned target = epoch * (unsigned)nb;
            unsigned v = 0;
            int n = 0;
            do {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
            } while ((int)(v - target) < 0 && ++n < polls);
            ok_s = (int)(v - target) >= 0;
            if (!ok_s) flags[kFlagStall] = 1;
        }
    }
    __syncthreads();
    return ok_s != 0;
}

// the sum over the blocks of one two-float value (stride: floats a block), by one warp
__device__ __forceinline__ F2 cr_sum(const float* vals, int stride, int nb, int lane)
{
    constexpr int K = (kCrBlocks + 31) / 32;
    float2 v[K];
#pragma unroll
    for (int u = 0; u < K; ++u) {
        const int k = lane + 32 * u;
        v[u] = k < nb ? __ldcg(reinterpret_cast<const float2*>(vals + (size_t)k * stride)) : make_float2(0.f, 0.f);
    }
    F2 s{v[0].x, v[0].y};
#pragma unroll
    for (int u = 1; u < K; ++u)
        if (32 * u < nb) s = f2_add(s, F2{v[u].x, v[u].y});
    return f2_warp_sum(s, 16);
}

// the new s of a row, own or staged: the same two operations everywhere
__device__ __forceinline__ float cr_new_s(float s, float a, float b, float alpha, float beta)
{
    return __fmaf_rn(-alpha, __fmaf_rn(beta, b, a), s);
}

// a row's published records (zeros for a wall), and the new s from them
struct CrRec { float4 r[3]; };
template <int D>
__device__ __forceinline__ CrRec cr_load(const float4* rec, int j, int Nf)
{
    CrRec R;
    R.r[0] = R.r[1] = R.r[2] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (j >= 0 && j < Nf) {
#pragma unroll
        for (int u = 0; u < D; ++u) R.r[u] = __ldcg(rec + 3 * (size_t)j + u);
    }
    return R;
}
template <int D>
__device__ __forceinline__ void cr_combine(const CrRec& R, float alpha, float beta, float* v)
{
    if (D == 3) {
        v[0] = cr_new_s(R.r[0].x, R.r[1].x, R.r[2].x, alpha, beta);
        v[1] = cr_new_s(R.r[0].y, R.r[1].y, R.r[2].y, alpha, beta);
        v[2] = cr_new_s(R.r[0].z, R.r[1].z, R.r[2].z, alpha, beta);
    } else {   // s, a in the first record
        v[0] = cr_new_s(R.r[0].x, R.r[0].z, R.r[1].x, alpha, beta);
        v[1] = cr_new_s(R.r[0].y, R.r[0].w, R.r[1].y, alpha, beta);
        v[2] = 0.f;
    }
}

template <int D>
__device__ __forceinline__ void cr_publish(float4* rec, int i, const float* s, const float* a, const float* b)
{
    if (D == 3) {
        rec[3 * (size_t)i] = make_float4(s[0], s[1], s[2], 0.f);
        rec[3 * (size_t)i + 1] = make_float4(a[0], a[1], a[2], 0.f);
        rec[3 * (size_t)i + 2] = make_float4(b[0], b[1], b[2], 0.f);
    } else {
        rec[3 * (size_t)i] = make_float4(s[0], s[1], a[0], a[1]);
        rec[3 * (size_t)i + 1] = make_float4(b[0], b[1], 0.f, 0.f);
    }
}

template <int D, int PF>
__global__ void __launch_bounds__(kCrThreads, PF > 1 ? 1 : 2) k_pen_cr(DevParams P, PenArgs A, PenCr C)
{
    extern __shared__ int4 pen_smem[];
    __shared__ float wred[3][kCrThreads / 32];
    __shared__ float part[kCrThreads * D];
    __shared__ F2 sum_s[3];
    __shared__ float val_s[6];
    __shared__ float ab_s[2];
    __shared__ F2 rr_s;
    __shared__ int stop_s;
    const int rows = blockDim.x, W = blockDim.y, w = threadIdx.y;
    const int tid = w * rows + threadIdx.x, nth = rows * W, lane = tid & 31, warp = tid >> 5;
    const int lb = blockIdx.x, nb = gridDim.x;
    const int i = lb * rows + threadIdx.x;
    unsigned epoch = 0;
    int4* sa = pen_smem;                                                 // position, and s (2-D) or its first component
    float2* sb = reinterpret_cast<float2*>(pen_smem + A.umax);           // 3-D: the other two
    float* st = reinterpret_cast<float*>(sb + (D == 3 ? A.umax : 0));    // lambda t
    int* ul = reinterpret_cast<int*>(st + A.umax);                       // the staged columns
    uint2* words = reinterpret_cast<uint2*>(ul + A.umax);                // the rows' ranks, word by word
    // what the phase keeps
    const int U = A.ucount ? A.ucount[lb] : -1;
    const int n = i < A.N ? A.ncp[i] : 0;
    for (int k = tid; k < U; k += nth) {
        const int j = A.uniq[(size_t)lb * A.ucap + k];
        ul[k] = j;
        sa[k] = A.ipos[j];
    }
    int j0[PF > 0 ? PF : 1];   // the thread's first staged neighbours
#pragma unroll
    for (int u = 0; u < PF; ++u) j0[u] = tid + u * nth < U ? ul[tid + u * nth] : -1;
    int ng = 0;
    if (U >= 0 && n > 0) {
        ng = A.groups[i >> 5];
        const uint2* ip = A.idx + ((long long)(i >> 5) * A.pw4) * 32 + (i & 31);
        for (int g = w; g < ng; g += W) words[(size_t)g * rows + threadIdx.x] = ip[(long long)g * 32];
    }
    const int4 pi = i < A.N ? A.ipos[i] : make_int4(0, 0, 0, 0);
    const int ui[3] = {pi.x, pi.y, pi.z};
    const bool fluid = i < A.Nf, mine = w == 0 && fluid;
    int it = A.flags[kFlagIter];
    const int it_end = it + C.iters;
    const F2 stop_rr = f2_of(A.scal[kSTol2] * A.scal[kSIn0]);
    // thread 0's: (s, y) and (q, D^-1 q) of the last iteration
    F2 rho = f2_of(A.scal[rho_slot32(it - 1)]), qu = f2_of(A.scal[kSQUPrev]);
    const float m = P.pen_diag32[pi.w], lam = P.pen_lam32[pi.w];
    float s[3] = {0.f, 0.f, 0.f}, a[3] = {0.f, 0.f, 0.f}, b[3] = {0.f, 0.f, 0.f};
    float p[3] = {0.f, 0.f, 0.f}, z[3] = {0.f, 0.f, 0.f}, dv[3] = {0.f, 0.f, 0.f};
    if (mine) {
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const size_t k = (size_t)i * D + d;
            s[d] = A.s[k];
            z[d] = A.z[k];
            dv[d] = A.invD[k];
            if (it > 0) {
                p[d] = A.p[k];
                b[d] = A.q[k];   // D^-1 q, as this kernel leaves it
            }
        }
        const float zero[3] = {0.f, 0.f, 0.f};
        cr_publish<D>(C.rec, i, s, zero, zero);
    }
    // the row's slots: staged records by rank, or columns
    auto slots = [&](auto&& term) {
        if (U >= 0) {
            for (int g = w; g < ng; g += W) {
                const uint2 v = words[(size_t)g * rows + threadIdx.x];
                term((int)(v.x & 0xffffu));
                term((int)(v.x >> 16));
                term((int)(v.y & 0xffffu));
                term((int)(v.y >> 16));
            }
        } else {
            const int* col = A.nindP + (i < A.N ? A.nptrP[i] : 0);
            for (int g = w; 4 * g < n; g += W)
                for (int k = 4 * g; k < min(n, 4 * g + 4); ++k) term(col[k]);
        }
    };
    float alpha = 0.f, beta = 0.f;
    bool first = true;
    if (tid < 6) val_s[tid] = 0.f;
    bool ok = cr_cross(C.count, C.v3, val_s, 6, ++epoch, lb, nb, tid, A.flags, C.polls);   // every row's s is out
    // a crossing's first loads: the thread's first neighbour's records, while
    // alpha and beta are formed
    CrRec pre[PF > 0 ? PF : 1];
#pragma unroll
    for (int u = 0; u < PF; ++u) pre[u] = cr_load<D>(C.rec, j0[u], A.Nf);
    while (ok) {
        // the new vectors of the own row (not before the phase's first iteration)
        if (!first) {
            float rs = 0.f;
            if (mine) {
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    p[d] = beta * p[d] + s[d];
                    z[d] += alpha * p[d];
                    s[d] = cr_new_s(s[d], a[d], b[d], alpha, beta);
                    b[d] = __fmaf_rn(beta, b[d], a[d]);
                    const float r = dv[d] != 0.f ? __fdividef(s[d], dv[d]) : 0.f;
                    rs += r * r;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) rs += __shfl_xor_sync(0xffffffffu, rs, o);
            if (lane == 0) wred[0][warp] = rs;
            ++it;
        }
        // the new s of the staged neighbours
        auto put = [&](int k, const CrRec& R) {
            float v[3];
            cr_combine<D>(R, alpha, beta, v);
            if (D == 3) {
                sa[k].w = __float_as_int(v[0]);
                sb[k] = make_float2(v[1], v[2]);
            } else {
                sa[k].z = __float_as_int(v[0]);
                sa[k].w = __float_as_int(v[1]);
            }
        };
#pragma unroll
        for (int u = 0; u < PF; ++u)
            if (tid + u * nth < U) put(tid + u * nth, pre[u]);
#pragma unroll 2
        for (int k = tid + PF * nth; k < U; k += nth) put(k, cr_load<D>(C.rec, ul[k], A.Nf));
        float si[3] = {s[0], s[1], s[2]};
        if (W > 1 && w > 0 && fluid && n > 0) cr_combine<D>(cr_load<D>(C.rec, i, A.Nf), alpha, beta, si);
        __syncthreads();
        if (!first && warp == 0) {
            const F2 v = f2_warp_sum(F2{lane < (nth >> 5) ? wred[0][lane] : 0.f, 0.f}, 8);
            if (lane == 0) {
                val_s[0] = v.h;
                val_s[1] = v.l;
            }
        }
        // lambda t
        float acc = 0.f;
        if (n > 0) {
            auto one = [&](const int* uj, const float* sj) {
                float dq[3];
                const float cf = pen_coef<D>(P, ui, uj, dq);
                float dot = __fmul_rn(dq[0], __fadd_rn(si[0], -sj[0]));
                dot = __fmaf_rn(dq[1], __fadd_rn(si[1], -sj[1]), dot);
                if (D == 3) dot = __fmaf_rn(dq[2], __fadd_rn(si[2], -sj[2]), dot);
                acc = __fmaf_rn(cf, dot, acc);
            };
            slots([&](int k) {
                if (U >= 0) {
                    const int4 pj = sa[k];
                    const int uj[3] = {pj.x, pj.y, pj.z};
                    if (D == 3) {
                        const float2 v = sb[k];
                        const float sj[3] = {__int_as_float(pj.w), v.x, v.y};
                        one(uj, sj);
                    } else {
                        const float sj[3] = {__int_as_float(pj.z), __int_as_float(pj.w), 0.f};
                        one(uj, sj);
                    }
                } else {
                    const int4 pj = A.ipos[k];
                    const int uj[3] = {pj.x, pj.y, pj.z};
                    float sj[3];
                    cr_combine<D>(cr_load<D>(C.rec, k, A.Nf), alpha, beta, sj);
                    one(uj, sj);
                }
            });
        }
        float ti = acc;
        if (W > 1) {   // the row's partial sums in the order of w
            part[tid] = acc;
            __syncthreads();
            ti = part[threadIdx.x];
            for (int v = 1; v < W; ++v) ti += part[v * rows + threadIdx.x];
        }
        ti = n > 0 ? lam * ti : 0.f;
        if (w == 0 && i < A.N) A.t[i] = ti;
        // every particle's lambda t (and every block's (r, r)) is out
        if (!(ok = cr_cross(C.count, C.v1, val_s, 2, ++epoch, lb, nb, tid, A.flags, C.polls))) break;
        if (!first && warp == (nth >> 5) - 1) {   // the stop test
            const F2 v = cr_sum(C.v1, 2, nb, lane);
            if (lane == 0) {
                const bool bad = !(v.h == v.h);
                const bool below = __fadd_rn(__fadd_rn(v.h, -stop_rr.h), __fadd_rn(v.l, -stop_rr.l)) < 0.f;
                rr_s = v;
                stop_s = (it >= A.cap || below || bad) ? (bad ? 3 : 1) : (it >= it_end ? 2 : 0);
            }
        }
#pragma unroll 2
        for (int k = tid; k < U; k += nth) st[k] = __ldcg(A.t + ul[k]);
        __syncthreads();
        if (!first && stop_s) break;   // the same in every block
        first = false;
        // y = M s
        float y[3] = {0.f, 0.f, 0.f};
        if (fluid && n > 0) {
            auto one = [&](const int* uj, float tj) {
                float dq[3];
                const float cf = __fmul_rn(pen_coef<D>(P, ui, uj, dq), __fadd_rn(tj, ti));
#pragma unroll
                for (int d = 0; d < D; ++d) y[d] = __fmaf_rn(cf, dq[d], y[d]);
            };
            slots([&](int k) {
                const int4 pj = U >= 0 ? sa[k] : A.ipos[k];
                const int uj[3] = {pj.x, pj.y, pj.z};
                one(uj, U >= 0 ? st[k] : __ldcg(A.t + k));
            });
        }
        if (W > 1) {
#pragma unroll
            for (int d = 0; d < D; ++d) part[tid * D + d] = y[d];
            __syncthreads();
            if (w == 0)
                for (int v = 1; v < W; ++v)
#pragma unroll
                    for (int d = 0; d < D; ++d) y[d] += part[(v * rows + threadIdx.x) * D + d];
        }
        float v[3] = {0.f, 0.f, 0.f};
        if (mine) {
#pragma unroll
            for (int d = 0; d < D; ++d) {
                y[d] = __fmaf_rn(m, s[d], __fmul_rn(P.pen_w32, y[d]));
                a[d] = dv[d] * y[d];
                v[0] += s[d] * y[d];
                v[1] += a[d] * y[d];
                v[2] += b[d] * y[d];
            }
            cr_publish<D>(C.rec, i, s, a, b);
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[c] += __shfl_xor_sync(0xffffffffu, v[c], o);
            if (lane == 0) wred[c][warp] = v[c];
        }
        __syncthreads();
        if (warp < 3) {
            const F2 x = f2_warp_sum(F2{lane < (nth >> 5) ? wred[warp][lane] : 0.f, 0.f}, 8);
            if (lane == 0) {
                val_s[2 * warp] = x.h;
                val_s[2 * warp + 1] = x.l;
            }
        }
        // every row's s, a, b and every block's dot products are out
        if (!(ok = cr_cross(C.count, C.v3, val_s, 6, ++epoch, lb, nb, tid, A.flags, C.polls))) break;
#pragma unroll
        for (int u = 0; u < PF; ++u) pre[u] = cr_load<D>(C.rec, j0[u], A.Nf);
        if (warp < 3) {
            const F2 v = cr_sum(C.v3 + 2 * warp, 6, nb, lane);
            if (lane == 0) sum_s[warp] = v;
        }
        __syncthreads();
        if (tid == 0) {
            const F2 x[3] = {sum_s[0], sum_s[1], sum_s[2]};
            // beta = rho / rho', (q, D^-1 q) = (y, a) + beta (2 (y, b) + beta (q', D^-1 q')), alpha = rho / (q, D^-1 q)
            F2 be{0.f, 0.f}, nq = x[1];
            if (it > 0) {
                be = f2_div(x[0], rho);
                nq = f2_add(nq, f2_mul(be, f2_add(F2{2.f * x[2].h, 2.f * x[2].l}, f2_mul(be, qu))));
            }
            rho = x[0];
            qu = nq;
            ab_s[0] = f2_div(rho, qu).h;
            ab_s[1] = be.h;
        }
        __syncthreads();
        alpha = ab_s[0];
        beta = ab_s[1];
    }
    if (mine) {
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const size_t k = (size_t)i * D + d;
            A.z[k] = z[d];
            A.p[k] = p[d];
            A.q[k] = b[d];
        }
        if (ok && stop_s != 3) {   // not after a NaN
#pragma unroll
            for (int d = 0; d < D; ++d) {
                const size_t k = (size_t)i * D + d;
                const double v = C.x[k] + C.scale * (double)z[d];
                C.x[k] = v;
                C.vel[(size_t)i * (D == 2 ? 2 : 4) + d] = v;
            }
            C.z4[i] = make_float4(z[0], z[1], z[2], 0.f);
        }
    }
    if (lb == 0 && tid == 0) {
        A.flags[kFlagIter] = it;
        if (ok) {
            A.scal[rho_slot32(it - 1)] = (double)rho.h + (double)rho.l;
            A.scal[kSQUPrev] = (double)qu.h + (double)qu.l;
            A.scal[kSIn] = (double)rr_s.h + (double)rr_s.l;
            if (stop_s != 2) A.flags[kFlagDone] = 1;   // 2: the launch's bound, the phase goes on
            if (stop_s == 3) A.flags[kFlagBad] = 1;
        }
    }
}

// ---- the system: C, b and D^-1 -------------------------------------------------------
// C of every particle's P-list (calculateMatrixC main.cpp:2462-2507; the wall
// rows' C_kj = - C_jk of fluid j give C^T its wall rows without a transposed
// list), and for the fluid rows in the same pass b = inertia v - C p (its wall
// velocities follow in k_pen_wall) and the FP32 D^-1.  Bound by the FP64
// pipe: 1.2 ms on 1.3 million particles.  C, the transposed lists (0.69 ms),
// b with the pair terms (2.06) and their slicing (1.04) took 5.0 ms in passes
// of their own.
// *near: the largest f / inertia of a P-list's viscous pair in FP32 bits where
// it is above kNearMin, infinite for a pair closer than MaxRadius / 256.  A
// lattice's pairs are some 1e-4; one pair close together has f ~ 1 / r, and a
// refinement phase leaves 2 f / inertia of the pair's own motion, so a phase
// asks for no more than that, and beyond kNearMax, or where the positions'
// units no longer hold the pair's direction to FP32, the step takes the
// pair-term operator (mph_case::pen_near; 0.01 spacings apart at mu = 0.1 in
// 180 particles of 2-D: not converged with the lattice's target).
constexpr float kNearMin = 2.5e-4f, kNearMax = 0.05f;
template <int D, int L>
__global__ void __launch_bounds__(128) k_pen_system(DevParams P, const int* __restrict__ type, const double* __restrict__ pos,
                                                    const double* __restrict__ vel, const int* __restrict__ ncp,
                                                    const long long* __restrict__ nptrP, const int* __restrict__ nindP,
                                                    const double* __restrict__ pvec, double* __restrict__ cval,
                                                    double* __restrict__ bvec, float* __restrict__ invD, int* __restrict__ near)
{
    const int i0 = (blockIdx.x * blockDim.x + threadIdx.x) / L, part = threadIdx.x % L;
    const int i = min(i0, P.N - 1);
    const bool fluid = i < P.Nf;
    double xi[3];
    load_vec<D>(pos, i, xi);
    const double rP2 = P.rP * P.rP, K = -P.kfp * P.m2h_rp;
    const long long b = nptrP[i];
    const int n = i0 < P.N ? ncp[i] : 0;
    double self[3] = {0, 0, 0}, cp[3] = {0, 0, 0};
    float dp[3] = {0.f, 0.f, 0.f}, nearest = 0.f;   // the row's f / inertia
    const int tf = fluid ? type[i] : 0;
    int selfk = 0;
    for (int a = part; a < n; a += L) {
        const int j = nindP[b + a];
        double cv[3] = {0, 0, 0};
        if (j == i) {
            selfk = a;
        } else if (fluid || j < P.Nf) {
            double xj[3], q[3];
            load_vec<D>(pos, j, xj);
            sep_vec<D>(P, xj, xi, q);
            const double r2 = norm2_fma<D>(q);
            if (r2_pos_below(r2, rP2)) {
                // w' / r = kf (-2 / RadiusP) (1 - r / RadiusP) / r
                const double inv = rsqrt(r2), f = K * (inv - P.inv_rp);
                const double pj = fluid ? pvec[j] : 0.0;
                const int tj = type[j];
                const float lam = P.lambda32[tj], turn = (float)inv * P.near_r;   // MaxRadius / |q|
                nearest = fmaxf(nearest, turn > 256.f ? __int_as_float(0x7f800000) : P.near_f[tf][tj] * (turn - P.near_k));
#pragma unroll
                for (int r = 0; r < D; ++r) {
                    cv[r] = q[r] * f;
                    self[r] += cv[r];
                    cp[r] += cv[r] * pj;
                    dp[r] += (float)cv[r] * (float)cv[r] * lam;
                }
            }
        }
        if (j == i && fluid) continue;   // the sum's slot: one store, by the lane that has it (nothing orders two lanes' stores)
#pragma unroll
        for (int r = 0; r < D; ++r) cval[(b + a) * D + r] = cv[r];
    }
#pragma unroll
    for (int r = 0; r < D; ++r) {
        self[r] = row_sum<L>(self[r]);
        cp[r] = row_sum<L>(cp[r]);
        dp[r] = row_sum<L>(dp[r]);
    }
    selfk = row_sum<L>(selfk);   // set by one lane
    const int warp_near = __reduce_max_sync(0xffffffffu, fluid ? __float_as_int(nearest) : 0);
    if ((threadIdx.x & 31) == 0 && warp_near > __float_as_int(kNearMin) && warp_near > *(volatile int*)near) atomicMax(near, warp_near);
    if (!fluid || i0 >= P.N || part != 0) return;
    const int ti = tf;
    const double pi = pvec[i];
    double v[3];
    load_vec<D>(vel, i, v);
#pragma unroll
    for (int r = 0; r < D; ++r) {
        if (n > 0) cval[(b + selfk) * D + r] = self[r];
        bvec[(size_t)i * D + r] = P.inert64[ti] * v[r] - (cp[r] + self[r] * pi);
        const float dg = P.inert32[ti] + P.pen_vd[ti] + dp[r] + (float)self[r] * (float)self[r] * P.lambda32[ti];
        invD[(size_t)i * D + r] = dg != 0.f ? 1.f / dg : 0.f;
    }
}

// The wall slots of the fluid rows in FP64 (main.cpp:2274-2303): the wall part
// of the row's viscous diagonal block (rows with wall slots only) and, with
// the wall velocities, into b; L threads a row.  f = visc mu_ij kf' (1/r -
// 1/RadiusV), and every term is one factor f / r^2 of q (x) q.  A warp a row
// took 0.61 ms on 1.3 million particles, most of it rows without any slots
// and sums over the warp; the assembly stage takes 2.26 ms there with 16
// threads a row, 2.32 with 4, which leave 15 slots in line a thread (0.18 ms
// on 22,000 particles, 0.15 with 16).  In 2-D a row has a dozen: 8.
template <int D, int L>
__global__ void __launch_bounds__(128) k_pen_wall(DevParams P, const int* __restrict__ type, const double* __restrict__ pos,
                                                  const double* __restrict__ vel, const int* __restrict__ nc,
                                                  const int* __restrict__ nfc, const long long* __restrict__ nptr,
                                                  const int* __restrict__ nind, double* __restrict__ bvec, double* __restrict__ sdiag64)
{
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) / L, part = threadIdx.x % L;
    const int nf = i < P.Nf ? nfc[i] : 0, n = i < P.Nf ? nc[i] : 0;
    if (!__any_sync(0xffffffffu, n > nf)) return;   // none of the warp's rows
    double v[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};      // xx xy xz yy yz zz, then b's
    if (n > nf) {
        const int ti = type[i];
        const long long nb = nptr[i];
        const double rV2 = P.rV * P.rV, K = -P.kfv * P.m2h_rv * P.visc;
        double xi[3];
        load_vec<D>(pos, i, xi);
        for (int k = nf + part; k < n; k += L) {
            const int j = nind[nb + k];
            double xj[3], vj[3], q[3] = {0.0, 0.0, 0.0}, qv = 0.0, fq[3] = {0.0, 0.0, 0.0};
            load_vec<D>(pos, j, xj);
            sep_vec<D>(P, xj, xi, q);
            const double r2 = norm2_fma<D>(q);
            if (!r2_pos_below(r2, rV2)) continue;
            load_vec<D>(vel, j, vj);
            const double inv = rsqrt(r2);
            const double f = (K * P.muij[ti][type[j]]) * (inv - P.inv_rv) * (inv * inv);
#pragma unroll
            for (int d = 0; d < D; ++d) {
                qv += q[d] * vj[d];
                fq[d] = f * q[d];
            }
#pragma unroll
            for (int d = 0; d < D; ++d) v[6 + d] += fq[d] * qv;
            v[0] += fq[0] * q[0];
            v[1] += fq[0] * q[1];
            v[3] += fq[1] * q[1];
            if (D == 3) {
                v[2] += fq[0] * q[2];
                v[4] += fq[1] * q[2];
                v[5] += fq[2] * q[2];
            }
        }
    }
#pragma unroll
    for (int t = 0; t < 9; ++t) {
        if (D == 2 && (t == 2 || t == 4 || t == 5 || t == 8)) continue;
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) v[t] += __shfl_xor_sync(0xffffffffu, v[t], o);
    }
    if (n == nf || part != 0) return;
#pragma unroll
    for (int t = 0; t < 6; ++t) sdiag64[(size_t)i * 8 + t] = v[t];
#pragma unroll
    for (int d = 0; d < D; ++d) bvec[(size_t)i * D + d] += v[6 + d];
}

// The diagonal with its row's own viscous pairs, as the other forms' D^-1 (a
// reader's request only: the point-Jacobi form keeps the lattice's).
template <int D>
__global__ void __launch_bounds__(256) k_pen_diag(DevParams P, const int* __restrict__ type, const double* __restrict__ pos,
                                                  const float* __restrict__ pos32, const float* __restrict__ poslo32,
                                                  const int* __restrict__ nc, const long long* __restrict__ nptr,
                                                  const int* __restrict__ nind, const int* __restrict__ ncp,
                                                  const long long* __restrict__ nptrP, const int* __restrict__ nindP,
                                                  const double* __restrict__ cval, int* __restrict__ unused, double* __restrict__ dinv)
{
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= P.Nf) return;
    const int ti = type[i];
    float hi[3], li[3], t[3] = {0.f, 0.f, 0.f};
    load_f32<D>(pos32, i, hi);
    load_f32<D>(poslo32, i, li);
    for (int k = lane; k < nc[i]; k += 32) {
        float e[3] = {0.f, 0.f, 0.f}, f = 0.f;
        pair_ef<D>(P, i, nind[nptr[i] + k], ti, hi, li, type, pos, pos32, poslo32, unused, e, f);
#pragma unroll
        for (int d = 0; d < D; ++d) t[d] += f * e[d] * e[d];
    }
    for (int a = lane; a < ncp[i]; a += 32)
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const double c = cval[(nptrP[i] + a) * D + d];
            t[d] += (float)(c * P.lambda[type[nindP[nptrP[i] + a]]]) * (float)c;
        }
#pragma unroll
    for (int d = 0; d < D; ++d) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t[d] += __shfl_xor_sync(0xffffffffu, t[d], o);
        const float dg = P.inert32[ti] + t[d];
        if (lane == 0) dinv[(size_t)i * D + d] = (double)(dg != 0.f ? 1.f / dg : 0.f);
    }
}

// ---- the FP64 outer residual ------------------------------------------------------------
// r = b - A x, with A x in three parts: inertia, C Lambda C^T and the wall
// part of the viscous diagonal in FP64 from x, the fluid pairs
// sum f e (e . (x_i - x_j)) added up in FP64 over the solve's corrections,
// V x = V x_0 + sum scale V z.  The pairs are evaluated from the positions in
// FP32 (coefficients and row sums as the stored pair terms had them): the
// differences of x_0 in two floats, those of the FP32 corrections z exactly.
//
// (x_0 comes as records (hi, lo) from k_x0.)  The update x += scale z, and z as records:
template <int D>
__global__ void __launch_bounds__(256) k_pen_pack(int Nf, double* __restrict__ x, const float* __restrict__ z, double scale,
                                                  const double* __restrict__ scale_src, const int* __restrict__ flags,
                                                  float4* __restrict__ rec)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= Nf) return;
    if (flags && flags[kFlagBad]) return;   // the device-driven solve: a phase that met a NaN ends the solve
    float h[3] = {0.f, 0.f, 0.f};
    const double sc = scale_src ? *scale_src : scale;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        const size_t k = (size_t)i * D + d;
        h[d] = z[k];
        x[k] += sc * (double)h[d];
    }
    rec[i] = make_float4(h[0], h[1], h[2], 0.f);
}

// lambda_k t_k, t = C^T x in FP64 from the particle's own P-list:
// C_jk = - C_kj (to the rounding of the minimum image), and C_kk for a fluid
// row itself
template <int D, int L>
__device__ __forceinline__ void pen_ct64(const DevParams& P, int tid, const int* __restrict__ type, const int* __restrict__ ncp,
                                         const long long* __restrict__ nptrP, const int* __restrict__ nindP,
                                         const double* __restrict__ cval, const double* __restrict__ x, double* __restrict__ t)
{
    const int k = tid / L, part = tid % L;
    const long long b = k < P.N ? nptrP[k] : 0;
    const int n = k < P.N ? ncp[k] : 0;
    double s = 0.0;
#pragma unroll 2
    for (int a = part; a < n; a += L) {
        const int j = nindP[b + a];
        if (j >= P.Nf) continue;
        double v = 0.0;
#pragma unroll
        for (int d = 0; d < D; ++d) v += cval[(b + a) * D + d] * x[(size_t)j * D + d];
        s = j == k ? s + v : s - v;
    }
    s = row_sum<L>(s);
    if (k < P.N && part == 0) t[k] = P.lambda[type[k]] * s;
}

// vacc_i (+)= scale sum over the fluid neighbours of f e (e . (x_i - x_j)),
// L lanes a row over its neighbour list.  A pair is two 16-byte gathers (three
// for x_0) and some 35 instructions; bound by the L1's gather rate.  Against
// the stored FP32 g and columns (16 bytes a slot streamed, x in six 4-byte
// gathers: 1.33 ms on 1.3 million particles with the P-part) it needs no pair
// terms, which took three passes to build: with C^T x in the same launch 0.92
// ms for x_0, 0.74 for z.
// The launch's first nbT blocks form lambda t of C^T x meanwhile (pen_ct64).
template <int D, int L, bool FIRST, int LT>
__global__ void __launch_bounds__(256) k_pen_visc(DevParams P, int nbT, const int4* __restrict__ ipos, const int* __restrict__ nfc,
                                                  const long long* __restrict__ nptr, const int* __restrict__ nind,
                                                  const float4* __restrict__ rec, const int* __restrict__ type, double scale,
                                                  const double* __restrict__ scale_src, double* __restrict__ vacc,
                                                  const int* __restrict__ ncp, const long long* __restrict__ nptrP,
                                                  const int* __restrict__ nindP, const double* __restrict__ cval,
                                                  const double* __restrict__ x, double* __restrict__ t)
{
    if ((int)blockIdx.x < nbT) {
        pen_ct64<D, LT>(P, blockIdx.x * blockDim.x + threadIdx.x, type, ncp, nptrP, nindP, cval, x, t);
        return;
    }
    const int i = ((blockIdx.x - nbT) * blockDim.x + threadIdx.x) / L, lane = threadIdx.x & (L - 1);
    float y[3] = {0.f, 0.f, 0.f};
    if (i < P.Nf) {
        const int n = nfc[i];
        const int* col = nind + nptr[i];
        const float4 hi = rec[i];
        const float4 li = FIRST ? rec[P.Nf + i] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4* lo = rec + P.Nf;
        const int4 pi = ipos[i];
        const float vm0 = pi.w ? P.pen_vm[1][0] : P.pen_vm[0][0], vm1 = pi.w ? P.pen_vm[1][1] : P.pen_vm[0][1];
#pragma unroll 4
        for (int k = lane; k < n; k += L) {
            const int j = col[k];
            const int4 pj = ipos[j];
            const float4 h = rec[j];
            const float q[3] = {fixed_sep_v(P, 0, pj.x, pi.x), fixed_sep_v(P, 1, pj.y, pi.y), D == 3 ? fixed_sep_v(P, 2, pj.z, pi.z) : 0.f};
            float dx[3] = {hi.x - h.x, hi.y - h.y, D == 3 ? hi.z - h.z : 0.f};
            if (FIRST) {
                const float4 l = lo[j];
                dx[0] += li.x - l.x;
                dx[1] += li.y - l.y;
                if (D == 3) dx[2] += li.z - l.z;
            }
            float r2 = q[0] * q[0] + q[1] * q[1];
            if (D == 3) r2 += q[2] * q[2];
            const float inv = rsqrtf(fmaxf(r2, 1e-18f));
            // mu_ij w' / |q|, w' = 1 - |q|, up to the constants in pen_v0; q / |q| twice (the row itself: 0)
            float dot = q[0] * dx[0] + q[1] * dx[1];
            if (D == 3) dot += q[2] * dx[2];
            const float t = (pj.w ? vm1 : vm0) * fmaxf(inv - 1.f, 0.f) * (dot * inv) * inv;
#pragma unroll
            for (int d = 0; d < D; ++d) y[d] += t * q[d];
        }
    }
#pragma unroll
    for (int d = 0; d < D; ++d)
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) y[d] += __shfl_xor_sync(0xffffffffu, y[d], o);
    if (i < P.Nf && lane < D) {
        const float yl = lane == 0 ? y[0] : (lane == 1 ? y[1] : y[2]);
        const size_t k = (size_t)i * D + lane;
        const double v = P.pen_v0 * (double)yl;
        vacc[k] = FIRST ? v : vacc[k] + (scale_src ? *scale_src : scale) * v;
    }
}

template <int D, int L>
__global__ void __launch_bounds__(128) k_pen_resid(DevParams P, const int* __restrict__ type, const int* __restrict__ nc,
                                                   const int* __restrict__ nfc, const int* __restrict__ ncp,
                                                   const long long* __restrict__ nptrP, const int* __restrict__ nindP,
                                                   const double* __restrict__ cval, const double* __restrict__ t,
                                                   const double* __restrict__ sdiag64, const double* __restrict__ vacc,
                                                   const double* __restrict__ x, const double* __restrict__ b, double* __restrict__ r,
                                                   double* __restrict__ partials, unsigned* __restrict__ counter, double* __restrict__ out)
{
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) / L, part = threadIdx.x % L;
    double acc = 0.0, y[3] = {0.0, 0.0, 0.0};
    if (i < P.Nf) {
        const long long pb = nptrP[i];
        const int np = ncp[i];
#pragma unroll 2
        for (int a = part; a < np; a += L) {
            const double lt = t[nindP[pb + a]];
#pragma unroll
            for (int d = 0; d < D; ++d) y[d] += cval[(pb + a) * D + d] * lt;
        }
    }
#pragma unroll
    for (int d = 0; d < D; ++d) y[d] = row_sum<L>(y[d]);
    if (i < P.Nf && part == 0) {
        double xi[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int d = 0; d < D; ++d) {
            xi[d] = x[(size_t)i * D + d];
            y[d] += vacc[(size_t)i * D + d];
        }
        if (nc[i] > nfc[i]) {   // wall neighbours: their part of the viscous diagonal
            const double2* sp = reinterpret_cast<const double2*>(sdiag64 + (size_t)i * 8);
            const double2 p = sp[0], q = sp[1], e = sp[2];   // (xx, xy), (xz, yy), (yz, zz)
            y[0] += p.x * xi[0] + p.y * xi[1] + q.x * xi[2];
            y[1] += p.y * xi[0] + q.y * xi[1] + e.x * xi[2];
            y[2] += q.x * xi[0] + e.x * xi[1] + e.y * xi[2];
        }
        const double inert = P.inert64[type[i]];
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const size_t k = (size_t)i * D + d;
            const double rv = b[k] - (inert * xi[d] + y[d]);
            r[k] = rv;
            acc += rv * rv;
        }
    }
    reduce_finalize(acc, partials, counter, out);
}

// Start of a refinement phase: r32 = r / scale, s = D^-1 r32, z = 0, the inner
// reference norm (r32, r32), the phase's target and the done flag.  The target
// is a reduction by tol_in or, in the phase that may meet the outer test with
// it (an iteration takes some 0.86, so a phase lands up to that much below its
// target), the fraction aim of what that test still asks for, less or more than
// tol_in, but no less than the inner operator leaves of the true residual
// (floor): where a solve lands under its tolerance then does not depend on
// where the phases before happened to end.
__global__ void __launch_bounds__(kReduceThreads) k_pen_phase(int n, const double* __restrict__ r, const float* __restrict__ invD,
                                                              float* __restrict__ s, float* __restrict__ z, double inv_scale,
                                                              const double* __restrict__ scale_src, double tol_in2, double tol_out2,
                                                              double aim2, double floor2, double* __restrict__ scal, int* __restrict__ flags,
                                                              double* __restrict__ partials, unsigned* __restrict__ counter,
                                                              unsigned* __restrict__ crossings)
{
    if (crossings && blockIdx.x == 0 && threadIdx.x == 0) *crossings = 0u;   // of the resident launch that follows
    const double sc = scale_src ? 1.0 / *scale_src : inv_scale;
    float acc = 0.f;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const float v = (float)(r[k] * sc);
        s[k] = invD[k] * v;
        z[k] = 0.f;
        acc += v * v;
    }
    if (reduce_finalize_last(acc, partials, counter, scal + kSIn0)) {
        const double left = tol_out2 * scal[kSRR0] / scal[kSRR];
        const double tol2 = 0.5 * tol_in2 < left ? fmax(aim2 * left, floor2) : tol_in2;
        scal[kSTol2] = tol2;
        const F2 stop = f2_of(tol2 * scal[kSIn0]);
        reinterpret_cast<float2*>(scal)[kSStop] = make_float2(stop.h, stop.l);
        scal[kSIn] = scal[kSIn0];
        flags[kFlagDone] = 0;
    }
}

// ---- host side ---------------------------------------------------------------------
constexpr int kPenBlocks = 152 * kPenResident;   // blocks of k_pen_y: what is resident at once

// Shared memory of the resident iteration for `umax` staged neighbours
static size_t cr_smem(const mph_case* c, int rows, int umax)
{
    return (size_t)umax * (c->dim == 3 ? 32 : 24) + (size_t)rows * ((c->pmax + 3) / 4) * sizeof(uint2) + 16;
}

// Blocks of the resident iteration that the device holds at once (0: none), two
// an SM and, in c->cr_alone, one an SM in the form with more registers
static int cr_capacity(mph_case* c)
{
    if (c->cr_cap < 0) {   // once a case: the attributes and the count belong to its device
        int sms = 0, coop = 0, nb = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device);
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c->device);
        const void* f[2] = {c->dim == 2 ? (const void*)k_pen_cr<2, kCrShared2> : (const void*)k_pen_cr<3, kCrShared3>,
                            c->dim == 2 ? (const void*)k_pen_cr<2, kCrAhead> : (const void*)k_pen_cr<3, kCrAhead>};
        for (const void* k : f) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kCrSmem);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, f[0], kCrThreads, kCrSmem);
        c->cr_cap = std::min(coop ? sms * nb : 0, kCrBlocks);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, f[1], kCrThreads, kCrSmem);
        c->cr_alone = coop && nb > 0 ? std::min(sms, kCrBlocks / 2) : 0;
    }
    return c->cr_cap;
}

static void pen_shape(mph_case* c)
{
    const int cap = cr_capacity(c);
    auto fits = [c](int r) { return r <= kCrThreads && cr_smem(c, r, (pen_ucap(r) + 127) / 128 * 128) <= (size_t)kCrSmem; };
    const PenShape S = pen_shape_for(c->dp.N, c->dim == 2 ? kCrMinRows2 : kCrMinRows3, kCrThreads, cap, c->cr_alone, fits);
    c->pen_rows = S.rows;
    c->pen_w = S.w;
    c->pen_resident = S.resident;
    c->pen_alone = S.alone;
}

// (The positions' unit is MaxRadius / 2^30, which stays fine in RadiusP.)
bool pen_applies(const mph_case* c)
{
    const DevParams& P = c->dp;
    if (!(c->step_pairs && mixed_jacobi(c) && P.maxR <= 16.0 * P.rP)) return false;
    for (int t = 0; t < 2; ++t)
        for (int u = 0; u < 2; ++u)
            if (!(P.pen_v0 * P.pen_vm[t][u] <= 1.0e25)) return false;   // unit systems far outside FP32's range
    return true;
}

template <typename T>
static int grow_t(T** p, long long* cap, long long need)
{
    if (need <= *cap) return MPH_OK;
    if (*p) cudaFree(*p);
    *p = nullptr;
    *cap = 0;
    const long long n = need + need / 8 + 1024;
    MPH_CUDA(cudaMalloc((void**)p, (size_t)n * sizeof(T)));
    *cap = n;
    return MPH_OK;
}

static int pen_smem_t(const mph_case* c) { return c->pen_umax * (c->dim == 3 ? 24 : 16); }
static int pen_smem_y(const mph_case* c) { return c->pen_umax * 16; }

// The P-lists' ranks of this step (c->pmax is the longest P-list).
static int launch_pen_lists(mph_case* c)
{
    DeviceState& d = c->d;
    const DevParams& P = c->dp;
    c->pen_staged = false;
    pen_shape(c);
    c->pen_pw4 = (c->pmax + 3) / 4;
    const int nsl = (P.N + 31) / 32, nb = (int)grid_for(P.N, c->pen_rows), ucap = pen_ucap(c->pen_rows);
    if (!d.pgroups) MPH_CUDA(cudaMalloc((void**)&d.pgroups, (size_t)nsl * sizeof(int)));
    MPH_TRY(grow_t(&d.puniq, &d.cap_puniq, (long long)nb * ucap));
    MPH_TRY(grow_t(&d.pucount, &d.cap_pucount, nb + 5));
    if (c->pen_resident) {   // each asked for on its own: one may have failed before
        if (!d.cr_rec) MPH_CUDA(cudaMalloc((void**)&d.cr_rec, (size_t)P.Nf * 3 * sizeof(float4)));
        if (!d.cr_vals) MPH_CUDA(cudaMalloc((void**)&d.cr_vals, (size_t)(8 * kCrBlocks + 32) * sizeof(float)));
    }
    MPH_TRY(grow_t(&d.pidx, &d.cap_pidx, (long long)nsl * c->pen_pw4 * 32));
    c->pen_umax = 0;
    c->loc_blocks[0] = 0;
    c->loc_blocks[1] = (int)grid_for(P.Nf, c->pen_rows);
    c->loc_cols = 0;
    c->loc_ct_blocks = 0;
    auto near_of = [](int bits) {   // rounded up to a quarter of an octave: small changes keep the captured solve
        float f;
        std::memcpy(&f, &bits, sizeof(f));
        return f > 0.f ? std::exp2(std::ceil(4.0 * std::log2((double)f)) / 4.0) : 0.0;
    };
    int h[5] = {};
    if (!c->inner_local) {
        MPH_CUDA(cudaMemcpyAsync(h, d.wrap32 + 2, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
        MPH_CUDA(cudaStreamSynchronize(c->stream));
        c->pen_near = near_of(h[0]);
        return MPH_OK;
    }
    const size_t smem = 2 * kPlWords * sizeof(unsigned);
    // (what the iteration's kernels stage is within a block's default limit)
    static_assert(pen_ucap(kMaxPenRows) % 128 == 0 && pen_ucap(kMaxPenRows) * 24 + 4096 <= 48 * 1024, "k_pen_t's shared memory");
    if (!c->pen_attr) {   // once a case: the attribute belongs to its device
        MPH_CUDA(cudaFuncSetAttribute(k_plist_ranks, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        c->pen_attr = true;
    }
    MPH_CUDA(cudaMemsetAsync(d.pucount + nb, 0, 5 * sizeof(int), c->stream));
    { k_plist_ranks<<<nb, c->pen_rows, smem, c->stream>>>(P.N, P.Nf, c->pen_pw4, ucap, d.ncp, d.nptrP, d.nindP, d.pidx, d.pgroups,
                                                         d.puniq, d.pucount, d.wrap32 + 2); MPH_COUNT_LAUNCH(); }
    MPH_CUDA(cudaMemcpyAsync(h, d.pucount + nb, sizeof(h), cudaMemcpyDeviceToHost, c->stream));
    MPH_CUDA(cudaStreamSynchronize(c->stream));
    c->pen_umax = (h[0] + 127) / 128 * 128;   // rounded up: small changes keep the captured graphs
    c->loc_ct_blocks = h[1];
    c->loc_blocks[0] = h[2];
    c->loc_blocks[1] -= h[2];
    c->loc_cols = (long long)(unsigned)h[3];
    c->pen_near = near_of(h[4]);
    c->pen_staged = true;
    return MPH_OK;
}

// The assembly stage of the point-Jacobi mixed form: no blocks, no pair terms,
// no slices and no transposed lists.  Leaves step_pen false where a pair is too
// close for the operator (the caller then assembles the pair terms).
int launch_pen_assemble(mph_case* c)
{
    DeviceState& d = c->d;
    const DevParams& P = c->dp;
    cudaStream_t st = c->stream;
    const size_t n = (size_t)P.Nf * c->dim;
    c->nslots = 0;
    c->level0_done = c->ct_ready = false;
    if (!d.ipos) MPH_CUDA(cudaMalloc((void**)&d.ipos, (size_t)P.N * sizeof(int4)));
    if (!d.z4) {   // components that a record does not use stay zero
        MPH_CUDA(cudaMalloc((void**)&d.z4, (size_t)P.Nf * 2 * sizeof(float4)));
        MPH_CUDA(cudaMemsetAsync(d.z4, 0, (size_t)P.Nf * 2 * sizeof(float4), st));
    }
    if (!d.vacc) MPH_CUDA(cudaMalloc((void**)&d.vacc, n * sizeof(double)));
    if (!d.v32) MPH_CUDA(cudaMalloc((void**)&d.v32, vec32_stride(n) * 8 * sizeof(float)));
    if (!d.tct) MPH_CUDA(cudaMalloc((void**)&d.tct, (size_t)(P.N + 1) * sizeof(double)));
    if (!d.tct32) MPH_CUDA(cudaMalloc((void**)&d.tct32, (size_t)(P.N + 1) * sizeof(float)));
    if (!d.sdiag64) MPH_CUDA(cudaMalloc((void**)&d.sdiag64, (size_t)P.Nf * 8 * sizeof(double)));
    MPH_TRY(grow_t(&d.cval, &d.cap_cval, c->nnbP * c->dim));
    launch_vector_p(c);
    const unsigned g = grid_for(P.N, 256);
    float* invD = d.v32 + 7 * vec32_stride(n);
    const int L = plist_lanes(P.N);
    auto system = [&](auto kern) {
        kern<<<grid_for((long long)P.N * L, 128), 128, 0, st>>>(P, d.type, d.pos, d.vel, d.ncp, d.nptrP, d.nindP, d.pvec, d.cval, d.bvec, invD, d.wrap32 + 2);
        MPH_COUNT_LAUNCH();
    };
    if (c->dim == 2) {
        { k_fixed_positions<2><<<g, 256, 0, st>>>(P, d.type, d.pos, d.ipos); MPH_COUNT_LAUNCH(); }
        L == 4 ? system(k_pen_system<2, 4>) : system(k_pen_system<2, 1>);
    } else {
        { k_fixed_positions<3><<<g, 256, 0, st>>>(P, d.type, d.pos, d.ipos); MPH_COUNT_LAUNCH(); }
        L == 4 ? system(k_pen_system<3, 4>) : system(k_pen_system<3, 1>);
    }
    auto walls = [&](auto kern, int lanes) {
        kern<<<grid_for((long long)P.Nf * lanes, 128), 128, 0, st>>>(P, d.type, d.pos, d.vel, d.nc, d.nfc, d.nptr, d.nind, d.bvec, d.sdiag64);
        MPH_COUNT_LAUNCH();
    };
    if (c->dim == 2) walls(k_pen_wall<2, 8>, 8);
    else walls(k_pen_wall<3, 16>, 16);
    MPH_TRY(launch_pen_lists(c));
    c->step_pen = c->pen_near <= kNearMax;
    return MPH_OK;
}

// D^-1 as a reader gets it (FP64 array), from the current step's lists and C
int pen_exact_diag(mph_case* c)
{
    DeviceState& d = c->d;
    const unsigned g = grid_for((long long)c->dp.Nf * 32, 256);
    if (c->dim == 2) k_pen_diag<2><<<g, 256, 0, c->stream>>>(c->dp, d.type, d.pos, d.pos32, d.poslo32, d.nc, d.nptr, d.nind, d.ncp, d.nptrP, d.nindP, d.cval, d.wrap32 + 1, d.invDiag);
    else k_pen_diag<3><<<g, 256, 0, c->stream>>>(c->dp, d.type, d.pos, d.pos32, d.poslo32, d.nc, d.nptr, d.nind, d.ncp, d.nptrP, d.nindP, d.cval, d.wrap32 + 1, d.invDiag);
    MPH_COUNT_LAUNCH();
    MPH_CUDA(cudaGetLastError());
    return MPH_OK;
}

// the viscous pairs' sum, C^T x and the residual, after k_pen_pack
template <int D, int L, bool FIRST, int LT>
static void pen_residual_t(mph_case* c, double scale, const double* scale_src)
{
    DeviceState& d = c->d;
    const DevParams& P = c->dp;
    cudaStream_t st = c->stream;
    const unsigned nbT = grid_for((long long)P.N * LT, 256);
    { k_pen_visc<D, L, FIRST, LT><<<nbT + grid_for((long long)P.Nf * L, 256), 256, 0, st>>>(
          P, (int)nbT, d.ipos, d.nfc, d.nptr, d.nind, d.z4, d.type, scale, scale_src, d.vacc,
          d.ncp, d.nptrP, d.nindP, d.cval, d.x, d.tct); MPH_COUNT_LAUNCH(); }
    { k_pen_resid<D, LT><<<grid_for((long long)P.Nf * LT, 128), 128, 0, st>>>(P, d.type, d.nc, d.nfc, d.ncp, d.nptrP, d.nindP, d.cval, d.tct, d.sdiag64, d.vacc,
                                                          d.x, d.bvec, d.r, d.partials, (unsigned*)(d.flags + kFlagCounter), d.scal + kSRR); MPH_COUNT_LAUNCH(); }
}

template <int D, int L, bool FIRST>
static void pen_residual(mph_case* c, double scale, const double* scale_src)
{
    if (plist_lanes(c->dp.N) == 4) pen_residual_t<D, L, FIRST, 4>(c, scale, scale_src);
    else pen_residual_t<D, L, FIRST, 1>(c, scale, scale_src);
}

// lanes a row of k_pen_visc: about 180 neighbours in 3-D, 37 in 2-D
constexpr int kVisc3 = 16, kVisc2 = 8;

// r = b - A x of the start value (its records are in z4, k_x0)
void launch_pen_start_residual(mph_case* c)
{
    if (c->dim == 2) pen_residual<2, kVisc2, true>(c, 0.0, nullptr);
    else pen_residual<3, kVisc3, true>(c, 0.0, nullptr);
}

// the residual after a resident phase, which has updated x and left z in z4
void launch_pen_residual(mph_case* c, double scale)
{
    if (c->dim == 2) pen_residual<2, kVisc2, false>(c, scale, nullptr);
    else pen_residual<3, kVisc3, false>(c, scale, nullptr);
}

// x += scale z and the residual after a phase
void launch_pen_refine(mph_case* c, double scale, const double* scale_src, const int* flags)
{
    DeviceState& d = c->d;
    const int Nf = c->dp.Nf;
    const float* z = d.v32 + vec32_stride((long long)Nf * c->dim);
    if (c->dim == 2) {
        { k_pen_pack<2><<<grid_for(Nf, 256), 256, 0, c->stream>>>(Nf, d.x, z, scale, scale_src, flags, d.z4); MPH_COUNT_LAUNCH(); }
        pen_residual<2, kVisc2, false>(c, scale, scale_src);
    } else {
        { k_pen_pack<3><<<grid_for(Nf, 256), 256, 0, c->stream>>>(Nf, d.x, z, scale, scale_src, flags, d.z4); MPH_COUNT_LAUNCH(); }
        pen_residual<3, kVisc3, false>(c, scale, scale_src);
    }
}

static unsigned* cr_count(const mph_case* c) { return (unsigned*)(c->d.cr_vals + 8 * kCrBlocks); }

// What the inner operator leaves of the true residual, at least: the viscous
// pairs outside it (the lattice's, or a close pair's).
double pen_floor(const mph_case* c) { return std::min(std::max(c->pen_tol, 2.0 * c->pen_near), 0.1); }

// The last phase aims at a quarter of the outer tolerance, and from 1e-10 down
// to 1e-11 at ever less, at a tenth beyond: such tolerances are asked for
// where forces and pressures are read off the velocities' divergence, which
// shows the solve's error enlarged (2-D frames at 1e-11: 4 to 11e-10 of the
// forces at a half, 1.4 to 3.5e-10 at an eighth).  At a half, solves refined to
// 1e-10 were up to 60% further from the 64-bit solution than with the pair-term
// operator (412,000 particles in 2-D 5.0e-11 and 3.2e-11; at a quarter 2.6e-11);
// a quarter takes some five of 150 iterations more (22,000 particles and three
// steps 6.0 -> 6.2 ms).
void launch_pen_phase(mph_case* c, double inv_scale, const double* scale_src, double tol_in2, double tol_out2)
{
    DeviceState& d = c->d;
    const double aim = std::max(0.1, 0.25 * std::min(1.0, std::pow(c->tol_outer * 1.0e10, 0.39794)));
    const double floor = pen_floor(c);
    const int n = c->dp.Nf * c->dim;
    float* v = d.v32;
    { k_pen_phase<<<std::min<int>(grid_for(n, kReduceThreads), kReduceBlocks), kReduceThreads, 0, c->stream>>>(
          n, d.r, v + 7 * vec32_stride(n), v + 2 * vec32_stride(n), v + vec32_stride(n), inv_scale, scale_src, tol_in2, tol_out2,
          aim * aim, floor * floor, d.scal, d.flags, d.partials,
          (unsigned*)(d.flags + kFlagCounter), c->pen_resident ? cr_count(c) : nullptr); MPH_COUNT_LAUNCH(); }
}

static PenArgs pen_args(const mph_case* c, int cap)
{
    const DeviceState& d = c->d;
    const size_t n = (size_t)c->dp.Nf * c->dim;
    PenArgs A{};
    A.N = c->dp.N;
    A.Nf = c->dp.Nf;
    A.pw4 = c->pen_pw4;
    A.ucap = pen_ucap(c->pen_rows);
    A.umax = c->pen_umax;
    A.cap = cap;
    A.ipos = d.ipos;
    A.idx = d.pidx;
    A.groups = d.pgroups;
    A.uniq = d.puniq;
    A.ucount = c->pen_staged ? d.pucount : nullptr;   // as the assembly built the lists: the option may have changed since
    A.ncp = d.ncp;
    A.nindP = d.nindP;
    A.nptrP = d.nptrP;
    const size_t ns = vec32_stride(n);
    A.z = d.v32 + ns;
    A.s = d.v32 + 2 * ns;
    A.y = d.v32 + 3 * ns;
    A.p = d.v32 + 4 * ns;
    A.q = d.v32 + 5 * ns;
    A.invD = d.v32 + 7 * ns;
    A.t = d.tct32;
    A.scal = d.scal;
    A.flags = d.flags;
    A.partials = d.partials;
    A.counter = (unsigned*)(d.flags + kFlagCounter);
    return A;
}

// The phase's iterations in one cooperative launch
int launch_pen_resident(mph_case* c, int cap, double scale)
{
    DeviceState& d = c->d;
    PenArgs A = pen_args(c, cap);
    const int nb = (int)grid_for(A.N, c->pen_rows);
    PenCr C{};
    C.rec = d.cr_rec;
    C.v3 = d.cr_vals;
    C.v1 = d.cr_vals + 6 * kCrBlocks;
    C.count = cr_count(c);   // zeroed by k_pen_phase
    C.scale = scale;
    C.iters = c->cr_iters;
    C.polls = c->cr_polls;
    C.x = d.x;
    C.vel = d.vel;
    C.z4 = d.z4;
    const dim3 blk(c->pen_rows, c->pen_w);
    void* args[] = {&c->dp, &A, &C};
    const size_t smem = cr_smem(c, c->pen_rows, c->pen_umax);
    // a block an SM and the device to itself (or too few SMs for the other form): the form with more registers
    const bool alone = c->pen_alone && (!c->shared_gpu || nb > c->cr_cap);
    const void* f = c->dim == 2 ? (alone ? (const void*)k_pen_cr<2, kCrAhead> : (const void*)k_pen_cr<2, kCrShared2>)
                                : (alone ? (const void*)k_pen_cr<3, kCrAhead> : (const void*)k_pen_cr<3, kCrShared3>);
    MPH_CUDA(cudaLaunchCooperativeKernel(f, dim3(nb), blk, args, smem, c->stream));
    MPH_COUNT_LAUNCH();
    return MPH_OK;
}

static unsigned vec_blocks(int n) { return std::min<unsigned>(grid_for(n / 4 + 1, kReduceThreads), kReduceBlocks); }

// y = M s and the iteration's scalars (two launches), then the vectors (one)
void launch_pen_operator(mph_case* c, int cap)
{
    const PenArgs A = pen_args(c, cap);
    const dim3 blk(c->pen_rows, c->pen_w);
    const int gt = (int)grid_for(A.N, c->pen_rows), nrb = (int)grid_for(A.Nf, c->pen_rows), gy = std::min(nrb, kPenBlocks);
    if (c->dim == 2) {
        { k_pen_t<2><<<gt, blk, pen_smem_t(c), c->stream>>>(c->dp, A); MPH_COUNT_LAUNCH(); }
        { k_pen_y<2><<<gy, blk, pen_smem_y(c), c->stream>>>(c->dp, A, nrb); MPH_COUNT_LAUNCH(); }
    } else {
        { k_pen_t<3><<<gt, blk, pen_smem_t(c), c->stream>>>(c->dp, A); MPH_COUNT_LAUNCH(); }
        { k_pen_y<3><<<gy, blk, pen_smem_y(c), c->stream>>>(c->dp, A, nrb); MPH_COUNT_LAUNCH(); }
    }
}

void launch_pen_vectors(mph_case* c, int cap, bool use_cond, cudaGraphConditionalHandle cond)
{
    const PenArgs A = pen_args(c, cap);
    const int n = A.Nf * c->dim;
    const unsigned rb = vec_blocks(n);
    if (use_cond) { k_pen_vec<true><<<rb, kReduceThreads, 0, c->stream>>>(A, n, 1, cond); MPH_COUNT_LAUNCH(); }
    else { k_pen_vec<false><<<rb, kReduceThreads, 0, c->stream>>>(A, n, 0, cond); MPH_COUNT_LAUNCH(); }
}

// ---- the iteration over the cases of a batch ------------------------------------------
struct BatchPen {
    DevParams P;
    PenArgs A;
    int n, t_nb, y_nb, y_nrb, v_nb;
};

template <int D>
__global__ void __launch_bounds__(kMaxPenRows) k_batch_pen_t(const BatchPen* __restrict__ cs, const int* __restrict__ b0, int nc)
{
    const int c = batch_case_of(b0, nc, (int)blockIdx.x);
    pen_t_body<D>(cs[c].P, cs[c].A, (int)blockIdx.x - b0[c]);
}
template <int D>
__global__ void __launch_bounds__(kMaxPenRows) k_batch_pen_y(const BatchPen* __restrict__ cs, const int* __restrict__ b0, int nc)
{
    const int c = batch_case_of(b0, nc, (int)blockIdx.x);
    pen_y_body<D>(cs[c].P, cs[c].A, (int)blockIdx.x - b0[c], cs[c].y_nb, cs[c].y_nrb);
}
__global__ void __launch_bounds__(kReduceThreads) k_batch_pen_vec(const BatchPen* __restrict__ cs, const int* __restrict__ b0, int nc)
{
    const int c = batch_case_of(b0, nc, (int)blockIdx.x);
    pen_vec_body<false>(cs[c].A, (int)blockIdx.x - b0[c], cs[c].v_nb, cs[c].n, 0, 0);
}
__global__ void k_batch_flags(const BatchPen* __restrict__ cs, int nc, int* __restrict__ out)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < nc * kFlagCount) out[t] = cs[t / kFlagCount].A.flags[t % kFlagCount];
}

size_t batch_pen_bytes() { return sizeof(BatchPen); }

// the case's record in a host table, and its block counts of the three launches
void batch_pen_fill(const mph_case* c, int cap, void* table, int k, int* nb)
{
    BatchPen& B = ((BatchPen*)table)[k];
    B.P = c->dp;
    B.A = pen_args(c, cap);
    B.n = c->dp.Nf * c->dim;
    B.t_nb = nb[0] = (int)grid_for(c->dp.N, c->pen_rows);
    B.y_nrb = (int)grid_for(c->dp.Nf, c->pen_rows);
    B.y_nb = nb[1] = std::min(B.y_nrb, kPenBlocks);
    B.v_nb = nb[2] = (int)vec_blocks(B.n);
}

// One CR iteration of the cases that still iterate (b0: the block starts of
// the three launches, nc + 1 each; nb: their block totals; umax: the largest
// staged count of the batch).
void launch_batch_pen(const void* table, const int* b0, int nc, int dim, int rows, int W, int umax, const int* nb, cudaStream_t st)
{
    const BatchPen* cs = (const BatchPen*)table;
    const dim3 blk(rows, W);
    if (nb[0] > 0) {
        if (dim == 2) k_batch_pen_t<2><<<nb[0], blk, umax * 16, st>>>(cs, b0, nc);
        else k_batch_pen_t<3><<<nb[0], blk, umax * 24, st>>>(cs, b0, nc);
        MPH_COUNT_LAUNCH();
    }
    if (nb[1] > 0) {
        if (dim == 2) k_batch_pen_y<2><<<nb[1], blk, umax * 16, st>>>(cs, b0 + (nc + 1), nc);
        else k_batch_pen_y<3><<<nb[1], blk, umax * 16, st>>>(cs, b0 + (nc + 1), nc);
        MPH_COUNT_LAUNCH();
    }
    if (nb[2] > 0) { k_batch_pen_vec<<<nb[2], kReduceThreads, 0, st>>>(cs, b0 + 2 * (nc + 1), nc); MPH_COUNT_LAUNCH(); }
}
void launch_batch_flags(const void* table, int nc, int* out, cudaStream_t st)
{
    { k_batch_flags<<<grid_for((long long)nc * kFlagCount, 256), 256, 0, st>>>((const BatchPen*)table, nc, out); MPH_COUNT_LAUNCH(); }
}

}  // namespace mph
