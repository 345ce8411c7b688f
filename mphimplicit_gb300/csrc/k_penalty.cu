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
// raised to that bound where the fluid is more viscous).
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
// Positions are fixed point in units of RadiusP / 2^22: their differences are
// exact (C_ik = -C_ki to the bit), good to 2^-22 of RadiusP, and become floats
// by an addition to the bits of 1.5 2^23 (integer-to-float conversions run on
// the quarter-rate pipe of the reciprocal square root).
//
// On 1,297,696 particles an application takes 98 us (k_pen_t 51, k_pen_y 47;
// the viscous pairs and stored records: 398) and the vectors 22 us in one
// kernel (43 in two), with 142 CR iterations where there were 140.
//
// A block of rows stages its distinct neighbours (position with s, or with
// lambda t) in shared memory; a block with too many of them gathers by the
// P-list's own columns.  Both evaluate pen_coef in the same order, so they
// give the same bits.
#include <algorithm>
#include <climits>
#include <mutex>
#include <type_traits>

#include "mph_device.cuh"
#include "mph_solver.cuh"

namespace mph {

constexpr int kSIn0 = 16, kSIn = 17, kSTol2 = 23;         // as in k_mixed.cu
constexpr int kSAlpha = 25, kSBeta = 26, kSQUPrev = 27;   // this iteration's alpha and beta, (q, D^-1 q) of the last one
__device__ __forceinline__ int rho_slot32(int it) { return 20 + (it & 1); }

constexpr int kPlWords = 1 << 13;   // bitmap of a row block's columns: 2^18 particles, fluid and wall window together
constexpr int kMaxPenRows = 256;   // threads of a row block (rows times threads a row)
// Staged neighbours a block of `rows` rows has room for.  Blocks of a
// 3.5-spacing cell order have about 2.8 (256 rows) to 3.9 (64) times their
// rows of them, against some 20 slots a row; one with more (a solve of 211
// blocks of 599 on average: 9.12 ms staged, 9.34 gathered) gains little.
static int pen_ucap(int rows) { return 4 * rows + 128; }

template <int D>
__global__ void k_fixed_positions(DevParams P, const int* __restrict__ type, const double* __restrict__ pos, int4* __restrict__ ipos)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    double x[3];
    load_vec<D>(pos, i, x);
    int u[3] = {0, 0, 0};
#pragma unroll
    for (int d = 0; d < D; ++d) u[d] = __double2int_rn((x[d] - P.dmin[d]) * P.fix_scale);
    ipos[i] = make_int4(u[0], u[1], u[2], type[i]);
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
__global__ void __launch_bounds__(kMaxPenRows) k_plist_ranks(int N, int Nf, int pw4, int ucap, const int* __restrict__ ncp,
                                                             const long long* __restrict__ nptrP, const int* __restrict__ nindP,
                                                             uint2* __restrict__ idx, int* __restrict__ groups,
                                                             int* __restrict__ uniq, int* __restrict__ ucount)
{
    extern __shared__ unsigned pl_smem[];
    unsigned* bm = pl_smem;
    unsigned* rank = pl_smem + kPlWords;
    __shared__ int red[4][32];
    __shared__ unsigned wsum[32];
    const int tid = threadIdx.x, lane = tid & 31, wl = tid >> 5, nwl = blockDim.x >> 5;
    const int i = blockIdx.x * blockDim.x + tid;
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

// q = x_j - x_i in the positions' units and cf = 1 / |q| - 1 / RadiusP (0
// beyond RadiusP), so that C_ij = kfp (2 / RadiusP) cf q.  um = u_i - kMagic.
// |q| = 0 (the row itself, coincident particles) gives a finite cf, and zero
// with its q.  WRAP: some pair of the step is a periodic image.
constexpr int kMagic = 0x4b400000;   // 1.5 2^23: adding d, |d| <= 2^22, gives the float 1.5 2^23 + d
template <int D, bool WRAP>
__device__ __forceinline__ float pen_coef(const DevParams& P, const int* um, const int* uj, float* q)
{
#pragma unroll
    for (int d = 0; d < D; ++d) {
        int v = uj[d] - um[d];
        if (WRAP) {
            const int w = v - kMagic;
            v += w > P.fix_h[d] ? -P.fix_w[d] : (w < -P.fix_h[d] ? P.fix_w[d] : 0);
        }
        q[d] = __fadd_rn(__int_as_float(v), -12582912.f);
    }
    float r2 = __fmul_rn(q[0], q[0]);
    r2 = __fmaf_rn(q[1], q[1], r2);
    if (D == 3) r2 = __fmaf_rn(q[2], q[2], r2);
    float inv;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(fmaxf(r2, 1.f)));
    return fmaxf(__fadd_rn(inv, -P.fix_inv), 0.f);
}

struct PenArgs {
    int N, Nf, pw4, ucap, umax, cap;
    const int4* ipos;
    const int* wrap;
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

// What a thread has in flight before its block's neighbours are staged: the
// first columns it stages and the first words of its row.  Their loads do not
// wait for the block's count or the row's length (both buffers have room for
// every index read here); what lies beyond is not used.  A block's time is
// this chain of loads, so nothing in it waits that need not.
constexpr int kPreCols = 3, kPreWords = 4;
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
    const int done = A.flags[kFlagDone], wrap = *A.wrap;
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
    const int um[3] = {pi.x - kMagic, pi.y - kMagic, pi.z - kMagic};
    auto sum = [&](auto WR) {
        auto one = [&](const int* uj, const float* sj) {
            float q[3];
            const float cf = pen_coef<D, decltype(WR)::value>(P, um, uj, q);
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
    };
    if (R.n > 0) {
        if (wrap) sum(std::true_type());
        else sum(std::false_type());
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

// Sums over the block of three FP32 values a thread: FP32 within a warp, FP64
// across the warps, as block_sum.
__device__ __forceinline__ void block_sum3(float (&v)[3], double (&out)[3])
{
    __shared__ double ws[3][32];
    const int tid = threadIdx.y * blockDim.x + threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int nw = (blockDim.x * blockDim.y + 31) >> 5;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[c] += __shfl_down_sync(0xffffffffu, v[c], o);
        if (lane == 0) ws[c][wid] = (double)v[c];
    }
    __syncthreads();
    if (wid == 0) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            double d = lane < nw ? ws[c][lane] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) d += __shfl_down_sync(0xffffffffu, d, o);
            out[c] = d;
        }
    }
    __syncthreads();
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
    const int done = A.flags[kFlagDone], it = A.flags[kFlagIter], wrap = *A.wrap;
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
        const int um[3] = {pi.x - kMagic, pi.y - kMagic, pi.z - kMagic};
        auto sum = [&](auto WR) {
            auto one = [&](const int* uj, float tj) {
                float q[3];
                const float c = __fmul_rn(pen_coef<D, decltype(WR)::value>(P, um, uj, q), __fadd_rn(tj, ti));
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
        };
        if (R.n > 0) {
            if (wrap) sum(std::true_type());
            else sum(std::false_type());
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
    double b[3];
    block_sum3(v, b);
    __shared__ bool last;
    if (tid == 0) {
#pragma unroll
        for (int c = 0; c < 3; ++c) A.partials[3 * (size_t)lb0 + c] = b[c];
        __threadfence();
        last = atomicAdd(A.counter, 1u) == (unsigned)nb - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double sum[3] = {0.0, 0.0, 0.0};
#pragma unroll 4
    for (int k = tid; k < nb; k += nth)
#pragma unroll
        for (int c = 0; c < 3; ++c) sum[c] += __ldcg(A.partials + 3 * (size_t)k + c);
    __shared__ double ws[3][32];
    const int lane = tid & 31, wid = tid >> 5, nwarp = (nth + 31) >> 5;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum[c] += __shfl_down_sync(0xffffffffu, sum[c], o);
        if (lane == 0) ws[c][wid] = sum[c];
    }
    __syncthreads();
    if (tid == 0) {
        double r[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            r[c] = ws[c][0];
            for (int w = 1; w < nwarp; ++w) r[c] += ws[c][w];
        }
        *A.counter = 0u;
        double beta = 0.0, qu = r[1];
        if (it > 0) {
            beta = r[0] / A.scal[rho_slot32(it - 1)];
            qu += beta * (2.0 * r[2] + beta * A.scal[kSQUPrev]);
        }
        A.scal[rho_slot32(it)] = r[0];
        A.scal[kSQUPrev] = qu;
        A.scal[kSBeta] = beta;
        A.scal[kSAlpha] = r[0] / qu;
    }
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
        ab[0] = (float)A.scal[kSAlpha];
        ab[1] = (float)A.scal[kSBeta];
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
    for (int k = lb * blockDim.x + threadIdx.x; k < n; k += nb * blockDim.x) {
        const float s = A.s[k], y = A.y[k], d = A.invD[k];
        const float p = it == 0 ? s : beta * A.p[k] + s;
        const float q = it == 0 ? y : beta * A.q[k] + y;
        A.p[k] = p;
        A.q[k] = q;
        A.z[k] += alpha * p;
        const float sn = s - alpha * (d * q);
        A.s[k] = sn;
        const float r = d != 0.f ? __fdividef(sn, d) : 0.f;
        acc += r * r;
    }
    const bool last = reduce_finalize_step(acc, A.partials, A.counter, A.scal + kSIn, A.flags + kFlagIter, lb, nb);
    if (last) {
        const double rr = A.scal[kSIn], rr0 = A.scal[kSIn0];
        const bool bad = !(rr == rr);
        const bool stop = it + 1 >= A.cap || rr / rr0 < A.scal[kSTol2] || bad;
        if (stop) {
            A.flags[kFlagDone] = 1;
            if (bad) A.flags[kFlagBad] = 1;
        }
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

// ---- host side ---------------------------------------------------------------------
constexpr int kPenBlocks = 152 * kPenResident;   // blocks of k_pen_y: what is resident at once

// Rows a block and threads a row.  A large case takes 256 rows a block (a
// row's share of the staged neighbours falls with the block: 5.2, 4.5 and 4.2
// times the rows of 128, 256 and 512); a small one fewer rows and four threads
// a row, so that its blocks reach every SM and a row's words are not one
// chain.
static void pen_shape(int N, int* rows, int* W)
{
    if (N > 152 * 512) { *rows = 256; *W = 1; }
    else if (N > 152 * 192) { *rows = 128; *W = 2; }
    else { *rows = 64; *W = 4; }
}

// The positions' unit is RadiusP / 2^20 or finer (domains up to about 1900
// RadiusP wide); in wider ones the stored operator's records are closer to C.
bool pen_applies(const mph_case* c) { return c->step_pairs && mixed_jacobi(c) && c->dp.fix_inv <= 1.0f / 1048576.0f; }

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

// Fixed-point positions and the P-lists' ranks of this step (after the
// neighbour stage; c->pmax is the longest P-list).
int launch_pen_lists(mph_case* c)
{
    DeviceState& d = c->d;
    const DevParams& P = c->dp;
    pen_shape(P.N, &c->pen_rows, &c->pen_w);
    c->pen_pw4 = (c->pmax + 3) / 4;
    const int nsl = (P.N + 31) / 32, nb = (int)grid_for(P.N, c->pen_rows), ucap = pen_ucap(c->pen_rows);
    if (!d.ipos) {
        MPH_CUDA(cudaMalloc((void**)&d.ipos, (size_t)P.N * sizeof(int4)));
        MPH_CUDA(cudaMalloc((void**)&d.pgroups, (size_t)nsl * sizeof(int)));
        MPH_CUDA(cudaMalloc((void**)&d.puniq, (size_t)nb * ucap * sizeof(int)));
        MPH_CUDA(cudaMalloc((void**)&d.pucount, (size_t)(nb + 4) * sizeof(int)));
    }
    if (!d.tct32) MPH_CUDA(cudaMalloc((void**)&d.tct32, (size_t)(P.N + 1) * sizeof(float)));
    MPH_TRY(grow_t(&d.pidx, &d.cap_pidx, (long long)nsl * c->pen_pw4 * 32));
    const unsigned g = grid_for(P.N, 256);
    if (c->dim == 2) { k_fixed_positions<2><<<g, 256, 0, c->stream>>>(P, d.type, d.pos, d.ipos); MPH_COUNT_LAUNCH(); }
    else { k_fixed_positions<3><<<g, 256, 0, c->stream>>>(P, d.type, d.pos, d.ipos); MPH_COUNT_LAUNCH(); }
    c->pen_umax = 0;
    c->loc_blocks[0] = 0;
    c->loc_blocks[1] = (int)grid_for(P.Nf, c->pen_rows);
    c->loc_cols = 0;
    c->loc_ct_blocks = 0;
    if (!c->inner_local) return MPH_OK;
    const size_t smem = 2 * kPlWords * sizeof(unsigned);
    static std::once_flag once;
    std::call_once(once, [smem] {   // fixed maxima: host threads of a batch would race on per-launch values
        cudaFuncSetAttribute(k_plist_ranks, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        const int t = (pen_ucap(kMaxPenRows) + 256) * 24, y = (pen_ucap(kMaxPenRows) + 256) * 16;
        cudaFuncSetAttribute(k_pen_t<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, t);
        cudaFuncSetAttribute(k_pen_t<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, t);
        cudaFuncSetAttribute(k_pen_y<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, y);
        cudaFuncSetAttribute(k_pen_y<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, y);
    });
    MPH_CUDA(cudaMemsetAsync(d.pucount + nb, 0, 4 * sizeof(int), c->stream));
    { k_plist_ranks<<<nb, c->pen_rows, smem, c->stream>>>(P.N, P.Nf, c->pen_pw4, ucap, d.ncp, d.nptrP, d.nindP, d.pidx, d.pgroups,
                                                         d.puniq, d.pucount); MPH_COUNT_LAUNCH(); }
    int h[4] = {};
    MPH_CUDA(cudaMemcpyAsync(h, d.pucount + nb, sizeof(h), cudaMemcpyDeviceToHost, c->stream));
    MPH_CUDA(cudaStreamSynchronize(c->stream));
    c->pen_umax = (h[0] + 127) / 128 * 128;   // rounded up: small changes keep the captured graphs
    c->loc_ct_blocks = h[1];
    c->loc_blocks[0] = h[2];
    c->loc_blocks[1] -= h[2];
    c->loc_cols = (long long)(unsigned)h[3];
    return MPH_OK;
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
    A.wrap = d.wrap32;
    A.idx = d.pidx;
    A.groups = d.pgroups;
    A.uniq = d.puniq;
    A.ucount = c->inner_local ? d.pucount : nullptr;
    A.ncp = d.ncp;
    A.nindP = d.nindP;
    A.nptrP = d.nptrP;
    A.z = d.v32 + n;
    A.s = d.v32 + 2 * n;
    A.y = d.v32 + 3 * n;
    A.p = d.v32 + 4 * n;
    A.q = d.v32 + 5 * n;
    A.invD = d.v32 + 7 * n;
    A.t = d.tct32;
    A.scal = d.scal;
    A.flags = d.flags;
    A.partials = d.partials;
    A.counter = (unsigned*)(d.flags + kFlagCounter);
    return A;
}

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
    const unsigned rb = std::min<int>(grid_for(n, kReduceThreads), kReduceBlocks);
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
    B.v_nb = nb[2] = std::min<int>(grid_for(B.n, kReduceThreads), kReduceBlocks);
}

// One CR iteration of the cases that still iterate (b0: the block starts of
// the three launches, nc + 1 each; nb: their block totals; umax: the largest
// staged count of the batch).
void launch_batch_pen(const void* table, const int* b0, int nc, int dim, int rows, int W, int umax, const int* nb, cudaStream_t st)
{
    static std::once_flag once;
    std::call_once(once, [] {
        const int t = (pen_ucap(kMaxPenRows) + 256) * 24, y = (pen_ucap(kMaxPenRows) + 256) * 16;
        cudaFuncSetAttribute(k_batch_pen_t<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, t);
        cudaFuncSetAttribute(k_batch_pen_t<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, t);
        cudaFuncSetAttribute(k_batch_pen_y<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, y);
        cudaFuncSetAttribute(k_batch_pen_y<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, y);
    });
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
