// k_particles.cu - particle motion and the cell list.
//
//   step_begin      : calculateConvection / calculateWall /
//                     calculatePeriodicBoundary / resetForce
//                     (main.cpp:1678, 2089, 4741, 1690), one pass per particle
//   cell keys       : main.cpp:1171-1186
//   bitonic network : the reference's compare-exchange network
//                     (main.cpp:1190-1211), stage by stage, with every stage
//                     whose partner distance is inside a tile run in shared
//                     memory; it reproduces the reference's permutation
//                     (the network is not stable, so a stable sort would not)
//   bucket ranges   : main.cpp:1213-1311 as one boundary scatter
//   permute         : main.cpp:1316-1378 as one SoA gather (+ the FP32
//                     position copy used by the neighbour pre-classification)
#include <algorithm>

#include "mph_device.cuh"

namespace mph {

struct WallMotion {
    double c[4][3], v[4][3], w[4][3], R[4][3][3];
};

template <int D>
__global__ void k_step_begin(DevParams P, WallMotion W, double* __restrict__ pos, double* __restrict__ vel,
                             double* __restrict__ force, int fB, int fE, int wB, int wE,
                             const int* __restrict__ type)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.N) return;
    double x[3], v[3];
    load_vec<D>(pos, i, x);
    load_vec<D>(vel, i, v);
    if (i >= fB && i < fE) {                                   // calculateConvection
#pragma unroll
        for (int d = 0; d < D; ++d) x[d] = DADD(x[d], DMUL(v[d], P.dt));
    } else if (i >= wB && i < wE) {                            // calculateWall
        const int t = type[i];
        double r[3];
#pragma unroll
        for (int d = 0; d < D; ++d) r[d] = DSUB(x[d], W.c[t][d]);
        const double (&R)[3][3] = W.R[t];
        const double* w = W.w[t];
        if (D == 3) {
            // rotated in place, component by component (main.cpp:2108-2110)
            r[0] = DADD(DADD(DMUL(R[0][0], r[0]), DMUL(R[0][1], r[1])), DMUL(R[0][2], r[2]));
            r[1] = DADD(DADD(DMUL(R[1][0], r[0]), DMUL(R[1][1], r[1])), DMUL(R[1][2], r[2]));
            r[2] = DADD(DADD(DMUL(R[2][0], r[0]), DMUL(R[2][1], r[1])), DMUL(R[2][2], r[2]));
            v[0] = DADD(DSUB(DMUL(w[1], r[2]), DMUL(w[2], r[1])), W.v[t][0]);
            v[1] = DADD(DSUB(DMUL(w[2], r[0]), DMUL(w[0], r[2])), W.v[t][1]);
            v[2] = DADD(DSUB(DMUL(w[0], r[1]), DMUL(w[1], r[0])), W.v[t][2]);
        } else {
            // 2D cases rotate about z only (checked at case creation), so the
            // z terms of the reference's expressions are exact zeros
            r[0] = DADD(DMUL(R[0][0], r[0]), DMUL(R[0][1], r[1]));
            r[1] = DADD(DMUL(R[1][0], r[0]), DMUL(R[1][1], r[1]));
            v[0] = DADD(-DMUL(w[2], r[1]), W.v[t][0]);
            v[1] = DADD(DMUL(w[2], r[0]), W.v[t][1]);
        }
#pragma unroll
        for (int d = 0; d < D; ++d) x[d] = DADD(DADD(r[d], W.c[t][d]), DMUL(W.v[t][d], P.dt));
        store_vec<D>(vel, i, v);
    }
#pragma unroll
    for (int d = 0; d < D; ++d) x[d] = DADD(mod_exact(DSUB(x[d], P.dmin[d]), P.dw[d]), P.dmin[d]);
    store_vec<D>(pos, i, x);
    const double z[3] = {0.0, 0.0, 0.0};
    store_vec<D>(force, i, z);
}

template <int D>
__global__ void k_cell_keys(DevParams P, const double* __restrict__ pos, const int* __restrict__ type,
                            int* __restrict__ key, int* __restrict__ perm, int* __restrict__ bbox, int* __restrict__ wrap)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 3) {   // what k_fluid_bbox and the assembly accumulate into
        bbox[i] = P.cc[i];
        bbox[3 + i] = 0;
        wrap[i] = 0;
        if (i == 0) bbox[8] = 0;
    }
    if (i >= P.nPow) return;
    if (i < P.N) {
        double x[3];
        load_vec<D>(pos, i, x);
        int c[3] = {0, 0, 0};
#pragma unroll
        for (int d = 0; d < D; ++d) c[d] = ((int)floor(DDIV(DSUB(x[d], P.dmin[d]), P.cw[d]))) % P.cc[d];
        key[i] = cell_id(P, c[0], c[1], c[2]) + (is_wall(type[i]) ? P.T : 0);
        perm[i] = i;
    } else {
        key[i] = 2 * P.T;
        perm[i] = P.N;
    }
}

// ---- bitonic network -------------------------------------------------------
// The reference's network, stage by stage: stage (m, dist) compares i and
// i | dist for every i without bit log2(dist), ascending where bit m + 1 of i
// is clear, and moves (key, index) pairs by their keys alone.  The stages of
// distance below a tile run in shared memory, a pair one 8-byte word, in
// passes of up to four: a thread takes the 16 elements that differ in the
// pass's four index bits, runs its four stages in registers and puts them
// back, so a pass costs one trip through shared memory and one barrier where
// a stage of two 4-byte arrays each had one.  The stages above a tile run
// three a launch in the same way, through global memory.  The whole cell-sort
// stage on 1.3 million particles 0.90 -> 0.55 ms, on 22,000 0.165 -> 0.11.
// Tiles of 2^12: 2^11, 2^13 and 2^14 took 0.121, 0.113 and 0.128 ms on 22,000
// (a tile is one block: larger ones leave SMs idle), 0.58, 0.57 and 0.52 on
// 1.3 million.
constexpr int kTileExp = 12;
constexpr int kTile = 1 << kTileExp;
constexpr int kTileThreads = kTile / 16;

__device__ __forceinline__ void pair_swap(unsigned long long& a, unsigned long long& b, bool asc)
{
    const bool sw = ((int)(a >> 32) > (int)(b >> 32)) == asc;
    const unsigned long long t = sw ? b : a;
    b = sw ? a : b;
    a = t;
}

// S stages of row m with distances 2^e, 2^(e-1), ... on the 2^S elements at
// base + j 2^(e-S+1), j = 0 .. 2^S - 1 (their position in the whole array
// decides the direction; bit m + 1 lies above every distance of the row)
template <int S>
__device__ __forceinline__ void pair_stages(unsigned long long* v, bool asc)
{
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const int d = 1 << (S - 1 - s);
#pragma unroll
        for (int j = 0; j < (1 << S); ++j)
            if (!(j & d)) pair_swap(v[j], v[j | d], asc);
    }
}

// base index of thread group t's elements: t with S zero bits inserted at bit lo
__device__ __forceinline__ int spread_bits(int t, int lo, int S) { return ((t >> lo) << (lo + S)) | (t & ((1 << lo) - 1)); }

// a word of padding every 16: the passes of small distances read 16 words in a
// row per thread, which without it all fall on the same banks
__device__ __forceinline__ int tile_at(int i) { return i + (i >> 4); }

template <int S>
__device__ __forceinline__ void tile_pass(unsigned long long* sh, int tile, int base, int m, int e)
{
    const int lo = e - S + 1;
    for (int t = threadIdx.x; t < (tile >> S); t += blockDim.x) {
        const int i = spread_bits(t, lo, S);
        unsigned long long v[1 << S];
#pragma unroll
        for (int j = 0; j < (1 << S); ++j) v[j] = sh[tile_at(i + (j << lo))];
        pair_stages<S>(v, (((base + i) >> m) & 2) == 0);
#pragma unroll
        for (int j = 0; j < (1 << S); ++j) sh[tile_at(i + (j << lo))] = v[j];
    }
    __syncthreads();
}

// Rows m0 .. m1 on one tile; row m runs its distances below the tile.
__global__ void __launch_bounds__(kTileThreads) k_bitonic_tile(int* __restrict__ key, int* __restrict__ perm, int tile, int tile_exp,
                                                               int m0, int m1)
{
    extern __shared__ unsigned long long tile_smem[];
    const int base = blockIdx.x * tile;
    for (int t = threadIdx.x; t < tile; t += blockDim.x)
        tile_smem[tile_at(t)] = ((unsigned long long)(unsigned)key[base + t] << 32) | (unsigned)perm[base + t];
    __syncthreads();
    for (int m = m0; m <= m1; ++m) {
        int e = min(m, tile_exp - 1);   // the row's largest distance inside the tile
        for (; e >= 3; e -= 4) tile_pass<4>(tile_smem, tile, base, m, e);
        if (e == 2) tile_pass<3>(tile_smem, tile, base, m, 2);
        else if (e == 1) tile_pass<2>(tile_smem, tile, base, m, 1);
        else if (e == 0) tile_pass<1>(tile_smem, tile, base, m, 0);
    }
    for (int t = threadIdx.x; t < tile; t += blockDim.x) {
        const unsigned long long v = tile_smem[tile_at(t)];
        key[base + t] = (int)(v >> 32);
        perm[base + t] = (int)(unsigned)v;
    }
}

// S stages of row m from distance 2^e down, in global memory
template <int S>
__global__ void __launch_bounds__(256) k_bitonic_global(int* __restrict__ key, int* __restrict__ perm, int groups, int m, int e)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= groups) return;
    const int lo = e - S + 1, i = spread_bits(t, lo, S);
    unsigned long long v[1 << S];
#pragma unroll
    for (int j = 0; j < (1 << S); ++j)
        v[j] = ((unsigned long long)(unsigned)key[i + (j << lo)] << 32) | (unsigned)perm[i + (j << lo)];
    pair_stages<S>(v, ((i >> m) & 2) == 0);
#pragma unroll
    for (int j = 0; j < (1 << S); ++j) {
        key[i + (j << lo)] = (int)(v[j] >> 32);
        perm[i + (j << lo)] = (int)(unsigned)v[j];
    }
}

// ---- counting sort (option cell_sort 1) ------------------------------------
// The production cell sort: the keys are cell indices in [0, 2T), so one
// counting pass sorts them.  A warp-aggregated histogram (lanes with equal
// keys, found with __match_any_sync, add their count once), the bucket
// offsets from the device scan (warp-level inclusive scans within a block),
// a warp-aggregated scatter, and last each bucket ordered by the particles'
// previous positions, so the permutation does not depend on the order in
// which the scatter's atomics were served: a stable sort.  Unlike the
// reference's bitonic network (main.cpp:1190-1211, not stable) it gives a
// different order inside a cell; cell ranges and per-cell particle sets are
// the same.
__global__ void k_count_keys(int N, const int* __restrict__ key, int* __restrict__ cnt)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const bool valid = i < N;
    const int k = valid ? key[i] : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, k);
    if (valid && lane == __ffs(peers) - 1) atomicAdd(cnt + k, __popc(peers));
}

__global__ void k_scatter_keys(int N, const int* __restrict__ key, const long long* __restrict__ off, int* __restrict__ cursor,
                               int* __restrict__ perm)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const bool valid = i < N;
    const int k = valid ? key[i] : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, k);
    const int leader = __ffs(peers) - 1;
    int base = 0;
    if (valid && lane == leader) base = atomicAdd(cursor + k, __popc(peers));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (valid) perm[off[k] + base + __popc(peers & ((1u << lane) - 1u))] = i;
}

// thread per bucket: its particles ordered by previous position (insertion
// sort: a bucket is one cell's fluid or wall particles), the sorted keys and
// the bucket starts
__global__ void k_bucket_order(int nb, const long long* __restrict__ off, int* __restrict__ key, int* __restrict__ perm,
                               int* __restrict__ bucket)
{
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    const long long s = off[b], e = off[b + 1];
    for (long long j = s + 1; j < e; ++j) {
        const int v = perm[j];
        long long k = j - 1;
        while (k >= s && perm[k] > v) {
            perm[k + 1] = perm[k];
            --k;
        }
        perm[k + 1] = v;
    }
    for (long long j = s; j < e; ++j) key[j] = b;
    bucket[b] = (int)s;
    if (b == nb - 1) bucket[nb] = (int)e;
}

// ---- bucket starts, permutation -------------------------------------------
// bucket[b] = first sorted position whose key >= b, b in [0, 2T].  A run of
// empty cells (the free space of a dam: tens of thousands) is filled by the
// warp together; by the one thread at its edge it took 171 us of a 5.7 ms
// step on 412,000 particles in 2-D.
__global__ void k_bucket_starts(const int* __restrict__ key, int N, int T, int* __restrict__ bucket)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    int lo = 1, hi = 0;
    if (i <= N) {
        lo = (i == 0) ? 0 : key[i - 1] + 1;
        hi = (i == N) ? 2 * T : key[i];
    }
    const bool wide = hi - lo >= 4;
    if (!wide)
        for (int b = lo; b <= hi; ++b) bucket[b] = i;
    for (unsigned m = __ballot_sync(0xffffffffu, wide); m; m &= m - 1) {
        const int src = __ffs(m) - 1;
        const int l = __shfl_sync(0xffffffffu, lo, src), h = __shfl_sync(0xffffffffu, hi, src), v = __shfl_sync(0xffffffffu, i, src);
        for (int b = l + lane; b <= h; b += 32) bucket[b] = v;
    }
}

template <int D>
__global__ void k_permute(int N, const int* __restrict__ perm, const int* __restrict__ id, const int* __restrict__ type,
                          const double* __restrict__ pos, const double* __restrict__ vel, int* __restrict__ id2,
                          int* __restrict__ type2, double* __restrict__ pos2, double* __restrict__ vel2,
                          float* __restrict__ pos32, float* __restrict__ poslo32, float4* __restrict__ pt2,
                          const double* __restrict__ prev, double* __restrict__ prev2, int history)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const int s = perm[i];
    id2[i] = id[s];
    type2[i] = type[s];
    double x[3], v[3];
    load_vec<D>(pos, s, x);
    load_vec<D>(vel, s, v);
    store_vec<D>(pos2, i, x);
    store_vec<D>(vel2, i, v);
    for (int h = 0; h < history; ++h) {   // the start velocities of the last steps follow the particles
        double a[3];
        load_vec<D>(prev + (size_t)h * N * VS<D>::v, s, a);
        store_vec<D>(prev2 + (size_t)h * N * VS<D>::v, i, a);
    }
    float h[3] = {0.f, 0.f, 0.f}, l[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int d = 0; d < D; ++d) {
        h[d] = (float)x[d];
        l[d] = (float)(x[d] - (double)h[d]);   // exact difference, rounded once
    }
    if (D == 2) {
        reinterpret_cast<float2*>(pos32)[i] = make_float2(h[0], h[1]);
        reinterpret_cast<float2*>(poslo32)[i] = make_float2(l[0], l[1]);
        pt2[i] = make_float4(h[0], h[1], 0.f, __int_as_float(type[s]));
    } else {
        // w: the type bits (read with the position by the pair-term operator)
        reinterpret_cast<float4*>(pos32)[i] = make_float4(h[0], h[1], h[2], __int_as_float(type[s]));
        reinterpret_cast<float4*>(poslo32)[i] = make_float4(l[0], l[1], l[2], 0.f);
    }
}

__global__ void k_fluid_bbox(const int* __restrict__ bucket, DevParams P, int* __restrict__ bbox)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c == 0) {   // the ends of the fluid and the wall particles, beside the box
        bbox[6] = bucket[P.T];
        bbox[7] = bucket[2 * P.T];
    }
    // and the most particles of a cell, fluid or wall
    const int most = c < P.T ? max(bucket[c + 1] - bucket[c], bucket[P.T + c + 1] - bucket[P.T + c]) : 0;
    const int warp_most = __reduce_max_sync(0xffffffffu, most);
    if ((threadIdx.x & 31) == 0 && warp_most > *(volatile int*)(bbox + 8)) atomicMax(bbox + 8, warp_most);
    if (c >= P.T) return;
    if (bucket[c + 1] - bucket[c] > 0) {
        const int p[3] = {(c / (P.cc[1] * P.cc[2])) % P.cc[0], (c / P.cc[2]) % P.cc[1], c % P.cc[2]};
        for (int d = 0; d < 3; ++d) {
            atomicMin(&bbox[d], p[d]);
            atomicMax(&bbox[3 + d], p[d]);
        }
    }
}

// ---- launchers -------------------------------------------------------------
void launch_step_begin(mph_case* c)
{
    WallMotion W;
    for (int t = 0; t < 4; ++t)
        for (int a = 0; a < 3; ++a) {
            W.c[t][a] = c->wallC[t][a];
            W.v[t][a] = c->wallV[t][a];
            W.w[t][a] = c->wallW[t][a];
            for (int b = 0; b < 3; ++b) W.R[t][a][b] = c->wallR[t][a][b];
        }
    const unsigned g = grid_for(c->dp.N, 256);
    if (c->dim == 2)
        { k_step_begin<2><<<g, 256, 0, c->stream>>>(c->dp, W, c->d.pos, c->d.vel, c->d.force, c->fB, c->fE, c->wB, c->wE, c->d.type); MPH_COUNT_LAUNCH(); }
    else
        { k_step_begin<3><<<g, 256, 0, c->stream>>>(c->dp, W, c->d.pos, c->d.vel, c->d.force, c->fB, c->fE, c->wB, c->wE, c->d.type); MPH_COUNT_LAUNCH(); }
}

void launch_cell_keys(mph_case* c)
{
    const unsigned g = grid_for(c->dp.nPow, 256);
    if (c->dim == 2) { k_cell_keys<2><<<g, 256, 0, c->stream>>>(c->dp, c->d.pos, c->d.type, c->d.key, c->d.perm, c->d.bbox, c->d.wrap32); MPH_COUNT_LAUNCH(); }
    else { k_cell_keys<3><<<g, 256, 0, c->stream>>>(c->dp, c->d.pos, c->d.type, c->d.key, c->d.perm, c->d.bbox, c->d.wrap32); MPH_COUNT_LAUNCH(); }
}

void launch_bitonic_sort(mph_case* c)
{
    const int n = c->dp.nPow, k = c->dp.powExp;
    if (k == 0) return;
    const int te = std::min(k, kTileExp), tile = 1 << te;
    const size_t smem = (size_t)(tile + tile / 16) * sizeof(unsigned long long);
    const int threads = std::max(32, std::min(kTileThreads, tile / 16));
    cudaStream_t st = c->stream;
    int *key = c->d.key, *perm = c->d.perm;
    // every row below the tile's exponent stays inside a tile
    { k_bitonic_tile<<<n / tile, threads, smem, st>>>(key, perm, tile, te, 0, te - 1); MPH_COUNT_LAUNCH(); }
    for (int m = te; m < k; ++m) {
        int e = m;
        while (e >= te) {
            const int s = std::min(3, e - te + 1);
            const int g = n >> s;
            if (s == 3) k_bitonic_global<3><<<grid_for(g, 256), 256, 0, st>>>(key, perm, g, m, e);
            else if (s == 2) k_bitonic_global<2><<<grid_for(g, 256), 256, 0, st>>>(key, perm, g, m, e);
            else k_bitonic_global<1><<<grid_for(g, 256), 256, 0, st>>>(key, perm, g, m, e);
            MPH_COUNT_LAUNCH();
            e -= s;
        }
        { k_bitonic_tile<<<n / tile, threads, smem, st>>>(key, perm, tile, te, m, m); MPH_COUNT_LAUNCH(); }
    }
}

int launch_counting_sort(mph_case* c)
{
    const int N = c->dp.N, nb = 2 * c->dp.T;
    DeviceState& d = c->d;
    if (!d.sort_cnt) {
        MPH_CUDA(cudaMalloc((void**)&d.sort_cnt, (size_t)(nb + 1) * sizeof(int)));
        MPH_CUDA(cudaMalloc((void**)&d.sort_off, (size_t)(nb + 1) * sizeof(long long)));
    }
    const unsigned g = grid_for(N, 256);
    MPH_CUDA(cudaMemsetAsync(d.sort_cnt, 0, (size_t)(nb + 1) * sizeof(int), c->stream));
    { k_count_keys<<<g, 256, 0, c->stream>>>(N, d.key, d.sort_cnt); MPH_COUNT_LAUNCH(); }
    MPH_TRY(launch_scan_i32_to_i64(c, d.sort_cnt, d.sort_off, nb));
    MPH_CUDA(cudaMemsetAsync(d.sort_cnt, 0, (size_t)(nb + 1) * sizeof(int), c->stream));
    { k_scatter_keys<<<g, 256, 0, c->stream>>>(N, d.key, d.sort_off, d.sort_cnt, d.perm); MPH_COUNT_LAUNCH(); }
    { k_bucket_order<<<grid_for(nb, 128), 128, 0, c->stream>>>(nb, d.sort_off, d.key, d.perm, d.bucket); MPH_COUNT_LAUNCH(); }
    return MPH_OK;
}

void launch_cell_ranges_and_permute(mph_case* c)
{
    const int N = c->dp.N;
    if (!c->cell_sort)   // the counting sort wrote the bucket starts already
        { k_bucket_starts<<<grid_for(N + 1, 256), 256, 0, c->stream>>>(c->d.key, N, c->dp.T, c->d.bucket); MPH_COUNT_LAUNCH(); }
    const unsigned g = grid_for(N, 256);
    DeviceState& d = c->d;
    const int history = d.vprev ? c->prev_valid : 0;
    if (c->dim == 2)
        { k_permute<2><<<g, 256, 0, c->stream>>>(N, d.perm, d.id, d.type, d.pos, d.vel, d.id_alt, d.type_alt, d.pos_alt, d.vel_alt, d.pos32,
                                                d.poslo32, d.pt32, d.vprev, d.vprev_alt, history); MPH_COUNT_LAUNCH(); }
    else
        { k_permute<3><<<g, 256, 0, c->stream>>>(N, d.perm, d.id, d.type, d.pos, d.vel, d.id_alt, d.type_alt, d.pos_alt, d.vel_alt, d.pos32,
                                                d.poslo32, nullptr, d.vprev, d.vprev_alt, history); MPH_COUNT_LAUNCH(); }
    std::swap(d.id, d.id_alt);
    std::swap(d.type, d.type_alt);
    std::swap(d.pos, d.pos_alt);
    std::swap(d.vel, d.vel_alt);
    if (history) std::swap(d.vprev, d.vprev_alt);
}

void launch_fluid_bbox(mph_case* c)
{
    { k_fluid_bbox<<<grid_for(c->dp.T, 256), 256, 0, c->stream>>>(c->d.bucket, c->dp, c->d.bbox); MPH_COUNT_LAUNCH(); }
}

}  // namespace mph
