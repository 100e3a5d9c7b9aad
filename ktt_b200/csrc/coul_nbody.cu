// coul_nbody.cu -- one leapfrog-style step of the direct N-body sum, the sibling of the Coulomb map
// that KTT tunes in Examples/Nbody (Nbody.cu:103-410 tuned kernel, NbodyReference.cu:36-75 reference).
//
// For every body i (position p_i, mass m_i, velocity v_i):
//     a_i = sum_j m_j d_ij / (|d_ij|^2 + eps^2)^(3/2),  d_ij = p_j - p_i   (j = i included: d = 0)
//     p_i' = p_i + dt v_i + damping dt^2 a_i,   v_i' = v_i + dt a_i,   w components: mass kept, 0
// The pair is the Coulomb pair with a softening term and a vector accumulator: one MUFU rsqrt and
// 12 FP32 operations (3 differences, 3 FMAs for r^2 + eps^2, 1/r^2, m/r, m/r^3, 3 FMAs into a).
// The FP32 pipe bounds it (F / 12 pairs/s), so all rsqrts stay on MUFU and the FP32 work runs as
// packed FFMA2/FMUL2/FADD2 on two bodies j per instruction.  A step without a configuration evaluates a
// pair once for both bodies from 4,096 bodies on (nbody_pair_kernel, 8.5 operations an interaction):
// 131,072 bodies in 5.17 ms = 3.32e12 interactions/s, against 8.51 ms by the configurable kernel's default and 6.99
// by its best configuration; the error of the accelerations falls from 2.7e-6 to 7e-8 with the shorter sums.
//
// Layout: each thread owns `BP` bodies i (strided by the block size so loads and stores coalesce) in
// registers; the bodies j stream through the CTA's TMA ring of 256-body float4 stages (the forward
// kernel's ring: one elected thread issues cp.async.bulk, mbarrier expect-tx, bounded waits), each
// stage is transposed once into x/y/z/m arrays, and every thread reads the bodies (j, j + 1) as
// 8-byte shared-memory broadcasts that meet a body i, held as a splat pair, in one packed
// instruction -- so no per-pair register moves are needed to form the packed operands.  With j_split = S >= 2 a
// thread-block cluster of S CTAs shares one tile of bodies i, each CTA taking 1/S of the bodies j,
// and rank 0 adds the partial accelerations from the peers' shared memory in rank order before it
// integrates and stores (for body counts too small to fill 148 SMs one tile per CTA).
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "coul_internal.h"

namespace coul {

namespace {

struct NbodyParams {
    const float4* pos;  // x, y, z, mass
    const float4* vel;  // x, y, z, (unused)
    float4* pos_new;
    float4* vel_new;
    int64_t n;
    float dt, damping, eps2;
    int* status;
};

// Body i's step from its acceleration.
__device__ __forceinline__ void integrate(const NbodyParams& p, const int64_t i, const float (&a)[3])
{
    const float dt = p.dt;
    const float half = p.damping * dt * dt;
    const float4 b = p.pos[i];
    const float4 v = p.vel[i];
    p.pos_new[i] = make_float4(fmaf(half, a[0], fmaf(dt, v.x, b.x)), fmaf(half, a[1], fmaf(dt, v.y, b.y)),
                               fmaf(half, a[2], fmaf(dt, v.z, b.z)), b.w);
    p.vel_new[i] = make_float4(fmaf(dt, a[0], v.x), fmaf(dt, a[1], v.y), fmaf(dt, a[2], v.z), 0.0f);
}

constexpr int kNbodyMaxThreads = 512;
constexpr int kNbodyMaxPortableSplit = 8;
constexpr int kNbodyMaxSplit = 16;  // above 8 the B200's non-portable cluster sizes
// dynamic shared memory: the TMA ring, its barriers, the transposed stage, the split's partial sums
constexpr int kNbodySoaOffset = kStages * kTileAtoms * 16 + 16;
constexpr int kNbodyRedOffset = kNbodySoaOffset + kTileAtoms * 16;
static_assert(kStages * 8 <= 16 && kNbodySoaOffset % 16 == 0, "ring barriers fit before the transposed stage");

// the widest register blocks (8 bodies i, each with three splat positions and three pair accumulators)
// need more than the 128 registers a 512-thread block leaves per thread
constexpr int nbody_max_threads(int bp) { return bp >= 8 ? 256 : kNbodyMaxThreads; }

template <int BP, int UNR, bool SPLIT>
__global__ void __launch_bounds__(nbody_max_threads(BP), 1) nbody_kernel(const NbodyParams p)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char* tiles = smem_raw;  // TMA ring of float4 (x, y, z, m) stages
    uint64_t* full = reinterpret_cast<uint64_t*>(smem_raw + kStages * kTileAtoms * 16);
    float* soa = reinterpret_cast<float*>(smem_raw + kNbodySoaOffset);  // x[256] y[256] z[256] m[256]
    const int tid = threadIdx.x;
    const int nthreads = blockDim.x;

    uint32_t S = 1, rank = 0;
    int tile = blockIdx.x;
    if constexpr (SPLIT) {
        S = cluster_size();
        rank = cluster_rank();
        tile = static_cast<int>(blockIdx.x / S);
    }

    // bodies i of this thread: tile * (nthreads * BP) + tid + k * nthreads, each held as a splat pair
    // (-x_i, -x_i) that meets the bodies (j, j + 1) in one packed instruction; the accumulators keep
    // the even-j and odd-j partial sums in their two lanes
    const int64_t ibase = static_cast<int64_t>(tile) * nthreads * BP + tid;
    float2 nx[BP], ny[BP], nz[BP], ax[BP], ay[BP], az[BP];
#pragma unroll
    for (int k = 0; k < BP; ++k) {
        const int64_t i = ibase + static_cast<int64_t>(k) * nthreads;
        const float4 b = i < p.n ? p.pos[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        nx[k] = splat(-b.x);
        ny[k] = splat(-b.y);
        nz[k] = splat(-b.z);
        ax[k] = ay[k] = az[k] = make_float2(0.0f, 0.0f);
    }
    const float2 eps2 = splat(p.eps2);

    // this CTA's share of the bodies j
    const int64_t chunk = (p.n + S - 1) / S;
    const int64_t jbegin = chunk * rank < p.n ? chunk * rank : p.n;
    const int64_t jcount = (p.n - jbegin) < chunk ? (p.n - jbegin) : chunk;
    const float4* src = p.pos + jbegin;
    const int64_t nst = (jcount + kTileAtoms - 1) / kTileAtoms;

    if (tid == 0) {
#pragma unroll
        for (int s = 0; s < kStages; ++s)
            mbar_init(&full[s], 1);
        fence_mbar_init();
    }
    __syncthreads();

    auto stage_count = [&](int64_t s) -> int {
        const int64_t rem = jcount - s * kTileAtoms;
        return static_cast<int>(rem < kTileAtoms ? rem : kTileAtoms);
    };
    auto issue = [&](int64_t s) {
        const int buf = static_cast<int>(s % kStages);
        const uint32_t bytes = static_cast<uint32_t>(stage_count(s)) * 16u;
        mbar_arrive_expect_tx(&full[buf], bytes);
        bulk_copy_g2s(tiles + buf * kTileAtoms * 16, src + s * kTileAtoms, bytes, &full[buf]);
    };
    if (tid == 0) {
        for (int64_t s = 0; s < nst && s < kStages; ++s)
            issue(s);
    }

    bool ok = true;
    for (int64_t s = 0; s < nst; ++s) {
        const int buf = static_cast<int>(s % kStages);
        const uint32_t parity = static_cast<uint32_t>((s / kStages) & 1);
        const bool arrived = mbar_wait_bounded(&full[buf], parity);
        if (__syncthreads_or(arrived ? 0 : 1)) {
            if (tid == 0) {
                report_status(p.status, kStatusTimeout);
                for (int64_t r = s; r < nst && r < s + kStages; ++r)
                    (void)mbar_wait_bounded(&full[r % kStages], static_cast<uint32_t>((r / kStages) & 1));
            }
            ok = false;
            break;
        }
        // Transpose the stage into four arrays (so a pair of bodies j is one 8-byte broadcast load);
        // the ragged last stage is padded with far-away massless bodies, so the loop needs no bound.
        const int cnt = stage_count(s);
        const float4* tile4 = reinterpret_cast<const float4*>(tiles + buf * kTileAtoms * 16);
        for (int j = tid; j < kTileAtoms; j += nthreads) {
            const float4 b = j < cnt ? tile4[j] : make_float4(kPadCoord, kPadCoord, kPadCoord, 0.0f);
            soa[0 * kTileAtoms + j] = b.x;
            soa[1 * kTileAtoms + j] = b.y;
            soa[2 * kTileAtoms + j] = b.z;
            soa[3 * kTileAtoms + j] = b.w;
        }
        // the TMA stage is free again: order the reads before its refill, which overlaps the math
        fence_proxy_async_smem();
        __syncthreads();
        if (tid == 0 && s + kStages < nst)
            issue(s + kStages);
        const float2* sx = reinterpret_cast<const float2*>(soa);
        const float2* sy = reinterpret_cast<const float2*>(soa + kTileAtoms);
        const float2* sz = reinterpret_cast<const float2*>(soa + 2 * kTileAtoms);
        const float2* sm = reinterpret_cast<const float2*>(soa + 3 * kTileAtoms);
#pragma unroll UNR
        for (int j = 0; j < kTileAtoms / 2; ++j) {
            const float2 bx = sx[j], by = sy[j], bz = sz[j], bm = sm[j];
#pragma unroll
            for (int k = 0; k < BP; ++k) {
                const float2 dx = __fadd2_rn(bx, nx[k]);
                const float2 dy = __fadd2_rn(by, ny[k]);
                const float2 dz = __fadd2_rn(bz, nz[k]);
                const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, eps2)));
                const float2 inv = make_float2(rsqrt_mufu(r2.x), rsqrt_mufu(r2.y));
                const float2 f = __fmul2_rn(__fmul2_rn(bm, inv), __fmul2_rn(inv, inv));
                ax[k] = __ffma2_rn(dx, f, ax[k]);
                ay[k] = __ffma2_rn(dy, f, ay[k]);
                az[k] = __ffma2_rn(dz, f, az[k]);
            }
        }
        __syncthreads();  // the four arrays are rewritten by the next stage
    }

    float a[BP][3];
#pragma unroll
    for (int k = 0; k < BP; ++k) {
        a[k][0] = ax[k].x + ax[k].y;
        a[k][1] = ay[k].x + ay[k].y;
        a[k][2] = az[k].x + az[k].y;
    }

    if constexpr (SPLIT) {
        // partial accelerations of the cluster, added by rank 0 in rank order
        float* red = reinterpret_cast<float*>(smem_raw + kNbodyRedOffset);
#pragma unroll
        for (int k = 0; k < BP; ++k)
#pragma unroll
            for (int c = 0; c < 3; ++c)
                red[(3 * k + c) * nthreads + tid] = a[k][c];
        cluster_sync();
        if (rank == 0) {
            for (uint32_t peer = 1; peer < S; ++peer) {
                const uint32_t base = cluster_map(red, peer);
#pragma unroll
                for (int k = 0; k < BP; ++k)
#pragma unroll
                    for (int c = 0; c < 3; ++c)
                        a[k][c] += ld_cluster_f32(base + 4u * static_cast<uint32_t>((3 * k + c) * nthreads + tid));
            }
        }
        cluster_sync();  // the peers' shared memory stays valid until rank 0 has read it
        if (rank != 0)
            return;
    }
    if (!ok)
        return;

#pragma unroll
    for (int k = 0; k < BP; ++k) {
        const int64_t i = ibase + static_cast<int64_t>(k) * nthreads;
        if (i < p.n)
            integrate(p, i, a[k]);
    }
}

// The step of a call that names no configuration.  A CTA takes 128 bodies i, four per lane, and its
// eight warps split the bodies j evenly, as do the CTAs of a cluster where there are few tiles (the
// configurable kernel's default, 512 bodies i a CTA and every j in turn, leaves 256 CTAs for 148 SMs at
// 131,072 bodies and 10 at 5,000).  A warp needs no other until the end: its lanes load 32 bodies j into
// registers while it evaluates the 32 before from its own shared memory, kept as pairs (x, x', y, y')
// (z, z', m, m') that two 16-byte broadcasts hand to the packed instructions.  The warps' accelerations
// are added in warp order, then over the ranks in rank order: deterministic.
constexpr int kStepWarps = 8;
constexpr int kStepBodies = 4;  // bodies i per lane
constexpr int kStepMaxSplit = 8;

__global__ void __launch_bounds__(32 * kStepWarps, 3) nbody_step_kernel(const NbodyParams p)
{
    constexpr int BP = kStepBodies;
    __shared__ float4 s_pairs[kStepWarps][32];          // a warp's 16 pairs of bodies j
    __shared__ float s_acc[kStepWarps][3 * BP * 32];
    const int lane = threadIdx.x % 32;
    const int warp = threadIdx.x / 32;
    const uint32_t ranks = cluster_size();
    const uint32_t rank = cluster_rank();
    const int64_t ibase = static_cast<int64_t>(blockIdx.x / ranks) * (32 * BP) + lane;
    float2 nx[BP], ny[BP], nz[BP], ax[BP], ay[BP], az[BP];
#pragma unroll
    for (int k = 0; k < BP; ++k) {
        const int64_t i = ibase + 32 * k;
        const float4 b = i < p.n ? p.pos[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        nx[k] = splat(-b.x);
        ny[k] = splat(-b.y);
        nz[k] = splat(-b.z);
        ax[k] = ay[k] = az[k] = make_float2(0.0f, 0.0f);
    }
    const float2 eps2 = splat(p.eps2);
    const int64_t shares = static_cast<int64_t>(ranks) * kStepWarps;
    const int64_t w = static_cast<int64_t>(rank) * kStepWarps + warp;
    const int64_t end = p.n / shares * (w + 1) + p.n % shares * (w + 1) / shares;
    int64_t b = p.n / shares * w + p.n % shares * w / shares;
    // a body past the share lies far away and has no mass
    const float4 none = make_float4(kPadCoord, kPadCoord, kPadCoord, 0.0f);
    float4 next = b + lane < end ? p.pos[b + lane] : none;
    float* pairs = reinterpret_cast<float*>(s_pairs[warp]);
    for (; b < end; b += 32) {
        const int count = static_cast<int>(end - b < 32 ? (end - b + 1) / 2 : 16);
        __syncwarp();  // the previous pairs have been read
        float* mine = pairs + lane / 2 * 8 + lane % 2;
        mine[0] = next.x;
        mine[2] = next.y;
        mine[4] = next.z;
        mine[6] = next.w;
        __syncwarp();
        next = b + 32 + lane < end ? p.pos[b + 32 + lane] : none;
#pragma unroll 2
        for (int j = 0; j < count; ++j) {
            const float4 xy = s_pairs[warp][2 * j];
            const float4 zm = s_pairs[warp][2 * j + 1];
            const float2 bx = make_float2(xy.x, xy.y), by = make_float2(xy.z, xy.w);
            const float2 bz = make_float2(zm.x, zm.y), bm = make_float2(zm.z, zm.w);
#pragma unroll
            for (int k = 0; k < BP; ++k) {
                const float2 dx = __fadd2_rn(bx, nx[k]);
                const float2 dy = __fadd2_rn(by, ny[k]);
                const float2 dz = __fadd2_rn(bz, nz[k]);
                const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, eps2)));
                const float2 inv = rsqrt_mufu_x2(r2);
                const float2 f = __fmul2_rn(__fmul2_rn(bm, inv), __fmul2_rn(inv, inv));
                ax[k] = __ffma2_rn(dx, f, ax[k]);
                ay[k] = __ffma2_rn(dy, f, ay[k]);
                az[k] = __ffma2_rn(dz, f, az[k]);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < BP; ++k) {
        s_acc[warp][(3 * k + 0) * 32 + lane] = ax[k].x + ax[k].y;
        s_acc[warp][(3 * k + 1) * 32 + lane] = ay[k].x + ay[k].y;
        s_acc[warp][(3 * k + 2) * 32 + lane] = az[k].x + az[k].y;
    }
    __syncthreads();
    const bool owner = warp < BP && warp % (ranks < BP ? ranks : BP) == rank;
    float a[3] = {0.0f, 0.0f, 0.0f};
    if (warp < BP) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int e = (3 * warp + c) * 32 + lane;
            a[c] = s_acc[0][e];
#pragma unroll
            for (int v = 1; v < kStepWarps; ++v)
                a[c] += s_acc[v][e];
            if (ranks > 1)
                s_acc[0][e] = a[c];  // only this thread reads or writes this entry
        }
    }
    if (ranks > 1) {
        cluster_sync();
        // warp k finishes the tile's k-th bodies, on the rank that owns them
        if (owner) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float* e = &s_acc[0][(3 * warp + c) * 32 + lane];
                float sum = ld_cluster_f32(cluster_map(e, 0));
                for (uint32_t r = 1; r < ranks; ++r)
                    sum += ld_cluster_f32(cluster_map(e, r));
                a[c] = sum;
            }
        }
        cluster_sync();  // the sums stay valid until every rank has read its share
    }
    if (!owner)
        return;
    const int64_t i = ibase + 32 * warp;
    if (i < p.n)
        integrate(p, i, a);
}

// The step with each pair of bodies evaluated once for both of them: 17 FP32 operations and one rsqrt for
// two interactions instead of 24 and two.  Bodies form blocks of 1,024; block I meets the blocks I + 1 ..
// I + B / 2 (mod B) -- for an even B the opposite block only where I < B / 2 -- so every pair of blocks
// meets once and every block has the same work.  A CTA takes a block I (128 bodies i a warp, four a lane)
// and a range of its tiles of 64 bodies j.  A lane starts with the j pair of its own number and moves on by
// one each step, reading the pair from shared memory and handing the pair's accelerations to the lane
// that meets it next by shuffles, so after 32 steps each j has met the warp's 128 bodies.  The warps'
// sums for a tile are added in warp order and go to the workspace, by the distance of the blocks; the
// bodies i keep their sums in registers over the CTA's whole range.  nbody_gather_kernel adds the parts of
// a body in a fixed order and integrates it.  Block I itself (distance 0) is evaluated one way.
constexpr int kPairBlock = 32 * kStepBodies * kStepWarps;
constexpr int kPairTile = 64;
constexpr int kPairTiles = kPairBlock / kPairTile;  // tiles of a block

struct NbodyPairParams {
    NbodyParams n;
    float* by_distance;  // [B / 2][3][padded]: on body j, from the block that many blocks before j's
    float* own;          // [parts][3][padded]: on body i, from its CTAs
    int64_t padded;      // B * kPairBlock
    int blocks, parts;
};

// Blocks of larger distance that block I meets: 1 .. this.
__host__ __device__ __forceinline__ int pair_reach(const int blocks, const int block)
{
    return blocks % 2 == 0 && block >= blocks / 2 ? blocks / 2 - 1 : blocks / 2;
}

__global__ void __launch_bounds__(32 * kStepWarps, 2) nbody_pair_kernel(const NbodyPairParams p)
{
    constexpr int BP = kStepBodies;
    __shared__ float4 s_xy[2][32], s_zm[2][32];                 // the tile's j pairs (x, x', y, y'), (z, z', m, m')
    __shared__ float s_j[2][kStepWarps][6 * 32];                // the warps' sums for a tile
    const int tid = threadIdx.x;
    const int lane = tid % 32;
    const int warp = tid / 32;
    const int block = blockIdx.x;
    const float4 none = make_float4(kPadCoord, kPadCoord, kPadCoord, 0.0f);  // far away, no mass
    const int64_t ibase = static_cast<int64_t>(block) * kPairBlock + warp * 32 * BP + lane;
    float2 nx[BP], ny[BP], nz[BP], nm[BP], ax[BP], ay[BP], az[BP];
#pragma unroll
    for (int k = 0; k < BP; ++k) {
        const int64_t i = ibase + 32 * k;
        const float4 b = i < p.n.n ? p.n.pos[i] : none;
        nx[k] = splat(-b.x);
        ny[k] = splat(-b.y);
        nz[k] = splat(-b.z);
        nm[k] = splat(-b.w);
        ax[k] = ay[k] = az[k] = make_float2(0.0f, 0.0f);
    }
    const float2 eps2 = splat(p.n.eps2);
    const int64_t total = static_cast<int64_t>(pair_reach(p.blocks, block) + 1) * kPairTiles;
    const int q_begin = static_cast<int>(total * blockIdx.y / p.parts);
    const int q_end = static_cast<int>(total * (blockIdx.y + 1) / p.parts);
    // tile q: the q % kPairTiles-th of the block at distance q / kPairTiles
    auto tile_base = [&](int q) -> int64_t {
        const int b = block + q / kPairTiles;
        return static_cast<int64_t>(b < p.blocks ? b : b - p.blocks) * kPairBlock + q % kPairTiles * kPairTile;
    };
    float4 next = none;
    auto fetch = [&](int q) {
        if (tid < kPairTile) {
            const int64_t j = tile_base(q) + tid;
            next = j < p.n.n ? p.n.pos[j] : none;
        }
    };
    auto stage = [&](int buf) {
        if (tid < kPairTile) {
            float* xy = reinterpret_cast<float*>(&s_xy[buf][tid / 2]) + tid % 2;
            float* zm = reinterpret_cast<float*>(&s_zm[buf][tid / 2]) + tid % 2;
            xy[0] = next.x;
            xy[2] = next.y;
            zm[0] = next.z;
            zm[2] = next.w;
        }
    };
    // the sums of tile q over the warps, to the workspace
    auto flush = [&](int q) {
        const int d = q / kPairTiles;
        if (d == 0 || tid >= 3 * kPairTile)
            return;
        const int c = tid / kPairTile;
        const int j = tid % kPairTile;
        const int e = (2 * c + j % 2) * 32 + j / 2;
        float sum = s_j[q & 1][0][e];
#pragma unroll
        for (int w = 1; w < kStepWarps; ++w)
            sum += s_j[q & 1][w][e];
        p.by_distance[(static_cast<int64_t>(d - 1) * 3 + c) * p.padded + tile_base(q) + j] = sum;
    };
    if (q_begin < q_end) {
        fetch(q_begin);
        stage(q_begin & 1);
    }
    for (int q = q_begin; q < q_end; ++q) {
        __syncthreads();  // tile q is staged, the warps' sums of tile q - 1 are complete
        if (q > q_begin)
            flush(q - 1);
        if (q + 1 < q_end)
            fetch(q + 1);
        const int buf = q & 1;
        float2 jx = make_float2(0.0f, 0.0f), jy = jx, jz = jx;
        auto meet = [&](auto both) {
#pragma unroll 1
            for (int step = 0; step < 32; ++step) {
                const int r = (lane + step) & 31;
                const float4 xy = s_xy[buf][r];
                const float4 zm = s_zm[buf][r];
                const float2 bx = make_float2(xy.x, xy.y), by = make_float2(xy.z, xy.w);
                const float2 bz = make_float2(zm.x, zm.y), bm = make_float2(zm.z, zm.w);
#pragma unroll
                for (int k = 0; k < BP; ++k) {
                    const float2 dx = __fadd2_rn(bx, nx[k]);
                    const float2 dy = __fadd2_rn(by, ny[k]);
                    const float2 dz = __fadd2_rn(bz, nz[k]);
                    const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, eps2)));
                    const float2 inv = rsqrt_mufu_x2(r2);
                    const float2 inv2 = __fmul2_rn(inv, inv);  // not 1/r^3: it leaves FP32's range before m/r^3 does
                    const float2 fi = __fmul2_rn(__fmul2_rn(bm, inv), inv2);
                    ax[k] = __ffma2_rn(dx, fi, ax[k]);
                    ay[k] = __ffma2_rn(dy, fi, ay[k]);
                    az[k] = __ffma2_rn(dz, fi, az[k]);
                    if constexpr (decltype(both)::value) {
                        const float2 fj = __fmul2_rn(__fmul2_rn(nm[k], inv), inv2);  // j is pulled the other way
                        jx = __ffma2_rn(dx, fj, jx);
                        jy = __ffma2_rn(dy, fj, jy);
                        jz = __ffma2_rn(dz, fj, jz);
                    }
                }
                if constexpr (decltype(both)::value) {
                    const int from = (lane + 1) & 31;  // that lane has met the pair this one meets next
                    jx.x = __shfl_sync(0xffffffffu, jx.x, from);
                    jx.y = __shfl_sync(0xffffffffu, jx.y, from);
                    jy.x = __shfl_sync(0xffffffffu, jy.x, from);
                    jy.y = __shfl_sync(0xffffffffu, jy.y, from);
                    jz.x = __shfl_sync(0xffffffffu, jz.x, from);
                    jz.y = __shfl_sync(0xffffffffu, jz.y, from);
                }
            }
        };
        if (q >= kPairTiles) {
            meet(std::true_type{});
            float* out = s_j[buf][warp];
            out[0 * 32 + lane] = jx.x;
            out[1 * 32 + lane] = jx.y;
            out[2 * 32 + lane] = jy.x;
            out[3 * 32 + lane] = jy.y;
            out[4 * 32 + lane] = jz.x;
            out[5 * 32 + lane] = jz.y;
        } else {
            meet(std::false_type{});
        }
        if (q + 1 < q_end)
            stage(buf ^ 1);
    }
    __syncthreads();
    if (q_begin < q_end)
        flush(q_end - 1);
    float* own = p.own + static_cast<int64_t>(blockIdx.y) * 3 * p.padded;
#pragma unroll
    for (int k = 0; k < BP; ++k) {
        own[0 * p.padded + ibase + 32 * k] = ax[k].x + ax[k].y;
        own[1 * p.padded + ibase + 32 * k] = ay[k].x + ay[k].y;
        own[2 * p.padded + ibase + 32 * k] = az[k].x + az[k].y;
    }
}

// A body's acceleration: its own CTAs' parts in order, then the parts by distance; then its step.  The
// parts are spread over a warp's four groups of eight distances' strides so that the loads of a body, one
// after another in memory only across bodies, are in flight together.
__global__ void __launch_bounds__(256) nbody_gather_kernel(const NbodyPairParams p)
{
    constexpr int kGroups = 8;  // warps of the block share 32 bodies
    __shared__ float s_sum[kGroups][3][32];
    const int lane = threadIdx.x % 32;
    const int group = threadIdx.x / 32;
    const int64_t i = static_cast<int64_t>(blockIdx.x) * 32 + lane;
    const int block = static_cast<int>(i / kPairBlock);
    // a body of the lower half of an even number of blocks has no part from the opposite block
    const int reach = p.blocks % 2 == 0 && block < p.blocks / 2 ? p.blocks / 2 - 1 : p.blocks / 2;
    float a[3] = {0.0f, 0.0f, 0.0f};
    const int rows = p.parts + reach;
#pragma unroll 4
    for (int r = group; r < rows; r += kGroups) {
        const float* src = r < p.parts ? p.own + static_cast<int64_t>(r) * 3 * p.padded
                                       : p.by_distance + static_cast<int64_t>(r - p.parts) * 3 * p.padded;
#pragma unroll
        for (int c = 0; c < 3; ++c)
            a[c] += src[c * p.padded + i];
    }
#pragma unroll
    for (int c = 0; c < 3; ++c)
        s_sum[group][c][lane] = a[c];
    __syncthreads();
    if (group != 0 || i >= p.n.n)
        return;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        a[c] = s_sum[0][c][lane];
        for (int g = 1; g < kGroups; ++g)
            a[c] += s_sum[g][c][lane];
    }
    integrate(p.n, i, a);
}

using NbodyLaunch = cudaError_t (*)(const NbodyParams&, dim3, dim3, size_t, int, cudaStream_t);

template <int BP, int UNR, bool SPLIT>
cudaError_t launch_nbody(const NbodyParams& p, dim3 grid, dim3 block, size_t smem, int split, cudaStream_t stream)
{
    auto kernel = nbody_kernel<BP, UNR, SPLIT>;
    if constexpr (!SPLIT) {
        (void)split;
        kernel<<<grid, block, smem, stream>>>(p);
        return cudaGetLastError();
    } else {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(grid.x * static_cast<unsigned>(split), grid.y, grid.z);
        cfg.blockDim = block;
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = static_cast<unsigned>(split);
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (split > kNbodyMaxPortableSplit) {
            cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
            if (e != cudaSuccess)
                return e;
            int clusters = 0;
            e = cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg);
            if (e != cudaSuccess)
                return e;
            if (clusters < 1)
                return cudaErrorLaunchOutOfResources;  // no SM group can hold such a cluster of these blocks
        }
        return cudaLaunchKernelEx(&cfg, kernel, p);
    }
}

struct NbodyVariant {
    int bp, unroll;
    bool split;
    NbodyLaunch launch;
};

template <int BP, int UNR>
void add_nbody(std::vector<NbodyVariant>& v)
{
    v.push_back({BP, UNR, false, &launch_nbody<BP, UNR, false>});
    v.push_back({BP, UNR, true, &launch_nbody<BP, UNR, true>});
}

const std::vector<NbodyVariant>& nbody_variants()
{
    static const std::vector<NbodyVariant> v = [] {
        std::vector<NbodyVariant> out;
        add_nbody<1, 1>(out);
        add_nbody<1, 2>(out);
        add_nbody<1, 4>(out);
        add_nbody<2, 1>(out);
        add_nbody<2, 2>(out);
        add_nbody<2, 4>(out);
        add_nbody<4, 1>(out);
        add_nbody<4, 2>(out);
        add_nbody<4, 4>(out);
        add_nbody<8, 1>(out);
        add_nbody<8, 2>(out);
        return out;
    }();
    return v;
}

int find_nbody(const coul_nbody_tune* t, const NbodyVariant** out)
{
    if (t == nullptr)
        return set_error(COUL_ERR_INVALID_ARGUMENT, "tune is NULL");
    if (t->block_x < 32 || t->block_x > kNbodyMaxThreads || t->block_x % 32 != 0)
        return set_error(COUL_ERR_DEVICE_LIMITS, "N-body block size must be a multiple of 32 in 32.." +
                                                     std::to_string(kNbodyMaxThreads));
    if (t->j_split < 0)
        return set_error(COUL_ERR_INVALID_ARGUMENT, "j_split must not be negative");
    if (t->j_split > kNbodyMaxSplit)  // beyond the largest cluster: no form
        return set_error(COUL_ERR_UNSUPPORTED, "j_split above " + std::to_string(kNbodyMaxSplit) + " is not supported");
    if (t->block_x > nbody_max_threads(t->bodies_per_thread))
        return set_error(COUL_ERR_DEVICE_LIMITS, "8 bodies per thread allow at most 256 threads per block");
    const int unroll = t->unroll <= 1 ? 1 : t->unroll;
    const bool split = t->j_split >= 2;
    for (const auto& e : nbody_variants()) {
        if (e.bp == t->bodies_per_thread && e.unroll == unroll && e.split == split) {
            if (out)
                *out = &e;
            return COUL_OK;
        }
    }
    return set_error(COUL_ERR_UNSUPPORTED, "no compiled N-body variant for bodies_per_thread=" +
                                               std::to_string(t->bodies_per_thread) + " unroll=" + std::to_string(unroll));
}

}  // namespace

}  // namespace coul

using namespace coul;

extern "C" {

COUL_API int coul_nbody_tune_default(coul_nbody_tune* t)
{
    if (t == nullptr)
        return set_error(COUL_ERR_INVALID_ARGUMENT, "tune is NULL");
    t->block_x = 128;
    t->bodies_per_thread = 4;
    t->unroll = 2;
    t->j_split = 0;
    return COUL_OK;
}

COUL_API int coul_nbody_tune_supported(const coul_nbody_tune* t) { return find_nbody(t, nullptr); }

// The checks and parameters of both entry points.
static int nbody_params(coul_ctx* ctx, const float* d_pos_mass, const float* d_vel, int64_t n, float dt, float damping,
                        float softening_sqr, float* d_pos_mass_new, float* d_vel_new, NbodyParams* p)
{
    if (n < 0 || (n > 0 && (!aligned16(d_pos_mass) || !aligned16(d_vel) || !aligned16(d_pos_mass_new) ||
                            !aligned16(d_vel_new) || !d_pos_mass || !d_vel || !d_pos_mass_new || !d_vel_new)))
        return set_error(COUL_ERR_INVALID_ARGUMENT, "bodies must be non-NULL, 16-byte aligned float4 arrays");
    if (d_pos_mass_new == d_pos_mass || d_vel_new == d_vel)
        return set_error(COUL_ERR_INVALID_ARGUMENT, "the step reads all old positions: outputs must not alias inputs");
    if (!(softening_sqr > 0.0f))
        return set_error(COUL_ERR_INVALID_ARGUMENT, "softening_sqr must be positive (the j = i term divides by it)");
    p->pos = reinterpret_cast<const float4*>(d_pos_mass);
    p->vel = reinterpret_cast<const float4*>(d_vel);
    p->pos_new = reinterpret_cast<float4*>(d_pos_mass_new);
    p->vel_new = reinterpret_cast<float4*>(d_vel_new);
    p->n = n;
    p->dt = dt;
    p->damping = damping;
    p->eps2 = softening_sqr;
    p->status = ctx->d_status;
    return COUL_OK;
}

COUL_API int coul_nbody_step(coul_ctx* ctx, const float* d_pos_mass, const float* d_vel, int64_t n, float dt, float damping,
                             float softening_sqr, const coul_nbody_tune* tune, float* d_pos_mass_new, float* d_vel_new)
{
    if (ctx == nullptr)
        return set_error(COUL_ERR_INVALID_ARGUMENT, "ctx is NULL");
    const NbodyVariant* v = nullptr;
    int rc = find_nbody(tune, &v);
    if (rc)
        return rc;
    NbodyParams p{};
    if ((rc = nbody_params(ctx, d_pos_mass, d_vel, n, dt, damping, softening_sqr, d_pos_mass_new, d_vel_new, &p)))
        return rc;
    if (n == 0)
        return COUL_OK;
    if ((rc = ctx_activate(ctx)))
        return rc;
    const int64_t per_tile = static_cast<int64_t>(tune->block_x) * tune->bodies_per_thread;
    const int64_t tiles = (n + per_tile - 1) / per_tile;
    const int split = tune->j_split >= 2 ? tune->j_split : 1;
    if (tiles * split > 2147483647LL)
        return set_error(COUL_ERR_DEVICE_LIMITS, "too many bodies for one launch");
    size_t smem = kNbodyRedOffset;
    if (split > 1)
        smem += static_cast<size_t>(tune->block_x) * 3 * tune->bodies_per_thread * sizeof(float);
    if ((rc = ctx_begin_timing(ctx)))
        return rc;
    cudaError_t e = v->launch(p, dim3(static_cast<unsigned>(tiles)), dim3(static_cast<unsigned>(tune->block_x)), smem, split,
                              ctx->stream);
    if (e == cudaErrorLaunchOutOfResources)
        return set_error(COUL_ERR_DEVICE_LIMITS, std::string("N-body launch: ") + cudaGetErrorString(e));
    if (e != cudaSuccess)
        return cuda_error(e, "N-body launch");
    return ctx_end_timing(ctx);
}

// From this many bodies on the pair form is faster than the one-way kernel (10,000
// bodies: 60 us, 65; 131,072: 5.17 ms, 7.16).
constexpr int64_t kPairBodies = 4096;
constexpr size_t kPairWorkspaceLimit = size_t{256} << 20;

// The pair form of the plain step.  Sets *done when it was launched; otherwise the caller launches the
// one-way kernel, which needs no workspace: under stream capture (a graph would hold as much again), beyond
// the workspace limit, or when the memory is not to be had.
static int nbody_pairs(coul_ctx* ctx, const NbodyParams& n, bool* done)
{
    *done = false;
    NbodyPairParams p{};
    p.n = n;
    const int64_t blocks = (n.n + kPairBlock - 1) / kPairBlock;
    p.padded = blocks * kPairBlock;
    // CTAs per block: up to 28 an SM (14 rounds of the resident two), 32 to 64 a block but about a tile at
    // least each; fewer leave long last rounds (131,072 bodies: 2 parts 6.3 ms, 8 5.3, 32 5.17; 10,000: 16
    // parts 77 us, 64 60)
    const int64_t want = std::max<int64_t>(32, std::min<int64_t>(64, 28LL * ctx->sm_count / blocks));
    p.parts = static_cast<int>(std::min<int64_t>(want, (blocks / 2 + 1) * kPairTiles));
    const int64_t rows = blocks / 2 + p.parts;
    const size_t need = static_cast<size_t>(rows) * 3 * static_cast<size_t>(p.padded) * sizeof(float);
    if (blocks < 2 || need > kPairWorkspaceLimit)
        return COUL_OK;
    p.blocks = static_cast<int>(blocks);
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(ctx->stream, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return COUL_OK;
    }
    void* mem = nullptr;
    bool own = false;
    int rc = workspace_begin(ctx, kWorkspacePairs, need, "N-body", &mem, &own);
    if (rc != COUL_OK)
        return rc == COUL_ERR_OUT_OF_MEMORY ? COUL_OK : rc;
    p.own = static_cast<float*>(mem);
    p.by_distance = p.own + static_cast<size_t>(p.parts) * 3 * static_cast<size_t>(p.padded);
    if ((rc = ctx_begin_timing(ctx)))
        return workspace_fail(ctx, rc);
    cudaError_t e;
    nbody_pair_kernel<<<dim3(static_cast<unsigned>(blocks), static_cast<unsigned>(p.parts)), 32 * kStepWarps, 0, ctx->stream>>>(p);
    if ((e = cudaGetLastError()) != cudaSuccess)
        return workspace_fail(ctx, cuda_error(e, "N-body launch"));
    nbody_gather_kernel<<<static_cast<unsigned>(p.padded / 32), 256, 0, ctx->stream>>>(p);
    if ((e = cudaGetLastError()) != cudaSuccess)
        return workspace_fail(ctx, cuda_error(e, "N-body launch"));
    *done = true;
    return ctx_end_timing(ctx);
}

COUL_API int coul_nbody_step_plain(coul_ctx* ctx, const float* d_pos_mass, const float* d_vel, int64_t n, float dt,
                                   float damping, float softening_sqr, float* d_pos_mass_new, float* d_vel_new)
{
    if (ctx == nullptr)
        return set_error(COUL_ERR_INVALID_ARGUMENT, "ctx is NULL");
    NbodyParams p{};
    int rc = nbody_params(ctx, d_pos_mass, d_vel, n, dt, damping, softening_sqr, d_pos_mass_new, d_vel_new, &p);
    if (rc || n == 0)
        return rc;
    if ((rc = ctx_activate(ctx)))
        return rc;
    if (n >= kPairBodies) {
        bool done = false;
        if ((rc = nbody_pairs(ctx, p, &done)) || done)
            return rc;
    }
    const int64_t tiles = (n + 32 * kStepBodies - 1) / (32 * kStepBodies);
    int split = 1;  // CTAs per tile: six CTAs an SM, two rounds of the resident three
    while (split < kStepMaxSplit && tiles * split < 6LL * ctx->sm_count)
        split *= 2;
    if (tiles * split > 2147483647LL)
        return set_error(COUL_ERR_DEVICE_LIMITS, "too many bodies for one launch");
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(tiles * split), 1, 1);
    cfg.blockDim = dim3(32 * kStepWarps, 1, 1);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(split);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = split > 1 ? 1 : 0;
    if ((rc = ctx_begin_timing(ctx)))
        return rc;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, nbody_step_kernel, p);
    if (e != cudaSuccess)
        return cuda_error(e, "N-body launch");
    return ctx_end_timing(ctx);
}

}  // extern "C"
