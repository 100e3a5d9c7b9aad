// coul_plain.cu -- the map and the slice of a call that names no configuration.
//
// KTT leaves the choice of a kernel to its tuner; a caller without one (the PyTorch binding's plain
// forward_3d / forward_2d) gets the kernels of this file, which suit every grid: a ligand's 40^3
// points, a slice, a 256^3 map.  The 3D kernel also runs the configurations of 2 x 8 and 2 x 16 points a
// thread with FP32 sums on maps of up to about 200^3 points (plain_tile).  (One CTA per point tile of a
// fixed shape, as the configurable forms have it, leaves most SMs idle on the small ones: 33 CTAs for a
// 37 x 41 x 33 map.)
//
// A warp evaluates one point tile -- 32 columns of x points (columns numbered row by row over the
// plane, so only a row's end and the plane's end are padded) by 16 or 8 z points, or by 4 rows of a
// slice -- against its own share of the atoms, and needs no other warp to do so: its lanes load 32
// atoms at a time straight into registers (the next 32 while these are evaluated), write what every
// lane will read of them to the warp's own shared memory, and the warp runs through them.  In 3D the
// record of an atom holds its z differences to the tile's planes, so the pair loop spends nothing on
// them.  The eight warps of a CTA share a tile and split the atoms evenly, as do the CTAs of a
// thread-block cluster where there are too few tiles for the GPU; their FP32 sums are added in a
// fixed order through shared memory (and distributed shared memory), so a map is the same from run to
// run, and a sum never runs over more than an eighth of the atoms.
//
// Bound: the MUFU unit and the FMA pipe together (5/16 of the reciprocal square roots on the FMA
// pipe in 3D, 2/8 in 2D).  On B200, against the default configuration's tile (128 x 4 x 16 points in
// 3D, 128 x 16 in 2D, all roots on MUFU): 37 x 41 x 33 x 211 atoms 15 us a call against 87; 96^3 x
// 4,096 0.644 ms against 1.39; 200^3 x 8,000 5.9 Tpair/s against 3.2; a 250 x 187 slice x 1,501 32
// against 176 us (with the conversion of its atoms).  What a thread's 32 points give in 3D: 16 points
// (8 planes) reach 5.4.  100 registers and 16 warps an SM: 80 registers (24 warps)
// spill a little and are 1 % slower, two atoms at a time are no faster.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "coul_forward.cuh"
#include "coul_internal.h"

namespace coul {

namespace {

constexpr int kPlainWarps = 8;
constexpr int kPlainThreads = 32 * kPlainWarps;
// The share of a call without a configuration, of 16 roots in 3D and of 8 in 2D, at MUFU's precision (rsqrt_full):
// 96^3 x 4,096 takes 644 us with 5/16 (2/16 745, 3/16 705, 4/16 659, 6/16 664; with
// rsqrt_fma, good to 4.6e-7 only, 629), 96^3 x 400 76 us (no share 94), a 1024 x 1024 slice x 20,000 3.83 ms with 2/8
// (1/8 or 3/8 4.19; rsqrt_fma 3.68).
constexpr int kPlainSoft = 5;
constexpr int kPlain2dSoft = 2;
constexpr int kPlainMaxSplit = 8;  // portable cluster size

// 3D: 2 x 16 points a thread; soft pairs spread over a thread's 16 lane pairs, SOFT of 16.
constexpr int kPlainX = 2;
constexpr int kPlainZ = 16;
constexpr int kPlainRecord = 4 + kPlainZ;  // floats per staged atom: x, y, q, q * kSoftRsqrtScale, dz of the planes

struct PlainParams {
    FwdParams f;
    int columns;  // columns of x points per row (2D: per group of rows)
    int depth;    // 3D: planes per tile, kPlainZ or half of it
    int vec_ok;
};

// This warp's share of the atoms: the w-th of all warps of all CTAs that share the tile.
__device__ __forceinline__ void warp_atoms(const int64_t n, const uint32_t ranks, int64_t& begin, int64_t& end)
{
    const int64_t total = static_cast<int64_t>(ranks) * kPlainWarps;
    const int64_t w = static_cast<int64_t>(cluster_rank()) * kPlainWarps + threadIdx.x / 32;
    begin = n / total * w + n % total * w / total;
    end = n / total * (w + 1) + n % total * (w + 1) / total;
}

// A tile's sums: every warp's values per lane (s[warp][(row * X + k) * 32 + lane], X points along x a
// row) are added in warp order, then over the ranks of the cluster in rank order; store(row, k, sums)
// gets the thread's own column's points once, X of a row or (C of them, C = 1) one at a time.
template <int X, int P, class Store>
__device__ __forceinline__ void reduce_tile(float (*s)[P * 32], const int rows, const uint32_t ranks, Store&& store)
{
    __syncthreads();
    const int lane = threadIdx.x % 32;
    const int warp = threadIdx.x / 32;
    if (ranks == 1) {
        for (int row = warp; row < rows; row += kPlainWarps) {
            float sum[X];
#pragma unroll
            for (int k = 0; k < X; ++k) {
                const int i = (row * X + k) * 32 + lane;
                sum[k] = s[0][i];
#pragma unroll
                for (int w = 1; w < kPlainWarps; ++w)
                    sum[k] += s[w][i];
            }
            store(row, 0, sum);
        }
        return;
    }
    const int values = rows * X;
    for (int v = warp; v < values; v += kPlainWarps) {
        float sum = s[0][v * 32 + lane];
#pragma unroll
        for (int w = 1; w < kPlainWarps; ++w)
            sum += s[w][v * 32 + lane];
        s[0][v * 32 + lane] = sum;  // only this thread reads or writes this entry
    }
    cluster_sync();
    for (int v = warp * static_cast<int>(ranks) + static_cast<int>(cluster_rank()); v < values;
         v += kPlainWarps * static_cast<int>(ranks)) {
        float part[kPlainMaxSplit];
#pragma unroll
        for (int r = 0; r < kPlainMaxSplit; ++r)  // independent loads, issued together
            if (r < static_cast<int>(ranks))
                part[r] = ld_cluster_f32(cluster_map(&s[0][v * 32 + lane], static_cast<uint32_t>(r)));
        float sum[1] = {part[0]};
#pragma unroll
        for (int r = 1; r < kPlainMaxSplit; ++r)
            if (r < static_cast<int>(ranks))
                sum[0] += part[r];
        store(v / X, v % X, sum);
    }
    cluster_sync();  // the sums stay valid until every rank has read its share
}

// 3D: `cnt` staged atoms against the tile's first D planes.
template <int SOFT, int D>  // SOFT: sixteenths (+ kSoftFull)
__device__ __forceinline__ void plain_batch(const float4* rec, const int cnt, const float (&gx)[kPlainX], const float gy,
                                            float2 (&acc)[kPlainX][kPlainZ / 2])
{
    constexpr int ZH = kPlainZ / 2;
#pragma unroll 1
    for (int j = 0; j < cnt; ++j) {
        const float4 a = rec[j * (kPlainRecord / 4)];  // x, y, q, scaled q
        const float dy = gy - a.y;
        const float dy2 = dy * dy;
        float2 dz[D / 2];
#pragma unroll
        for (int m = 0; m < D / 4; ++m) {
            const float4 d = rec[j * (kPlainRecord / 4) + 1 + m];
            dz[2 * m] = make_float2(d.x, d.y);
            dz[2 * m + 1] = make_float2(d.z, d.w);
        }
        const float2 q = splat(a.z), qs = splat(a.w);
#pragma unroll
        for (int k = 0; k < kPlainX; ++k) {
            const float dx = gx[k] - a.x;
            const float2 dxy = splat(fmaf(dx, dx, dy2));
#pragma unroll
            for (int m = 0; m < D / 2; ++m) {
                const float2 r2 = __ffma2_rn(dz[m], dz[m], dxy);
                if (SOFT != 0 && spread_soft(k * ZH + m, soft_share(SOFT)))
                    pair_update<true, SOFT >= kSoftFull, false>(r2, q, qs, acc[k][m]);
                else
                    pair_update<false, false, false>(r2, q, qs, acc[k][m]);
            }
        }
    }
}

template <int SOFT>
__global__ void __launch_bounds__(kPlainThreads, 2) plain_3d_kernel(const PlainParams p)
{
    constexpr int P = kPlainX * kPlainZ;
    // a warp's staged atoms, later its sums
    __shared__ __align__(16) float s_warp[kPlainWarps][P * 32];
    __shared__ float4 s_gz[kPlainZ / 4];  // the tile's planes
    static_assert(32 * kPlainRecord <= P * 32 && kPlainRecord % 4 == 0, "the records fit where the sums go");
    const int lane = threadIdx.x % 32;
    const int warp = threadIdx.x / 32;
    const uint32_t ranks = cluster_size();
    const int64_t tile = blockIdx.x / ranks;
    const int64_t column = tile * 32 + lane;
    const int yrow = static_cast<int>(column / p.columns);
    const int x0 = static_cast<int>(column % p.columns) * kPlainX;
    // tiles start at multiples of the depth on the whole grid, whichever planes a slab asks for
    const int z0 = (p.f.z_base / p.depth + static_cast<int>(blockIdx.y)) * p.depth;
    const int planes = p.f.nz - z0 < p.depth ? p.f.nz - z0 : p.depth;
    float gx[kPlainX];
#pragma unroll
    for (int k = 0; k < kPlainX; ++k)
        gx[k] = fmaf(static_cast<float>(x0 + k), p.f.h, p.f.ox);
    const float gy = fmaf(static_cast<float>(yrow), p.f.h, p.f.oy);
    if (threadIdx.x < kPlainZ)
        reinterpret_cast<float*>(s_gz)[threadIdx.x] = fmaf(static_cast<float>(z0 + static_cast<int>(threadIdx.x)), p.f.h, p.f.oz);
    __syncthreads();
    float2 acc[kPlainX][kPlainZ / 2];
#pragma unroll
    for (int k = 0; k < kPlainX; ++k)
#pragma unroll
        for (int m = 0; m < kPlainZ / 2; ++m)
            acc[k][m] = make_float2(0.0f, 0.0f);

    int64_t b, end;
    warp_atoms(p.f.n_atoms, ranks, b, end);
    const bool soft_grid = SOFT != 0 && soft_axis(p.f.nx, p.f.h, p.f.ox) && soft_axis(p.f.ny, p.f.h, p.f.oy);
    float4* rec = reinterpret_cast<float4*>(s_warp[warp]);
    float4 a = b + lane < end ? p.f.atoms[b + lane] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (; b < end; b += 32) {
        const int cnt = static_cast<int>(end - b < 32 ? end - b : 32);
        __syncwarp();  // the previous records have been read
        rec[lane * (kPlainRecord / 4)] = make_float4(a.x, a.y, a.w, a.w * kSoftRsqrtScale);
        float dz_min = kSoftFar, dz_max = 0.0f;  // over the planes of the tile, whichever of them a slab asks for
#pragma unroll
        for (int m = 0; m < kPlainZ / 4; ++m) {
            const float4 g = s_gz[m];
            const float4 dz = make_float4(g.x - a.z, g.y - a.z, g.z - a.z, g.w - a.z);
            rec[lane * (kPlainRecord / 4) + 1 + m] = dz;
            if (4 * m < p.depth)
                dz_range(dz, dz_min, dz_max);
        }
        const bool ok = lane >= cnt || (soft_grid && soft_place(a, dz_max));
        bool soft = SOFT != 0 && __all_sync(0xffffffffu, ok && (lane >= cnt || dz_min >= kSoftNear));
        __syncwarp();
        if (SOFT != 0 && !soft && __all_sync(0xffffffffu, ok)) {
            const float y[1] = {gy};
            soft = !on_columns(0xffffffffu, rec, kPlainRecord / 4, cnt, gx, y);
        }
        if (b + 32 + lane < end)
            a = p.f.atoms[b + 32 + lane];
        // a tile that overhangs the grid by half or more evaluates its first half
        if (planes <= kPlainZ / 2) {
            if (soft)
                plain_batch<SOFT, kPlainZ / 2>(rec, cnt, gx, gy, acc);
            else
                plain_batch<0, kPlainZ / 2>(rec, cnt, gx, gy, acc);
        } else if (soft) {
            plain_batch<SOFT, kPlainZ>(rec, cnt, gx, gy, acc);
        } else {
            plain_batch<0, kPlainZ>(rec, cnt, gx, gy, acc);
        }
    }
    __syncwarp();
#pragma unroll
    for (int m = 0; m < kPlainZ; ++m)
#pragma unroll
        for (int k = 0; k < kPlainX; ++k)
            s_warp[warp][(m * kPlainX + k) * 32 + lane] = coul::lane(acc[k][m / 2], m & 1);
    const FwdParams& f = p.f;
    reduce_tile<kPlainX, P>(s_warp, planes, ranks, [&](int row, int k, const auto& sum) {
        constexpr int N = sizeof(sum) / sizeof(float);
        const int z = z0 + row;
        if (yrow < f.ny && z >= f.z_base)
            store_points<N>(f.out + (static_cast<int64_t>(z - f.z_base) * f.ny + yrow) * f.nx, x0 + k, f.nx, sum,
                            f.accumulate, p.vec_ok);
    });
}

// 2D: 4 x 4 points a thread.
constexpr int kPlain2dX = 4;
constexpr int kPlain2dY = 4;

template <int SOFT>
__global__ void __launch_bounds__(kPlainThreads, 4) plain_2d_kernel(const PlainParams p)
{
    constexpr int P = kPlain2dX * kPlain2dY;
    constexpr int YH = kPlain2dY / 2;
    __shared__ __align__(16) float s_warp[kPlainWarps][P * 32];
    const int lane = threadIdx.x % 32;
    const int warp = threadIdx.x / 32;
    const uint32_t ranks = cluster_size();
    const int64_t column = static_cast<int64_t>(blockIdx.x / ranks) * 32 + lane;
    const int y0 = static_cast<int>(column / p.columns) * kPlain2dY;
    const int x0 = static_cast<int>(column % p.columns) * kPlain2dX;
    float gx[kPlain2dX];
#pragma unroll
    for (int k = 0; k < kPlain2dX; ++k)
        gx[k] = fmaf(static_cast<float>(x0 + k), p.f.h, p.f.ox);
    float2 gy[YH], acc[kPlain2dX][YH];
    float unused;
    blocked_coords<YH, kModeSlice2d>(p.f, y0, 0, unused, gy);
#pragma unroll
    for (int k = 0; k < kPlain2dX; ++k)
#pragma unroll
        for (int i = 0; i < YH; ++i)
            acc[k][i] = make_float2(0.0f, 0.0f);

    int64_t b, end;
    warp_atoms(p.f.n_atoms, ranks, b, end);
    const bool soft_grid = SOFT != 0 && soft_axis(p.f.nx, p.f.h, p.f.ox) && soft_axis(p.f.ny, p.f.h, p.f.oy);
    float4* rec = reinterpret_cast<float4*>(s_warp[warp]);
    float4 a = b + lane < end ? p.f.atoms[b + lane] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (; b < end; b += 32) {
        const int cnt = static_cast<int>(end - b < 32 ? end - b : 32);
        __syncwarp();
        rec[lane] = a;
        // an atom's .z is its dz^2 to the slice
        const bool ok = lane >= cnt || (soft_grid && fabsf(a.x) < kSoftFar && fabsf(a.y) < kSoftFar && a.z >= 0.0f &&
                                        a.z < kSoftFar * kSoftFar);
        bool soft = SOFT != 0 && __all_sync(0xffffffffu, ok && (lane >= cnt || a.z >= kSoftNear * kSoftNear));
        __syncwarp();
        if (SOFT != 0 && !soft && __all_sync(0xffffffffu, ok)) {
            float y[kPlain2dY];
#pragma unroll
            for (int m = 0; m < kPlain2dY; ++m)
                y[m] = coul::lane(gy[m / 2], m & 1);
            soft = !on_columns(0xffffffffu, rec, 1, cnt, gx, y);
        }
        if (b + 32 + lane < end)
            a = p.f.atoms[b + 32 + lane];
        if (soft) {
#pragma unroll 2
            for (int j = 0; j < cnt; ++j)
                pair_block_2d<kPlain2dX, YH, YH, SOFT, 0, false>(gx, gy, rec[j], acc);
        } else {
#pragma unroll 2
            for (int j = 0; j < cnt; ++j)
                pair_block_2d<kPlain2dX, YH, YH, 0, 0, false>(gx, gy, rec[j], acc);
        }
    }
    __syncwarp();
#pragma unroll
    for (int m = 0; m < kPlain2dY; ++m)
#pragma unroll
        for (int k = 0; k < kPlain2dX; ++k)
            s_warp[warp][(m * kPlain2dX + k) * 32 + lane] = coul::lane(acc[k][m / 2], m & 1);
    const FwdParams& f = p.f;
    reduce_tile<kPlain2dX, P>(s_warp, kPlain2dY, ranks, [&](int row, int k, const auto& sum) {
        constexpr int N = sizeof(sum) / sizeof(float);
        const int y = y0 + row;
        if (y < f.ny)
            store_points<N>(f.out + static_cast<int64_t>(y) * f.nx, x0 + k, f.nx, sum, f.accumulate, p.vec_ok);
    });
}

int launch_plain(coul_ctx* ctx, void (*kernel)(PlainParams), const PlainParams& p, int64_t tiles_xy, int64_t tiles_z,
                 int split)
{
    if (tiles_xy * split > 2147483647LL || tiles_z > 65535)
        return set_error(COUL_ERR_DEVICE_LIMITS, "grid too large for one launch");
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(tiles_xy * split), static_cast<unsigned>(tiles_z), 1);
    cfg.blockDim = dim3(kPlainThreads, 1, 1);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(split);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = split > 1 ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, p);
    return e == cudaSuccess ? COUL_OK : cuda_error(e, "forward launch");
}

// CTAs that share a tile: twice as many while they leave half of the SMs without one, and while a
// launch of fewer than `fill` CTAs an SM would leave each warp 16 atoms or more.
int plain_split(const coul_ctx* ctx, int64_t tiles, int64_t n, int fill)
{
    int split = 1;
    while (split < kPlainMaxSplit) {
        const int64_t atoms = n / (2 * split * kPlainWarps);  // a warp's share after doubling
        const bool idle = tiles * split < ctx->sm_count / 2 && atoms >= 3;
        const bool thin = tiles * split < static_cast<int64_t>(ctx->sm_count) * fill && atoms >= 16;
        if (!idle && !thin)
            break;
        split *= 2;
    }
    return split;
}

int check_call(const float* d_atoms, int64_t n_atoms, const float* d_out)
{
    if (n_atoms < 0)
        return set_error(COUL_ERR_INVALID_ARGUMENT, "negative atom count");
    if (d_out == nullptr)
        return set_error(COUL_ERR_INVALID_ARGUMENT, "output pointer is NULL");
    if (n_atoms > 0 && (d_atoms == nullptr || !aligned16(d_atoms)))
        return set_error(COUL_ERR_INVALID_ARGUMENT, "atoms must be a non-NULL, 16-byte aligned float4 array");
    return COUL_OK;
}

}  // namespace

int launch_plain_3d(coul_ctx* ctx, const FwdParams& f, int nz, int soft)
{
    void (*kernel)(PlainParams) = nullptr;
    switch (soft) {
    case 0: kernel = plain_3d_kernel<0>; break;
    case 2: kernel = plain_3d_kernel<2>; break;
    case 3: kernel = plain_3d_kernel<3>; break;
    case 4: kernel = plain_3d_kernel<4>; break;
    case 5: kernel = plain_3d_kernel<5>; break;
    case 6: kernel = plain_3d_kernel<6>; break;
    case 8: kernel = plain_3d_kernel<8>; break;
    case 10: kernel = plain_3d_kernel<10>; break;
    case kPlainSoft + kSoftFull: kernel = plain_3d_kernel<kPlainSoft + kSoftFull>; break;
    default: return set_error(COUL_ERR_UNSUPPORTED, "no kernel for this share of FMA-pipe roots");
    }
    PlainParams p{};
    p.f = f;
    p.columns = (f.nx + kPlainX - 1) / kPlainX;
    const int64_t tiles_xy = (static_cast<int64_t>(p.columns) * f.ny + 31) / 32;
    // The depth and the split follow from the whole grid, so that a slab's values are the map's.
    p.vec_ok = f.nx % kPlainX == 0 && reinterpret_cast<uintptr_t>(f.out) % (kPlainX * sizeof(float)) == 0;
    // Half the depth where full tiles would give a GPU of two CTAs an SM less than two rounds of them:
    // 64^3 x 4,000 takes 203 us instead of 235.
    const auto tiles_at = [&](int depth) { return tiles_xy * ((nz + depth - 1) / depth); };
    p.depth = kPlainZ;
    if (tiles_at(kPlainZ) < 4LL * ctx->sm_count && nz / (kPlainZ / 2) < 65535)
        p.depth = kPlainZ / 2;
    const int split = plain_split(ctx, tiles_at(p.depth), f.n_atoms, 5);
    const int64_t tiles_z = (f.nz + p.depth - 1) / p.depth - f.z_base / p.depth;
    return launch_plain(ctx, kernel, p, tiles_xy, tiles_z, split);
}

}  // namespace coul

using namespace coul;

extern "C" {

COUL_API int coul_forward_3d_plain(coul_ctx* ctx, const float* d_atoms, int64_t n_atoms, const coul_grid* grid,
                                   int z_begin, int z_end, int accumulate, float* d_out)
{
    if (ctx == nullptr)
        return set_error(COUL_ERR_INVALID_ARGUMENT, "ctx is NULL");
    int rc = validate_grid(grid);
    if (rc)
        return rc;
    // the limits of the default configuration's launch
    if ((grid->ny + 3) / 4 > 65535 || (grid->nz + 15) / 16 > 65535)
        return set_error(COUL_ERR_DEVICE_LIMITS, "grid too large for one launch");
    if (z_begin < 0 || z_begin >= z_end || z_end > grid->nz)
        return set_error(COUL_ERR_INVALID_ARGUMENT, "slab [z_begin, z_end) must be a non-empty range inside the grid");
    if ((rc = check_call(d_atoms, n_atoms, d_out)) || (rc = ctx_activate(ctx)))
        return rc;
    FwdParams f{};
    f.atoms = reinterpret_cast<const float4*>(d_atoms);
    f.n_atoms = n_atoms;
    f.nx = grid->nx;
    f.ny = grid->ny;
    f.nz = z_end;
    f.z_base = z_begin;
    f.h = grid->spacing;
    f.ox = grid->origin[0];
    f.oy = grid->origin[1];
    f.oz = grid->origin[2];
    f.out = d_out;
    f.accumulate = accumulate ? 1 : 0;
    if ((rc = ctx_begin_timing(ctx)) || (rc = launch_plain_3d(ctx, f, grid->nz, kPlainSoft + kSoftFull)))
        return rc;
    return ctx_end_timing(ctx);
}

COUL_API int coul_forward_2d_plain(coul_ctx* ctx, const float* d_atoms, int64_t n_atoms, float spacing, int nx, int ny,
                                   int accumulate, float* d_out)
{
    if (ctx == nullptr)
        return set_error(COUL_ERR_INVALID_ARGUMENT, "ctx is NULL");
    const coul_grid g{nx, ny, 1, spacing, {0.0f, 0.0f, 0.0f}};
    int rc = validate_grid(&g);
    if (rc || (rc = check_call(d_atoms, n_atoms, d_out)) || (rc = ctx_activate(ctx)))
        return rc;
    if ((ny + 15) / 16 > 65535)
        return set_error(COUL_ERR_DEVICE_LIMITS, "grid too large for one launch");
    PlainParams p{};
    p.f.atoms = reinterpret_cast<const float4*>(d_atoms);
    p.f.n_atoms = n_atoms;
    p.f.nx = nx;
    p.f.ny = ny;
    p.f.nz = 1;
    p.f.h = spacing;
    p.f.out = d_out;
    p.f.accumulate = accumulate ? 1 : 0;
    p.columns = (nx + kPlain2dX - 1) / kPlain2dX;
    p.vec_ok = nx % kPlain2dX == 0 && aligned16(d_out);
    const int64_t tiles = (static_cast<int64_t>(p.columns) * ((ny + kPlain2dY - 1) / kPlain2dY) + 31) / 32;
    const int split = plain_split(ctx, tiles, n_atoms, 4);
    if ((rc = ctx_begin_timing(ctx)) ||
        (rc = launch_plain(ctx, plain_2d_kernel<kPlain2dSoft + kSoftFull>, p, tiles, 1, split)))
        return rc;
    return ctx_end_timing(ctx);
}

}  // extern "C"
