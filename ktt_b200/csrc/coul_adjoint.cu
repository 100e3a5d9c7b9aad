// coul_adjoint.cu -- gradient of a loss on the 3D map with respect to charges and positions.
//
// For V_i = sum_j q_j / |r_i - r_j| and any loss L(V) with G_i = dL/dV_i (for the weighted
// least-squares loss 0.5 sum_i w_i (V_i - T_i)^2, G_i = w_i (V_i - T_i)):
//     dL/dq_j = sum_i G_i / r_ij
//     dL/dr_j = q_j sum_i G_i (r_i - r_j) / r_ij^3
// Nothing is stored per pair: 1/r is recomputed.  KTT has no adjoint; this is the B200 form of the
// transposed sum.  A thread owns one atom, a CTA kAdjThreads atoms and a chunk of grid rows; the rows'
// G values pass through shared memory in blocks of kRows rows x X points, and while a block of
// X columns is processed the thread holds its X differences dx = x - a.x in registers, so a
// pair costs six FP32 operations -- r^2 = fma(dx, dx, dy^2 + dz^2), t = G/r, 1/r^2, the sum of t (for the
// charge), and two FMAs that add t/r^2 by column (its sum times dx gives the x component) and by row
// (its sum times dy and dz gives the other two) -- and one MUFU rsqrt.  Two neighbouring columns share
// each packed instruction: dx, the column sums and the four-point loads of G come in pairs as they
// are.  A row is summed by itself, the rows of a block are added in FP32 and the block's sums go into FP64
// sums per atom; each (atom tile, row chunk) writes its FP64 partials, and a second kernel adds the
// chunks in a fixed order, so the result is deterministic.
//
// An FP32 sum is thus no longer than a row of 25 points and more: chains of a row's 16 lane pairs (8), then of
// the block's 8 rows (16); column sums of 16 rows.  Rows of up to 24 points (SHORT) would not be: theirs go
// into FP64 one by one, and G dx/r^3 is added along the row (eight operations a pair).  With rows of 64 terms
// in one chain the charge gradient was 1.2 to 1.7 times less exact than row by row for nx <= 32.
//
// Bound: the MUFU unit (one rsqrt a pair at 16 a clock and SM, 4.64e12 pairs/s; the six FP32
// operations alone would allow 5.9e12).  128^3 x 8,192 atoms: 4.38 ms = 3.93 Tpair/s, against 4.86 ms for a form
// with the atoms in pairs, eight FP32 operations a pair and whole rows per thread; 61 x 57 x 50 x 777 atoms: 59 us
// for the call against 174; rows of 1 point, 447 x 447 of them, x 3,000 atoms: 1.30 ms against 1.75.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "coul_internal.h"

namespace coul {

constexpr int kAdjThreads = 128;

// Shapes of the kernel by the grid columns X a thread holds in registers: rows per staged block and resident
// CTAs per SM.  32 columns share a row's dy^2 + dz^2, its sums and its loads of G among twice as many pairs as
// 16, which stay for row lengths that 32 would pad (16 warps of 126 registers against 20 of 94).  SHORT, us with
// 3,000 atoms and 200,000 points, against the form with whole rows per thread: 4 columns, rows of 1, 2, 4 points
// 1,300, 660, 340 (1,744, 1,044, 668); 8, rows of 8 256 (502); 16, rows of 16 211 (418); 24, rows of 24 205 (393).
template <int X, bool SHORT>
struct AdjShape {
    static constexpr int kRows = X == 24 ? 16 : 256 / X;
    static constexpr int kBlocksPerSm = X == 32 ? 4 : SHORT && X < 24 ? 6 : 5;
};
constexpr int kAdjFoldRows = 16;  // terms of a column sum before it goes into FP64
constexpr int kAdjReduceWarps = 8;

struct AdjParams {
    const float4* atoms;
    int64_t n_atoms;
    int nx, ny, nz;
    float h, ox, oy, oz;
    const float* grad_map;   // G, nx*ny*nz, x fastest
    double* partial;         // [chunks][n_atoms][4]: sum G/r, sum G dx/r^3, sum G dy/r^3, sum G dz/r^3
    int64_t rows_per_chunk;
    int chunks;
};

template <int X, bool SHORT>
__global__ void __launch_bounds__(kAdjThreads, AdjShape<X, SHORT>::kBlocksPerSm) adjoint_kernel(const AdjParams p)
{
    constexpr int kRows = AdjShape<X, SHORT>::kRows;
    constexpr int M = X / 2;                              // lane pairs of columns
    constexpr int C = SHORT ? 2 : 1;                      // chains of a row's sums
    constexpr int kPerThread = kRows * X / kAdjThreads;   // staged values per thread
    static_assert(kRows * X % kAdjThreads == 0 && X % 4 == 0 && kRows <= kAdjThreads, "block shape");
    // two buffers: a block is staged while slower warps still read the one before, one barrier a block
    __shared__ __align__(16) float s_g[2][kRows * X];
    __shared__ float2 s_row[2][kRows];  // the rows' (y, z)
    const int tid = threadIdx.x;
    const int64_t j = static_cast<int64_t>(blockIdx.x) * kAdjThreads + tid;
    // a thread past the last atom evaluates one far away and writes nothing
    const float4 a = j < p.n_atoms ? p.atoms[j] : make_float4(kPadCoord, kPadCoord, kPadCoord, 0.0f);
    const int64_t rows = static_cast<int64_t>(p.ny) * p.nz;
    const int64_t r_begin = static_cast<int64_t>(blockIdx.y) * p.rows_per_chunk;
    const int64_t r_end = r_begin + p.rows_per_chunk < rows ? r_begin + p.rows_per_chunk : rows;
    double tq = 0.0, tx = 0.0, ty = 0.0, tz = 0.0;

    // the next block's values travel through registers while the current one is evaluated
    float next[kPerThread];
    auto fetch = [&](int64_t row0, int x0) {
#pragma unroll
        for (int i = 0; i < kPerThread; ++i) {
            const int e = tid + i * kAdjThreads;
            const int64_t row = row0 + e / X;
            const int x = x0 + e % X;
            next[i] = row < r_end && x < p.nx ? p.grad_map[row * p.nx + x] : 0.0f;
        }
    };
    fetch(r_begin, 0);
    int buf = 0;
    for (int x0 = 0; x0 < p.nx; x0 += X) {
        float2 dx[M], s3x[M];
#pragma unroll
        for (int m = 0; m < M; ++m) {
            float d[2];
#pragma unroll
            for (int l = 0; l < 2; ++l) {
                const int x = x0 + 2 * m + l;
                // a column past the row's end lies far away (its staged G is zero)
                d[l] = (x < p.nx ? fmaf(static_cast<float>(x), p.h, p.ox) : kPadCoord) - a.x;
            }
            dx[m] = make_float2(d[0], d[1]);
            s3x[m] = make_float2(0.0f, 0.0f);
        }
        // the column sums into FP64: at the end of the rows, and every kAdjFoldRows rows
        auto fold_x = [&]() {
            float2 sx[4];
#pragma unroll
            for (int m = 0; m < M; ++m) {
                sx[m % 4] = m < 4 ? __fmul2_rn(dx[m], s3x[m]) : __ffma2_rn(dx[m], s3x[m], sx[m % 4]);
                s3x[m] = make_float2(0.0f, 0.0f);
            }
            const float2 sum = __fadd2_rn(__fadd2_rn(sx[0], sx[1]), __fadd2_rn(sx[2 % M], sx[3 % M]));
            tx += static_cast<double>(sum.x + sum.y);
        };
        int unfolded = 0;
        for (int64_t row0 = r_begin; row0 < r_end; row0 += kRows) {
            const int count = static_cast<int>(r_end - row0 < kRows ? r_end - row0 : kRows);
            buf ^= 1;
#pragma unroll
            for (int i = 0; i < kPerThread; ++i)
                s_g[buf][tid + i * kAdjThreads] = next[i];
            if (tid < count) {
                const int64_t row = row0 + tid;
                s_row[buf][tid] = make_float2(fmaf(static_cast<float>(static_cast<int>(row % p.ny)), p.h, p.oy),
                                         fmaf(static_cast<float>(static_cast<int>(row / p.ny)), p.h, p.oz));
            }
            __syncthreads();
            if (row0 + kRows < r_end)
                fetch(row0 + kRows, x0);
            else
                fetch(r_begin, x0 + X);
            float2 sq = make_float2(0.0f, 0.0f);
            float sy = 0.0f, sz = 0.0f;
            for (int r = 0; r < count; ++r) {
                const float2 yz = s_row[buf][r];
                const float dy = yz.x - a.y;
                const float dz = yz.y - a.z;
                const float2 dyz2 = splat(fmaf(dy, dy, dz * dz));
                const float4* g4 = reinterpret_cast<const float4*>(s_g[buf] + r * X);
                float2 q[C], s3[C], sx[C];  // the row's sums
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    const float4 gq = g4[m / 2];
                    const float2 g = m & 1 ? make_float2(gq.z, gq.w) : make_float2(gq.x, gq.y);
                    const float2 r2 = __ffma2_rn(dx[m], dx[m], dyz2);
                    const float2 inv = rsqrt_mufu_x2(r2);
                    const float2 t = __fmul2_rn(g, inv);  // not 1/r^3 first: it leaves FP32's range before G/r^3 does
                    const float2 inv2 = __fmul2_rn(inv, inv);
                    q[m % C] = m < C ? t : __fadd2_rn(q[m % C], t);
                    if constexpr (SHORT) {
                        const float2 t3 = __fmul2_rn(t, inv2);
                        s3[m % C] = m < C ? t3 : __fadd2_rn(s3[m % C], t3);
                        sx[m % C] = m < C ? __fmul2_rn(t3, dx[m]) : __ffma2_rn(t3, dx[m], sx[m % C]);
                    } else {
                        s3x[m] = __ffma2_rn(t, inv2, s3x[m]);
                        s3[m % C] = m < C ? __fmul2_rn(t, inv2) : __ffma2_rn(t, inv2, s3[m % C]);
                    }
                }
                const float2 qr = SHORT ? __fadd2_rn(q[0], q[C - 1]) : q[0];
                const float2 v2 = SHORT ? __fadd2_rn(s3[0], s3[C - 1]) : s3[0];
                const float v = v2.x + v2.y;
                if constexpr (SHORT) {
                    const float2 xr = __fadd2_rn(sx[0], sx[C - 1]);
                    tq += static_cast<double>(qr.x + qr.y);
                    tx += static_cast<double>(xr.x + xr.y);
                    ty = fma(static_cast<double>(dy), static_cast<double>(v), ty);
                    tz = fma(static_cast<double>(dz), static_cast<double>(v), tz);
                } else {
                    sq = __fadd2_rn(sq, qr);
                    sy = fmaf(dy, v, sy);
                    sz = fmaf(dz, v, sz);
                }
            }
            if constexpr (!SHORT) {
                tq += static_cast<double>(sq.x + sq.y);
                ty += static_cast<double>(sy);
                tz += static_cast<double>(sz);
                unfolded += kRows;
                if (unfolded >= kAdjFoldRows) {
                    fold_x();
                    unfolded = 0;
                }
            }
        }
        if constexpr (!SHORT)
            fold_x();
    }
    if (j < p.n_atoms) {
        double2* dst = reinterpret_cast<double2*>(p.partial + (static_cast<int64_t>(blockIdx.y) * p.n_atoms + j) * 4);
        dst[0] = make_double2(tq, tx);
        dst[1] = make_double2(ty, tz);
    }
}

// dq_j = sum over chunks of the partial sum; dr_j = q_j * (sum of the three position partials).  A
// warp's lanes are the 4 components of 8 consecutive atoms (256 contiguous bytes of each chunk); warp
// w of the block adds the chunks w, w + 8, ... in order, then the warps' sums are added in warp order.
// One thread per atom over all chunks took as long as the gradient itself for a small molecule.
__global__ void __launch_bounds__(32 * kAdjReduceWarps) adjoint_reduce_kernel(
    const float4* __restrict__ atoms, const double* __restrict__ partial, int64_t n, int chunks,
    float* __restrict__ grad_q, float* __restrict__ grad_xyz, float4* __restrict__ grad)
{
    __shared__ double s_sum[kAdjReduceWarps][32];
    const int lane = threadIdx.x % 32;
    const int warp = threadIdx.x / 32;
    const int64_t e = static_cast<int64_t>(blockIdx.x) * 32 + lane;  // element (atom, component)
    double s = 0.0;
    if (e < 4 * n) {
#pragma unroll 8
        for (int c = warp; c < chunks; c += kAdjReduceWarps)
            s += partial[static_cast<int64_t>(c) * 4 * n + e];
    }
    s_sum[warp][lane] = s;
    __syncthreads();
    if (warp != 0 || e >= 4 * n)
        return;
    s = s_sum[0][lane];
#pragma unroll
    for (int w = 1; w < kAdjReduceWarps; ++w)
        s += s_sum[w][lane];
    const int64_t j = e / 4;
    const int k = static_cast<int>(e % 4);
    const float v = static_cast<float>(k == 0 ? s : static_cast<double>(atoms[j].w) * s);
    if (grad)
        reinterpret_cast<float*>(grad)[4 * j + (k == 0 ? 3 : k - 1)] = v;  // (dx, dy, dz, dq)
    if (k == 0 && grad_q)
        grad_q[j] = v;
    if (k != 0 && grad_xyz)
        grad_xyz[3 * j + k - 1] = v;
}

}  // namespace coul

using namespace coul;

template <int X, bool SHORT>
static void launch_adjoint(const AdjParams& p, int64_t tiles, cudaStream_t stream)
{
    adjoint_kernel<X, SHORT><<<dim3(static_cast<unsigned>(tiles), static_cast<unsigned>(p.chunks)), kAdjThreads, 0, stream>>>(p);
}

// The kernel for rows of nx points.
struct AdjForm {
    void (*launch)(const AdjParams&, int64_t, cudaStream_t);
    int blocks_per_sm;
};

template <int X, bool SHORT>
static AdjForm adjoint_form()
{
    return AdjForm{&launch_adjoint<X, SHORT>, AdjShape<X, SHORT>::kBlocksPerSm};
}

static AdjForm adjoint_form(int64_t nx)
{
    if (nx <= 24)  // the fewest columns that hold a row
        return nx <= 4 ? adjoint_form<4, true>() : nx <= 8 ? adjoint_form<8, true>() : nx <= 16 ? adjoint_form<16, true>() : adjoint_form<24, true>();
    // 32 columns a thread unless they pad the rows by more than the 4 % they gain over 16
    const auto padded = [&](int64_t x) { return (nx + x - 1) / x * x; };
    return padded(32) * 100 <= padded(16) * 104 ? adjoint_form<32, false>() : adjoint_form<16, false>();
}

// The call of both entry points: any of the three outputs may be NULL.
static int adjoint_3d(coul_ctx* ctx, const float* d_atoms, int64_t n_atoms, const coul_grid* grid, const float* d_grad_map,
                      float* d_grad_q, float* d_grad_xyz, float* d_grad)
{
    if (ctx == nullptr)
        return set_error(COUL_ERR_INVALID_ARGUMENT, "ctx is NULL");
    int rc = validate_grid(grid);
    if (rc)
        return rc;
    if (n_atoms < 0 || d_grad_map == nullptr || (n_atoms > 0 && (d_atoms == nullptr || !aligned16(d_atoms))) ||
        (d_grad_q == nullptr && d_grad_xyz == nullptr && d_grad == nullptr))
        return set_error(COUL_ERR_INVALID_ARGUMENT, "bad atoms, gradient map or outputs");
    if (n_atoms == 0)
        return COUL_OK;
    if ((rc = ctx_activate(ctx)))
        return rc;

    const int64_t tiles = (n_atoms + kAdjThreads - 1) / kAdjThreads;
    const int64_t rows = static_cast<int64_t>(grid->ny) * grid->nz;
    const AdjForm form = adjoint_form(grid->nx);
    // Equal (tile, chunk) CTAs in whole waves of the resident ones, rounded down so that no wave is
    // nearly empty: as many waves (at most 8; the SMs' warps drift apart within one) as leave a chunk
    // 32 rows, else one wave.
    const int64_t slots = static_cast<int64_t>(ctx->sm_count) * form.blocks_per_sm;
    int64_t chunks = 1;
    for (int64_t waves = 8; waves >= 1; --waves) {
        chunks = std::max<int64_t>(1, waves * slots / tiles);
        if (rows / chunks >= 32)
            break;
    }
    chunks = std::max<int64_t>(1, std::min<int64_t>(chunks, std::min<int64_t>((rows + 3) / 4, 65535)));
    const int64_t rows_per_chunk = (rows + chunks - 1) / chunks;
    chunks = (rows + rows_per_chunk - 1) / rows_per_chunk;
    if (tiles > 2147483647LL)
        return set_error(COUL_ERR_DEVICE_LIMITS, "too many atoms");

    void* partial = nullptr;
    bool own = false;
    if ((rc = workspace_begin(ctx, kWorkspaceAdjoint,
                              static_cast<size_t>(chunks) * static_cast<size_t>(n_atoms) * 4 * sizeof(double), "adjoint",
                              &partial, &own)))
        return rc;

    AdjParams p{};
    p.atoms = reinterpret_cast<const float4*>(d_atoms);
    p.n_atoms = n_atoms;
    p.nx = grid->nx;
    p.ny = grid->ny;
    p.nz = grid->nz;
    p.h = grid->spacing;
    p.ox = grid->origin[0];
    p.oy = grid->origin[1];
    p.oz = grid->origin[2];
    p.grad_map = d_grad_map;
    p.partial = static_cast<double*>(partial);
    p.rows_per_chunk = rows_per_chunk;
    p.chunks = static_cast<int>(chunks);
    if ((rc = ctx_begin_timing(ctx)))
        return workspace_fail(ctx, rc);
    cudaError_t e;
    form.launch(p, tiles, ctx->stream);
    if ((e = cudaGetLastError()) != cudaSuccess)
        return workspace_fail(ctx, cuda_error(e, "adjoint launch"));
    adjoint_reduce_kernel<<<static_cast<unsigned>((n_atoms + 7) / 8), 32 * kAdjReduceWarps, 0, ctx->stream>>>(
        p.atoms, p.partial, n_atoms, p.chunks, d_grad_q, d_grad_xyz, reinterpret_cast<float4*>(d_grad));
    if ((e = cudaGetLastError()) != cudaSuccess)
        return workspace_fail(ctx, cuda_error(e, "adjoint reduction launch"));
    return ctx_end_timing(ctx);
}

extern "C" {

COUL_API int coul_adjoint_3d(coul_ctx* ctx, const float* d_atoms, int64_t n_atoms, const coul_grid* grid,
                             const float* d_grad_map, float* d_grad_q, float* d_grad_xyz)
{
    return adjoint_3d(ctx, d_atoms, n_atoms, grid, d_grad_map, d_grad_q, d_grad_xyz, nullptr);
}

COUL_API int coul_adjoint_3d_packed(coul_ctx* ctx, const float* d_atoms, int64_t n_atoms, const coul_grid* grid,
                                    const float* d_grad_map, float* d_grad)
{
    return adjoint_3d(ctx, d_atoms, n_atoms, grid, d_grad_map, nullptr, nullptr, d_grad);
}

}  // extern "C"
