"""Maps and slices of calls that name no configuration (coul_forward_3d_plain, coul_forward_2d_plain):
against the FP64 oracle at the edges of tiles (64 x-y points by 16 or 8 planes, 4 x 4 points by 32
columns), of the atom batches and shares (32 atoms, 8 warps, 1 .. 8 CTAs a tile) and of the FMA-pipe
share (512 atoms); run-to-run and slab equality bit for bit; accumulation.

Tolerance: an FP32 pair term is good to 4.6e-7 (the FMA-pipe root) plus three FP32 roundings, and a sum
of n terms in eight or more parts rounds by less than n / 8 * 2^-24 of its largest partial sum; with
the charges' random signs both stay below 1e-5 of the largest value for the sizes here."""
import numpy as np
import pytest

import oracle
from ktt_b200 import errors
import ktt_b200

pytestmark = pytest.mark.gpu

TOL = 1e-5


def _atoms(n, seed, box=20.0):
    rng = np.random.default_rng(seed)
    a = np.empty((n, 4), dtype=np.float32)
    a[:, :3] = rng.uniform(0.0, box, (n, 3))
    a[:, 3] = rng.uniform(-1.0, 1.0, n)
    return a


def _cuda(a):
    import torch
    return torch.from_numpy(a).cuda() if a.shape[0] else torch.zeros((0, 4), device="cuda")


@pytest.mark.parametrize("n", [0, 1, 31, 211, 511, 512, 2049])
@pytest.mark.parametrize("dims", [(1, 1, 1), (63, 1, 8), (64, 2, 9), (65, 3, 16), (37, 41, 33), (130, 90, 70)])
def test_plain_map(ctx, dims, n):
    import torch
    a, h, origin = _atoms(n, seed=n + dims[0]), 0.5, (-1.0, 0.5, 2.0)
    out = torch.full((dims[2], dims[1], dims[0]), float("nan"), device="cuda")
    ctx.forward_3d(_cuda(a), dims, h, origin, out=out)
    if n == 0:
        assert torch.count_nonzero(out) == 0
    else:
        assert errors.report(out.cpu().numpy(), oracle.grid3d(a, h, dims, origin))["rel_norm"] <= TOL
    assert torch.equal(out, ctx.forward_3d(_cuda(a), dims, h, origin))
    base = torch.linspace(-2, 2, out.numel(), device="cuda").reshape(out.shape)
    acc = base.clone()
    ctx.forward_3d(_cuda(a), dims, h, origin, out=acc, accumulate=True)
    assert torch.equal(acc, base + out)
    # slabs at any boundary, whatever the tiles' depth
    cuts = sorted({0, dims[2] // 3, dims[2] // 2 + 1 if dims[2] > 2 else 0, dims[2]})
    parts = [ctx.forward_3d_slab(_cuda(a), dims, h, z0, z1, origin) for z0, z1 in zip(cuts, cuts[1:])]
    assert torch.equal(torch.cat(parts), out)


@pytest.mark.parametrize("n", [0, 1, 33, 511, 513, 4000])
@pytest.mark.parametrize("shape", [(1, 1), (127, 3), (128, 4), (129, 5), (250, 187), (3, 1000)])
def test_plain_slice(ctx, shape, n):
    import torch
    a, h = _atoms(n, seed=n + shape[0]), 0.5
    a[:, 2] = (np.float32(7.3) - a[:, 2]) ** 2
    out = torch.full((shape[1], shape[0]), float("nan"), device="cuda")
    ctx.forward_2d(_cuda(a), h, shape[0], shape[1], out=out)
    if n == 0:
        assert torch.count_nonzero(out) == 0
    else:
        assert errors.report(out.cpu().numpy(), oracle.slice2d(a, h, shape[0], shape[1]))["rel_norm"] <= TOL
    assert torch.equal(out, ctx.forward_2d(_cuda(a), h, shape[0], shape[1]))
    base = torch.linspace(-2, 2, out.numel(), device="cuda").reshape(out.shape)
    acc = base.clone()
    ctx.forward_2d(_cuda(a), h, shape[0], shape[1], out=acc, accumulate=True)
    assert torch.equal(acc, base + out)


def test_plain_call_keeps_the_refusals(ctx):
    import torch
    a = _cuda(_atoms(8, seed=1))
    flat = torch.zeros(33, device="cuda")
    with pytest.raises(ktt_b200.CoulombError) as e:
        ctx.forward_3d(flat[1:].view(-1, 4), (8, 8, 8), 0.5)  # 4-byte offset: not 16-byte aligned
    assert e.value.status == ktt_b200.COUL_ERR_INVALID_ARGUMENT
    with pytest.raises(ktt_b200.CoulombError) as e:
        ctx.forward_3d(a, (1, 262141, 1), 0.5)
    assert e.value.status == ktt_b200.COUL_ERR_DEVICE_LIMITS
    for z0, z1 in ((-1, 4), (5, 5), (6, 3), (0, 9)):
        with pytest.raises(ktt_b200.CoulombError):
            ctx.forward_3d_slab(a, (8, 8, 8), 0.5, z0, z1, out=torch.empty((max(z1 - z0, 1), 8, 8), device="cuda"))


@pytest.mark.parametrize("n", [0, 1, 33, 300, 700])
@pytest.mark.parametrize("dims", [(1, 1, 1), (63, 2, 8), (65, 1, 9), (37, 41, 17), (130, 40, 31)])
@pytest.mark.parametrize("shape,soft", [((8, 2, 2), 2), ((8, 2, 1), 0), ((16, 2, 1), 12), ((8, 2, 1), 5)])
def test_fp32_configurations_on_the_plain_kernel(ctx, n, dims, shape, soft):
    """FP32 configurations of 8 x 2 and 16 x 2 points on a small map: a warp's sum of n / 8 terms, each
    with the root's error (2.3e-7 rms, bias below 2^-21) and 2^-24 a step: below n / 8 * 2^-24 + 1e-6 of the
    point's sum |q| / r.  Slabs at multiples of the configuration's depth equal the map; a sum adds to out."""
    import torch
    rng = np.random.default_rng(n + dims[0])
    a = np.empty((n, 4), dtype=np.float32)
    a[:, :3] = rng.uniform(0.0, 20.0, (n, 3))
    a[:, 3] = rng.uniform(0.1, 1.0, n)
    h, origin = 0.5, (-1.0, 0.5, 2.0)
    tune = ktt_b200.Tune(block_x=64, block_y=1, z_iterations=shape[0], x_points=shape[1], unroll=shape[2],
                         rsqrt_soft=soft)
    atoms = torch.from_numpy(a).cuda() if n else torch.zeros((0, 4), device="cuda")
    out = torch.full((dims[2], dims[1], dims[0]), float("nan"), device="cuda")
    ctx.forward_3d(atoms, dims, h, origin, tune=tune, out=out)
    if n == 0:
        assert torch.count_nonzero(out) == 0
        return
    ref = oracle.grid3d(a, h, dims, origin)
    assert np.max(np.abs(out.cpu().numpy() - ref) / np.abs(ref)) <= n / 8 * 2.0**-24 + 1e-6
    if dims[2] > shape[0]:
        slab = ctx.forward_3d_slab(atoms, dims, h, shape[0], dims[2], origin, tune=tune)
        assert torch.equal(slab, out[shape[0]:])
    base = torch.linspace(-2, 2, out.numel(), device="cuda").reshape(out.shape)
    acc = base.clone()
    ctx.forward_3d(atoms, dims, h, origin, tune=tune, out=acc, accumulate=True)
    assert torch.equal(acc, base + out)


def _places(n, seed):
    """n atoms of which 32 lie on grid points (spacing 0.5, origin 0), one for every place in a tile of 2 x 16
    points a thread, and 8 without charge lie beyond FP32's r^2: what pads a molecule."""
    a = _atoms(n, seed)
    rng = np.random.default_rng(seed + 1)
    pick = rng.permutation(n)
    for i in range(32):
        a[pick[i], :3] = 0.5 * np.array([i, i % 7, (5 * i + i // 16) % 16])
    far = np.array([[1e20, 0, 0], [0, -1e20, 0], [0, 0, 1e20], [np.inf, 1, 2], [1, -np.inf, 2], [1, 2, np.inf],
                    [3e38, 3e38, 3e38], [-np.inf, np.inf, -np.inf]], dtype=np.float32)
    a[pick[32:40], :3] = far
    a[pick[32:40], 3] = 0.0
    return a, pick[:32]


def _check_places(out, a, hits, exact):
    """`out` (last axis x, spacing 0.5) is q * inf on the atoms `hits` and the exact map elsewhere."""
    at = np.round(a[hits, :3] * 2).astype(int)
    mask = np.zeros(out.shape, dtype=bool)
    for (x, y, z), q in zip(at, a[hits, 3]):
        index = (z, y, x) if out.ndim == 3 else (y, x)
        assert out[index] == np.copysign(np.inf, q), (x, y, z)
        mask[index] = True
    assert np.all(np.isfinite(out[~mask]))
    ref = exact[~mask]
    assert np.linalg.norm(out[~mask] - ref) <= TOL * np.linalg.norm(ref)


@pytest.mark.parametrize("n", [100, 511, 512, 2049])
@pytest.mark.parametrize("dims", [(40, 9, 16), (37, 13, 41), (96, 64, 48)])
@pytest.mark.parametrize("fields", [None, dict(z_iterations=8, x_points=2, unroll=2, rsqrt_soft=2),
                                    dict(z_iterations=16, x_points=2, rsqrt_soft=12, precision=4)])
def test_atoms_on_grid_points_and_beyond_range(ctx, dims, n, fields):
    """A point on an atom is +-inf and an atom without charge adds nothing wherever it lies, also where a pair's
    root runs on the FMA pipe, whose arithmetic holds for r^2 in 2^-100 .. 2^101 only."""
    import torch
    a, hits = _places(n, n)
    tune = ktt_b200.Tune(block_x=16, block_y=2, **fields) if fields else None
    out = ctx.forward_3d(_cuda(a), dims, 0.5, tune=tune)
    with np.errstate(divide="ignore"):
        ref = oracle.grid3d(np.delete(a, np.where(a[:, 3] == 0)[0], axis=0), 0.5, dims)
    _check_places(out.cpu().numpy(), a, hits, ref)
    if dims[2] > 16:
        assert torch.equal(ctx.forward_3d_slab(_cuda(a), dims, 0.5, 16, dims[2], tune=tune), out[16:])
    if fields and n == 512:
        batch = ktt_b200.Batch(ctx, [(_cuda(a), dims, 0.5, (0.0, 0.0, 0.0))],
                               ktt_b200.Tune(block_x=7, block_y=3, z_iterations=16, x_points=2, rsqrt_soft=12, precision=4))
        batch.run()
        ctx.synchronize()
        _check_places(batch.outputs[0].cpu().numpy(), a, hits, ref)
        batch.close()


@pytest.mark.parametrize("n", [100, 511, 512, 2049])
def test_atoms_on_slice_points_and_beyond_range(ctx, n):
    a, hits = _places(n, n)
    flat = a.copy()
    with np.errstate(over="ignore"):
        flat[:, 2] = (np.float32(7.3) - a[:, 2]) ** 2
    flat[hits, 2] = 0.0
    flat[hits, 1] = 0.5 * (np.arange(32) % 7)
    out = ctx.forward_2d(_cuda(flat), 0.5, 61, 30).cpu().numpy()
    with np.errstate(divide="ignore"):
        ref = oracle.slice2d(np.delete(flat, np.where(flat[:, 3] == 0)[0], axis=0), 0.5, 61, 30)
    _check_places(out, flat, hits, ref)


@pytest.mark.parametrize("n", [600, 3000])
def test_atoms_closer_than_the_range_of_the_root(ctx, n):
    """Distances whose square is small, subnormal or zero in FP32, at the origin's point: MUFU's value, which
    flushes a subnormal r^2 to zero.  One charge near the point dominates it by 1e10 and more."""
    a = _atoms(n, seed=n) + np.array([1, 1, 1, 0], dtype=np.float32)
    for k in range(32):  # the point's place in its tile
        origin = (-0.5 * (k % 2), 0.0, -0.5 * (k // 2))
        for r, want in ((1e-14, 1e14), (3e-16, 1 / 3e-16), (1e-18, 1e18), (1e-20, np.inf), (1e-30, np.inf)):
            a[7] = ((0.0, 0.0, r, 1.0), (r, 0.0, 0.0, 1.0))[k % 2]
            got = ctx.forward_3d(_cuda(a), (96, 64, 32), 0.5, origin)[k // 2, 0, k % 2].item()
            assert got == want or abs(got / want - 1) <= 1e-6, (k, r)


@pytest.mark.parametrize("fields", [None, dict(z_iterations=16, x_points=2, rsqrt_soft=12, precision=2),
                                    dict(z_iterations=16, x_points=2, rsqrt_soft=2, precision=4)])
def test_root_of_one_pair_at_mufu_precision(ctx, fields):
    """One charge of 1 among 600 charge-free atoms, every coordinate a multiple of 1/16 below 64: differences of
    10 bits, r^2 exact in FP32, the sum the root itself.  rsqrt.approx's documented bound, 2^-22.9, holds for every
    root of a call whose caller did not choose another; with FP64 sums also in a batch."""
    rng = np.random.default_rng(5)
    dims, h = (80, 64, 48), 0.5
    gz, gy, gx = np.meshgrid(*(np.arange(d) * h for d in dims[::-1]), indexing="ij")
    tune = ktt_b200.Tune(block_x=16, block_y=2, **fields) if fields else None
    for i in range(8):
        a = np.zeros((600, 4), dtype=np.float32)
        a[:, :3] = (2 * rng.integers(0, 8 * 32, (600, 3)) + 1) / 16
        j = int(rng.integers(0, 600))
        a[j, 3] = 1.0
        exact = 1.0 / np.sqrt((gx - a[j, 0]) ** 2 + (gy - a[j, 1]) ** 2 + (gz - a[j, 2]) ** 2)
        maps = [ctx.forward_3d(_cuda(a), dims, h, tune=tune).cpu().numpy()]
        if fields and fields["precision"] == 4:
            batch = ktt_b200.Batch(ctx, [(_cuda(a), dims, h, (0.0, 0.0, 0.0))],
                                   ktt_b200.Tune(block_x=8, block_y=4, **dict(fields, rsqrt_soft=12)))
            batch.run()
            ctx.synchronize()
            maps.append(batch.outputs[0].cpu().numpy())
            batch.close()
        if fields is None:
            flat = a.copy()
            flat[:, 2] = a[:, 2] ** 2
            maps.append(ctx.forward_2d(_cuda(flat), h, dims[0], dims[1]).cpu().numpy())
        for v in maps:
            assert np.max(np.abs(v / (exact if v.ndim == 3 else exact[0]) - 1)) <= 2.0**-22.9 + 2.0**-30


@pytest.mark.parametrize("h,origin", [(0.5, (-7.25, 3.0, 1e3)), (0.01, (1e6, -1e6, 1e6)), (0.01, (0.0, 3e4, 0.0)),
                                      (2.0**-44, (0.0, 0.0, 0.0)), (-0.5, (9.0, 9.0, 9.0)), (1e3, (-2e4, 0.0, 1e5))])
@pytest.mark.parametrize("dims", [(40, 9, 16), (97, 40, 33)])
@pytest.mark.parametrize("fields", [None, dict(z_iterations=16, x_points=2, rsqrt_soft=12, precision=4)])
def test_atoms_on_points_of_fine_and_far_grids(ctx, h, origin, dims, fields):
    """Eight charges of 1 on grid points among 600 atoms, some of them in a plane or a column of the grid: +inf at every
    point whose FP32 coordinates equal a charge's (several, where the spacing is finer than the origin's rounding), the
    oracle's value elsewhere."""
    rng = np.random.default_rng(dims[0])
    g = [(np.arange(d) * np.float64(np.float32(h)) + np.float64(np.float32(o))).astype(np.float32)
         for d, o in zip(dims, origin)]
    lo = np.array([min(x[0], x[-1]) for x in g], dtype=np.float64)
    hi = np.array([max(x[0], x[-1]) for x in g], dtype=np.float64)
    a = np.zeros((600, 4), dtype=np.float32)
    a[:, :3] = lo + (hi - lo) * rng.uniform(-0.3, 1.3, (600, 3))
    a[:, 3] = rng.uniform(-1.0, 1.0, 600)
    for j in range(100):  # in one or two of a point's coordinates
        for c in ((2,), (0, 1), (1, 2), (0, 2))[j % 4]:
            a[j, c] = rng.choice(g[c])
    a[600 - 8:, :3] = np.stack([rng.choice(x, 8) for x in g], 1)
    a[600 - 8:, 3] = 1.0
    tune = ktt_b200.Tune(block_x=16, block_y=2, **fields) if fields else None
    out = ctx.forward_3d(_cuda(a), dims, h, origin, tune=tune).cpu().numpy()
    hit = np.zeros(dims[::-1], dtype=bool)
    for x, y, z, q in a:
        hit |= (g[2] == z)[:, None, None] & (g[1] == y)[None, :, None] & (g[0] == x)[None, None, :]
    assert hit.any()
    plus = np.zeros(dims[::-1], dtype=bool)
    for x, y, z, q in a[600 - 8:]:
        plus |= (g[2] == z)[:, None, None] & (g[1] == y)[None, :, None] & (g[0] == x)[None, None, :]
    only = plus & np.isposinf(out)
    assert np.array_equal(only, plus) or (hit & ~plus).any()
    assert np.all(np.isfinite(out[~hit]))
    with np.errstate(divide="ignore", invalid="ignore"):
        ref = oracle.grid3d(a, h, dims, origin)
    assert np.linalg.norm(out[~hit] - ref[~hit]) <= TOL * np.linalg.norm(ref[~hit])
