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
