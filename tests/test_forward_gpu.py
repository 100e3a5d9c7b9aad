"""Parity of the sm_100a forward kernels with the FP64 oracle (and KTT's golden output).

Tolerances: every form stays within 1e-5 relative error normwise (max|dV| / max|V*|) of the FP64
oracle; the precise forms also pointwise, max|dV| / max(|V*|, floor) <= 1e-5, at the floors of
ktt_b200/errors.py (rms(V*) for the FP32-pair forms with compensated or FP64-merged sums, 1e-3 rms(V*)
for FP64 pairs).  KTT's own known-answer threshold is 0.01 absolute
(Examples/JSON/CoulombSum3d.json:172-181).
"""
import json
import os

import numpy as np
import pytest

import oracle
from ktt_b200 import errors, workloads
import ktt_b200

pytestmark = pytest.mark.gpu

TOL_NORM = 1e-5


def _t(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _np(t):
    return t.detach().cpu().numpy()


@pytest.fixture(scope="module")
def kat(golden_dir):
    with open(os.path.join(golden_dir, "coulomb3d_kat.json")) as f:
        return json.load(f)


def test_kat_full_map_matches_reference_output(ctx, kat):
    cells = kat["cells"]
    atoms = oracle.kat_atoms(64)
    out = ctx.forward_3d(_t(atoms), (cells, cells, cells), kat["grid_spacing_f32"])
    ctx.synchronize()
    v = _np(out).reshape(-1)
    idx = np.asarray(kat["index"], dtype=np.int64)
    golden = np.asarray(kat["bits"], dtype=np.uint32).view(np.float32)
    assert np.max(np.abs(v[idx] - golden)) <= kat["validation_threshold"]
    ref = oracle.grid3d(atoms, kat["grid_spacing_f32"], (cells, cells, cells)).reshape(-1)
    rep = errors.report(v, ref)
    assert rep["rel_norm"] <= TOL_NORM, rep
    assert rep["rel_point"] <= 1e-5, rep


def test_slice2d_against_oracle_and_device_prep(ctx):
    w = workloads.slice_2d()
    ka = w.ktt_atoms()
    ref = oracle.slice2d(ka, w.spacing, w.nx, w.ny)
    got = _np(ctx.forward_2d(_t(ka), w.spacing, w.nx, w.ny))
    rep = errors.report(got, ref)
    assert rep["rel_norm"] <= TOL_NORM, rep
    dev = ctx.slice_atoms(_t(w.atoms), w.z_slice)
    assert np.array_equal(_np(dev).view(np.uint32), ka.view(np.uint32))


def _small_case(n_atoms=300, seed=7):
    rng = np.random.default_rng(seed)
    a = np.empty((n_atoms, 4), dtype=np.float32)
    a[:, :3] = rng.uniform(-2.0, 14.0, (n_atoms, 3))
    a[:, 3] = rng.uniform(-1, 1, n_atoms)
    return a, (37, 11, 19), 0.5, (-1.0, 2.0, 0.25)


@pytest.fixture(scope="module")
def small_ref():
    a, dims, h, origin = _small_case()
    return a, dims, h, origin, oracle.grid3d(a, h, dims, origin)


def test_every_3d_variant_on_ragged_grid(ctx, small_ref):
    import torch
    a, dims, h, origin, ref = small_ref
    ta = _t(a)
    soa = [_t(np.ascontiguousarray(a[:, k])) for k in range(4)]
    shapes = [(32, 4), (64, 2), (16, 8), (128, 1), (32, 1)]
    failures = []
    count = 0
    for i, (tune, is2d, is_soa) in enumerate(ktt_b200.variants()):
        if is2d:
            continue
        tune.block_x, tune.block_y = shapes[i % len(shapes)]
        out = torch.full((dims[2], dims[1], dims[0]), float("nan"), device="cuda")
        if is_soa:
            ctx.forward_3d_soa(*soa, dims, h, origin, tune=tune, out=out)
        else:
            ctx.forward_3d(ta, dims, h, origin, tune=tune, out=out)
        ctx.synchronize()
        rep = errors.report(_np(out), ref)
        if not rep["rel_norm"] <= TOL_NORM:
            failures.append((tune.as_dict(), is_soa, rep))
        count += 1
    assert count > 250
    assert not failures, failures[:5]


def test_every_2d_variant(ctx):
    import torch
    w = workloads.slice_2d(seed=9, n_atoms=333, n=45)
    ka = w.ktt_atoms()
    ref = oracle.slice2d(ka, w.spacing, 45, 29)
    ta = _t(ka)
    failures = []
    for i, (tune, is2d, _) in enumerate(ktt_b200.variants()):
        if not is2d:
            continue
        tune.block_x, tune.block_y = [(32, 4), (16, 2), (8, 8), (64, 1)][i % 4]
        out = torch.full((29, 45), float("nan"), device="cuda")
        ctx.forward_2d(ta, w.spacing, 45, 29, tune=tune, out=out)
        ctx.synchronize()
        rep = errors.report(_np(out), ref)
        if not rep["rel_norm"] <= TOL_NORM:
            failures.append((tune.as_dict(), rep))
    assert not failures, failures[:5]


@pytest.mark.parametrize("n_atoms", [0, 1, 3, 255, 256, 257, 513, 4097, 8195])
@pytest.mark.parametrize("form", ["tma", "soa", "const", "fp64", "comp"])
def test_ragged_atom_counts(ctx, n_atoms, form):
    import torch
    a, dims, h, origin = _small_case(n_atoms=max(n_atoms, 1), seed=n_atoms + 3)
    a = a[:n_atoms]
    ref = oracle.grid3d(a, h, dims, origin) if n_atoms else np.zeros(dims[::-1])
    tune = ktt_b200.Tune(block_x=32, block_y=2, z_iterations=4, x_points=2)
    out = torch.full((dims[2], dims[1], dims[0]), float("nan"), device="cuda")
    if form == "soa":
        cols = [_t(np.ascontiguousarray(a[:, k])) if n_atoms else torch.zeros(1, device="cuda") for k in range(4)]
        ctx.forward_3d_soa(*cols, dims, h, origin, tune=tune, out=out)
    else:
        if form == "const":
            tune.atom_source = ktt_b200.ATOMS_CONSTANT
        elif form == "fp64":
            tune.precision = ktt_b200.PREC_FP64_MERGE
        elif form == "comp":
            tune.precision = ktt_b200.PREC_COMPENSATED
        ta = _t(a) if n_atoms else torch.zeros((0, 4), device="cuda")
        ctx.forward_3d(ta, dims, h, origin, tune=tune, out=out)
    ctx.synchronize()
    got = _np(out)
    if n_atoms == 0:
        assert np.all(got == 0.0)
    else:
        rep = errors.report(got, ref)
        assert rep["rel_norm"] <= TOL_NORM, rep


def test_accumulate_semantics(ctx, small_ref):
    import torch
    a, dims, h, origin, ref = small_ref
    base = torch.linspace(-3, 3, dims[0] * dims[1] * dims[2], device="cuda").reshape(dims[2], dims[1], dims[0])
    out = base.clone()
    ctx.forward_3d(_t(a), dims, h, origin, out=out, accumulate=True)
    out2 = ctx.forward_3d(_t(a), dims, h, origin)
    ctx.synchronize()
    np.testing.assert_allclose(_np(out), _np(base) + _np(out2), rtol=0, atol=2e-6)
    # constant-memory path accumulates across its chunks and onto the caller's data
    out3 = base.clone()
    t = ktt_b200.Tune(atom_source=ktt_b200.ATOMS_CONSTANT, z_iterations=2, x_points=1)
    ctx.forward_3d(_t(a), dims, h, origin, tune=t, out=out3, accumulate=True)
    ctx.synchronize()
    np.testing.assert_allclose(_np(out3), _np(base) + ref, rtol=0, atol=1e-4)


def test_reference_kernel(ctx, small_ref):
    a, dims, h, origin, ref = small_ref
    out = ctx.forward_3d_reference(_t(a), dims, h, origin)
    ctx.synchronize()
    assert errors.report(_np(out), ref)["rel_norm"] <= TOL_NORM


def test_host_buffer_call_matches_device_call(ctx, small_ref):
    a, dims, h, origin, ref = small_ref
    host = ctx.forward_3d_host(a, dims, h, origin)
    dev = _np(ctx.forward_3d(_t(a), dims, h, origin))
    ctx.synchronize()
    assert np.array_equal(host, dev)


def test_invalid_arguments_rejected_before_launch(ctx, small_ref):
    import torch
    a, dims, h, origin, _ = small_ref
    ta = _t(np.concatenate([np.zeros(1, np.float32), a.reshape(-1)]))
    mis = ta[1:].view(-1, 4)  # 4-byte offset: not 16-byte aligned
    with pytest.raises(ktt_b200.CoulombError) as e:
        ctx.forward_3d(mis, dims, h, origin)
    assert e.value.status == ktt_b200.COUL_ERR_INVALID_ARGUMENT
    with pytest.raises(ktt_b200.CoulombError) as e:
        ctx.forward_3d(_t(a), dims, h, origin, tune=ktt_b200.Tune(z_iterations=3))
    assert e.value.status == ktt_b200.COUL_ERR_UNSUPPORTED
    with pytest.raises(ktt_b200.CoulombError) as e:
        ctx.forward_3d(_t(a), (0, 4, 4), h, origin)
    assert e.value.status == ktt_b200.COUL_ERR_INVALID_ARGUMENT
    ctx.synchronize()


def test_bounded_wait_expiry_is_reported_and_context_survives(ctx, small_ref):
    assert ctx.probe_bounded_wait(True, 10_000_000) == ktt_b200.COUL_OK
    assert ctx.probe_bounded_wait(False, 20_000_000) == ktt_b200.COUL_ERR_TIMEOUT
    # the context (and the device) stays usable
    a, dims, h, origin, ref = small_ref
    out = ctx.forward_3d(_t(a), dims, h, origin)
    ctx.synchronize()
    assert errors.report(_np(out), ref)["rel_norm"] <= TOL_NORM


def test_full_map_uniform_subset(ctx):
    """The benchmark's 256^3 x 65,536-atom map against FP64 on a seeded 0.1% subset: plain FP32
    normwise; the form bench.py benches (ktt_b200/tuned/b200_map3d.json) and the FP64-merge form
    normwise and pointwise at the gate floor; FP64 pairs pointwise at the strict floor."""
    w = workloads.uniform_map()
    ta = _t(w.atoms)
    total = int(np.prod(w.dims))
    idx = workloads.subset_indices(total, 0.001)
    ref, sabs = oracle.points3d(w.atoms, w.spacing, w.dims, idx, want_sumabs=True)
    bench_form = ktt_b200.tuned("b200_map3d")
    assert bench_form is not None and bench_form.precision in (ktt_b200.PREC_COMPENSATED, ktt_b200.PREC_FP64_MERGE,
                                                               ktt_b200.PREC_FP64_MERGE_SHARED)
    forms = [(ktt_b200.Tune(), "norm"),
             (ktt_b200.Tune(precision=ktt_b200.PREC_FP64_MERGE, z_iterations=8), "point"),
             (bench_form, "point"),
             (ktt_b200.Tune(block_x=64, block_y=1, z_iterations=8, x_points=4, precision=ktt_b200.PREC_FP64_PAIRS),
              "strict")]
    for tune, gate in forms:
        out = ctx.forward_3d(ta, w.dims, w.spacing, tune=tune)
        ctx.synchronize()
        rep = errors.gate(_np(out).reshape(-1)[idx], ref, sumabs=sabs)
        assert rep["passes_norm"], (tune, rep)
        if gate in ("point", "strict"):
            assert rep["passes_point"], (tune, rep)
        if gate == "strict":
            assert rep["passes_point_strict"], (tune, rep)


def test_precision_forms_on_the_clustered_map(ctx):
    """The cancellation-heavy map (65,536 atoms in 64 Gaussian clusters of alternating +1/-1 charges,
    net charge 0, sum |q|/r about 1000 |V|; 256^3 grid) against FP64 on a seeded 0.1% subset.  The
    compensated and FP64-merge forms (FP64 sums in registers or in shared memory) -- all rsqrts on
    MUFU, 2/8 on the FMA pipe, and the alternating 5/16 share -- meet the gate (1e-5 normwise and pointwise at the floor rms(V*)); FP64 pairs meet
    1e-5 pointwise at the strict floor (1e-3 rms(V*)); FP32 accumulation, with or without the FMA-pipe
    share, misses the pointwise gate, which is why the precise forms exist."""
    w = workloads.clustered_map()
    ta = _t(w.atoms)
    total = int(np.prod(w.dims))
    idx = workloads.subset_indices(total, 0.001, seed=23)
    ref, sabs = oracle.points3d(w.atoms, w.spacing, w.dims, idx, want_sumabs=True)
    tile = dict(block_x=64, block_y=1, z_iterations=8, x_points=2, unroll=2)
    precise = [dict(precision=p, rsqrt_soft=s) for p in (ktt_b200.PREC_COMPENSATED, ktt_b200.PREC_FP64_MERGE,
                                                          ktt_b200.PREC_FP64_MERGE_SHARED)
               for s in (0, 2, 12)]
    reports = {}
    for fields in precise + [dict(precision=ktt_b200.PREC_FP32, rsqrt_soft=s) for s in (0, 2)]:
        tune = ktt_b200.Tune(**tile, **fields)
        out = ctx.forward_3d(ta, w.dims, w.spacing, tune=tune)
        ctx.synchronize()
        reports[(fields["precision"], fields["rsqrt_soft"])] = errors.gate(_np(out).reshape(-1)[idx], ref, sumabs=sabs)
    for fields in precise:
        rep = reports[(fields["precision"], fields["rsqrt_soft"])]
        assert rep["passes_norm"] and rep["passes_point"], (fields, rep)
    for s in (0, 2):
        assert not reports[(ktt_b200.PREC_FP32, s)]["passes_point"], reports[(ktt_b200.PREC_FP32, s)]
    exact = ktt_b200.Tune(block_x=64, block_y=1, z_iterations=8, x_points=4, precision=ktt_b200.PREC_FP64_PAIRS)
    out = ctx.forward_3d(ta, w.dims, w.spacing, tune=exact)
    ctx.synchronize()
    rep = errors.gate(_np(out).reshape(-1)[idx], ref, sumabs=sabs)
    assert rep["passes_norm"] and rep["passes_point"] and rep["passes_point_strict"], rep


def test_fp64_pair_variants_on_a_ragged_grid(ctx):
    """Every compiled FP64-pair variant on a grid whose sides are not multiples of the tile, with an
    origin: the map equals the FP64 oracle to the rounding of its FP32 store (pointwise 2e-7 relative
    above a floor of 1e-6 rms(V*))."""
    rng = np.random.default_rng(41)
    n, dims, h, origin = 1337, (45, 29, 23), 0.5, (-3.25, 1.5, 0.75)
    a = np.empty((n, 4), dtype=np.float32)
    a[:, :3] = rng.uniform(-4.0, 24.0, (n, 3))
    a[:, 3] = rng.uniform(-1.0, 1.0, n)
    ref = oracle.grid3d(a, h, dims, origin)
    rms = float(np.sqrt(np.mean(ref * ref)))
    count = 0
    for tune, is2d, is_soa in ktt_b200.variants():
        if is2d or is_soa or tune.precision != ktt_b200.PREC_FP64_PAIRS:
            continue
        tune.block_x, tune.block_y = 32, 4
        out = ctx.forward_3d(_t(a), dims, h, origin, tune=tune)
        ctx.synchronize()
        rep = errors.report(_np(out), ref, floor=1e-6 * rms)
        assert rep["rel_point"] <= 2e-7, (tune.as_dict(), rep)
        count += 1
    assert count >= 16


@pytest.mark.parametrize("tune", [
    dict(block_x=32, block_y=1, z_iterations=8, x_points=2, unroll=2, rsqrt_soft=2),
    dict(block_x=32, block_y=4, z_iterations=8, x_points=2, unroll=1, rsqrt_soft=12),
    dict(block_x=64, block_y=2, z_iterations=16, x_points=1, unroll=1, rsqrt_soft=0),
    dict(block_x=16, block_y=8, z_iterations=4, x_points=4, unroll=1, rsqrt_soft=3),
])
def test_fp64_merge_shared_sums_equal_register_sums(ctx, tune):
    """The FP64 merge with its sums in shared memory is the same arithmetic as with the sums in
    registers: the maps agree bit for bit, and both meet the FP64 oracle."""
    import torch
    rng = np.random.default_rng(41)
    a = np.zeros((5000, 4), dtype=np.float32)
    a[:, :3] = rng.uniform(0.0, 30.0, (5000, 3))
    a[:, 3] = rng.uniform(-1.0, 1.0, 5000)
    dims, h, origin = (61, 37, 45), 0.5, (0.3, -0.2, 1.0)
    atoms = torch.from_numpy(a).cuda()
    reg = ctx.forward_3d(atoms, dims, h, origin, tune=ktt_b200.Tune(precision=ktt_b200.PREC_FP64_MERGE, **tune))
    shr = ctx.forward_3d(atoms, dims, h, origin,
                         tune=ktt_b200.Tune(precision=ktt_b200.PREC_FP64_MERGE_SHARED, **tune))
    assert torch.equal(reg, shr)
    ref = oracle.grid3d(a, h, dims, origin)
    assert errors.report(shr.cpu().numpy(), ref)["rel_norm"] <= 1e-5


@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 300, 1), (131, 3, 9), (129, 7, 17), (257, 2, 8), (96, 33, 5)])
@pytest.mark.parametrize("tune", [
    ktt_b200.Tune(block_x=64, block_y=1, z_iterations=8, x_points=2, unroll=2, rsqrt_soft=2),
    ktt_b200.Tune(block_x=64, block_y=1, z_iterations=8, x_points=4, precision=ktt_b200.PREC_FP64_PAIRS),
    ktt_b200.Tune(block_x=7, block_y=3, z_iterations=4, x_points=1, atom_source=ktt_b200.ATOMS_CONSTANT),
    ktt_b200.Tune(block_x=16, block_y=8, z_iterations=16, x_points=2, rsqrt_soft=12,
                  precision=ktt_b200.PREC_FP64_MERGE_SHARED),
])
def test_linear_and_rectangular_tiles(ctx, dims, tune):
    """Planes that the block's rectangles pad by a little, a lot and not at all (the launch picks linear
    x-y tiles or the rectangles): within the norm tolerance of the oracle, and the points of a
    row-by-row launch (block of one row, no linear tile can be fewer) bit for bit."""
    import torch
    rng = np.random.default_rng(sum(dims))
    a = np.empty((77, 4), dtype=np.float32)
    a[:, :3] = rng.uniform(0.0, 0.5 * max(dims), (77, 3))
    a[:, 3] = rng.uniform(-1.0, 1.0, 77)
    h, origin = 0.5, (-1.0, 0.5, 2.0)
    out = torch.full((dims[2], dims[1], dims[0]), float("nan"), device="cuda")
    ctx.forward_3d(_t(a), dims, h, origin, tune=tune, out=out)
    assert errors.report(_np(out), oracle.grid3d(a, h, dims, origin))["rel_norm"] <= TOL_NORM
    row = ktt_b200.Tune(**dict(tune.as_dict(), block_x=1, block_y=1))
    assert torch.equal(out, ctx.forward_3d(_t(a), dims, h, origin, tune=row))


@pytest.mark.parametrize("n", [0, 1, 23, 24, 25, 48, 191, 193, 400])
@pytest.mark.parametrize("block", [(32, 4), (7, 3), (16, 1), (64, 4)])
@pytest.mark.parametrize("nz", [7, 8, 9, 33])
def test_record_tiles(ctx, n, block, nz):
    """2 x 16 points a thread, atoms as records in shared memory: atom counts around the batches (24), the
    FP32 partials (48) and the stages (192), blocks with a partial warp, depths that use half a tile;
    within the norm tolerance of the oracle, FP64 sums in registers and in shared memory bit for bit
    alike, slabs equal to the map."""
    import torch
    a = np.empty((n, 4), dtype=np.float32)
    rng = np.random.default_rng(n + nz)
    a[:, :3] = rng.uniform(0.0, 18.0, (n, 3))
    a[:, 3] = rng.uniform(-1.0, 1.0, n)
    atoms = _t(a) if n else torch.zeros((0, 4), device="cuda")
    dims, h, origin = (35, 11, nz), 0.5, (-1.0, 0.5, 2.0)
    ref = oracle.grid3d(a, h, dims, origin) if n else None
    maps = {}
    for prec in (ktt_b200.PREC_FP32, ktt_b200.PREC_FP64_MERGE, ktt_b200.PREC_FP64_MERGE_SHARED):
        for soft in (2, 12):
            tune = ktt_b200.Tune(block_x=block[0], block_y=block[1], z_iterations=16, x_points=2, precision=prec,
                                 rsqrt_soft=soft)
            out = torch.full((nz, 11, 35), float("nan"), device="cuda")
            ctx.forward_3d(atoms, dims, h, origin, tune=tune, out=out)
            if n:
                assert errors.report(_np(out), ref)["rel_norm"] <= TOL_NORM
            else:
                assert torch.count_nonzero(out) == 0
            if nz > 16:
                slab = ctx.forward_3d_slab(atoms, dims, h, 16, nz, origin, tune=tune)
                assert torch.equal(slab, out[16:])
            maps[prec, soft] = out
    for soft in (2, 12):
        assert torch.equal(maps[ktt_b200.PREC_FP64_MERGE, soft], maps[ktt_b200.PREC_FP64_MERGE_SHARED, soft])


@pytest.mark.parametrize("n", [0, 1, 31, 33, 255, 257, 700])
@pytest.mark.parametrize("dims", [(1, 1, 1), (63, 2, 8), (65, 1, 9), (37, 41, 17), (130, 40, 21)])
@pytest.mark.parametrize("shape", [(4, 1), (4, 4), (8, 4), (16, 1), (16, 2)])
def test_fp64_pairs_shared_tiles(ctx, n, dims, shape):
    """FP64 pairs, a tile's atoms split over warps and clusters: atom counts around the batches of 32 and
    the warps' shares, tiles at the edges of the columns and planes.  Every point to the rounding of its
    FP32 store (2^-24) plus the Newton step's 2^-40: 1.2e-7 with room for a sum's FP64 rounding; slabs
    equal the map."""
    import torch
    rng = np.random.default_rng(n + dims[0])
    a = np.empty((n, 4), dtype=np.float32)
    a[:, :3] = rng.uniform(0.0, 20.0, (n, 3))
    a[:, 3] = rng.uniform(0.1, 1.0, n)
    h, origin = 0.5, (-1.0, 0.5, 2.0)
    tune = ktt_b200.Tune(block_x=64, block_y=1, z_iterations=shape[0], x_points=shape[1],
                         precision=ktt_b200.PREC_FP64_PAIRS)
    atoms = _t(a) if n else torch.zeros((0, 4), device="cuda")
    out = torch.full((dims[2], dims[1], dims[0]), float("nan"), device="cuda")
    ctx.forward_3d(atoms, dims, h, origin, tune=tune, out=out)
    if n == 0:
        assert torch.count_nonzero(out) == 0
        return
    ref = oracle.grid3d(a, h, dims, origin)
    assert np.max(np.abs(_np(out) - ref) / np.abs(ref)) <= 1.2e-7
    if dims[2] > 16:
        assert torch.equal(ctx.forward_3d_slab(atoms, dims, h, 16, dims[2], origin, tune=tune), out[16:])
    base = torch.linspace(-2, 2, out.numel(), device="cuda").reshape(out.shape)
    acc = base.clone()
    ctx.forward_3d(atoms, dims, h, origin, tune=tune, out=acc, accumulate=True)
    assert torch.equal(acc, base + out)


@pytest.mark.parametrize("dims,n", [((130, 129, 33), 300), ((128, 128, 32), 5000), ((96, 90, 97), 1), ((90, 96, 100), 0),
                                    ((257, 128, 47), 2000)])
@pytest.mark.parametrize("fields", [None, dict(block_x=16, block_y=2, z_iterations=16, x_points=2, precision=4, rsqrt_soft=12),
                                    dict(block_x=64, block_y=1, z_iterations=8, x_points=2, unroll=2, rsqrt_soft=2),
                                    dict(block_x=64, block_y=1, z_iterations=32, x_points=1),
                                    dict(block_x=64, block_y=1, z_iterations=8, x_points=4, precision=3),
                                    dict(block_x=64, block_y=1, z_iterations=4, x_points=2, atom_source=1)])
def test_host_buffer_call_in_slabs(ctx, dims, n, fields):
    """Larger maps are evaluated and copied out in slabs of whole tiles: the host's map equals the device's bit
    for bit, also with a last slab of one plane, and for forms that are not cut; the call is timed."""
    rng = np.random.default_rng(n)
    a = np.empty((n, 4), dtype=np.float32)
    a[:, :3] = rng.uniform(0.0, 40.0, (n, 3))
    a[:, 3] = rng.uniform(-1.0, 1.0, n)
    tune = ktt_b200.Tune(**fields) if fields else None
    import torch
    atoms = _t(a) if n else torch.zeros((0, 4), device="cuda")
    dev = ctx.forward_3d(atoms, dims, 0.5, (0.5, 0.25, -1.0), tune=tune)
    ctx.synchronize()
    for _ in range(2):
        host = ctx.forward_3d_host(a, dims, 0.5, (0.5, 0.25, -1.0), tune=tune)
        assert np.array_equal(host, _np(dev))
        assert ctx.elapsed_ms() > 0.0


def test_fp64_pairs_on_a_column_deeper_than_one_grid(ctx):
    """A configuration of 16 planes a tile takes maps of up to 65,535 of them; the 8-plane tiles it runs then
    need more than one grid's 65,535 along z.  To the FP32 store's rounding, 2^-24 and the Newton step's
    2^-40: 1.2e-7."""
    dims = (1, 1, 524_291)
    a = np.array([[0.3, 0.2, 10.0, 1.0], [0.1, -0.4, 262_140.2, 0.5], [0.0, 0.1, 524_280.7, 0.25]], dtype=np.float32)
    tune = ktt_b200.Tune(block_x=64, block_y=1, z_iterations=16, x_points=2, precision=ktt_b200.PREC_FP64_PAIRS)
    out = _np(ctx.forward_3d(_t(a), dims, 1.0, tune=tune))
    ref = oracle.grid3d(a, 1.0, dims)
    assert np.max(np.abs(out - ref) / np.abs(ref)) <= 1.2e-7


def test_host_buffer_call_refuses_what_the_device_call_refuses(ctx):
    """A map of more planes of tiles than a grid holds is refused as a whole, also where the host-buffer call would
    have cut it into slabs that fit."""
    a = np.zeros((2000, 4), dtype=np.float32)
    tune = ktt_b200.Tune(block_x=32, block_y=1, z_iterations=1, x_points=1)
    dims = (16, 1, 70_000)
    with pytest.raises(ktt_b200.CoulombError) as e:
        ctx.forward_3d(_t(a), dims, 0.5, tune=tune)
    assert e.value.status == ktt_b200.COUL_ERR_DEVICE_LIMITS
    with pytest.raises(ktt_b200.CoulombError) as e:
        ctx.forward_3d_host(a, dims, 0.5, tune=tune)
    assert e.value.status == ktt_b200.COUL_ERR_DEVICE_LIMITS


def _signed_atoms(n, seed, box):
    rng = np.random.default_rng(seed)
    a = np.empty((n, 4), dtype=np.float32)
    a[:, :3] = rng.uniform(0.0, box, (n, 3))
    a[:, 3] = rng.uniform(-1.0, 1.0, n)
    return a


@pytest.mark.parametrize("dims,n", [((96, 96, 96), 15), ((96, 96, 96), 30), ((96, 96, 96), 60), ((128, 128, 128), 73),
                                    ((128, 128, 128), 250), ((131, 117, 125), 500), ((160, 160, 160), 97),
                                    ((160, 160, 161), 250), ((224, 224, 224), 19), ((224, 224, 209), 60)])
@pytest.mark.parametrize("prec", [ktt_b200.PREC_FP64_MERGE, ktt_b200.PREC_FP64_MERGE_SHARED])
def test_record_tiles_by_warps_a_tile(ctx, dims, n, prec):
    """FP64-merge record tiles with 1, 2, 4 and 8 warps a tile (by the map's tiles and the atom count), shares of one
    atom more or less, some empty: within the norm tolerance of the oracle, slabs equal to the map, a sum adds to
    out."""
    import torch
    a = _signed_atoms(n, n + dims[2], 0.5 * dims[0])
    h, origin = 0.5, (-1.0, 0.5, 2.0)
    tune = ktt_b200.Tune(block_x=16, block_y=2, z_iterations=16, x_points=2, precision=prec, rsqrt_soft=12)
    out = torch.full(dims[::-1], float("nan"), device="cuda")
    ctx.forward_3d(_t(a), dims, h, origin, tune=tune, out=out)
    assert errors.report(_np(out), oracle.grid3d(a, h, dims, origin))["rel_norm"] <= TOL_NORM
    assert torch.equal(ctx.forward_3d_slab(_t(a), dims, h, 48, dims[2], origin, tune=tune), out[48:])
    base = torch.linspace(-2, 2, out.numel(), device="cuda").reshape(out.shape)
    acc = base.clone()
    ctx.forward_3d(_t(a), dims, h, origin, tune=tune, out=acc, accumulate=True)
    assert torch.equal(acc, base + out)


@pytest.mark.parametrize("n", [1, 24, 47, 49, 200])
@pytest.mark.parametrize("block", [(32, 4), (7, 3), (16, 1), (8, 4)])
@pytest.mark.parametrize("shape,prec,soft", [((16, 2, 1), ktt_b200.PREC_FP64_MERGE_SHARED, 12),
                                             ((16, 2, 1), ktt_b200.PREC_FP32, 2)])
def test_record_tiles_of_one_warp_in_a_batch(ctx, n, block, shape, prec, soft):
    """Record tiles whose warp runs through all atoms, blocks with a partial warp, grids that overhang a tile by
    every number of planes: persistent and separate launches bit for bit, within the norm tolerance of the oracle."""
    import torch
    tune = ktt_b200.Tune(block_x=block[0], block_y=block[1], z_iterations=shape[0], x_points=shape[1], unroll=shape[2],
                         precision=prec, rsqrt_soft=soft)
    mols = [(_signed_atoms(n, n + nz, 18.0), (35 - nz % 3, 11, nz), 0.5, (-1.0, 0.5, 2.0)) for nz in range(1, 36, 3)]
    batch = ktt_b200.Batch(ctx, [(_t(a), *rest) for a, *rest in mols], tune)
    batch.run()
    ctx.synchronize()
    maps = [out.clone() for out in batch.outputs]
    for (a, dims, h, origin), out in zip(mols, maps):
        assert errors.report(_np(out), oracle.grid3d(a, h, dims, origin))["rel_norm"] <= TOL_NORM
    for out in batch.outputs:
        out.zero_()
    batch.run(ktt_b200.BATCH_SEPARATE)
    ctx.synchronize()
    assert all(torch.equal(x, y) for x, y in zip(maps, batch.outputs))
    batch.close()


@pytest.mark.parametrize("block", [(64, 1), (7, 3)])
@pytest.mark.parametrize("shape,soft", [((8, 2, 2), 2), ((8, 2, 1), 0), ((16, 2, 1), 12), ((16, 2, 4), 0)])
def test_fp32_tiles_on_a_map_too_large_for_the_plain_kernel(ctx, block, shape, soft):
    """FP32 configurations of 2 x 8 and 2 x 16 points from 64 tiles an SM on run their own tile: within the norm
    tolerance of the oracle, slabs equal to the map."""
    import torch
    dims, h, origin = (223, 224, 209), 0.5, (-1.0, 0.5, 2.0)
    a = _signed_atoms(37, 3, 100.0)
    tune = ktt_b200.Tune(block_x=block[0], block_y=block[1], z_iterations=shape[0], x_points=shape[1], unroll=shape[2],
                         rsqrt_soft=soft)
    out = torch.full(dims[::-1], float("nan"), device="cuda")
    ctx.forward_3d(_t(a), dims, h, origin, tune=tune, out=out)
    assert errors.report(_np(out), oracle.grid3d(a, h, dims, origin))["rel_norm"] <= TOL_NORM
    assert torch.equal(ctx.forward_3d_slab(_t(a), dims, h, 96, dims[2], origin, tune=tune), out[96:])


@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 300, 1), (131, 3, 9), (129, 7, 17), (257, 2, 8), (96, 33, 5)])
@pytest.mark.parametrize("tune", [
    dict(z_iterations=8, x_points=1, unroll=2, rsqrt_soft=2), dict(z_iterations=8, x_points=4, rsqrt_soft=3),
    dict(z_iterations=16, x_points=1), dict(z_iterations=4, x_points=4),
    dict(z_iterations=8, x_points=2, precision=ktt_b200.PREC_COMPENSATED),
    dict(z_iterations=8, x_points=2, precision=ktt_b200.PREC_FP64_MERGE, rsqrt_soft=2)])
def test_linear_tiles_of_the_one_cta_kernels(ctx, dims, tune):
    """As test_linear_and_rectangular_tiles, for tiles that run a CTA each on maps of this size: blocks of 64 x 1 and
    7 x 3 against a block of one thread, bit for bit."""
    import torch
    a = _signed_atoms(77, sum(dims), 0.5 * max(dims))
    h, origin = 0.5, (-1.0, 0.5, 2.0)
    one = ctx.forward_3d(_t(a), dims, h, origin, tune=ktt_b200.Tune(block_x=1, block_y=1, **tune))
    assert errors.report(_np(one), oracle.grid3d(a, h, dims, origin))["rel_norm"] <= TOL_NORM
    for block in ((64, 1), (7, 3)):
        out = torch.full(dims[::-1], float("nan"), device="cuda")
        ctx.forward_3d(_t(a), dims, h, origin, tune=ktt_b200.Tune(block_x=block[0], block_y=block[1], **tune), out=out)
        assert torch.equal(out, one)
