"""The adjoint kernel and its torch.autograd.Function against FP64 references.

L = 0.5 sum_i w_i (V_i - T_i)^2 with w = 0 within 1.5 A of any atom.  The GPU gradient (forward map
in the FP64-merge form, adjoint with FP64 partial sums) is compared with the oracle's FP64 gradient
and with FP64 central finite differences (h = 1e-4) of the oracle's FP64 loss; tolerance 1e-4
relative (normwise over the checked atoms, per component kind).
"""
import numpy as np
import pytest

import oracle
from ktt_b200 import workloads
import ktt_b200

pytestmark = pytest.mark.gpu

TOL = 1e-4
FORWARD = dict(z_iterations=8, x_points=2, precision=ktt_b200.PREC_FP64_MERGE)


def _gpu_loss_and_grad(ctx, atoms, dims, h, target, weight, origin=None):
    import torch
    a = torch.from_numpy(atoms).cuda().requires_grad_(True)
    t = torch.from_numpy(target.reshape(dims[::-1])).cuda()
    w = torch.from_numpy(weight.reshape(dims[::-1])).cuda()
    v = ktt_b200.coulomb_map(a, ctx, dims, h, origin, ktt_b200.Tune(**FORWARD))
    loss = 0.5 * (w.double() * (v.double() - t.double()) ** 2).sum()
    loss.backward()
    return float(loss.item()), a.grad.cpu().numpy().astype(np.float64)


def _rel(got, ref):
    return float(np.max(np.abs(got - ref)) / max(np.max(np.abs(ref)), 1e-300))


def test_adjoint_small_against_fp64_gradient(ctx):
    rng = np.random.default_rng(3)
    n, dims, h, origin = 300, (40, 33, 27), 0.5, (-2.0, 1.0, 0.5)
    atoms = np.empty((n, 4), dtype=np.float32)
    atoms[:, :3] = rng.uniform(0.0, 16.0, (n, 3))
    atoms[:, 3] = rng.uniform(-1, 1, n)
    target = rng.normal(0, 1, dims[::-1]).astype(np.float32)
    weight = workloads.exclusion_weights(atoms, dims, h, 1.5, origin)
    loss, grad = _gpu_loss_and_grad(ctx, atoms, dims, h, target, weight, origin)
    ref_loss, dq, dr = oracle.adjoint3d(atoms, h, dims, target, weight, origin=origin)
    assert abs(loss - ref_loss) <= 1e-5 * ref_loss
    assert _rel(grad[:, 3], dq) <= TOL
    assert _rel(grad[:, :3], dr) <= TOL


def test_adjoint_config5_finite_differences_and_reference(ctx):
    """8,192 atoms in a 64 A cube, 128^3 grid at 0.5 A; the target map from charges perturbed by
    N(0, 0.1); FD and FP64 gradient on 64 seeded atoms."""
    import torch
    atoms, q_target, dims, h, excl = workloads.adjoint_problem()
    weight = workloads.exclusion_weights(atoms, dims, h, excl)
    target_atoms = atoms.copy()
    target_atoms[:, 3] = q_target
    target = ctx.forward_3d(torch.from_numpy(target_atoms).cuda(), dims, h,
                            tune=ktt_b200.Tune(**FORWARD)).cpu().numpy()
    loss, grad = _gpu_loss_and_grad(ctx, atoms, dims, h, target, weight)

    sel = np.sort(np.random.default_rng(17).choice(atoms.shape[0], 64, replace=False))
    ref_loss, dq, dr, vmap = oracle.adjoint3d(atoms, h, dims, target, weight, sel=sel, want_map=True)
    assert abs(loss - ref_loss) <= 1e-5 * ref_loss
    assert _rel(grad[sel, 3], dq) <= TOL
    assert _rel(grad[sel, :3], dr) <= TOL

    eps = 1e-4
    fd = np.empty((sel.size, 4))
    for n_, j in enumerate(sel):
        base = atoms[j].astype(np.float64)
        for c in range(4):
            plus, minus = base.copy(), base.copy()
            plus[c] += eps
            minus[c] -= eps
            lp = oracle.loss_perturbed(atoms, int(j), plus, h, dims, target, vmap, weight)
            lm = oracle.loss_perturbed(atoms, int(j), minus, h, dims, target, vmap, weight)
            fd[n_, c] = (lp - lm) / (2 * eps)
    assert _rel(grad[sel, 3], fd[:, 3]) <= TOL
    assert _rel(grad[sel, :3], fd[:, :3]) <= TOL


def _adam_fp64(a_mat, w, target, q0, lr, steps, b1=0.9, b2=0.999, eps=1e-8):
    """Adam (the update torch.optim.Adam makes) on L(q) = 0.5 sum w (A q - T)^2 in FP64; the map is
    linear in the charges, A[i, j] = 1 / |r_i - r_j|.  Returns the loss before each step."""
    q = q0.astype(np.float64).copy()
    m = np.zeros_like(q)
    v = np.zeros_like(q)
    losses = []
    for s in range(1, steps + 1):
        r = a_mat @ q - target
        losses.append(0.5 * float((w * r * r).sum()))
        g = a_mat.T @ (w * r)
        m = b1 * m + (1 - b1) * g
        v = b2 * v + (1 - b2) * g * g
        q -= lr * (m / (1 - b1 ** s)) / (np.sqrt(v / (1 - b2 ** s)) + eps)
    return np.array(losses), q


def test_adam_charge_fitting(ctx):
    """100 Adam steps (lr 0.005) on the charges of 512 atoms through the autograd function.  The loss
    falls below 15% of its start (the fit of charges to a smooth 1/r map is ill-posed, so the charges
    themselves are only required not to drift away), and the loss trajectory follows the same Adam run
    made in FP64 on the explicit 110,592 x 512 map matrix within 1% at every tenth step."""
    import torch
    steps, lr = 100, 0.005
    atoms, q_target, dims, h, excl = workloads.adjoint_problem(seed=6, n_atoms=512, n=48, box=24.0)
    w_np = workloads.exclusion_weights(atoms, dims, h, excl)
    weight = torch.from_numpy(w_np).cuda().double()
    target_atoms = atoms.copy()
    target_atoms[:, 3] = q_target
    tune = ktt_b200.Tune(**FORWARD)
    target = ctx.forward_3d(torch.from_numpy(target_atoms).cuda(), dims, h, tune=tune).double()
    xyz = torch.from_numpy(atoms[:, :3].copy()).cuda()
    q = torch.from_numpy(atoms[:, 3].copy()).cuda().requires_grad_(True)
    opt = torch.optim.Adam([q], lr=lr)
    losses = []
    for _ in range(steps):
        opt.zero_grad()
        v = ktt_b200.coulomb_map(torch.cat([xyz, q[:, None]], dim=1), ctx, dims, h, None, tune)
        loss = 0.5 * (weight * (v.double() - target) ** 2).sum()
        loss.backward()
        opt.step()
        losses.append(float(loss.item()))
    losses = np.array(losses)

    g = np.arange(dims[0], dtype=np.float64) * h
    zz, yy, xx = np.meshgrid(g, g, g, indexing="ij")
    pts = np.stack([xx.ravel(), yy.ravel(), zz.ravel()], 1)
    a_mat = np.empty((pts.shape[0], atoms.shape[0]))
    for j in range(atoms.shape[0]):
        a_mat[:, j] = 1.0 / np.sqrt(((pts - atoms[j, :3].astype(np.float64)) ** 2).sum(1))
    ref_losses, _ = _adam_fp64(a_mat, w_np.ravel().astype(np.float64),
                               a_mat @ q_target.astype(np.float64), atoms[:, 3], lr, steps)

    q_err0 = np.abs(atoms[:, 3] - q_target).mean()
    q_err = np.abs(q.detach().cpu().numpy() - q_target).mean()
    assert losses[-1] < 0.15 * losses[0], losses[::10]
    assert q_err <= q_err0, (q_err, q_err0)
    rel = np.abs(losses[::10] - ref_losses[::10]) / ref_losses[::10]
    assert rel.max() <= 1e-2, (losses[::10], ref_losses[::10])


def test_adam_charge_fitting_full_size(ctx):
    """The charge fit at its stated size: 100 Adam steps (lr 0.005) on the charges of 8,192 atoms on
    the 128^3 grid through the autograd function (each step one forward map and one adjoint).  At
    every tenth step the loss the GPU computed equals the FP64 oracle's loss for the same charges
    within 1e-4 relative; the loss falls below half its start and the charges do not drift away."""
    import time

    import torch
    steps, lr = 100, 0.005
    atoms, q_target, dims, h, excl = workloads.adjoint_problem()
    w_np = workloads.exclusion_weights(atoms, dims, h, excl)
    weight = torch.from_numpy(w_np).cuda().double()
    target_atoms = atoms.copy()
    target_atoms[:, 3] = q_target
    tune = ktt_b200.Tune(**FORWARD)
    target32 = ctx.forward_3d(torch.from_numpy(target_atoms).cuda(), dims, h, tune=tune)
    target = target32.double()
    xyz = torch.from_numpy(atoms[:, :3].copy()).cuda()
    q = torch.from_numpy(atoms[:, 3].copy()).cuda().requires_grad_(True)
    opt = torch.optim.Adam([q], lr=lr)
    losses, snapshots = [], []
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for s in range(steps):
        opt.zero_grad()
        v = ktt_b200.coulomb_map(torch.cat([xyz, q[:, None]], dim=1), ctx, dims, h, None, tune)
        loss = 0.5 * (weight * (v.double() - target) ** 2).sum()
        loss.backward()
        if s % 10 == 0:
            snapshots.append((s, q.detach().clone()))
        losses.append(loss.detach())
        opt.step()
    torch.cuda.synchronize()
    seconds = time.perf_counter() - t0
    losses = np.array([float(x) for x in losses])
    print(f"\n100 Adam steps, 8192 atoms, 128^3 grid: {seconds:.3f} s ({1e3 * seconds / steps:.2f} ms per step)")

    target_np = target32.cpu().numpy()
    for s, qs in snapshots:
        a = atoms.copy()
        a[:, 3] = qs.cpu().numpy()
        ref_loss, _, _ = oracle.adjoint3d(a, h, dims, target_np, w_np, sel=np.array([0]))
        assert abs(losses[s] - ref_loss) <= 1e-4 * ref_loss, (s, losses[s], ref_loss)
    q_err0 = np.abs(atoms[:, 3] - q_target).mean()
    q_err = np.abs(q.detach().cpu().numpy() - q_target).mean()
    assert losses[-1] < 0.5 * losses[0], losses[::10]
    assert q_err <= q_err0, (q_err, q_err0)


@pytest.mark.parametrize("n", [1, 128, 129, 400])
@pytest.mark.parametrize("dims", [(1, 1, 1), (16, 3, 5), (31, 9, 4), (32, 8, 9), (33, 40, 3), (49, 2, 37), (65, 130, 1)])
def test_adjoint_block_edges(ctx, dims, n):
    """Row lengths around the kernel's column blocks (16 and 32), row counts around its staged blocks
    and chunks, atom counts around a CTA's 128, against the FP64 gradient.  L = 0.5 sum V^2 with T = 0
    and w = 1, so G = V: an FP32 pair chain is good to about 4e-7 of its own magnitude and the sums
    here cancel by less than a factor of ten in the largest component; 1e-5 of it."""
    import torch
    rng = np.random.default_rng(1000 * n + dims[0])
    atoms = np.empty((n, 4), dtype=np.float32)
    atoms[:, :3] = rng.uniform(-4.0, 0.5 * max(dims) + 4.0, (n, 3))
    atoms[:, 3] = rng.uniform(0.2, 1.0, n)
    h, origin = 0.5, (0.25, -0.5, 1.0)
    v = oracle.grid3d(atoms, h, dims, origin).astype(np.float32)
    zero, one = np.zeros_like(v), np.ones_like(v)
    _, dq, dr = oracle.adjoint3d(atoms, h, dims, zero, one, origin=origin)
    got = ktt_b200.adjoint_3d(ctx, torch.from_numpy(atoms).cuda(), dims, h, torch.from_numpy(v).cuda(), origin)
    got = got.cpu().numpy().astype(np.float64)
    assert _rel(got[:, 3], dq) <= 1e-5
    assert _rel(got[:, :3], dr) <= 1e-5


def _gradient_fp64(atoms, dims, h, grad_map):
    """dL/dq and dL/dr of every atom with G = grad_map, in FP64; a point with G = 0 adds nothing."""
    g = [np.arange(d, dtype=np.float64) * h for d in dims]
    points = np.stack([c.ravel() for c in np.meshgrid(*g[::-1], indexing="ij")], 1)[:, ::-1]
    w = grad_map.astype(np.float64).ravel()
    points, w = points[w != 0], w[w != 0]
    dq, dr = np.empty(atoms.shape[0]), np.empty((atoms.shape[0], 3))
    for j, a in enumerate(atoms.astype(np.float64)):
        d = points - a[:3]
        r = np.sqrt((d * d).sum(1))
        dq[j] = (w / r).sum()
        dr[j] = a[3] * ((w / r ** 3)[:, None] * d).sum(0)
    return dq, dr


@pytest.mark.parametrize("dims", [(8, 4, 4), (40, 6, 5), (64, 3, 3)])
def test_adjoint_masked_point_close_to_an_atom(ctx, dims):
    """A point with G = 0 (a fit's mask) adds nothing however close the atom lies: 1 / r^3 leaves FP32's range
    below 1.4e-13, G / r * (1 / r^2) does not before r^2 does.  An FP32 pair chain is good to about 4e-7: 1e-5."""
    import torch
    rng = np.random.default_rng(dims[0])
    atoms = np.empty((40, 4), dtype=np.float32)
    atoms[:, :3] = rng.uniform(-3.0, 3.0, (40, 3))
    atoms[:, 3] = rng.uniform(0.2, 1.0, 40)
    for j, r in enumerate((1e-13, 1e-14, 1e-16, 2e-18)):
        atoms[j, :3] = np.roll((r, 0.0, 0.0), j % 3)  # next to the origin's point
    grad_map = rng.uniform(0.5, 1.0, dims[::-1]).astype(np.float32)
    grad_map[0, 0, 0] = 0.0
    dq, dr = _gradient_fp64(atoms, dims, 0.5, grad_map)
    got = ktt_b200.adjoint_3d(ctx, torch.from_numpy(atoms).cuda(), dims, 0.5, torch.from_numpy(grad_map).cuda())
    got = got.cpu().numpy().astype(np.float64)
    assert np.all(np.isfinite(got))
    assert _rel(got[:, 3], dq) <= 1e-5
    assert _rel(got[:, :3], dr) <= 1e-5


@pytest.mark.parametrize("n", [1, 128, 300])
@pytest.mark.parametrize("dims", [(1, 90, 7), (2, 65, 1), (3, 9, 8), (4, 64, 65), (5, 33, 2), (8, 32, 9), (9, 17, 3),
                                  (16, 16, 17), (17, 5, 16), (23, 7, 7), (24, 33, 16), (25, 8, 9), (47, 17, 1)])
def test_adjoint_short_rows(ctx, dims, n):
    """Rows around the kernel's widths (4, 8, 16, 24, then blocks of 16 and 32), row counts around its staged blocks
    (64, 32, 16, 8), against the FP64 gradient.  G in [0.5, 1]: the charge sums do not cancel, the position sums by
    less than a factor of ten in the largest component: 1e-5 as above."""
    import torch
    rng = np.random.default_rng(1000 * n + dims[0])
    atoms = np.empty((n, 4), dtype=np.float32)
    atoms[:, :3] = rng.uniform(-4.0, 0.5 * max(dims) + 4.0, (n, 3))
    atoms[:, 3] = rng.uniform(0.2, 1.0, n)
    grad_map = rng.uniform(0.5, 1.0, dims[::-1]).astype(np.float32)
    dq, dr = _gradient_fp64(atoms, dims, 0.5, grad_map)
    got = ktt_b200.adjoint_3d(ctx, torch.from_numpy(atoms).cuda(), dims, 0.5, torch.from_numpy(grad_map).cuda())
    got = got.cpu().numpy().astype(np.float64)
    assert _rel(got[:, 3], dq) <= 1e-5
    assert _rel(got[:, :3], dr) <= 1e-5


@pytest.mark.parametrize("nx", [1, 2, 3, 4])
def test_adjoint_short_rows_are_summed_in_fp64(ctx, nx):
    """Charge gradient of rows of a few points, G normal.  Rounding errors in units of u = 2^-24, rms of a rounding
    0.42 u (uniform over a binade): differences and r^2 0.42 and 0.36, the root 1 (documented below 2.15), G / r and the
    store 0.42 each, together 1.3 u; a row's sum adds 0.42 u times the square root of its log2(nx) levels, and FP64
    sums of rows add nothing.  Sums of 64 rows in FP32 would come to 1.6 u and more."""
    import torch
    u = 2.0**-24
    rng = np.random.default_rng(nx)
    ny = int((200_000 // nx) ** 0.5)
    dims = (nx, ny, ny)
    atoms = np.empty((200, 4), dtype=np.float32)
    atoms[:, :3] = rng.uniform(0.0, 1.0, (200, 3)) * 0.5 * np.array(dims)
    atoms[:, 3] = rng.uniform(-1.0, 1.0, 200)
    grad_map = rng.normal(0.0, 1.0, dims[::-1]).astype(np.float32)
    dq, _ = _gradient_fp64(atoms, dims, 0.5, grad_map)
    got = ktt_b200.adjoint_3d(ctx, torch.from_numpy(atoms).cuda(), dims, 0.5, torch.from_numpy(grad_map).cuda())
    error = np.linalg.norm(got[:, 3].cpu().numpy().astype(np.float64) - dq) / np.linalg.norm(dq)
    assert error <= u * np.sqrt(1.3**2 + 0.42**2 * np.log2(nx))


def test_adjoint_on_two_streams_and_captured(ctx):
    """The context's partial sums are one stream's at a time (gradients of two sizes on two streams, nothing waited
    for between); captured calls, on two streams forked within one capture as well, keep memory of their own: their
    replays equal the eager calls bit for bit after later calls have grown the context's, beside eager calls on another
    stream, and for a second graph made when the first is gone."""
    import torch
    rng = np.random.default_rng(12)
    data, want = [], []
    for n, dims in ((3000, (61, 57, 50)), (700, (40, 90, 33))):
        atoms = np.empty((n, 4), dtype=np.float32)
        atoms[:, :3] = rng.uniform(0.0, 25.0, (n, 3))
        atoms[:, 3] = rng.uniform(-1.0, 1.0, n)
        g = rng.normal(0.0, 1.0, dims[::-1]).astype(np.float32)
        data.append((torch.from_numpy(atoms).cuda(), dims, 0.5, torch.from_numpy(g).cuda()))
        want.append(ktt_b200.adjoint_3d(ctx, *data[-1]))
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]

    def eager():
        got = []
        for i in range(8):
            with torch.cuda.stream(streams[i % 2]):
                got.append((i % 2, ktt_b200.adjoint_3d(ctx, *data[i % 2])))
        return got

    got = eager()
    torch.cuda.synchronize()
    for k, grad in got:
        assert torch.equal(grad, want[k])
    for _ in range(2):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            fork, side = torch.cuda.current_stream(), torch.cuda.Stream()
            first = ktt_b200.adjoint_3d(ctx, *data[0])
            side.wait_stream(fork)
            with torch.cuda.stream(side):
                beside = [ktt_b200.adjoint_3d(ctx, *data[1]) for _ in range(2)]
            again = ktt_b200.adjoint_3d(ctx, *data[0])
            fork.wait_stream(side)
        big = torch.cat([data[0][0]] * 8)
        ktt_b200.adjoint_3d(ctx, big, *data[0][1:])
        for _ in range(3):
            for out in (first, again, *beside):
                out.zero_()
            graph.replay()
            got = eager()
            torch.cuda.synchronize()
            assert torch.equal(first, want[0]) and torch.equal(again, want[0])
            assert all(torch.equal(b, want[1]) for b in beside)
            for k, grad in got:
                assert torch.equal(grad, want[k])
        del graph, first, again, beside
