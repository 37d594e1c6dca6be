"""Differentiable float32 SGM: CUDA forward/backward vs a plain-PyTorch reference (autograd) and
FP64 finite differences, on 64x48x32 crops of a seeded scene (Hamming cost + U(0,0.5) jitter)."""
import numpy as np
import pytest
import torch

from fasterstereocuda_b200 import scenes
from fasterstereocuda_b200.float_sgm import reference_sgm


def jittered_cost(oracle_mod, W, H, D, B=1, seed=70):
    vols = []
    rng = np.random.Generator(np.random.PCG64(seed))
    for b in range(B):
        L, R, _ = scenes.planar_pair(seed + b, W, H, dmin=2.0, dmax=D - 6.0)
        cfg = oracle_mod.Config(width=W, height=H, disp_range=D, do_lr_check=0, do_median=0)
        c = oracle_mod.match(cfg, L, R, dump=True)["cost"].astype(np.float64)
        vols.append(c + rng.uniform(0.0, 0.5, size=c.shape))
    return np.stack(vols)


def fd_check(f, x, idx, g_analytic, h=1e-6):
    """central differences of the scalar f at flat indices idx of x (float64, modified in place)"""
    fd = []
    flat = x.view(-1)
    for i in idx:
        old = flat[i].item()
        flat[i] = old + h
        fp = f().item()
        flat[i] = old - h
        fm = f().item()
        flat[i] = old
        fd.append((fp - fm) / (2 * h))
    fd = np.array(fd)
    ga = g_analytic.reshape(-1)[idx]
    return np.linalg.norm(ga - fd) / max(np.linalg.norm(fd), 1e-12)


def test_reference_autograd_matches_fp64_finite_differences(oracle_mod):
    """CPU: the PyTorch restatement's autograd gradient equals central differences in FP64."""
    c = torch.tensor(jittered_cost(oracle_mod, 14, 11, 32), dtype=torch.float64, requires_grad=True)
    p1 = torch.full(c.shape[:-1], 10.0, dtype=torch.float64, requires_grad=True)
    p2 = torch.full(c.shape[:-1], 150.0, dtype=torch.float64, requires_grad=True)
    w = torch.randn(c.shape[:-1], dtype=torch.float64, generator=torch.Generator().manual_seed(0))
    (reference_sgm(c, p1, p2) * w).sum().backward()
    with torch.no_grad():
        f = lambda: (reference_sgm(c, p1, p2) * w).sum()  # noqa: E731
        gc = c.grad.numpy()
        idx = np.argsort(-np.abs(gc.reshape(-1)))[:20]
        assert fd_check(f, c, idx, gc) < 1e-6
        g1 = p1.grad.numpy()
        idx = np.argsort(-np.abs(g1.reshape(-1)))[:8]
        assert fd_check(f, p1, idx, g1) < 1e-6


@pytest.mark.gpu
def test_forward_matches_reference(oracle_mod):
    c64 = torch.tensor(jittered_cost(oracle_mod, 64, 48, 32, B=2), dtype=torch.float64)
    p1 = torch.full(c64.shape[:-1], 10.0, dtype=torch.float64)
    p2 = torch.full(c64.shape[:-1], 150.0, dtype=torch.float64)
    from fasterstereocuda_b200.float_sgm import float_sgm
    d = float_sgm(c64.float().cuda(), p1.float().cuda(), p2.float().cuda()).cpu().double()
    ref = reference_sgm(c64, p1, p2)
    assert torch.allclose(d, ref, rtol=1e-4, atol=1e-4), (d - ref).abs().max()


@pytest.mark.gpu
@pytest.mark.parametrize("D", [32, 64])
def test_backward_matches_fp64_finite_differences_and_autograd(oracle_mod, D):
    from fasterstereocuda_b200.float_sgm import float_sgm
    c64 = torch.tensor(jittered_cost(oracle_mod, 64, 48, D), dtype=torch.float64)
    gen = torch.Generator().manual_seed(1)
    p1 = (10.0 + torch.rand(c64.shape[:-1], generator=gen, dtype=torch.float64))
    p2 = (150.0 + 10 * torch.rand(c64.shape[:-1], generator=gen, dtype=torch.float64))
    w = torch.randn(c64.shape[:-1], generator=gen, dtype=torch.float64)
    # kernel gradients (float32)
    c = c64.float().cuda().requires_grad_()
    q1 = p1.float().cuda().requires_grad_()
    q2 = p2.float().cuda().requires_grad_()
    (float_sgm(c, q1, q2) * w.float().cuda()).sum().backward()
    gk = [c.grad.cpu().double().numpy(), q1.grad.cpu().double().numpy(), q2.grad.cpu().double().numpy()]
    # autograd reference (FP64)
    cr, r1, r2 = (t.clone().requires_grad_() for t in (c64, p1, p2))
    (reference_sgm(cr, r1, r2) * w).sum().backward()
    gr = [cr.grad.numpy(), r1.grad.numpy(), r2.grad.numpy()]
    for a, b, name in zip(gk, gr, ("cost", "p1", "p2")):
        rel = np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-12)
        assert rel < 1e-3, (name, rel)
    # FP64 finite differences on the largest entries
    with torch.no_grad():
        xs = [c64.clone(), p1.clone(), p2.clone()]
        f = lambda: (reference_sgm(xs[0], xs[1], xs[2]) * w).sum()  # noqa: E731
        for k, n in ((0, 24), (1, 8), (2, 8)):
            idx = np.argsort(-np.abs(gk[k].reshape(-1)))[:n]
            assert fd_check(f, xs[k], idx, gk[k]) < 1e-3, k


@pytest.mark.gpu
@pytest.mark.parametrize("D", [32, 64])
def test_ragged_sizes_match_autograd_and_repeat(oracle_mod, D):
    """Line counts that leave part of a warp idle and scanlines ending inside a segment: forward
    and gradients against the FP64 autograd reference; a second run gives the same bits."""
    from fasterstereocuda_b200.float_sgm import float_sgm
    c64 = torch.tensor(jittered_cost(oracle_mod, 37, 29, D, B=2, seed=91), dtype=torch.float64)
    gen = torch.Generator().manual_seed(3)
    p1 = 8.0 + 4 * torch.rand(c64.shape[:-1], generator=gen, dtype=torch.float64)
    p2 = 100.0 + 60 * torch.rand(c64.shape[:-1], generator=gen, dtype=torch.float64)
    w = torch.randn(c64.shape[:-1], generator=gen, dtype=torch.float64)

    def run():
        c = c64.float().cuda().requires_grad_()
        q1 = p1.float().cuda().requires_grad_()
        q2 = p2.float().cuda().requires_grad_()
        d = float_sgm(c, q1, q2)
        (d * w.float().cuda()).sum().backward()
        return [t.detach().cpu() for t in (d, c.grad, q1.grad, q2.grad)]
    first, again = run(), run()
    for a, b in zip(first, again):
        assert torch.equal(a, b)
    cr, r1, r2 = (t.clone().requires_grad_() for t in (c64, p1, p2))
    dr = reference_sgm(cr, r1, r2)
    assert torch.allclose(first[0].double(), dr.detach(), rtol=1e-4, atol=1e-4), (first[0].double() - dr).abs().max()
    (dr * w).sum().backward()
    for a, b, name in zip(first[1:], (cr.grad, r1.grad, r2.grad), ("cost", "p1", "p2")):
        rel = (a.double() - b).norm() / max(b.norm(), 1e-12)
        assert rel < 1e-3, (name, rel)


@pytest.mark.gpu
def test_fitting_penalty_maps_reduces_l1(oracle_mod):
    """Demo: fit per-pixel P1/P2 maps to the ground-truth disparity under an L1 loss."""
    from fasterstereocuda_b200.float_sgm import float_sgm
    W, H, D = 128, 96, 64
    L, R, gt = scenes.planar_pair(80, W, H, dmin=4.0, dmax=50.0)
    cfg = oracle_mod.Config(width=W, height=H, disp_range=D, do_lr_check=0, do_median=0)
    cost = torch.tensor(oracle_mod.match(cfg, L, R, dump=True)["cost"], dtype=torch.float32).cuda()[None]
    cost = cost + torch.rand(cost.shape, generator=torch.Generator(device="cuda").manual_seed(0), device="cuda") * 0.5
    gt = torch.tensor(gt).cuda()[None]
    lp1 = torch.full((1, H, W), np.log(10.0), device="cuda", requires_grad=True)
    lp2 = torch.full((1, H, W), np.log(150.0), device="cuda", requires_grad=True)
    opt = torch.optim.Adam([lp1, lp2], lr=0.05)
    losses = []
    inner = (slice(None), slice(8, H - 8), slice(8, W - 8))
    for _ in range(40):
        opt.zero_grad()
        disp = float_sgm(cost, lp1.exp(), lp2.exp())
        loss = (disp[inner] - gt[inner]).abs().mean()
        loss.backward()
        opt.step()
        losses.append(loss.item())
    assert losses[-1] < losses[0] * 0.98, losses[::10]


def first_candidate_adjoint(cost, p1, p2, w):
    """Disparity and gradients of sum(w * disp) in float64 with the documented order of equal
    candidates (same d, d-1, d+1, jump; the lowest k of the minimum); autograd splits ties."""
    D = cost.shape[-1]
    pad = torch.nn.functional.pad

    def candidates(q, m, a, b):
        return torch.stack([q, pad(q, (1, 0), value=np.inf)[..., :-1] + a, pad(q, (0, 1), value=np.inf)[..., 1:] + a,
                            (m + b).expand_as(q)])
    disp, total = reference_sgm(cost, p1, p2, return_sum=True)
    weight = torch.softmax(-total, -1)
    g_sum = -w[..., None] * weight * (torch.arange(D, dtype=cost.dtype) - disp[..., None])
    gc, g1, g2 = torch.zeros_like(cost), torch.zeros_like(p1), torch.zeros_like(p2)
    for dim, rev in ((1, False), (2, False), (1, True), (2, True)):
        order = list(range(cost.shape[dim]))[::-1 if rev else 1]
        L = [cost.select(dim, order[0])]
        for k in order[1:]:
            m = L[-1].min(-1, keepdim=True).values
            a, b = p1.select(dim, k)[..., None], p2.select(dim, k)[..., None]
            L.append(cost.select(dim, k) + candidates(L[-1], m, a, b).min(0).values - m)
        g = torch.zeros_like(L[0])
        for i in range(len(order) - 1, -1, -1):
            k = order[i]
            g = g + g_sum.select(dim, k)
            gc.select(dim, k).add_(g)
            if i == 0:
                break
            q = L[i - 1]
            m, at = q.min(-1, keepdim=True)
            pick = candidates(q, m, p1.select(dim, k)[..., None], p2.select(dim, k)[..., None]).min(0).indices
            same, dn, up, jump = (torch.where(pick == n, g, 0.0) for n in range(4))
            g1.select(dim, k).add_((dn + up).sum(-1))
            g2.select(dim, k).add_(jump.sum(-1))
            back = same + pad(dn, (0, 1))[..., 1:] + pad(up, (1, 0))[..., :-1]
            g = back.scatter_add(-1, at, jump.sum(-1, keepdim=True) - g.sum(-1, keepdim=True))
    return disp, gc, g1, g2


@pytest.mark.gpu
@pytest.mark.parametrize("D", [32, 64])
@pytest.mark.parametrize("H,W", [(1, 1), (1, 9), (8, 1), (7, 8), (8, 16), (17, 33)])
def test_segment_edges_and_disparity_alone(D, H, W):
    """Lines that end before, at and past a segment (8) and a chunk (16): gradients against the FP64
    adjoint, on half-integer costs and penalties so that equal candidates occur and every path sum is
    exact; the call without gradients gives the same disparities."""
    from fasterstereocuda_b200.float_sgm import float_sgm
    gen = torch.Generator().manual_seed(100 * H + W + D)
    c64 = torch.rand(2, H, W, D, generator=gen, dtype=torch.float64).argsort(-1).double() * 0.5
    p1 = torch.randint(3, 7, (2, H, W), generator=gen).double() + 0.25
    p2 = torch.randint(20, 40, (2, H, W), generator=gen).double() + 0.125
    w = torch.randn(2, H, W, generator=gen, dtype=torch.float64)
    c, q1, q2 = (t.float().cuda().requires_grad_() for t in (c64, p1, p2))
    d = float_sgm(c, q1, q2)
    (d * w.float().cuda()).sum().backward()
    with torch.no_grad():
        assert torch.equal(float_sgm(c, q1, q2), d)
    dr, *expected = first_candidate_adjoint(c64, p1, p2, w)
    assert torch.allclose(d.detach().cpu().double(), dr, rtol=1e-4, atol=1e-4)
    for a, b, name in zip((c.grad, q1.grad, q2.grad), expected, ("cost", "p1", "p2")):
        if b.norm() == 0:
            assert a.abs().max() == 0, name
            continue
        assert (a.cpu().double() - b).norm() / b.norm() < 1e-3, name


@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("shape", [(), (1,), (5, 7), (1, 5, 7), (2, 1, 7), (2, 5, 1), (2, 5, 8), (4, 5, 7), None])
def test_penalties_of_other_sizes_or_devices_are_refused(shape, grad):
    """Penalty maps without one value a pixel, or on the host (None): an error before any kernel. On
    tensors without storage, so that no call can reach a GPU."""
    from torch._subclasses.fake_tensor import FakeTensorMode
    from fasterstereocuda_b200.float_sgm import float_sgm
    with FakeTensorMode():
        cost = torch.empty(2, 5, 7, 32, device="cuda").requires_grad_(grad)
        good = torch.empty(2, 5, 7, device="cuda")
        bad = torch.empty(2, 5, 7) if shape is None else torch.empty(shape, device="cuda")
        for p1, p2 in ((bad, good), (good, bad)):
            with pytest.raises(ValueError, match="p1 and p2"):
                float_sgm(cost, p1, p2)


def undefined_aware_adjoint(cost, p1, p2, w):
    """As first_candidate_adjoint, with the documented handling of values that compare with nothing: a minimum
    passes over NaN, and a candidate takes the place of "same d" only where it is smaller."""
    D = cost.shape[-1]
    pad = torch.nn.functional.pad

    def least(q):
        m = q[..., :1]
        for k in range(1, D):
            m = torch.fmin(m, q[..., k:k + 1])
        return m

    def chosen(q, m, a, b):
        t, pick = q, torch.zeros(q.shape, dtype=torch.long)
        for n, c in enumerate((pad(q, (1, 0), value=np.inf)[..., :-1] + a, pad(q, (0, 1), value=np.inf)[..., 1:] + a,
                               (m + b).expand_as(q)), 1):
            pick = torch.where(c < t, n, pick)
            t = torch.where(c < t, c, t)
        return pick
    total = 0
    states = []
    for dim, rev in ((1, False), (2, False), (1, True), (2, True)):
        order = list(range(cost.shape[dim]))[::-1 if rev else 1]
        L = [cost.select(dim, order[0])]
        for k in order[1:]:
            m = least(L[-1])
            a, b = p1.select(dim, k)[..., None], p2.select(dim, k)[..., None]
            t = torch.fmin(L[-1], pad(L[-1], (1, 0), value=np.inf)[..., :-1] + a)
            t = torch.fmin(torch.fmin(t, pad(L[-1], (0, 1), value=np.inf)[..., 1:] + a), m + b)
            L.append(cost.select(dim, k) + t - m)
        states.append((dim, order, L))
        total = total + torch.stack([L[order.index(k)] for k in range(len(order))], dim)
    weight = torch.softmax(-total, -1)
    levels = torch.arange(D, dtype=cost.dtype)
    disp = (weight * levels).sum(-1)
    g_sum = -w[..., None] * weight * (levels - disp[..., None])
    gc, g1, g2 = torch.zeros_like(cost), torch.zeros_like(p1), torch.zeros_like(p2)
    for dim, order, L in states:
        g = torch.zeros_like(L[0])
        for i in range(len(order) - 1, -1, -1):
            k = order[i]
            g = g + g_sum.select(dim, k)
            gc.select(dim, k).add_(g)
            if i == 0:
                break
            q = L[i - 1]
            m = least(q)
            pick = chosen(q, m, p1.select(dim, k)[..., None], p2.select(dim, k)[..., None])
            same, dn, up, jump = (torch.where(pick == n, g, 0.0) for n in range(4))
            g1.select(dim, k).add_((dn + up).sum(-1))
            g2.select(dim, k).add_(jump.sum(-1))
            at = (q == m) & ((q == m).cumsum(-1) == 1)  # the lowest k, or none
            back = same + pad(dn, (0, 1))[..., 1:] + pad(up, (1, 0))[..., :-1]
            g = torch.where(at, back - (same + dn + up).sum(-1, keepdim=True), back)
    return disp, gc, g1, g2


def masked_inputs(case, D):
    gen = torch.Generator().manual_seed(D)
    c = torch.rand(2, 21, 37, D, generator=gen, dtype=torch.float64) * 60
    if case == "voxels":
        c[torch.rand(c.shape, generator=gen) < 0.3] = np.inf
        c[..., 5] = 7.0  # a candidate left in every pixel
    elif case == "pixel":
        c[0, 10, 20] = np.inf
    else:
        c[0, 10, 20, 3] = np.nan
    p1 = 10.0 + torch.rand(2, 21, 37, generator=gen, dtype=torch.float64)
    p2 = 150.0 + torch.rand(2, 21, 37, generator=gen, dtype=torch.float64)
    w = torch.randn(2, 21, 37, generator=gen, dtype=torch.float64)
    return [t.float().double() for t in (c, p1, p2, w)]


@pytest.mark.parametrize("D", [32, 64])
def test_masked_cost_model_agrees_with_the_plain_adjoint_where_all_is_finite(D):
    c, p1, p2, w = masked_inputs("voxels", D)
    for a, b in zip(undefined_aware_adjoint(c, p1, p2, w), first_candidate_adjoint(c, p1, p2, w)):
        assert torch.allclose(a, b, rtol=1e-12, atol=1e-12)


@pytest.mark.gpu
@pytest.mark.parametrize("D", [32, 64])
@pytest.mark.parametrize("case", ["voxels", "pixel", "nan"])
def test_masked_costs(case, D):
    """Infinite costs in some voxels, in all of one pixel, and one NaN: the same undefined entries as the
    model of the documented order, the others within 1e-3 of it in norm (as the tests above)."""
    from fasterstereocuda_b200.float_sgm import float_sgm
    c64, p1, p2, w = masked_inputs(case, D)
    c, q1, q2 = (t.float().cuda().requires_grad_() for t in (c64, p1, p2))
    d = float_sgm(c, q1, q2)
    grads = torch.autograd.grad(d, (c, q1, q2), w.float().cuda())
    with torch.no_grad():
        assert torch.equal(torch.nan_to_num(float_sgm(c, q1, q2), nan=-1.0), torch.nan_to_num(d, nan=-1.0))
    for a, b, name in zip((d.detach(), *grads), undefined_aware_adjoint(c64, p1, p2, w), ("disp", "cost", "p1", "p2")):
        a = a.cpu().double()
        assert torch.equal(a.isnan(), b.isnan()), (name, int(a.isnan().sum()), int(b.isnan().sum()))
        ok = ~b.isnan()
        assert (a[ok] - b[ok]).norm() <= 1e-3 * b[ok].norm() + 1e-30, name


@pytest.mark.gpu
@pytest.mark.parametrize("D", [32, 64])
def test_backward_after_the_inputs_changed(D):
    """The gradients come from what the forward pass recorded: inputs that are overwritten in place
    before the backward pass neither raise nor change them."""
    from fasterstereocuda_b200.float_sgm import float_sgm
    c64, p1, p2, w = masked_inputs("voxels", D)
    w = w.float().cuda()

    def run(change):
        leaves = [t.float().cuda().requires_grad_() for t in (c64, p1, p2)]
        inputs = [t * 1 for t in leaves]
        d = float_sgm(*inputs)
        if change:
            for t in inputs:
                t.zero_()
        return torch.autograd.grad(d, leaves, w)
    for a, b in zip(run(True), run(False)):
        assert torch.equal(a, b)


@pytest.mark.gpu
def test_penalty_maps_of_another_shape_with_a_value_a_pixel():
    """Such maps are taken in the order of their values; their gradients have their shape."""
    from fasterstereocuda_b200.float_sgm import float_sgm
    c64, p1, p2, w = masked_inputs("voxels", 32)
    w = w.float().cuda()
    grads = []
    for s1, s2 in (((2, 21, 37), (2, 21, 37)), ((2, 1, 21, 37), (2, 21, 37)), ((2 * 21 * 37,), (2, 21, 37, 1))):
        c, q1, q2 = c64.float().cuda().requires_grad_(), *(p.float().cuda().view(s).requires_grad_()
                                                          for p, s in ((p1, s1), (p2, s2)))
        g = torch.autograd.grad(float_sgm(c, q1, q2), (c, q1, q2), w)
        assert g[1].shape == s1 and g[2].shape == s2
        grads.append([t.reshape(-1) for t in g])
    for other in grads[1:]:
        assert all(torch.equal(a, b) for a, b in zip(grads[0], other))
