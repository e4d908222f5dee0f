"""Interpolation and MoE routing kernels on the GPU against their CPU /
PyTorch references."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nd,mode,ac", [(1, "linear", False), (2, "linear", True), (3, "linear", False),
                                        (2, "nearest", False)])
def test_interpolate_cuda_matches_cpu_oracle(nd, mode, ac):
    from distdl_b200.functional.interpolate import interpolate
    torch.manual_seed(0)
    ins, outs = [9, 7, 6][:nd], [20, 15, 11][:nd]
    x = torch.randn(3, 4, *ins)
    # a slab of the output computed from a slab of the input, in global coordinates
    x_lo = [2] + [0] * (nd - 1)
    y_lo = [8] + [0] * (nd - 1)
    xs = x[:, :, 2:].contiguous()
    args = (x_lo, ins, ins, y_lo, outs, outs, None, mode, ac)
    xc = xs.clone().requires_grad_()
    yc = interpolate(xc, *args)
    xg = xs.cuda().requires_grad_()
    yg = interpolate(xg, *args)
    assert torch.allclose(yg.cpu(), yc, atol=1e-5)
    g = torch.randn_like(yc)
    yc.backward(g)
    yg.backward(g.cuda())
    assert torch.allclose(xg.grad.cpu(), xc.grad, atol=1e-4)


def test_moe_routing_kernels_match_torch():
    from distdl_b200.ops import moe
    torch.manual_seed(0)
    T, d, E, k, C = 300, 256, 8, 2, 96
    x = torch.randn(T, d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    ids = torch.randint(0, E, (T * k,), device="cuda", dtype=torch.int32)
    w = torch.rand(T, k, device="cuda", requires_grad=True)
    slot, counts = moe.assign_slots(ids, E, C)
    assert int(counts.sum()) == T * k
    ref_slot, ref_counts = moe.assign_slots(ids.cpu(), E, C)
    assert torch.equal(slot.cpu(), ref_slot) and torch.equal(counts.cpu(), ref_counts)
    for e in range(E):
        s = slot[(ids == e)]
        kept = s[s >= 0]
        assert kept.numel() == min(C, int(counts[e])) and kept.unique().numel() == kept.numel()
    buf = moe.dispatch(x, ids, slot, E, C, k)
    y = moe.combine(buf * 2, w, ids, slot, T, k)
    keep = (slot >= 0).reshape(T, k).float()
    ref = (2 * x.detach().float()) * (w.detach() * keep).sum(1, keepdim=True)
    assert (y.float() - ref).abs().max().item() < 3e-2 * ref.abs().max().item()
    g = torch.randn_like(y)
    y.backward(g)
    gx_ref = 2 * g.float() * (w.detach() * keep).sum(1, keepdim=True)
    assert (x.grad.float() - gx_ref).abs().max().item() < 3e-2 * gx_ref.abs().max().item()
    gw_ref = (2 * x.detach().float() * g.float()).sum(1, keepdim=True) * keep
    assert (w.grad - gw_ref).abs().max().item() < 3e-2 * gw_ref.abs().max().item() + 1e-3


@pytest.mark.parametrize("E,k,ld", [(8, 2, 8), (6, 1, 8), (16, 4, 16), (40, 8, 40), (64, 2, 64)])
def test_router_kernel_matches_softmax_topk_renormalisation(E, k, ld):
    """The router kernels (softmax, top-k, renormalised weights, probability sums; slots in pair-index
    order) and the backward kernel against the same computation written with PyTorch ops in fp32."""
    from distdl_b200.ops import moe
    torch.manual_seed(E * 10 + k)
    T, C = 777, 10_000
    logits = (torch.randn(T, ld, device="cuda") * 2).to(torch.bfloat16).requires_grad_()
    w, prob_sum, ids, slot, counts = moe.route(logits, E, k, C)
    lr = logits.detach().float()[:, :E].requires_grad_()
    probs = torch.softmax(lr, dim=-1)
    topw, topi = probs.topk(k, dim=-1)
    topw = topw / topw.sum(-1, keepdim=True)
    assert torch.equal(ids.reshape(T, k).long().sort(-1).values, topi.sort(-1).values)
    order = ids.reshape(T, k).long().argsort(-1), topi.argsort(-1)
    assert torch.allclose(w.gather(1, order[0]), topw.gather(1, order[1]), atol=1e-5)
    assert torch.allclose(prob_sum, probs.sum(0), rtol=1e-4, atol=1e-3)
    assert torch.equal(counts.long(), torch.bincount(ids.long(), minlength=E))
    # every pair has its own slot within its expert (nothing dropped at this capacity)
    assert (slot >= 0).all()
    key = ids.long() * C + slot.long()
    assert key.unique().numel() == key.numel()
    # gradients through the weights and through the probability sums (the auxiliary loss)
    gw = torch.randn(T, k, device="cuda")
    gp = torch.randn(E, device="cuda")
    (w * gw).sum().add((prob_sum * gp).sum()).backward()
    gw_ref = torch.zeros_like(gw).scatter(1, order[1], gw.gather(1, order[0]))     # same pairing as the kernel's order
    ((topw * gw_ref).sum() + (probs.sum(0) * gp).sum()).backward()
    got = logits.grad.float()
    assert torch.allclose(got[:, :E], lr.grad, atol=2e-2, rtol=2e-2), (got[:, :E] - lr.grad).abs().max()
    assert (got[:, E:] == 0).all()
    # a small capacity drops the late arrivals only
    _, _, ids2, slot2, _ = moe.route(logits.detach(), E, k, 8)
    for e in range(min(E, 4)):
        kept = (slot2[ids2 == e] >= 0).sum().item()
        assert kept == min(8, int((ids2 == e).sum()))
    # the slots are the arrival order by pair index (the same in every run): compare with the
    # index-ordered assignment written with PyTorch ops on the host
    ref_slot, ref_counts = moe.assign_slots(ids2.cpu(), E, 8)
    assert torch.equal(slot2.cpu(), ref_slot)
    ref_slot, ref_counts = moe.assign_slots(ids.cpu(), E, C)
    assert torch.equal(slot.cpu(), ref_slot) and torch.equal(counts.cpu(), ref_counts)


@pytest.mark.parametrize("dtype,shape", [(torch.float32, (6, 5, 7, 9)), (torch.bfloat16, (8, 16, 33)),
                                         (torch.float32, (3, 64, 4, 4, 5))])
def test_batch_norm_kernels_match_the_pytorch_formulation(dtype, shape):
    """Per-feature sum, sum of squared deviations and the normalise + affine map (forward and backward)
    against the same expressions written with PyTorch operations in fp32."""
    from distdl_b200.ops import batchnorm as bn
    torch.manual_seed(3)
    F = shape[1]
    stat = (1, F) + (1,) * (len(shape) - 2)
    x = torch.randn(*shape, device="cuda").to(dtype).requires_grad_()
    mean = torch.randn(stat, device="cuda").mul(0.1).to(dtype).requires_grad_()
    var = (torch.rand(stat, device="cuda") + 0.5).to(dtype).requires_grad_()
    gamma = (1 + 0.1 * torch.randn(stat, device="cuda")).to(dtype).requires_grad_()
    beta = (0.1 * torch.randn(stat, device="cuda")).to(dtype).requires_grad_()
    dims = [d for d in range(len(shape)) if d != 1]
    tol = 1e-4 if dtype == torch.float32 else 3e-2

    def close(a, b):
        err = (a.float() - b.float()).abs().max().item() / (b.float().abs().max().item() + 1e-6)
        assert err < tol, err

    ref = [t.detach().float().requires_grad_() for t in (x, mean, var, gamma, beta)]
    s, sr = bn.channel_sum(x), ref[0].sum(dims, keepdim=True)
    q, qr = bn.channel_sqdev(x, mean), ((ref[0] - ref[1]) ** 2).sum(dims, keepdim=True)
    y = bn.normalize(x, mean, var, gamma, beta, 1e-5)
    yr = ref[3] * (ref[0] - ref[1]) / torch.sqrt(ref[2] + 1e-5) + ref[4]
    close(s, sr)
    close(q, qr)
    close(y, yr)
    gs, gq, gy = torch.randn_like(sr), torch.randn_like(qr), torch.randn_like(yr)
    torch.autograd.backward([s, q, y], [gs.to(dtype), gq.to(dtype), gy.to(dtype)])
    torch.autograd.backward([sr, qr, yr], [gs.to(dtype).float(), gq.to(dtype).float(), gy.to(dtype).float()])
    for got, want in zip((x, mean, var, gamma, beta), ref):
        close(got.grad, want.grad)


@pytest.mark.parametrize("nd,kind,kernel,stride,dilation", [
    (1, "avg", (3,), (2,), (1,)), (1, "max", (3,), (1,), (2,)),
    (2, "avg", (2, 3), (2, 1), (1, 1)), (2, "max", (3, 3), (2, 2), (1, 1)), (2, "max", (2, 2), (1, 1), (2, 3)),
    (3, "avg", (2, 2, 2), (2, 2, 2), (1, 1, 1)), (3, "max", (3, 2, 3), (1, 2, 1), (1, 1, 2))])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_pooling_kernels_match_torch_on_a_cropped_view(nd, kind, kernel, stride, dilation, dtype):
    import torch.nn.functional as F

    from distdl_b200.ops import pooling
    torch.manual_seed(3)
    space = {1: (37,), 2: (19, 23), 3: (9, 11, 13)}[nd]
    full = torch.randn(3, 5, *[n + 3 for n in space], device="cuda").to(dtype)
    crop = (slice(None), slice(None)) + tuple(slice(1, 1 + n) for n in space)
    x = full.clone().requires_grad_()
    xr = full.float().clone().requires_grad_()
    view = x[crop]
    assert pooling.usable(view) and not view.is_contiguous()
    y = pooling.pool(view, kind, kernel, stride, dilation)
    if kind == "avg":
        fn = {1: F.avg_pool1d, 2: F.avg_pool2d, 3: F.avg_pool3d}[nd]
        yr = fn(xr[crop], kernel, stride=stride)
    else:
        fn = {1: F.max_pool1d, 2: F.max_pool2d, 3: F.max_pool3d}[nd]
        yr = fn(xr[crop], kernel, stride=stride, dilation=dilation)
    assert y.shape == yr.shape
    tol = 1e-6 if dtype == torch.float32 else 1e-2
    assert (y.float() - yr).abs().max().item() <= tol * (1 + yr.abs().max().item())
    dy = torch.randn_like(yr)
    y.backward(dy.to(dtype))
    yr.backward(dy)
    assert (x.grad.float() - xr.grad).abs().max().item() <= tol * (1 + xr.grad.abs().max().item()) * 4


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.bfloat16])
@pytest.mark.parametrize("mode,ac,n_in,n_out", [
    ("linear", False, (7, 9, 11), (14, 18, 22)),       # two outputs per input: four take an inner input
    ("linear", True, (5, 6, 7), (8, 9, 10)),
    ("linear", False, (9, 8, 6), (4, 5, 3)),           # fewer outputs than inputs: some inputs are taken by none
    ("linear", True, (3, 4, 2), (40, 60, 90)),         # more outputs per input than a thread keeps weights for
    ("linear", False, (1, 5, 3), (6, 1, 16)),          # extents of one
    ("nearest", False, (5, 3, 4), (10, 7, 33))])
def test_interpolation_kernels_over_scales(mode, ac, n_in, n_out, dtype):
    """1-, 2- and 3-dimensional, few planes and more planes than a thread takes at once, sub-ranges of the output,
    against the CPU code in fp64; an infinity reaches the outputs whose weight for it is not zero, and no other."""
    from distdl_b200.functional.interpolate import interpolate
    torch.manual_seed(5)
    tol = {torch.float32: 2e-6, torch.float64: 1e-13, torch.bfloat16: 8e-3}[dtype]     # a few roundings of the type
    for nd, planes, cut in ((1, 3, 0), (2, 70, 1), (3, 5, 1)):
        gi, go = list(n_in[3 - nd:]), list(n_out[3 - nd:])
        lo = [0] * nd
        hi = [max(1, n - cut) for n in go]
        x = torch.randn(1, planes, *gi).to(dtype)
        args = (lo, gi, gi, lo, hi, go, None, mode, ac)
        xc, xg = x.double().clone().requires_grad_(), x.cuda().requires_grad_()
        yc, yg = interpolate(xc, *args), interpolate(xg, *args)
        assert yg.dtype == dtype and yg.shape == yc.shape
        assert (yg.double().cpu() - yc).abs().max() <= tol * yc.abs().max()
        dy = torch.randn(yc.shape).to(dtype)
        yc.backward(dy.double())
        yg.backward(dy.cuda())
        assert (xg.grad.double().cpu() - xc.grad).abs().max() <= tol * (1 + xc.grad.abs().max())
        bad = x.clone()
        bad[:, :, -1] = float("inf")
        assert torch.equal(interpolate(bad.cuda(), *args).isfinite().cpu(), interpolate(bad.double(), *args).isfinite())


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.bfloat16])
@pytest.mark.parametrize("mode,ac,planes,n_in,n_out", [
    ("linear", False, 700, (35, 41), (70, 81)),          # rows: two segments of outputs, the last one shorter
    ("linear", True, 90, (34, 17, 9), (68, 34, 18)),     # sheets: nearly half a step, so that five outputs take some inputs
    ("linear", True, 40, (46, 23, 22), (69, 35, 33)),
    ("linear", False, 300, (70, 33, 30), (35, 16, 15)),  # fewer outputs than inputs: inputs that none takes
    ("nearest", False, 120, (33, 10, 9), (99, 21, 10))])
def test_interpolation_marches_over_large_tensors(mode, ac, planes, n_in, n_out, dtype):
    """A million outputs and more, most of which a thread takes sheet by sheet of a volume (row by row of an image):
    sub-ranges of the output, infinities; against the CPU code in fp64 with the bounds of the test above."""
    from distdl_b200.functional.interpolate import interpolate
    torch.manual_seed(6)
    tol = {torch.float32: 2e-6, torch.float64: 1e-13, torch.bfloat16: 8e-3}[dtype]
    gi, go = list(n_in), list(n_out)
    lo = [0] * len(gi)
    hi = [n - 1 for n in go]
    hi[-1] += go[-1] % 2                                   # an even extent at the end for some: pairs of bf16
    x = torch.randn(1, planes, *gi).to(dtype)
    args = (lo, gi, gi, lo, hi, go, None, mode, ac)
    xc, xg = x.double().clone().requires_grad_(), x.cuda().requires_grad_()
    yc, yg = interpolate(xc, *args), interpolate(xg, *args)
    assert (yg.double().cpu() - yc).abs().max() <= tol * yc.abs().max()
    dy = torch.randn(yc.shape).to(dtype)
    yc.backward(dy.double())
    yg.backward(dy.cuda())
    assert (xg.grad.double().cpu() - xc.grad).abs().max() <= tol * (1 + xc.grad.abs().max())
    bad = x.clone()
    bad[:, :, -1] = float("inf")
    assert torch.equal(interpolate(bad.cuda(), *args).isfinite().cpu(), interpolate(bad.double(), *args).isfinite())


@pytest.mark.parametrize("mode,ac,planes,n_in,n_out,forward,adjoint", [
    ("linear", False, 110, (35, 81), (70, 162), "fp32 fp64 bf16", ""),       # rows: three segments, the last one shorter
    ("linear", True, 140, (41, 120), (82, 161), "fp32 fp64 bf16", ""),       # rows of an odd length
    ("nearest", False, 60, (33, 20, 9), (99, 21, 20), "fp32 bf16", ""),
    ("linear", False, 70, (34, 12, 14), (51, 18, 21), "fp32 bf16", "fp32 fp64"),           # three outputs take an input
    ("linear", False, 235, (33, 8, 8), (66, 16, 16), "fp32 fp64 bf16", "fp32 fp64"),            # four
    ("linear", True, 85, (34, 17, 10), (68, 34, 20), "fp32 bf16", "fp32 fp64 bf16"),      # five
    ("linear", False, 160, (70, 33, 34), (35, 16, 17), "", "fp32 fp64")])                      # two, of some none
@pytest.mark.parametrize("slab", [False, True])
def test_interpolation_sheet_by_sheet(mode, ac, planes, n_in, n_out, forward, adjoint, slab):
    """Where the rules say that sheets (rows) are walked, whole tensors and slabs that begin and end inside, with a halo of
    their own input: segments and their ends, infinities; against the CPU code in fp64 with the bounds of the test above."""
    from test_interpolate_routes import marches

    from distdl_b200.functional.interpolate import interpolate
    for name, dtype, code in (("fp32", torch.float32, 0), ("fp64", torch.float64, 1), ("bf16", torch.bfloat16, 2)):
        torch.manual_seed(6)
        tol = {torch.float32: 2e-6, torch.float64: 1e-13, torch.bfloat16: 8e-3}[dtype]
        gi, go = list(n_in), list(n_out)
        lo, hi, x_lo, x_hi = [0] * len(gi), list(go), [0] * len(gi), list(gi)
        if slab:                                          # the leading dimension cut off at both ends, the last at its end
            lo[0], hi[0], hi[-1] = 3, go[0] - 2, go[-1] - 2
            step = (gi[0] - 1) / (go[0] - 1) if ac else gi[0] / go[0]
            at = lambda o: o * step if ac or mode == "nearest" else max(0.0, (o + 0.5) * step - 0.5)  # noqa: E731
            x_lo[0], x_hi[0] = int(at(lo[0])), min(int(at(hi[0] - 1)) + 2, gi[0])
        n_x, n_y = [b - a for a, b in zip(x_lo, x_hi)], [b - a for a, b in zip(lo, hi)]
        route = dict(linear=int(mode == "linear"), corners=int(ac), x_off=x_lo, y_off=lo, in_global=gi, out_global=go)
        assert marches(0, code, planes, n_x, n_y, **route) or name not in forward
        assert marches(1, code, planes, n_x, n_y, **route) or name not in adjoint
        x = torch.randn(1, planes, *n_x).to(dtype)
        args = (x_lo, x_hi, gi, lo, hi, go, None, mode, ac)
        xc, xg = x.double().clone().requires_grad_(), x.cuda().requires_grad_()
        yc, yg = interpolate(xc, *args), interpolate(xg, *args)
        assert (yg.double().cpu() - yc).abs().max() <= tol * yc.abs().max()
        dy = torch.randn(yc.shape).to(dtype)
        yc.backward(dy.double())
        yg.backward(dy.cuda())
        assert (xg.grad.double().cpu() - xc.grad).abs().max() <= tol * (1 + xc.grad.abs().max())
        bad = x.clone()
        bad[:, :, -1] = float("inf")
        assert torch.equal(interpolate(bad.cuda(), *args).isfinite().cpu(), interpolate(bad.double(), *args).isfinite())


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.bfloat16])
@pytest.mark.parametrize("mode", ["linear", "nearest"])
@pytest.mark.parametrize("n_in", [(0,), (0, 5), (4, 0), (0, 3, 4), (3, 0, 4), (3, 4, 0)])
def test_interpolation_of_an_empty_slab(n_in, mode, dtype):
    """A worker may hold none of the input's entries along a dimension: zeros, as the CPU code writes them, and a
    gradient without elements."""
    from distdl_b200.functional.interpolate import interpolate
    nd = len(n_in)
    n_global, n_out = [6] * nd, [7] * nd
    args = ([2] * nd, [2 + n for n in n_in], n_global, [0] * nd, n_out, n_out, None, mode, False)
    x = torch.empty(2, 3, *n_in, device="cuda", dtype=dtype, requires_grad=True)
    y = interpolate(x, *args)
    assert y.dtype == dtype and torch.equal(y.double().cpu(), interpolate(x.detach().double().cpu(), *args))
    assert y.shape == (2, 3, *n_out) and not y.any()
    assert torch.autograd.grad(y.sum(), x)[0].shape == x.shape


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape,affine,track", [
    ((6, 5, 7, 9), True, True),             # planes of 63: units shared between neighbours
    ((4, 3, 64), True, False),
    ((3, 70, 2), False, True),              # many features, planes smaller than a unit
    ((2, 2, 37, 41, 13), True, True),       # several CTAs per plane
    ((5, 4), True, True)])                  # no dimension besides batch and feature
def test_batch_norm_layer_fused_on_one_worker(shape, affine, track, dtype):
    """Output, gradients and running statistics of the layer against PyTorch in fp64, with a mean far from zero."""
    import distdl_b200
    from distdl_b200 import backends
    from distdl_b200.nn import DistributedBatchNorm
    distdl_b200.config.set_backend("native", "cupy")
    torch.manual_seed(9)
    P = backends.backend.Partition().create_partition_inclusive([0]).create_cartesian_topology_partition([1] * len(shape))
    F = shape[1]
    layer = DistributedBatchNorm(P, F, affine=affine, track_running_stats=track, device="cuda", dtype=dtype)
    x = (torch.randn(shape, device="cuda") * 2 + (50 if dtype == torch.float32 else 5)).to(dtype).requires_grad_()
    w = torch.ones(F, dtype=torch.float64, device="cuda")
    b = torch.zeros(F, dtype=torch.float64, device="cuda")
    if affine:
        with torch.no_grad():
            layer.gamma.add_(torch.randn_like(layer.gamma), alpha=0.3)
            layer.beta.add_(torch.randn_like(layer.beta), alpha=0.3)
        w, b = layer.gamma.detach().double().flatten(), layer.beta.detach().double().flatten()
    xr, w, b = x.detach().double().requires_grad_(), w.requires_grad_(), b.requires_grad_()
    rm, rv = torch.zeros(F, device="cuda").double(), torch.ones(F, device="cuda").double()
    yr = torch.nn.functional.batch_norm(xr, rm, rv, w, b, True, 0.1, layer.eps)
    y = layer(x)
    dy = torch.randn(shape, device="cuda").to(dtype)
    y.backward(dy)
    yr.backward(dy.double())
    # fp32: subtracting a mean of 50 from values of spread 2 leaves 25 eps; bf16: the statistics are bf16 as well
    # (a mean of 5 to 2^-8 beside a spread of 2: 0.01)
    tol = 2e-5 if dtype == torch.float32 else 2e-2

    def close(a, r, floor=0.0):
        assert (a.double().flatten() - r.flatten()).abs().max() <= tol * (r.abs().max() + floor)

    close(y, yr)
    close(x.grad, xr.grad, floor=float(dy.double().abs().max()))
    if affine:
        close(layer.gamma.grad, w.grad, floor=1.0)
        close(layer.beta.grad, b.grad, floor=1.0)
    if track:
        close(layer.running_mean, rm)
        close(layer.running_var, rv)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("space,pads", [((7,), (0, 1)), ((5, 8), (1, 1, 1, 1)), ((6, 5), (0, 3, 2, 0)),
                                        ((3, 4, 13), (2, 1, 0, 0, 1, 0)), ((4, 300), (4, 0, 0, 0))])
def test_padding_kernel_moves_the_same_bits(space, pads, dtype):
    """Widths on either side, row lengths of every divisibility, few and many planes, 0 and -inf; gradients of
    the first and second order; an input that is not contiguous and a function transform take the library's way."""
    import torch.nn.functional as F

    from distdl_b200.ops.pad import pad
    torch.manual_seed(8)
    for planes in (1, 37):
        x = torch.randn(2, planes, *space, device="cuda").to(dtype).requires_grad_()
        xr = x.detach().clone().requires_grad_()
        for value in (0.0, float("-inf")):
            y, yr = pad(x, pads, value), F.pad(xr, pads, value=value)
            assert "ShiftCopy" in type(y.grad_fn).__name__ and torch.equal(y, yr)
        dy = torch.randn_like(yr)
        g, = torch.autograd.grad((pad(x, pads) * 1).pow(2).mul(dy).sum(), x, create_graph=True)
        gr, = torch.autograd.grad((F.pad(xr, pads) * 1).pow(2).mul(dy).sum(), xr, create_graph=True)
        assert torch.equal(g, gr)
        assert torch.equal(torch.autograd.grad(g.sum(), x)[0], torch.autograd.grad(gr.sum(), xr)[0])
    assert torch.equal(pad(x.transpose(0, 1), pads), F.pad(x.transpose(0, 1), pads))
    assert torch.equal(pad(x, pads[:2]), F.pad(x, pads[:2]))              # the last dimension alone
    assert torch.equal(torch.func.vmap(lambda t: pad(t, pads))(x.detach()[None]), F.pad(x.detach(), pads)[None])
    assert "pad" in str(torch.jit.trace(lambda t: pad(t, pads), x.detach()).graph)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("kind,kernel,stride,space", [
    ("max", (2, 2), (2, 2), (12, 14)), ("avg", (2, 2), (2, 2), (6, 6)), ("max", (3, 2), (1, 2), (9, 8)),
    ("avg", (3, 3, 2), (2, 2, 2), (7, 9, 6)), ("max", (2, 2, 2), (2, 2, 2), (4, 5, 130)), ("max", (2,), (2,), (10,))])
def test_pooling_backward_by_pairs(kind, kernel, stride, space, dtype):
    """Windows of two that tile the last dimension, with every form of window along the others."""
    import torch.nn.functional as F

    from distdl_b200.ops import pooling
    torch.manual_seed(10)
    nd = len(space)
    x = torch.randn(3, 70, *space, device="cuda").to(dtype).requires_grad_()
    xr = x.detach().double().requires_grad_()
    fn = getattr(F, f"{kind}_pool{nd}d")
    y, yr = pooling.pool(x, kind, kernel, stride), fn(xr, kernel, stride=stride)
    dy = torch.randn(yr.shape, device="cuda").to(dtype)
    y.backward(dy)
    yr.backward(dy.double())
    tol = 1e-6 if dtype == torch.float32 else 8e-3           # fp32 sums of a few terms; one rounding to bf16
    assert (y.double() - yr).abs().max() <= tol * yr.abs().max()
    if dtype == torch.float32 or kind == "avg" or stride == kernel:
        assert (x.grad.double() - xr.grad).abs().max() <= tol * xr.grad.abs().max()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("space,pads,C", [((5, 7), (1, 1, 1, 1), 8), ((64, 3), (0, 2, 1, 0), 72), ((3, 4, 13), (1, 1, 0, 0, 2, 1), 136),
                                          ((9, 9, 9), (0, 0, 0, 0, 0, 0), 24)])
def test_padding_into_channels_last_and_back(space, pads, C, dtype):
    """Channels below, on and beyond a tile, positions beyond a tile; the bits of padding and crop, to the second
    order."""
    import torch.nn.functional as F

    from distdl_b200.ops.pad import channels_first, channels_last_usable, pad_channels_last
    torch.manual_seed(12)
    x = torch.randn(3, C, *space, device="cuda").to(dtype).requires_grad_()
    xr = x.detach().clone().requires_grad_()
    nd = len(space)
    w = torch.empty(16, C, *[3] * nd, device="cuda", dtype=dtype)
    assert channels_last_usable(x, pads, w) and not channels_last_usable(x.float(), pads, w.float())
    y, yr = pad_channels_last(x, pads), F.pad(xr, pads)
    fmt = torch.channels_last if len(space) == 2 else torch.channels_last_3d
    assert y.is_contiguous(memory_format=fmt) and torch.equal(y, yr)
    z = channels_first(y)
    assert z.is_contiguous() and torch.equal(z, yr)
    dy = torch.randn_like(yr)
    g, = torch.autograd.grad((z * 1).pow(2).mul(dy).sum(), x, create_graph=True)
    gr, = torch.autograd.grad((yr * 1).pow(2).mul(dy).sum(), xr, create_graph=True)
    assert g.is_contiguous() and torch.equal(g, gr)
    assert torch.equal(torch.autograd.grad(g.sum(), x)[0], torch.autograd.grad(gr.sum(), xr)[0])


@pytest.mark.parametrize("space,C", [((2, 17, 19), 8), ((30, 21), 64), ((5, 300), 16), ((11, 13, 7), 40), ((33, 34), 48),
                                     ((12, 31), 56), ((65, 3), 128), ((330, 301), 8), ((17, 77, 79), 24), ((301, 333), 40),
                                     ((221, 247), 88)])
def test_channel_tiles_follow_the_number_of_channels(space, C):
    """Tiles of 4 to 32 pairs of channels, positions on and beyond their edges, channels that do not fill the last one; the
    narrow ones into channels-last memory only for the last sizes, back for all."""
    import torch.nn.functional as F

    from distdl_b200.ops.pad import channels_first, pad_channels_last
    torch.manual_seed(13)
    x = torch.randn(2, C, *space, device="cuda").bfloat16()
    pads = (1, 0, 2, 1) + ((1, 1) if len(space) == 3 else ())
    y = pad_channels_last(x, pads)
    assert torch.equal(y, F.pad(x, pads)) and torch.equal(channels_first(y), F.pad(x, pads))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("batch,space,cin,cout,kernel,stride,bias", [
    (2, (13, 17), 16, 24, 3, 1, True), (2, (12, 12), 8, 8, 1, 1, False), (2, (14, 14), 16, 16, 3, 2, False),
    (2, (9, 9), 12, 8, 3, 1, True), (5, (1, 40), 32, 16, 3, 1, False), (2, (11, 9, 10), 24, 16, 3, 1, True),
    (16, (3, 3, 3), 48, 48, 3, 1, False), (1, (5, 86, 1), 32, 32, 3, 1, True), (1, (24, 84, 73), 64, 56, 3, 1, False),
    (3, (16, 1, 24), 40, 128, 3, 1, False)])
def test_feature_convolution_on_one_worker(batch, space, cin, cout, kernel, stride, bias, dtype):
    """Layouts in and out, and output and gradients as close to fp64 as the library's convolution of the padded input,
    channels first: whatever precision that has for this shape.  Channel counts that keep this way too, extents of one,
    slabs, small volumes of a large batch."""
    import torch.nn.functional as F

    import distdl_b200
    from distdl_b200 import backends, nn
    distdl_b200.config.set_backend("native", "cupy")
    torch.manual_seed(13)
    nd = len(space)
    P = backends.backend.Partition().create_partition_inclusive([0]).create_cartesian_topology_partition([1] * (nd + 2))
    cls = {2: nn.DistributedFeatureConv2d, 3: nn.DistributedFeatureConv3d}[nd]
    layer = cls(P, cin, cout, kernel, stride=stride, padding=kernel // 2, bias=bias, device="cuda", dtype=dtype)
    x = torch.randn(batch, cin, *space, device="cuda").to(dtype).requires_grad_()
    params = [layer.weight] + ([layer.bias] if bias else [])
    conv = getattr(F, f"conv{nd}d")
    results = []
    y = layer(x)
    dy = torch.randn(y.shape, device="cuda").to(dtype)
    results.append([y, *torch.autograd.grad(y, [x] + params, dy)])
    assert y.is_contiguous() and y.dtype == dtype and results[0][1].is_contiguous()
    for t in ([x] + params, [t.detach().double().requires_grad_() for t in [x] + params]):
        z = conv(F.pad(t[0], (kernel // 2,) * 2 * nd), *t[1:], stride=stride)
        results.append([z, *torch.autograd.grad(z, t, dy.to(z.dtype))])
    for a, b, r in zip(*results):
        assert a.shape == r.shape
        # (sums in another order, where the layouts differ or the library adds atomically)
        assert (a.double() - r).norm() <= 1.1 * (b.double() - r).norm() + 1e-7 * r.norm()


def test_feature_convolution_with_the_precision_of_fp32_set_for_convolutions_alone():
    """``torch.backends.cudnn.conv.fp32_precision``, beside which the older ``allow_tf32`` cannot be read."""
    import distdl_b200
    from distdl_b200 import backends, nn
    distdl_b200.config.set_backend("native", "cupy")
    P = backends.backend.Partition().create_partition_inclusive([0]).create_cartesian_topology_partition([1] * 5)
    layer = nn.DistributedFeatureConv3d(P, 16, 16, 3, padding=1, device="cuda")
    x = torch.randn(1, 16, 30, 30, 30, device="cuda")
    want = torch.nn.functional.conv3d(x.double(), layer.weight.double(), layer.bias.double(), padding=1)
    before = torch.backends.cudnn.conv.fp32_precision
    try:
        torch.backends.cudnn.conv.fp32_precision = "ieee"
        y = layer(x)
    finally:
        torch.backends.cudnn.conv.fp32_precision = before
    assert (y.double() - want).norm() <= 1e-6 * want.norm()


def test_batch_norm_on_one_worker_matches_the_passes_between_workers():
    """bf16: the fused passes round where the exchange between workers does: the same outputs, statistics and gradients
    bit for bit, but for features whose sums, added in another order, fall on the other side of a rounding."""
    import distdl_b200
    from distdl_b200 import backends
    from distdl_b200.nn import DistributedBatchNorm
    distdl_b200.config.set_backend("native", "cupy")
    P = backends.backend.Partition().create_partition_inclusive([0]).create_cartesian_topology_partition([1] * 4)
    outs = []
    for fused in (True, False):
        torch.manual_seed(21)
        layer = DistributedBatchNorm(P, 48, device="cuda", dtype=torch.bfloat16)
        if not fused:
            layer._alone = lambda *a: False
        x = (torch.randn(4, 48, 37, 29, device="cuda") * 2 + 1).bfloat16().requires_grad_()
        dy = torch.randn(4, 48, 37, 29, device="cuda").bfloat16()
        for _ in range(2):
            y = layer(x)
        g = torch.autograd.grad(y, [x, layer.gamma, layer.beta], dy)
        outs.append([y.detach(), layer.running_mean.clone(), layer.running_var.clone(), *g])
    for a, b in zip(*outs):
        assert (a != b).float().mean() < 0.1
        assert (a.double() - b.double()).norm() <= 8e-3 * b.double().norm()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(4, 3, 16), (2, 5, 3, 64)])
def test_batch_norm_of_large_constant_features(shape, dtype):
    """Values whose square is beyond fp32, but whose deviations from the mean are not."""
    import distdl_b200
    from distdl_b200 import backends
    from distdl_b200.nn import DistributedBatchNorm
    distdl_b200.config.set_backend("native", "cupy")
    P = backends.backend.Partition().create_partition_inclusive([0]).create_cartesian_topology_partition([1] * len(shape))
    layer = DistributedBatchNorm(P, shape[1], device="cuda", dtype=dtype)
    x = torch.full(shape, 2.0 ** 66, device="cuda", dtype=dtype).requires_grad_()
    y = layer(x)
    assert not y.any()                                    # powers of two: sums and means are exact
    y.backward(torch.ones_like(y))
    assert x.grad.isfinite().all() and (layer.running_mean.float() - 0.1 * 2.0 ** 66).abs().max() < 2.0 ** 58
    assert (layer.running_var.float() - 0.9).abs().max() < 0.01


@pytest.mark.parametrize("nd,dtype", [(2, torch.bfloat16), (3, torch.bfloat16), (3, torch.float32)])
def test_feature_convolution_with_batched_gradients(nd, dtype):
    """Gradients of several incoming ones at once (a function transform around the backward pass only)."""
    import distdl_b200
    from distdl_b200 import backends, nn
    from distdl_b200.ops.pad import pad
    distdl_b200.config.set_backend("native", "cupy")
    torch.manual_seed(18)
    P = backends.backend.Partition().create_partition_inclusive([0]).create_cartesian_topology_partition([1] * (nd + 2))
    cls = {2: nn.DistributedFeatureConv2d, 3: nn.DistributedFeatureConv3d}[nd]
    layer = cls(P, 16, 16, 3, padding=1, device="cuda", dtype=dtype)
    x = torch.randn(1, 16, *[5] * nd, device="cuda").to(dtype).requires_grad_()
    y = layer(x)
    dys = torch.randn(3, *y.shape, device="cuda").to(dtype)
    got = torch.autograd.grad(y, (x, layer.weight), dys, is_grads_batched=True, retain_graph=True)
    assert got[0].is_contiguous()
    for k in range(3):
        for a, b in zip(got, torch.autograd.grad(y, (x, layer.weight), dys[k], retain_graph=True)):
            # the same products in another order: bf16 results, or tf32 operands
            assert (a[k].double() - b.double()).norm() <= 8e-3 * b.double().norm()
    p = pad(x, (1, 1, 0, 2, 1, 0)[:2 * nd])
    dys = torch.randn(3, *p.shape, device="cuda").to(dtype)
    got, = torch.autograd.grad(p, x, dys, is_grads_batched=True, retain_graph=True)
    for k in range(3):
        assert torch.equal(got[k], torch.autograd.grad(p, x, dys[k], retain_graph=True)[0])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_batch_norm_weights_may_change_before_the_backward_pass(dtype):
    """The gradient is that of the weights of the forward pass."""
    import distdl_b200
    from distdl_b200 import backends
    from distdl_b200.nn import DistributedBatchNorm
    distdl_b200.config.set_backend("native", "cupy")
    torch.manual_seed(20)
    P = backends.backend.Partition().create_partition_inclusive([0]).create_cartesian_topology_partition([1] * 4)
    layer = DistributedBatchNorm(P, 6, device="cuda", dtype=dtype)
    x = torch.randn(3, 6, 5, 7, device="cuda").to(dtype).requires_grad_()
    dy = torch.randn(3, 6, 5, 7, device="cuda").to(dtype)
    want = torch.autograd.grad(layer(x), (x, layer.gamma, layer.beta), dy)
    y = layer(x)
    with torch.no_grad():
        layer.gamma.mul_(3)
        layer.beta.add_(1)
    for a, b in zip(torch.autograd.grad(y, (x, layer.gamma, layer.beta), dy), want):
        assert torch.equal(a, b)
