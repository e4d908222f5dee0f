"""Memory-bound kernels against plain fp32 PyTorch references."""
import pytest
import torch

from distdl_b200 import _native
from distdl_b200.ops._util import stream_ptr

pytestmark = pytest.mark.gpu


def _close(a, b, tol=2e-2):
    err = (a.float() - b.float()).abs().max().item()
    scale = b.float().abs().max().item() + 1e-6
    assert err / scale < tol, f"err {err} scale {scale}"


@pytest.mark.parametrize("d", [1024, 1600, 4096])
@pytest.mark.parametrize("rms", [True, False])
def test_norm_fwd_bwd(d, rms):
    from distdl_b200.ops import layer_norm, rms_norm
    torch.manual_seed(0)
    rows = 777
    x = torch.randn(rows, d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = (1 + 0.1 * torch.randn(d, device="cuda")).to(torch.bfloat16).requires_grad_()
    b = None if rms else (0.1 * torch.randn(d, device="cuda")).to(torch.bfloat16).requires_grad_()
    y = rms_norm(x, w, 1e-5) if rms else layer_norm(x, w, b, 1e-5)
    dy = torch.randn_like(y)
    y.backward(dy)
    xr = x.detach().float().requires_grad_()
    wr = w.detach().float().requires_grad_()
    if rms:
        yr = xr * torch.rsqrt(xr.pow(2).mean(-1, keepdim=True) + 1e-5) * wr
    else:
        br = b.detach().float().requires_grad_()
        yr = torch.nn.functional.layer_norm(xr, (d,), wr, br, 1e-5)
    yr.backward(dy.float())
    _close(y, yr)
    _close(x.grad, xr.grad)
    _close(w.grad, wr.grad)
    if not rms:
        _close(b.grad, br.grad)


@pytest.mark.parametrize("rms", [True, False])
def test_add_norm_returns_sum_and_norm_with_the_gradient_of_both(rms):
    """The residual add fused into the norm: both outputs and, in backward, gradients arriving on both."""
    from distdl_b200.ops import add_layer_norm, add_rms_norm
    torch.manual_seed(1)
    rows, d = 515, 4096
    x = torch.randn(rows, d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    r = torch.randn(rows, d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = (1 + 0.1 * torch.randn(d, device="cuda")).to(torch.bfloat16).requires_grad_()
    b = None if rms else (0.1 * torch.randn(d, device="cuda")).to(torch.bfloat16).requires_grad_()
    s, y = add_rms_norm(x, r, w, 1e-5) if rms else add_layer_norm(x, r, w, b, 1e-5)
    ds, dy = torch.randn_like(s), torch.randn_like(y)
    torch.autograd.backward([s, y], [ds, dy])
    xr, rr = x.detach().float().requires_grad_(), r.detach().float().requires_grad_()
    wr = w.detach().float().requires_grad_()
    sr = (xr + rr).detach().to(torch.bfloat16).float() + (xr + rr - (xr + rr).detach())     # the stored sum is bf16
    if rms:
        yr = sr * torch.rsqrt(sr.pow(2).mean(-1, keepdim=True) + 1e-5) * wr
    else:
        br = b.detach().float().requires_grad_()
        yr = torch.nn.functional.layer_norm(sr, (d,), wr, br, 1e-5)
    torch.autograd.backward([sr, yr], [ds.float(), dy.float()])
    _close(s, sr)
    _close(y, yr)
    _close(x.grad, xr.grad)
    _close(r.grad, rr.grad)
    _close(w.grad, wr.grad)
    # only the sum is used downstream: the gradient passes through untouched
    x2 = x.detach().requires_grad_()
    s2, _ = add_rms_norm(x2, r.detach(), w.detach(), 1e-5)
    s2.backward(ds)
    assert torch.equal(x2.grad, ds)


def test_rope_on_the_projection_output_rotates_in_place_without_copying_gradients():
    from distdl_b200.ops import rope_
    torch.manual_seed(0)
    b, seq, hq, hk, hd = 2, 64, 4, 2, 128
    lin = torch.randn(b, seq, (hq + 2 * hk) * hd, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    y = lin * 1.0                                                     # a non-leaf, like a projection's output
    ref = rope_(y.detach().clone().reshape(b * seq, hq + 2 * hk, hd), seq, hq + hk, theta=10000.0)
    out = rope_(y, seq, hq + hk, theta=10000.0, layout=(b * seq, hq + 2 * hk, hd))
    assert out.shape == lin.shape and torch.equal(out.reshape(ref.shape), ref)
    g = torch.randn_like(out)
    out.backward(g.clone())           # the node rotates the gradient it is handed in place
    # the adjoint of a rotation is the inverse rotation: rotating the gradient forward again gives g
    back = rope_(lin.grad.clone().reshape(b * seq, hq + 2 * hk, hd), seq, hq + hk, theta=10000.0)
    _close(back, g.reshape(back.shape), 1e-2)


def test_swiglu_gelu():
    from distdl_b200.ops import gelu, swiglu
    torch.manual_seed(0)
    gu = torch.randn(300, 2 * 512, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    y = swiglu(gu)
    dy = torch.randn_like(y)
    y.backward(dy)
    r = gu.detach().float().requires_grad_()
    yr = torch.nn.functional.silu(r[:, :512]) * r[:, 512:]
    yr.backward(dy.float())
    _close(y, yr)
    _close(gu.grad, r.grad)
    x = torch.randn(300, 640, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    y = gelu(x)
    y.backward(dy[:, :1].expand(300, 640).contiguous())
    r = x.detach().float().requires_grad_()
    yr = torch.nn.functional.gelu(r, approximate="tanh")
    yr.backward(dy[:, :1].expand(300, 640).float())
    _close(y, yr)
    _close(x.grad, r.grad)


def test_rope_roundtrip_and_reference():
    from distdl_b200.ops import rope_, rope_table
    torch.manual_seed(0)
    seq, hq, hk, hd = 64, 4, 2, 128
    tokens = 2 * seq
    qkv = torch.randn(tokens, hq + 2 * hk, hd, device="cuda", dtype=torch.bfloat16)
    ref_in = qkv.clone()
    out = rope_(qkv.clone(), seq, hq + hk, theta=10000.0)
    table = rope_table(seq, hd, 10000.0, qkv.device)
    pos = torch.arange(tokens, device="cuda") % seq
    cos = table[pos, :, 0].unsqueeze(1)
    sin = table[pos, :, 1].unsqueeze(1)
    x = ref_in[:, : hq + hk].float()
    a, b = x[..., : hd // 2], x[..., hd // 2:]
    ref = torch.cat([a * cos - b * sin, b * cos + a * sin], -1)
    _close(out[:, : hq + hk], ref)
    assert torch.equal(out[:, hq + hk:], ref_in[:, hq + hk:])


def test_embedding_and_xent():
    from distdl_b200.ops import cross_entropy_, embedding
    torch.manual_seed(0)
    V, d, T = 1000, 256, 333
    table = torch.randn(V, d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    ids = torch.randint(0, V, (T,), device="cuda")
    e = embedding(ids, table)
    assert torch.equal(e, table.detach()[ids])
    g = torch.randn_like(e)
    e.backward(g)
    ref = torch.zeros(V, d, device="cuda")
    ref.index_add_(0, ids, g.float())
    _close(table.grad, ref)

    ld = 1008
    logits = torch.randn(T, ld, device="cuda", dtype=torch.bfloat16)
    lr = logits[:, :V].detach().float().requires_grad_()
    tgt = torch.randint(0, V, (T,), device="cuda")
    loss_ref = torch.nn.functional.cross_entropy(lr, tgt)
    loss_ref.backward()
    lg = logits.clone().requires_grad_()
    work = lg * 1  # non-leaf that the op may overwrite
    loss = cross_entropy_(work, tgt, vocab=V, unit_grad=True)
    loss.backward()
    assert abs(loss.item() - loss_ref.item()) < 2e-2
    _close(lg.grad[:, :V], lr.grad, tol=3e-2)
    assert lg.grad[:, V:].abs().max().item() == 0


def test_adamw_matches_torch():
    from distdl_b200.ops import adamw_step_, sumsq_
    torch.manual_seed(0)
    n = 100003
    p = torch.randn(n, device="cuda")
    g = torch.randn(n, device="cuda")
    ref = torch.nn.Parameter(p.clone())
    opt = torch.optim.AdamW([ref], lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    m = torch.zeros_like(p)
    v = torch.zeros_like(p)
    pb = torch.empty(n, device="cuda", dtype=torch.bfloat16)
    master = p.clone()
    for step in range(1, 4):
        ref.grad = g.clone()
        opt.step()
        gg = g.clone()
        adamw_step_(master, m, v, gg, pb, lr=1e-2, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=step)
        assert gg.abs().max().item() == 0
    assert (master - ref.detach()).abs().max().item() < 1e-5
    _close(pb, master)
    out = torch.zeros(1, device="cuda")
    sumsq_(g, out)
    assert abs(out.item() - (g.double() ** 2).sum().item()) / n < 1e-3


def test_accumulate_into_fp32_buffer():
    """acc(fp32) += scale * g(bf16): the cast-and-add kernel of the gradient accumulators."""
    from distdl_b200.ops.optim import accumulate_f32_
    torch.manual_seed(2)
    n = 1 << 20
    acc = torch.randn(n, device="cuda")
    g = torch.randn(n, device="cuda").to(torch.bfloat16)
    want = acc + 0.5 * g.float()
    accumulate_f32_(acc, g, 0.5)
    assert torch.allclose(acc, want, atol=1e-6)
    g32 = torch.randn(1000, device="cuda")                # other dtypes take the PyTorch path
    acc2 = torch.zeros(1000, device="cuda")
    accumulate_f32_(acc2, g32)
    assert torch.equal(acc2, g32)


@pytest.mark.parametrize("rows,n", [(1, 8), (33, 264), (7, 6400), (4096, 256), (5000, 1600)])
def test_column_sum(rows, n):
    """Fewer rows than a CTA takes, columns beyond the last full group of 256, accumulation; the same bits in
    every run."""
    from distdl_b200.ops.gemm import column_sum
    torch.manual_seed(4)
    x = torch.randn(rows, n, device="cuda").bfloat16()
    ref = x.double().sum(0)
    tol = 2e-6 * x.double().abs().sum(0).max()            # fp32 sums of bf16 values, in blocks
    out = column_sum(x)
    assert (out.double() - ref).abs().max() <= tol and torch.equal(out, column_sum(x))
    acc = torch.randn(n, device="cuda")
    want = acc.double() + ref
    assert column_sum(x, acc) is acc and (acc.double() - want).abs().max() <= tol + 1e-6


@pytest.mark.parametrize("zero,kept", [(True, False), (True, True), (False, False)])
def test_embedding_and_linear_gradients_reach_the_fp32_accumulator(zero, kept):
    """Parameters with an optimizer's accumulator: two backward passes add up there in fp32 and leave no .grad;
    repeated ids, an accumulator that is not 16-byte aligned."""
    import distdl_b200
    from distdl_b200 import backends, nn
    distdl_b200.config.set_backend("native", "cupy")
    torch.manual_seed(6)
    world = backends.backend.Partition().create_partition_inclusive([0])
    P = world.create_cartesian_topology_partition([1, 1, 1])
    V, d, out = 50, 24, 40
    kw = dict(dtype=torch.bfloat16, auto_clear_buffer=not kept)
    embed = nn.DistributedEmbeddingZero(P, V, d, **kw)
    if zero:
        ag = nn.DistributedLinearAllGatherZero(P, d, out, bias=True, **kw)
        rs = nn.DistributedLinearReduceScatterZero(P, out, d, bias=True, **kw)
    else:
        ag = nn.DistributedLinearAllGather(P, d, out, bias=True, dtype=torch.bfloat16)
        rs = nn.DistributedLinearReduceScatter(P, out, d, bias=True, dtype=torch.bfloat16)
    params = [embed.weight, ag.weight, ag.bias, rs.weight, rs.bias]
    for p in params:
        shift = 1 if p is embed.weight else 0
        p.main_grad_view = torch.zeros(p.numel() + 8, device="cuda")[shift:shift + p.numel()]
    ids = torch.randint(0, 7, (2, 64), device="cuda")
    gs = [torch.randn(2, 64, d, device="cuda").bfloat16() for _ in range(2)]
    w = [p.detach().double().requires_grad_() for p in params]
    w1 = (lambda t: t.reshape(d, out)) if zero else (lambda t: t.reshape(out, d).t())
    for g in gs:
        rs(ag(embed(ids))).backward(g)
        h = torch.nn.functional.embedding(ids, w[0].reshape(V, d)) @ w1(w[1]) + w[2].reshape(out)
        (h @ w[3].reshape(d, out).t() + w[4].reshape(d)).backward(g.double())
    for m in (embed, ag, rs):
        if hasattr(m, "clear_weight_buffer"):
            m.clear_weight_buffer()
    for p, r in zip(params, w):
        assert p.grad is None
        err = (p.main_grad_view.double() - r.grad.flatten()).norm() / r.grad.norm()
        assert err < 1e-2, err                  # bf16 activations and incoming gradients


@pytest.mark.parametrize("V,ld", [(5, 8), (4099, 4104), (40003, 40008), (16384, 16384)])
@pytest.mark.parametrize("fill", [torch.finfo(torch.bfloat16).min, float("-inf"), torch.finfo(torch.bfloat16).max, -1e38])
def test_xent_with_masked_and_extreme_logits(V, ld, fill):
    """Masks over whole and partial vectors, over all columns but one, in front of and behind what a thread reads
    first, masked targets and ignored rows, in rows of less and of more than one sweep of the CTA: loss and gradient
    of each row against fp64."""
    from distdl_b200 import _native
    from distdl_b200.ops._util import stream_ptr
    torch.manual_seed(11)
    low, rows = fill < 0, 8
    lg = torch.randn(rows, ld, device="cuda").mul_(3).bfloat16()
    third = V // 3
    if low:                                                 # (fp32 has no room for a log beside several of 3e38)
        lg[0, :third] = fill                                # whole vectors and one in part, seen first; the target
        lg[1, -(ld - V) - third - 1:] = fill                # seen last, up to the partial vector
        lg[2, torch.rand(ld, device="cuda") < 0.9] = fill   # here and there
        lg[3, :] = fill                                     # all but one column
        lg[3, V - 1] = 2.0
        lg[4, :third] = -torch.finfo(torch.bfloat16).max    # two kinds of mask beside each other
        lg[4, third:2 * third] = float("-inf")
    lg[5, 0] = fill                                         # one logit
    tgt = torch.tensor([0, 0, V // 2, V - 1, V - 1, 0, -100, V], device="cuda")
    lg[2, V // 2] = 1.0
    scale = 0.5
    a = lg[:, :V].double()
    ok = (tgt >= 0) & (tgt < V)
    t = tgt.clamp(0, V - 1)
    lse = torch.logsumexp(a, 1)
    want = torch.where(ok, lse - a.gather(1, t[:, None])[:, 0], 0.0)
    grad = torch.softmax(a, 1)
    grad[torch.arange(rows), t] -= 1.0
    grad = torch.where(ok[:, None], grad * scale, 0.0)
    loss = torch.empty(rows, device="cuda")
    _native.call("dd_xent", lg.data_ptr(), tgt.data_ptr(), loss.data_ptr(), rows, V, ld, scale, stream_ptr())
    same = (loss.double() == want) | (torch.isinf(want) & (loss == want.float()))
    # fp32: a few roundings of the largest value that takes part, and of a sum of V terms added in blocks
    assert (same | ((loss.double() - want).abs() <= 1e-6 * (lse.abs() + want.abs()) + 1e-5)).all(), (loss, want)
    # probabilities carry the rounding of lse (2^-24 |lse|) and are rounded to bf16
    tol = grad.abs() * (2 ** -8 + 4e-7 * lse.abs().clamp(max=1e4)[:, None]) + 1e-6
    assert ((lg[:, :V].double() - grad).abs() <= tol).all()
    assert (lg[:, V:] == 0).all()


@pytest.mark.parametrize("zero,kept", [(True, False), (True, True), (False, False)])
def test_hooks_and_partial_backward_passes_see_the_gradients(zero, kept):
    """Parameters with an optimizer's accumulator: hooks run, also those registered after the forward pass, and what
    they return reaches the accumulator; ``torch.autograd.grad`` finds the gradients, and passes that are not asked
    for them leave the accumulators alone."""
    import distdl_b200
    from distdl_b200 import backends, nn
    from distdl_b200.parallel.optimizer import FlatAdamW
    distdl_b200.config.set_backend("native", "cupy")
    torch.manual_seed(6)
    world = backends.backend.Partition().create_partition_inclusive([0])
    P = world.create_cartesian_topology_partition([1, 1, 1])
    V, d, out = 50, 24, 40
    kw = dict(dtype=torch.bfloat16, auto_clear_buffer=not kept)
    embed = nn.DistributedEmbeddingZero(P, V, d, **kw)
    if zero:
        ag = nn.DistributedLinearAllGatherZero(P, d, out, bias=True, **kw)
        rs = nn.DistributedLinearReduceScatterZero(P, out, d, bias=True, **kw)
    else:
        ag = nn.DistributedLinearAllGather(P, d, out, bias=True, dtype=torch.bfloat16)
        rs = nn.DistributedLinearReduceScatter(P, out, d, bias=True, dtype=torch.bfloat16)
    model = torch.nn.ModuleList([embed, ag, rs])
    opt = FlatAdamW(model)
    params = [embed.weight, ag.bias, rs.bias] + ([] if zero else [ag.weight, rs.weight])
    ids = torch.randint(0, 7, (2, 64), device="cuda")
    g = torch.randn(2, 64, d, device="cuda").bfloat16()

    def gradients():
        for m in model:
            if hasattr(m, "clear_weight_buffer"):
                m.clear_weight_buffer()
        got = [p.main_grad_view.clone() for p in params]
        opt.grad.zero_()
        return got

    def leaves():                                # where autograd's gradients arrive
        return [embed.weight_buffer, ag.bias_buffer, rs.bias_buffer] if kept else params

    rs(ag(embed(ids))).backward(g)
    want = gradients()
    assert all(w.any() for w in want)
    y = rs(ag(embed(ids)))
    got = torch.autograd.grad(y, leaves(), g, retain_graph=True)
    assert not any(p.main_grad_view.any() for p in params)
    for a, w in zip(got, want):
        assert (a.float().flatten() - w).norm() <= 2 ** -8 * w.norm()         # rounded to bf16 once
    y.backward(g, inputs=[leaves()[0]])
    assert all(p is params[0] or not v.any() for p, v in zip(params, gradients()))
    if kept:
        return
    seen = []
    handles = [p.register_hook(lambda t: 2 * t) for p in params[:2]]
    y = rs(ag(embed(ids)))
    handles += [p.register_post_accumulate_grad_hook(lambda p: seen.append(p.shape)) for p in params[2:]]
    y.backward(g)
    assert sorted(seen) == sorted(p.shape for p in params[2:])
    for k, (a, w) in enumerate(zip(gradients(), want)):
        w = 2 * w if k < 2 else w
        assert (a - w).norm() <= 2 ** -8 * w.norm()
    for h in handles:
        h.remove()
    rs(ag(embed(ids))).backward(g)
    assert all(p.grad is None and torch.equal(a, w) for p, a, w in zip(params[1:], gradients()[1:], want[1:]))


@pytest.mark.parametrize("d", [264, 4096, 8192])
def test_norm_backward_takes_a_scratch_that_starts_anywhere(d):
    """The partial sums go to any 4-byte address of the caller's, with the same bits, and nothing beside them."""
    from distdl_b200 import _native
    from distdl_b200.ops._util import stream_ptr
    torch.manual_seed(17)
    rows = 37
    x, dy, w = (torch.randn(n, d, device="cuda").bfloat16() for n in (rows, rows, 1))
    stats = torch.stack([x.float().mean(1), (x.float().var(1, unbiased=False) + 1e-5).rsqrt()], 1).contiguous()
    parts = _native.lib().dd_norm_bwd_parts(rows) * 2 * d
    results = []
    for shift in (0, 1, 2):
        scratch = torch.full((parts + 4,), 7.0, device="cuda")
        dx, dw, db = torch.empty_like(x), torch.empty(d, device="cuda"), torch.empty(d, device="cuda")
        _native.call("dd_norm_bwd", 0, dy.data_ptr(), x.data_ptr(), w.data_ptr(), stats.data_ptr(), None, dx.data_ptr(),
                     dw.data_ptr(), db.data_ptr(), scratch[shift:].data_ptr(), 0, rows, d, stream_ptr())
        assert (scratch[:shift] == 7.0).all() and (scratch[shift + parts:] == 7.0).all()
        results.append((dx, dw, db))
    for other in results[1:]:
        assert all(torch.equal(a, b) for a, b in zip(results[0], other))


@pytest.mark.parametrize("n", [1, 3, 4, 1023, 4099, (1 << 20) + 7])
@pytest.mark.parametrize("shift", [0, 1])
def test_sum_of_squares_at_any_length_and_address(n, shift):
    """16-byte loads where the address allows them, single ones otherwise and at the end.  fp32 sums of n non-negative
    terms over thousands of threads: at most a few hundred roundings in a row, 512 * 2**-24."""
    from distdl_b200.ops import sumsq_
    torch.manual_seed(21)
    x = torch.randn(n + shift, device="cuda")[shift:]
    out = torch.full((1,), 2.0, device="cuda")
    sumsq_(x, out)
    want = x.double().pow(2).sum().item() + 2.0
    assert abs(out.item() - want) <= 512 * 2 ** -24 * want


def test_wide_grids_match_narrow_ones():
    """Beyond 32768 CTAs a thread takes one vector: the bits of AdamW and SwiGLU on parts that a grid in strides takes,
    with a remainder behind the last vector."""
    from distdl_b200 import ops
    torch.manual_seed(0)
    n = 4 * 256 * 32768 + 4 * 256 + 7
    state = [torch.rand(n, device="cuda") for _ in range(4)] + [torch.zeros(n, device="cuda", dtype=torch.bfloat16)]
    parts = [t.clone() for t in state]
    kw = dict(lr=1e-3, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=3, grad_scale=0.5)
    ops.adamw_step_(*state, **kw)
    for lo in range(0, n, 1 << 23):
        ops.adamw_step_(*[t[lo:lo + (1 << 23)] for t in parts], **kw)
    assert all(torch.equal(a, b) for a, b in zip(state, parts)) and not state[3].any()
    h = torch.randn(4099, 2 * 16400, device="cuda", dtype=torch.bfloat16).requires_grad_()
    dy = torch.randn(4099, 16400, device="cuda", dtype=torch.bfloat16)
    y = ops.swiglu(h)
    dh, = torch.autograd.grad(y, h, dy)
    for rows in (slice(0, 1000), slice(3099, 4099)):
        part = h.detach()[rows].clone().requires_grad_()
        want = ops.swiglu(part)
        assert torch.equal(y[rows], want) and torch.equal(dh[rows], torch.autograd.grad(want, part, dy[rows])[0])
    n = 8 * 256 * 32768 + 8 * 256
    a, b, y = (torch.randn(n, device="cuda").bfloat16() for _ in range(3))
    _native.call("dd_add_bf16", a.data_ptr(), b.data_ptr(), y.data_ptr(), n, stream_ptr())
    assert torch.equal(y, a + b)
    x = a.requires_grad_()
    y = ops.gelu(x)
    dx, = torch.autograd.grad(y, x, b)
    for part in (slice(0, 1 << 20), slice(n - (1 << 20), n)):
        p = x.detach()[part].clone().requires_grad_()
        want = ops.gelu(p)
        assert torch.equal(y[part], want) and torch.equal(dx[part], torch.autograd.grad(want, p, b[part])[0])


def _replay_ms(fn, calls):
    """The shortest of five replays of a graph of ``calls`` calls."""
    fn()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(calls):
            fn()
    best = float("inf")
    for _ in range(5):
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        graph.replay()
        end.record()
        end.synchronize()
        best = min(best, start.elapsed_time(end))
    return best


@pytest.mark.parametrize("cast", ["fp32 to bf16", "bf16 to fp32", "bf16 added to fp32"])
def test_a_cast_takes_no_longer_than_its_parts(cast):
    """16e6 values in one call against four calls of a quarter each: threads of one value each must not bring a grid of as
    many CTAs (3.3 to 3.5 times as long; 1.8 where the sum is read as well)."""
    n = 1 << 24
    f, h = torch.randn(n, device="cuda"), torch.randn(n, device="cuda").bfloat16()

    def run(part):
        for lo in range(0, n, part):
            if cast == "fp32 to bf16":
                _native.call("dd_cast_f32_bf16", f[lo:].data_ptr(), h[lo:].data_ptr(), part, 1.0, stream_ptr())
            else:
                _native.call("dd_cast_bf16_f32", h[lo:].data_ptr(), f[lo:].data_ptr(), part, 1.0, int("added" in cast),
                             stream_ptr())
    assert _replay_ms(lambda: run(n), 5) < 1.2 * _replay_ms(lambda: run(n // 4), 5)


@pytest.mark.parametrize("rms", [True, False])
def test_norm_gradients_without_a_residual_hold_no_registers_for_it(rms):
    """Against an addition that moves as many bytes: 1.5 and 1.6 times as long, 2.2 and 2.5 where the registers of a
    residual that is not there leave one CTA per SM."""
    rows, d = 16384, 2560
    dy, x, dx = (torch.randn(rows, d, device="cuda").bfloat16() for _ in range(3))
    w, stats = torch.ones(d, device="cuda").bfloat16(), torch.rand(rows, 2, device="cuda")
    part = torch.empty(_native.lib().dd_norm_bwd_parts(rows) * 2 * d, device="cuda")
    dw, db = torch.zeros(2, d, device="cuda")

    def norm():
        _native.call("dd_norm_bwd", int(rms), dy.data_ptr(), x.data_ptr(), w.data_ptr(), stats.data_ptr(), 0, dx.data_ptr(),
                     dw.data_ptr(), 0 if rms else db.data_ptr(), part.data_ptr(), 1, rows, d, stream_ptr())

    def add():
        _native.call("dd_add_bf16", dy.data_ptr(), x.data_ptr(), dx.data_ptr(), rows * d, stream_ptr())
    assert _replay_ms(norm, 5) < 1.9 * _replay_ms(add, 5)
