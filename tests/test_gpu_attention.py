"""Flash attention kernels against fp32 PyTorch scaled-dot-product attention."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(q, k, v, batch, seq, causal):
    from distdl_b200.ops.attention import _reference
    return _reference(q.float(), k.float(), v.float(), batch, seq, causal, 1.0 / math.sqrt(q.shape[-1]))


@pytest.mark.parametrize("batch,seq,Hq,Hkv,D,causal", [
    (1, 128, 1, 1, 128, True), (2, 256, 4, 2, 128, True), (1, 512, 8, 2, 128, False), (2, 384, 5, 5, 64, True),
    (1, 1024, 4, 1, 128, True), (2, 512, 6, 3, 64, True), (1, 256, 2, 2, 64, False)])
def test_attention_forward(batch, seq, Hq, Hkv, D, causal):
    from distdl_b200 import _native
    from distdl_b200.ops import attention_forward
    torch.manual_seed(0)
    T = batch * seq
    qkv = torch.randn(T, Hq + 2 * Hkv, D, device="cuda", dtype=torch.bfloat16)
    q, k, v = qkv[:, :Hq], qkv[:, Hq:Hq + Hkv], qkv[:, Hq + Hkv:]
    out, lse = attention_forward(q, k, v, batch, seq, causal)
    torch.cuda.synchronize()
    assert _native.read_status()[0] == 0
    ref = _ref(q, k, v, batch, seq, causal)
    err = (out.float() - ref).abs().max().item()
    assert err < 2e-2, err
    # log-sum-exp of the scaled scores
    qh = q.float().reshape(batch, seq, Hq, D).transpose(1, 2)
    kh = k.float().reshape(batch, seq, Hkv, D).transpose(1, 2).repeat_interleave(Hq // Hkv, 1)
    s = qh @ kh.transpose(-1, -2) / math.sqrt(D)
    if causal:
        s = s.masked_fill(torch.triu(torch.ones(seq, seq, device="cuda", dtype=torch.bool), 1), float("-inf"))
    assert (torch.logsumexp(s, -1) - lse).abs().max().item() < 2e-2


@pytest.mark.parametrize("batch,seq,Hq,Hkv,D,causal", [
    (1, 128, 1, 1, 128, True), (2, 256, 4, 2, 128, True), (1, 512, 4, 1, 128, False), (2, 384, 3, 3, 64, True),
    (2, 512, 4, 2, 64, True)])
def test_attention_backward(batch, seq, Hq, Hkv, D, causal):
    from distdl_b200 import _native
    from distdl_b200.ops import attention
    torch.manual_seed(1)
    T = batch * seq
    qkv = torch.randn(T, Hq + 2 * Hkv, D, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    q, k, v = qkv[:, :Hq], qkv[:, Hq:Hq + Hkv], qkv[:, Hq + Hkv:]
    out = attention(q, k, v, batch, seq, causal)
    dout = torch.randn_like(out)
    out.backward(dout)
    torch.cuda.synchronize()
    assert _native.read_status()[0] == 0
    ref_in = qkv.detach().float().requires_grad_()
    qr, kr, vr = ref_in[:, :Hq], ref_in[:, Hq:Hq + Hkv], ref_in[:, Hq + Hkv:]
    ref = _ref(qr, kr, vr, batch, seq, causal)
    ref.backward(dout.float())
    for name, sl in (("dq", slice(0, Hq)), ("dk", slice(Hq, Hq + Hkv)), ("dv", slice(Hq + Hkv, None))):
        g, gr = qkv.grad[:, sl].float(), ref_in.grad[:, sl]
        err = (g - gr).abs().max().item()
        scale = gr.abs().max().item()
        assert err / scale < 3e-2, f"{name}: err {err} scale {scale}"


@pytest.mark.parametrize("D,Hq,Hkv,B,S", [(64, 3, 1, 2, 128), (128, 4, 2, 1, 384), (64, 25, 25, 1, 256)])
def test_backward_with_an_output_that_is_not_16_byte_aligned(D, Hq, Hkv, B, S):
    """The row sums of O * dO read O in whatever width its address allows: the same bits either way."""
    from distdl_b200.ops.attention import attention_backward, attention_forward
    torch.manual_seed(14)
    q, k, v = (torch.randn(B * S, h, D, device="cuda").bfloat16() for h in (Hq, Hkv, Hkv))
    dout = torch.randn(B * S, Hq, D, device="cuda").bfloat16()
    out, lse = attention_forward(q, k, v, B, S, True)
    shifted = torch.empty(out.numel() + 4, device="cuda", dtype=torch.bfloat16)[4:].view(out.shape).copy_(out)
    assert shifted.data_ptr() % 16 == 8
    for a, b in zip(attention_backward(dout, q, k, v, out, lse, B, S), attention_backward(dout, q, k, v, shifted, lse, B, S)):
        assert torch.equal(a, b)


def test_backward_with_an_output_of_any_stride_but_no_odd_address():
    """Rows that lie apart are gathered first; an address between two 4-byte words is refused on the host."""
    from distdl_b200 import _native
    from distdl_b200.ops.attention import attention_backward, attention_forward
    torch.manual_seed(16)
    B, S, H, D = 2, 128, 3, 64
    q, k, v, dout = (torch.randn(B * S, H, D, device="cuda").bfloat16() for _ in range(4))
    out, lse = attention_forward(q, k, v, B, S, True)
    apart = torch.cat([out, torch.randn_like(out)], dim=2)[..., :D]
    for a, b in zip(attention_backward(dout, q, k, v, out, lse, B, S), attention_backward(dout, q, k, v, apart, lse, B, S)):
        assert torch.equal(a, b)
    odd = torch.empty(out.numel() + 8, device="cuda", dtype=torch.bfloat16)[1:1 + out.numel()].view(out.shape)
    with pytest.raises(_native.NativeError):
        attention_backward(dout, q, k, v, odd, lse, B, S)


def test_backward_of_more_sequences_than_a_grid_dimension_holds():
    """65 537 windows of 128 tokens: the first, the last and those around the limit of a grid's second and third
    dimension have the bits that a call of their own gives them."""
    from distdl_b200 import _native
    from distdl_b200.ops.attention import attention_backward, attention_forward
    torch.manual_seed(15)
    B, S, D = 65537, 128, 64
    q, k, v, dout = (torch.randn(B * S, 1, D, device="cuda", dtype=torch.bfloat16) for _ in range(4))
    out, lse = attention_forward(q, k, v, B, S, True)
    grads = attention_backward(dout, q, k, v, out, lse, B, S)
    for b in (0, 40000, 65534, 65535, 65536):
        sl = slice(b * S, (b + 1) * S)
        one = attention_backward(dout[sl], q[sl], k[sl], v[sl], out[sl], lse[b:b + 1], 1, S)
        for a, r in zip(grads, one):
            assert torch.equal(a[sl], r)
    assert _native.read_status()[0] == 0


@pytest.mark.parametrize("batch,seq,Hq,Hkv,D,causal", [
    (1, 7, 2, 2, 128, True),            # less than a tile
    (2, 128, 40, 40, 64, False),        # one key tile: nothing is handed on
    (3, 129, 4, 2, 128, True),          # one query and one key in the last tile, heads of a group on CTAs of their own
    (2, 1000, 8, 4, 128, True),
    (1, 641, 4, 1, 128, True),
    (1, 512, 6, 2, 64, False),          # split groups, the last key tile finishes every query tile
    (8, 384, 20, 20, 64, True),         # more key tiles than SMs: nobody starts together
    (8, 640, 40, 20, 64, True),         # heads of a group one after the other
    (1, 8192, 18, 9, 128, True),        # the same, the long sweeps at head dim 128
    (2, 2048, 16, 16, 64, True)])       # four key tiles of a head start together
def test_backward_in_one_pass(batch, seq, Hq, Hkv, D, causal):
    """All three gradients from one kernel, against 64 bits.  P and dS are rounded to bf16 (2**-9 each at most) before the
    products and the gradients after them: 2-norm errors of about 2**-9 * sqrt(2) = 0.28 %; 0.5 % allowed.  Twice the same
    bits: the partial sums have an order."""
    from distdl_b200 import _native
    from distdl_b200.ops.attention import _one_pass, attention_backward, attention_forward
    assert _one_pass(batch, seq, Hq, Hkv, D, causal)
    torch.manual_seed(17)
    T = batch * seq
    qkv = torch.randn(T, Hq + 2 * Hkv, D, device="cuda", dtype=torch.bfloat16)
    q, k, v = qkv[:, :Hq], qkv[:, Hq:Hq + Hkv], qkv[:, Hq + Hkv:]
    dout = torch.randn(T, Hq, D, device="cuda", dtype=torch.bfloat16)
    out, lse = attention_forward(q, k, v, batch, seq, causal)
    grads = attention_backward(dout, q, k, v, out, lse, batch, seq, causal)
    again = attention_backward(dout, q, k, v, out, lse, batch, seq, causal)
    assert _native.read_status()[0] == 0
    mask = torch.triu(torch.ones(seq, seq, device="cuda", dtype=torch.bool), 1) if causal else None
    G, err, size = Hq // Hkv, [0.0] * 4, [0.0] * 4
    for n in range(Hkv):                                      # one group of heads at a time: [batch, G or 1, seq, D]
        heads = [slice(n * G, (n + 1) * G), slice(n, n + 1), slice(n, n + 1)]
        four = lambda t, sl: t[:, sl].double().reshape(batch, seq, -1, D).transpose(1, 2)  # noqa: E731
        ins = [four(t, sl).requires_grad_() for t, sl in zip((q, k, v), heads)]
        s = ins[0] @ ins[1].transpose(-1, -2) / math.sqrt(D)
        ref = (s if mask is None else s.masked_fill(mask, float("-inf"))).softmax(-1) @ ins[2]
        want = [ref, *torch.autograd.grad(ref, ins, four(dout, heads[0]))]
        for i, (t, w, sl) in enumerate(zip((out, *grads), want, [heads[0], *heads])):
            err[i] += (four(t, sl) - w).pow(2).sum().item()
            size[i] += w.pow(2).sum().item()
    assert all(e < 5e-3 ** 2 * z for e, z in zip(err, size)), (err, size)
    assert all(torch.equal(g, a) for g, a in zip(grads, again))


def test_ragged_projection_in_training():
    """Sequences that are not whole tiles run natively where a gradient is wanted, with a gradient at any address of
    its own; without one they keep the library's operators."""
    from distdl_b200.ops import attention_packed
    from distdl_b200.ops.attention import _ragged_ok, _reference
    torch.manual_seed(18)
    B, S, Hq, Hkv, D = 2, 100, 4, 2, 128
    x = torch.randn(B * S, Hq + 2 * Hkv, D, device="cuda", dtype=torch.bfloat16).requires_grad_()
    dout = torch.randn(B * S, Hq, D, device="cuda", dtype=torch.bfloat16)
    y = attention_packed(x, Hq, Hkv, B, S)
    assert type(y.grad_fn).__name__ == "_PackedAttnFnBackward"
    w = x.detach().clone().requires_grad_()
    h, = torch.autograd.grad(_reference(w[:, :Hq], w[:, Hq:Hq + Hkv], w[:, Hq + Hkv:], B, S, True, 1.0 / math.sqrt(D)), w, dout)
    shifted = torch.empty(dout.numel() + 8, device="cuda", dtype=torch.bfloat16)[4:4 + dout.numel()].view(dout.shape).copy_(dout)
    for d in (dout, shifted):
        g, = torch.autograd.grad(y, x, d, retain_graph=True)
        # two kernels, both with gradients of 0.28 % (see above)
        assert (g.float() - h.float()).norm() < 8e-3 * h.float().norm()
    with torch.no_grad():
        assert attention_packed(x, Hq, Hkv, B, S).grad_fn is None
        assert not _ragged_ok(x, Hq, Hkv, B, S)
    odd = torch.empty(x.numel() + 8, device="cuda", dtype=torch.bfloat16)[1:1 + x.numel()].view(x.shape).requires_grad_()
    assert not _ragged_ok(odd, Hq, Hkv, B, S)          # (and the library's kernels are not called with it here)


@pytest.mark.parametrize("scale", [0.0, -0.1])
def test_ragged_projection_with_a_scale_that_is_not_positive(scale):
    """The scores in masked places are -inf before the scale: such calls keep the library's operators, which take it."""
    from distdl_b200.ops import attention_packed
    torch.manual_seed(19)
    B, S, H, D = 2, 100, 2, 128
    x = torch.randn(B * S, 3 * H, D, device="cuda", dtype=torch.bfloat16).requires_grad_()
    dout = torch.randn(B * S, H, D, device="cuda", dtype=torch.bfloat16)
    y = attention_packed(x, H, H, B, S, causal=True, scale=scale)
    g, = torch.autograd.grad(y, x, dout)
    w = x.detach().double().requires_grad_()
    q, k, v = (w[:, i * H:(i + 1) * H].reshape(B, S, H, D).transpose(1, 2) for i in range(3))
    s = (q @ k.transpose(-1, -2) * scale).masked_fill(torch.ones(S, S, device="cuda", dtype=torch.bool).triu(1), -math.inf)
    ref = (s.softmax(-1) @ v).transpose(1, 2).reshape(B * S, H, D)
    h, = torch.autograd.grad(ref, w, dout.double())
    # bf16 probabilities and results: 0.28 % (see above)
    assert (y.double() - ref).norm() < 5e-3 * ref.norm() and (g.double() - h).norm() < 5e-3 * h.norm()


def test_backward_in_one_pass_holds_no_more_than_it_uses():
    """Grouped-query heads that one CTA sweeps one after the other need no partial sums of dK and dV."""
    from distdl_b200.ops.attention import _one_pass, attention_backward, attention_forward
    B, S, Hq, Hkv, D = 8, 1024, 32, 8, 64
    words = _one_pass(B, S, Hq, Hkv, D, True)
    assert words
    q, k, v, dout = (torch.randn(B * S, h, D, device="cuda", dtype=torch.bfloat16) for h in (Hq, Hkv, Hkv, Hq))
    out, lse = attention_forward(q, k, v, B, S, True)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    base = torch.cuda.memory_allocated()
    grads = attention_backward(dout, q, k, v, out, lse, B, S, True)
    held = torch.cuda.max_memory_allocated() - base
    gradients = sum(g.numel() * 2 for g in grads)
    # 4 bytes per element of dQ, statistics and counters; the allocator rounds each of four blocks up to 2 MB at most
    assert held <= gradients + 4 * q.numel() + B * Hq * S * 8 + (1 << 20) + 4 * (2 << 20)
    assert gradients + 4 * words <= held


def test_backward_without_room_for_the_sums_of_one_pass(monkeypatch):
    """A call that fits in memory with the two kernels, which need no sums, still runs."""
    from distdl_b200.ops.attention import _one_pass, attention_backward, attention_forward
    B, S, Hq, Hkv, D = 1, 512, 8, 2, 128
    words = _one_pass(B, S, Hq, Hkv, D, True)
    assert words
    torch.manual_seed(20)
    q, k, v, dout = (torch.randn(B * S, h, D, device="cuda", dtype=torch.bfloat16) for h in (Hq, Hkv, Hkv, Hq))
    out, lse = attention_forward(q, k, v, B, S, True)
    want = attention_backward(dout, q, k, v, out, lse, B, S, True)
    real = torch.empty

    def full(*size, **kw):
        if size == (words,):
            raise torch.OutOfMemoryError("no room")
        return real(*size, **kw)
    monkeypatch.setattr(torch, "empty", full)
    got = attention_backward(dout, q, k, v, out, lse, B, S, True)
    for a, b in zip(got, want):
        # two ways with errors of 0.28 % (see above)
        assert (a.float() - b.float()).norm() < 8e-3 * b.float().norm()


@pytest.mark.parametrize("batch,seq,Hq,Hkv,D", [(1, 384, 32, 8, 64), (2, 640, 4, 4, 128), (1, 1152, 3, 1, 128)])
def test_forward_with_a_tile_per_cta(batch, seq, Hq, Hkv, D):
    """Full attention over an odd number of tiles that all fit the SMs at once."""
    from distdl_b200 import _native
    from distdl_b200.ops.attention import _two_tiles, attention_forward
    assert not _two_tiles(0, batch, seq, Hq, False)
    torch.manual_seed(22)
    q, k, v = (torch.randn(batch * seq, h, D, device="cuda", dtype=torch.bfloat16) for h in (Hq, Hkv, Hkv))
    out, lse = attention_forward(q, k, v, batch, seq, False)
    assert _native.read_status()[0] == 0
    four = lambda t: t.double().reshape(batch, seq, -1, D).transpose(1, 2)  # noqa: E731
    K, V = (four(t).repeat_interleave(Hq // Hkv, 1) for t in (k, v))
    s = four(q) @ K.transpose(-1, -2) / math.sqrt(D)
    # probabilities and output rounded to bf16: 0.28 % (see above)
    assert (four(out) - s.softmax(-1) @ V).norm() < 5e-3 * (s.softmax(-1) @ V).norm()
    assert (lse - s.logsumexp(-1)).abs().max() < 1e-3


def _backward_errors(batch, seq, Hq, Hkv, D, causal, shift=0):
    """Relative 2-norm errors of output and gradients against 64 bits, and whether a second run has the same bits."""
    from distdl_b200 import _native
    from distdl_b200.ops.attention import attention_backward, attention_forward
    torch.manual_seed(23)
    q, k, v, dout = (torch.randn(batch * seq, h, D, device="cuda", dtype=torch.bfloat16) for h in (Hq, Hkv, Hkv, Hq))
    out, lse = attention_forward(q, k, v, batch, seq, causal)
    if shift:                                # an output that starts between two 16-byte units
        out = torch.empty(out.numel() + shift, device="cuda", dtype=torch.bfloat16)[shift:].view(out.shape).copy_(out)
    grads = attention_backward(dout, q, k, v, out, lse, batch, seq, causal)
    again = attention_backward(dout, q, k, v, out, lse, batch, seq, causal)
    assert _native.read_status()[0] == 0
    leaves = [t.double().requires_grad_() for t in (q, k, v)]
    Q, K, V = (t.reshape(batch, seq, -1, D).transpose(1, 2) for t in leaves)
    s = Q @ K.repeat_interleave(Hq // Hkv, 1).transpose(-1, -2) / math.sqrt(D)
    if causal:
        s = s.masked_fill(torch.ones(seq, seq, device="cuda", dtype=torch.bool).triu(1), float("-inf"))
    ref = (s.softmax(-1) @ V.repeat_interleave(Hq // Hkv, 1)).transpose(1, 2).reshape(out.shape)
    want = [ref, *torch.autograd.grad(ref, leaves, dout.double())]
    errors = [((t.double() - w).norm() / w.norm()).item() for t, w in zip((out, *grads), want)]
    return errors, all(torch.equal(a, b) for a, b in zip(grads, again))


@pytest.mark.parametrize("batch,seq,Hq,Hkv,D,causal,shift", [
    (2, 512, 4, 4, 128, True, 0), (1, 384, 5, 5, 128, False, 0),
    (4, 512, 32, 8, 128, True, 0),           # grouped heads, more key tiles than the one kernel takes
    (1, 512, 8, 2, 128, False, 0), (2, 384, 6, 2, 128, False, 0),
    (1, 512, 4, 2, 64, False, 0), (3, 384, 3, 3, 64, False, 0), (2, 256, 4, 4, 64, True, 0),
    (1, 512, 4, 4, 128, True, 4), (1, 512, 4, 2, 64, False, 4)])
def test_backward_in_two_kernels(batch, seq, Hq, Hkv, D, causal, shift):
    """The same bounds as in one pass (see there), at sizes that the rule leaves to the two kernels."""
    from distdl_b200.ops.attention import _one_pass
    assert not _one_pass(batch, seq, Hq, Hkv, D, causal)
    errors, same = _backward_errors(batch, seq, Hq, Hkv, D, causal, shift)
    assert max(errors) < 5e-3, errors
    assert same


@pytest.mark.parametrize("batch,seq,Hq,Hkv,causal", [(2, 7, 2, 2, True), (3, 100, 4, 2, False), (2, 129, 4, 1, True),
                                                     (1, 1000, 6, 3, False), (1, 641, 4, 4, True)])
def test_ragged_lengths_at_head_dim_64(batch, seq, Hq, Hkv, causal):
    errors, same = _backward_errors(batch, seq, Hq, Hkv, 64, causal)
    assert max(errors) < 5e-3, errors
    assert same


def test_two_kernels_over_more_sequences_than_a_grid_dimension_holds(monkeypatch):
    """The sequences around the limit have the bits of a call of their own, as in one pass (see above)."""
    import importlib
    A = importlib.import_module("distdl_b200.ops.attention")
    monkeypatch.setattr(A, "_one_pass", lambda *sizes: 0)
    torch.manual_seed(24)
    B, S, D = 65537, 128, 64
    q, k, v, dout = (torch.randn(B * S, 1, D, device="cuda", dtype=torch.bfloat16) for _ in range(4))
    out, lse = A.attention_forward(q, k, v, B, S, True)
    grads = A.attention_backward(dout, q, k, v, out, lse, B, S)
    for b in (0, 65534, 65535, 65536):
        sl = slice(b * S, (b + 1) * S)
        one = A.attention_backward(dout[sl], q[sl], k[sl], v[sl], out[sl], lse[b:b + 1], 1, S)
        assert all(torch.equal(a[sl], r) for a, r in zip(grads, one))


@pytest.mark.parametrize("batch,seq,Hq,Hkv,D,causal", [(1, 128, 2, 2, 128, True), (2, 384, 6, 2, 64, False),
                                                       (1, 512, 4, 1, 128, True), (2, 256, 3, 3, 64, True)])
def test_kernels_behind_a_switch(batch, seq, Hq, Hkv, D, causal, monkeypatch):
    """A tile per CTA forward, P and dS through shared memory backward."""
    monkeypatch.setenv("DISTDL_ATTN_FWD2", "0")
    monkeypatch.setenv("DISTDL_ATTN_BWD2", "0")
    errors, same = _backward_errors(batch, seq, Hq, Hkv, D, causal)
    assert max(errors) < 5e-3, errors
    assert same


def test_ragged_projection_differentiated_twice_and_in_batches():
    """A gradient that is itself differentiated, and batched gradients, are the library's operators': the same as where the
    forward pass was the library's too.  Two bf16 ways to the same numbers: 0.28 % each, 0.56 % after another pass."""
    from torch.nn.attention import SDPBackend, sdpa_kernel

    from distdl_b200.ops import attention_packed
    from distdl_b200.ops.attention import _reference
    torch.manual_seed(25)
    B, S, Hq, Hkv, D = 1, 100, 4, 2, 128
    x = torch.randn(B * S, Hq + 2 * Hkv, D, device="cuda", dtype=torch.bfloat16).requires_grad_()
    douts = torch.randn(3, B * S, Hq, D, device="cuda", dtype=torch.bfloat16)
    u = torch.randn_like(x)
    y = attention_packed(x, Hq, Hkv, B, S)
    assert type(y.grad_fn).__name__ == "_PackedAttnFnBackward"
    w = x.detach().double().requires_grad_()
    ref = _reference(w[:, :Hq], w[:, Hq:Hq + Hkv].repeat_interleave(2, 1), w[:, Hq + Hkv:].repeat_interleave(2, 1), B, S, True,
                     1.0 / math.sqrt(D))
    with sdpa_kernel(SDPBackend.MATH):                       # (the library's fused kernels have no second derivative)
        g, = torch.autograd.grad(y, x, douts[0], create_graph=True)
        gg, = torch.autograd.grad(g, x, u, retain_graph=True)
        batched, = torch.autograd.grad(y, x, douts, is_grads_batched=True, retain_graph=True)
    h, = torch.autograd.grad(ref, w, douts[0].double(), create_graph=True)
    hh, = torch.autograd.grad(h, w, u.double(), retain_graph=True)
    assert (g.double() - h).norm() < 1e-2 * h.norm()
    assert (gg.double() - hh).norm() < 2e-2 * hh.norm()
    for got, d in zip(batched, douts):
        want, = torch.autograd.grad(ref, w, d.double(), retain_graph=True)
        assert (got.double() - want).norm() < 1e-2 * want.norm()
