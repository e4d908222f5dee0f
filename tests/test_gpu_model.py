"""The decoder on one GPU through the native kernels: the model trains, the
native path agrees with the library path, and the weight-gradient GEMM that
accumulates straight into the optimizer's fp32 buffer matches autograd."""
import os

import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(seed=0, **over):
    import distdl_b200
    from distdl_b200 import models
    from distdl_b200.parallel import FlatAdamW
    distdl_b200.config.set_backend("native", "cupy")
    torch.manual_seed(seed)
    cfg = models.llama_tiny(d_model=256, n_heads=4, n_kv_heads=2, ffn_dim=512, max_seq=128, vocab_size=1024, **over)
    model = models.Decoder(cfg, models.ParallelLayout(1, 1))
    return cfg, model, FlatAdamW(model, lr=1e-3)


def _tokens(cfg, batch=2, seed=1):
    g = torch.Generator().manual_seed(seed)
    return torch.randint(0, cfg.vocab_size, (batch, cfg.max_seq + 1), generator=g).cuda()


def _grads(env):
    old = {k: os.environ.get(k) for k in env}
    os.environ.update(env)
    try:
        cfg, model, opt = _model()
        tok = _tokens(cfg)
        for _ in range(2):                              # two micro-batches accumulate
            model.loss(tok[:, :-1], tok[:, 1:], scale=1.0 / tok[:, 1:].numel()).backward()
        model.release_gathered()
        torch.cuda.synchronize()
        return opt.grad.clone(), opt.names
    finally:
        for k, v in old.items():
            if v is None:
                os.environ.pop(k, None)
            else:
                os.environ[k] = v


def test_direct_main_grad_matches_autograd():
    a, names = _grads({"DISTDL_DIRECT_MAIN_GRAD": "1"})
    b, _ = _grads({"DISTDL_DIRECT_MAIN_GRAD": "0"})
    assert a.abs().max() > 0
    for name, o, n in names:
        x, y = a[o:o + n], b[o:o + n]
        # the autograd path rounds every micro-batch gradient to bf16 first
        tol = 2e-2 * y.abs().max().item() + 1e-7
        assert (x - y).abs().max().item() <= tol, name


def test_native_matches_library_path():
    a, names = _grads({})
    b, _ = _grads({"DISTDL_FORCE_TORCH": "1"})
    for name, o, n in names:
        x, y = a[o:o + n], b[o:o + n]
        tol = 5e-2 * y.abs().max().item() + 1e-6
        assert (x - y).abs().max().item() <= tol, name


def test_decoder_trains_on_repeated_batch():
    from distdl_b200.parallel import Trainer
    cfg, model, _ = _model()
    # a second optimizer would re-home the parameters again: build the trainer on a fresh model
    import distdl_b200.models as models
    torch.manual_seed(0)
    model = models.Decoder(cfg, models.ParallelLayout(1, 1))
    trainer = Trainer(model, global_tokens_per_step=4 * cfg.max_seq, micro_batch=2, lr=3e-3, warmup_steps=0)
    tok = _tokens(cfg, batch=4)
    losses = [trainer.step_device(tok).item() for _ in range(8)]
    assert all(v == v for v in losses)
    assert losses[-1] < losses[0] - 0.5, losses


def _gpt2_grads(env, hook=False):
    import distdl_b200
    from distdl_b200 import models
    from distdl_b200.parallel import FlatAdamW
    distdl_b200.config.set_backend("native", "cupy")
    old = {k: os.environ.get(k) for k in env}
    os.environ.update(env)
    try:
        torch.manual_seed(3)
        cfg = models.gpt2_xl(d_model=256, n_heads=4, n_kv_heads=4, ffn_dim=512, max_seq=128, vocab_size=1000, n_layers=2)
        model = models.Decoder(cfg, models.ParallelLayout(1, 1))
        with torch.no_grad():
            for n, p in model.named_parameters():
                if "norm" in n:
                    p.add_(torch.randn_like(p) * 0.1)
        seen = []
        if hook:
            for n, p in model.named_parameters():
                if "norm2" in n:
                    p.register_hook(lambda g, n=n: seen.append((n, g.float().norm().item())))
        opt = FlatAdamW(model, lr=1e-3)
        tok = _tokens(cfg)
        for _ in range(2):
            model.loss(tok[:, :-1], tok[:, 1:], scale=1.0 / tok[:, 1:].numel()).backward()
        model.release_gathered()
        torch.cuda.synchronize()
        return opt.grad.clone(), opt.names, seen
    finally:
        for k, v in old.items():
            if v is None:
                os.environ.pop(k, None)
            else:
                os.environ[k] = v


def test_layer_norms_of_a_decoder_accumulate_directly():
    """LayerNorm weights and biases: straight into the fp32 accumulators, the same as through autograd (which rounds
    the gradient of every micro-batch to bf16 first) and as the library path; a hook of the user's still sees them."""
    a, names, _ = _gpt2_grads({"DISTDL_DIRECT_MAIN_GRAD": "1"})
    for env in ({"DISTDL_DIRECT_MAIN_GRAD": "0"}, {"DISTDL_FORCE_TORCH": "1"}):
        b, _, _ = _gpt2_grads(env)
        for name, o, n in names:
            x, y = a[o:o + n], b[o:o + n]
            assert (x - y).abs().max().item() <= 3e-2 * y.abs().max().item() + 1e-7, (env, name)
    c, _, seen = _gpt2_grads({"DISTDL_DIRECT_MAIN_GRAD": "1"}, hook=True)
    assert len(seen) == 2 * 2 * 2 and all(v > 0 for _, v in seen)
    for name, o, n in names:
        x, y = a[o:o + n], c[o:o + n]
        assert (x - y).abs().max().item() <= 2e-2 * y.abs().max().item() + 1e-7, name


@pytest.mark.parametrize("affine,shape", [(True, (3, 37, 256)), (True, (1, 1, 1600)), (False, (2, 5, 264))])
def test_layer_norm_layer_takes_a_residual(affine, shape):
    import distdl_b200
    from distdl_b200 import backends, nn
    distdl_b200.config.set_backend("native", "cupy")
    P = backends.backend.Partition().create_partition_inclusive([0]).create_cartesian_topology_partition([1, 1, 1])
    torch.manual_seed(4)
    layer = nn.DistributedLayerNorm(P, shape[-1], elementwise_affine=affine, device="cuda", dtype=torch.bfloat16)
    if affine:
        with torch.no_grad():
            layer.weight.normal_()
            layer.bias.normal_()
    x, r = (torch.randn(shape, device="cuda").bfloat16().requires_grad_() for _ in range(2))
    ds, dy = (torch.randn(shape, device="cuda").bfloat16() for _ in range(2))
    leaves = [x, r, *layer.parameters()]
    s, y = layer(x, residual=r)
    got = torch.autograd.grad([s, y], leaves, [ds, dy])
    s2 = x + r
    want = torch.autograd.grad([s2, layer(s2)], leaves, [ds, dy])
    assert torch.equal(s, s2)
    for a, b in zip(got, want):
        # the separate form rounds the two gradients of the sum to bf16 before it adds them
        assert (a.float() - b.float()).norm() <= 1e-2 * b.float().norm()


@pytest.mark.parametrize("late", ["weight", "bias"])
def test_norm_parameter_unfrozen_after_the_optimizer_was_built(late):
    """The one without an accumulator gets its gradient from autograd, the other reaches the optimizer all the same."""
    import distdl_b200
    from distdl_b200 import backends, nn
    from distdl_b200.parallel import FlatAdamW
    distdl_b200.config.set_backend("native", "cupy")
    P = backends.backend.Partition().create_partition_inclusive([0]).create_cartesian_topology_partition([1, 1, 1])
    torch.manual_seed(6)
    layer = nn.DistributedLayerNorm(P, 256, device="cuda", dtype=torch.bfloat16)
    getattr(layer, late).requires_grad_(False)
    opt = FlatAdamW(layer, lr=1e-3)
    getattr(layer, late).requires_grad_(True)
    x, dy = (torch.randn(2, 37, 256, device="cuda").bfloat16() for _ in range(2))
    layer(x).backward(dy)
    xh = torch.nn.functional.layer_norm(x.double(), (256,), eps=layer.eps)
    want = {"weight": (xh * dy.double()).sum((0, 1)), "bias": dy.double().sum((0, 1))}
    got = getattr(layer, late).grad.double().view(-1)
    other = "bias" if late == "weight" else "weight"
    # fp32 sums, then rounded to bf16 (2**-9 of a value at most)
    assert (got - want[late]).norm() <= 4e-3 * want[late].norm()
    assert (opt.grad[:256].double() - want[other]).norm() <= 4e-3 * want[other].norm()
