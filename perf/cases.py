"""The work that a user of this framework has one GPU do, as cases that can be timed and compared.

Five kinds of work, each through the entry points that a user's program calls:

* ``train``      ``parallel.Trainer.step`` on a ``models.Decoder``: host tokens in, one optimizer step done;
* ``score``      a ``Decoder`` in inference: logits of whole prompts, or of the next token only;
* ``attention``  ``ops.attention`` / ``ops.attention_packed`` with its backward pass, for models of the user's own;
* ``moe``        ``models.moe.MoEFeedForward``, routed expert layers, trained or only evaluated;
* ``spatial``    convolution, batch norm, pooling and up-sampling layers of a network on images or volumes.

``listed()`` names twelve cases, ``draw(rng)`` gives more of the same ranges.
"""
import math

import torch

import distdl_b200
from distdl_b200 import backends, models, nn, ops
from distdl_b200.models.moe import MoEFeedForward
from distdl_b200.parallel import Trainer

# The widths of the decoder configurations that the package ships (models/llama.py, gpt2.py, mixtral.py).
_LLAMA_8B = dict(family="llama", d_model=4096, n_heads=32, n_kv_heads=8, ffn=14336, vocab=128256)
_GPT2_XL = dict(family="gpt2", d_model=1600, n_heads=25, n_kv_heads=25, ffn=6400, vocab=50257)


def listed():
    return [
        # the smallest training job (the package's own smoke run): every kernel is tiny, launches and host work count
        dict(name="train_tiny", kind="train", family="llama", d_model=512, n_heads=4, n_kv_heads=2, ffn=1024,
             vocab=4096, layers=2, seq=256, batch=2, micro=1),
        # GPT-2-XL widths: LayerNorm, GELU, biases, learned positions, head dim 64; two micro-batches accumulate
        dict(name="train_gpt2", kind="train", layers=4, seq=1024, batch=8, micro=4, **_GPT2_XL),
        # the benchmark's model (Llama-3-8B widths, full vocabulary, sequence 4096) cut to two layers: the largest case
        dict(name="train_llama", kind="train", layers=2, seq=4096, batch=2, micro=2, **_LLAMA_8B),
        # a mid-sized decoder on documents whose length is not a multiple of any tile
        dict(name="train_ragged", kind="train", family="llama", d_model=2048, n_heads=16, n_kv_heads=4, ffn=5632,
             vocab=32000, layers=4, seq=1000, batch=3, micro=3),
        # evaluation of a model: logits of every position of prompts of an odd length
        dict(name="score_prompts", kind="score", layers=2, batch=2, seq=1531, last=False, **_LLAMA_8B),
        # the next token after one short prompt: few rows against all the weights, what every step of generate() does
        dict(name="score_next", kind="score", layers=4, batch=1, seq=33, last=True, **_LLAMA_8B),
        # long-context training: one long sequence, grouped-query heads, causal, packed projection
        dict(name="attention_long", kind="attention", batch=1, seq=16384, n_heads=32, n_kv_heads=8, head_dim=128,
             causal=True, packed=True),
        # an encoder: full attention, head dim 64, ragged length, separate q / k / v
        dict(name="attention_encoder", kind="attention", batch=8, seq=1500, n_heads=16, n_kv_heads=16, head_dim=64,
             causal=False, packed=False),
        # one expert layer of Mixtral widths in training
        dict(name="moe_train", kind="moe", d_model=4096, ffn=14336, experts=8, top_k=2, tokens=4096, backward=True),
        # the same layer evaluated on a handful of tokens: the experts' weights are what is moved
        dict(name="moe_eval", kind="moe", d_model=4096, ffn=14336, experts=8, top_k=2, tokens=64, backward=False),
        # one level of an image network in bf16: convolution, batch norm, max pooling, up-sampling back
        dict(name="spatial_2d", kind="spatial", nd=2, batch=8, channels=64, size=256, kernel=3, pool="max", window=2,
             stride=2, up=2.0, mode="linear", align=False, dtype="bf16"),
        # one level of a network on volumes in fp32, the type that such solvers use; overlapping windows, odd size
        dict(name="spatial_3d", kind="spatial", nd=3, batch=1, channels=32, size=93, kernel=3, pool="avg", window=3,
             stride=2, up=1.5, mode="linear", align=True, dtype="fp32"),
    ]


# ------------------------------------------------------------------------------------------------ drawing
def _log(rng, lo, hi):
    """An integer between lo and hi, spread over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_decoder(rng, family):
    head_dim = rng.choice((64, 128))
    heads = _log(rng, 2, 4096 // head_dim)
    kv = heads if family == "gpt2" else rng.choice([k for k in range(1, heads + 1) if heads % k == 0])
    d = heads * head_dim
    return dict(family=family, d_model=d, n_heads=heads, n_kv_heads=kv, ffn=max(64, int(d * rng.uniform(2, 4)) // 64 * 64),
                vocab=_log(rng, 500, 128256), layers=rng.randint(1, 6))


def _draw_one(rng):
    kind = rng.choice(("train", "train", "score", "attention", "moe", "spatial"))
    c = dict(kind=kind)
    if kind == "train":
        c.update(_draw_decoder(rng, rng.choice(("llama", "gpt2"))))
        c["seq"] = _log(rng, 64, 4096)
        c["batch"] = _log(rng, 1, max(1, 8192 // c["seq"]))
        c["micro"] = rng.choice([m for m in range(1, c["batch"] + 1) if c["batch"] % m == 0 and c["batch"] <= 4 * m])
    elif kind == "score":
        c.update(_draw_decoder(rng, rng.choice(("llama", "gpt2"))))
        c["seq"] = _log(rng, 1, 4096)
        c["batch"] = _log(rng, 1, max(1, min(16, 4096 // c["seq"])))
        c["last"] = rng.random() < 0.5
    elif kind == "attention":
        c["head_dim"] = rng.choice((64, 128))
        c["n_heads"] = _log(rng, 4, 32)
        c["n_kv_heads"] = rng.choice([k for k in range(1, c["n_heads"] + 1) if c["n_heads"] % k == 0])
        c["seq"] = _log(rng, 100, 16384) if rng.random() < 0.5 else 128 * _log(rng, 1, 128)
        c["batch"] = _log(rng, 1, max(1, 16384 // c["seq"]))
        c["causal"] = rng.random() < 0.7
        c["packed"] = rng.random() < 0.5
    elif kind == "moe":
        c["d_model"] = 64 * _log(rng, 8, 64)
        c["ffn"] = 64 * _log(rng, 16, 224)
        c["experts"] = rng.choice((4, 8, 16))
        c["top_k"] = rng.choice((1, 2))
        c["tokens"] = _log(rng, 64, 4096)
        c["backward"] = rng.random() < 0.6
    else:
        c["nd"] = rng.choice((2, 3))
        c["batch"] = _log(rng, 1, 8)
        c["channels"] = 8 * _log(rng, 1, 16)
        c["size"] = _log(rng, 16, 400 if c["nd"] == 2 else 96)
        c["kernel"] = rng.choice((1, 3))
        c["pool"] = rng.choice(("avg", "max"))
        c["window"] = rng.choice((2, 3))
        c["stride"] = rng.choice((1, 2))
        c["up"] = rng.choice((1.5, 2.0))
        c["mode"] = rng.choice(("linear", "linear", "nearest"))
        c["align"] = c["mode"] == "linear" and rng.random() < 0.5
        c["dtype"] = rng.choice(("bf16", "fp32"))
    return c


def _cost(case):
    """Seconds that the work takes at rates that every kind of it can reach: to compare cases only."""
    w = work(case)
    return w["bytes"] / 4e12 + w["flops"] / 0.8e15


_LIMIT = None


def draw(rng):
    global _LIMIT
    if _LIMIT is None:
        _LIMIT = max(_cost(c) for c in listed())
    while True:
        c = _draw_one(rng)
        elements = c["batch"] * c["channels"] * c["size"] ** c["nd"] if c["kind"] == "spatial" else 0
        if _cost(c) <= _LIMIT and elements <= 8 * 64 * 256 ** 2:
            return c


# ------------------------------------------------------------------------------------------------ preparing
def _backend():
    torch.cuda.set_device(0)
    distdl_b200.config.set_backend("native", "cupy")


def _config(case):
    kw = dict(d_model=case["d_model"], n_heads=case["n_heads"], n_kv_heads=case["n_kv_heads"], ffn_dim=case["ffn"],
              vocab_size=case["vocab"], n_layers=case["layers"], max_seq=max(64, case["seq"]))
    return models.llama3_8b(**kw) if case["family"] == "llama" else models.gpt2_xl(**kw)


def _grid(dims):
    world = backends.backend.Partition()
    return world.create_partition_inclusive([0]).create_cartesian_topology_partition([1] * dims)


def _tokens(gen, rows, columns, vocab):
    """Token ids as in text: the frequency falls with the rank r as 1 / (r + 32)."""
    u = torch.rand(rows, columns, generator=gen, device="cuda", dtype=torch.float64)
    return (32.0 * ((vocab / 32.0 + 1.0) ** u - 1.0)).long().clamp_(max=vocab - 1)


class _Spatial(torch.nn.Module):
    def __init__(self, case, dtype):
        super().__init__()
        nd = case["nd"]
        P = _grid(nd + 2)
        conv = {2: nn.DistributedFeatureConv2d, 3: nn.DistributedFeatureConv3d}[nd]
        pool = {("avg", 2): nn.DistributedAvgPool2d, ("avg", 3): nn.DistributedAvgPool3d,
                ("max", 2): nn.DistributedMaxPool2d, ("max", 3): nn.DistributedMaxPool3d}[case["pool"], nd]
        c = case["channels"]
        self.conv = conv(P, c, c, case["kernel"], padding=case["kernel"] // 2, bias=False, device="cuda", dtype=dtype)
        self.norm = nn.DistributedBatchNorm(P, c, device="cuda", dtype=dtype)
        self.pool = pool(P, case["window"], stride=case["stride"])
        self.up = nn.DistributedUpsample(P, scale_factor=case["up"], mode=case["mode"], align_corners=case["align"])

    def forward(self, x):
        return self.up(self.pool(self.norm(self.conv(x))))


def prepare(case, seed):
    _backend()
    torch.manual_seed(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    st = {"case": case}

    def normal(*shape, dtype=torch.bfloat16):
        return torch.randn(*shape, generator=gen, device="cuda").to(dtype)

    if kind == "train":
        model = models.Decoder(_config(case), models.ParallelLayout(1, 1))
        st["trainer"] = Trainer(model, global_tokens_per_step=case["batch"] * case["seq"], micro_batch=case["micro"],
                                lr=3e-4, warmup_steps=10, total_steps=100000)
        st["tokens"] = _tokens(gen, case["batch"], case["seq"] + 1, case["vocab"]).cpu().pin_memory()
    elif kind == "score":
        st["model"] = models.Decoder(_config(case), models.ParallelLayout(1, 1)).eval()
        st["tokens"] = _tokens(gen, case["batch"], case["seq"], case["vocab"])
    elif kind == "attention":
        T, hq, hkv, hd = case["batch"] * case["seq"], case["n_heads"], case["n_kv_heads"], case["head_dim"]
        if case["packed"]:
            st["inputs"] = [normal(T, hq + 2 * hkv, hd).requires_grad_()]
        else:
            st["inputs"] = [normal(T, h, hd).requires_grad_() for h in (hq, hkv, hkv)]
        st["dout"] = normal(T, hq, hd)
    elif kind == "moe":
        cfg = models.mixtral_8x7b(d_model=case["d_model"], ffn_dim=case["ffn"], n_experts=case["experts"],
                                  top_k=case["top_k"])
        st["layer"] = MoEFeedForward(cfg, models.ParallelLayout(1, 1))
        with torch.no_grad():
            st["layer"].router.weight.normal_(0.0, cfg.init_std)
        st["x"] = normal(1, case["tokens"], case["d_model"]).requires_grad_(case["backward"])
        st["dy"] = normal(1, case["tokens"], case["d_model"])
        st["aux_weight"] = torch.tensor(0.01 * case["tokens"], device="cuda")
    else:
        dtype = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
        st["net"] = _Spatial(case, dtype)
        st["x"] = normal(case["batch"], case["channels"], *[case["size"]] * case["nd"], dtype=dtype).requires_grad_()
        st["dy"] = normal(case["batch"], case["channels"], *[_sizes(case)[1]] * case["nd"], dtype=dtype)
    return st


# ------------------------------------------------------------------------------------------------ running
def run(st):
    return {"train": _run_train, "score": _run_score, "attention": _run_attention, "moe": _run_moe,
            "spatial": _run_spatial}[st["case"]["kind"]](st)


def _run_train(st):
    loss = st["trainer"].step(st["tokens"])
    opt = st["trainer"].opt.state_dict()
    return [loss, opt["master"], opt["exp_avg"], opt["exp_avg_sq"]]


def _run_score(st):
    model = st["model"]
    with torch.no_grad():
        h = model(st["tokens"])
        return model.head(h[:, -1:] if st["case"]["last"] else h)


def _run_attention(st):
    case, ins = st["case"], st["inputs"]
    if case["packed"]:
        out = ops.attention_packed(ins[0], case["n_heads"], case["n_kv_heads"], case["batch"], case["seq"],
                                   causal=case["causal"])
    else:
        out = ops.attention(*ins, case["batch"], case["seq"], causal=case["causal"])
    return [out.detach(), *torch.autograd.grad(out, ins, st["dout"])]


def _run_moe(st):
    layer, x = st["layer"], st["x"]
    if not st["case"]["backward"]:
        with torch.no_grad():
            return [layer(x), layer.aux_loss]
    y = layer(x)
    params = [layer.router.weight, layer.w_up, layer.w_down]
    grads = torch.autograd.grad([y, layer.aux_loss], [x, *params], [st["dy"], st["aux_weight"]])
    return [y.detach(), layer.aux_loss.detach(), *grads]


def _run_spatial(st):
    net, x = st["net"], st["x"]
    y = net(x)
    grads = torch.autograd.grad(y, [x, net.conv.weight, net.norm.gamma, net.norm.beta], st["dy"])
    return [y.detach(), *grads, net.norm.running_mean, net.norm.running_var]


# ------------------------------------------------------------------------------------------------ counting
def _sizes(case):
    """Extent of every spatial dimension after pooling, and after up-sampling."""
    pooled = (case["size"] - case["window"]) // case["stride"] + 1
    return pooled, int(math.floor(pooled * case["up"]))


def _attention_flops(batch, seq, heads, head_dim, causal):
    return 4.0 * batch * heads * seq * seq * head_dim * (0.5 if causal else 1.0)


def _weights(case):
    """(matrix elements of the blocks, of the head, all parameters)."""
    cfg = _config(case)
    d, hd = cfg.d_model, cfg.head_dim
    block = d * (cfg.n_heads + 2 * cfg.n_kv_heads) * hd + cfg.n_heads * hd * d \
        + (3 if cfg.activation == "swiglu" else 2) * d * cfg.ffn_dim
    return cfg.n_layers * block, cfg.vocab_size * d, cfg.num_parameters()


def work(case):
    """Inputs read once and outputs written once; the products of the model (not of padding or of anything
    computed twice)."""
    kind = case["kind"]
    if kind == "train":
        cfg = _config(case)
        tokens = case["batch"] * case["seq"]
        # parameters in bf16, master weights and both moments in fp32: each read and written
        return {"bytes": 28.0 * cfg.num_parameters() + 8.0 * tokens,
                "flops": cfg.train_flops_per_token(case["seq"]) * tokens}
    if kind == "score":
        blocks, head, _ = _weights(case)
        tokens = case["batch"] * case["seq"]
        rows = case["batch"] if case["last"] else tokens
        hd = case["d_model"] // case["n_heads"]
        return {"bytes": 2.0 * (blocks + head + rows * case["vocab"] + tokens * case["d_model"]),
                "flops": 2.0 * (blocks * tokens + head * rows)
                + case["layers"] * _attention_flops(case["batch"], case["seq"], case["n_heads"], hd, True)}
    if kind == "attention":
        T = case["batch"] * case["seq"]
        # q, k, v, dout read; out, dq, dk, dv written
        return {"bytes": 2.0 * T * case["head_dim"] * (4 * case["n_heads"] + 4 * case["n_kv_heads"]),
                "flops": 3.5 * _attention_flops(case["batch"], case["seq"], case["n_heads"], case["head_dim"],
                                                case["causal"])}
    if kind == "moe":
        weights = 3.0 * case["experts"] * case["d_model"] * case["ffn"]
        rows = float(case["tokens"] * case["d_model"])
        flops = 2.0 * 3 * case["tokens"] * case["top_k"] * case["d_model"] * case["ffn"]
        if case["backward"]:
            return {"bytes": 2.0 * (2 * weights + 4 * rows), "flops": 3 * flops}
        return {"bytes": 2.0 * (weights + 2 * rows), "flops": flops}
    e = 2.0 if case["dtype"] == "bf16" else 4.0
    planes = case["batch"] * case["channels"]
    n_in, n_out = case["size"] ** case["nd"], _sizes(case)[1] ** case["nd"]
    # x and dy read, y and dx written
    return {"bytes": 2 * e * planes * (n_in + n_out),
            "flops": 3 * 2.0 * planes * n_in * case["channels"] * case["kernel"] ** case["nd"]}


def tolerance(case):
    """About four times the difference between this package's kernels and the same work on library kernels
    (``DISTDL_FORCE_TORCH=1``), which round at other places, over the listed and ten drawn cases."""
    kind = case["kind"]
    if kind == "train":
        # seen: gradients 0.0166 (their squares 0.022) through five layers in bf16; the largest differences are
        # sums with cancellation in the embedding rows of frequent tokens, next to rows that are zero
        return {"rel": 0.03, "max": 0.99}
    if kind == "score":
        return {"rel": 0.03, "max": 0.22}           # seen 0.0124 and 0.055
    if kind == "attention":
        return {"rel": 0.013, "max": 0.94}          # seen 0.0032 and 0.234 (gradients of the first, sharpest rows)
    if kind == "moe":
        return {"rel": 0.022, "max": 0.47}          # seen 0.0056 and 0.117
    if case["dtype"] == "bf16":
        return {"rel": 0.03, "max": 0.99}           # seen 0.026 and 0.999: equal values in a pooling window
    if case["pool"] == "max":
        return {"rel": 2e-3, "max": 0.99}           # one window in about 1e6 has its two largest values 1e-6 apart
    return {"rel": 4e-5, "max": 1e-3}               # seen 8e-6 and 2e-4
