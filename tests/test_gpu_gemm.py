"""tcgen05 GEMM against a plain fp32 PyTorch reference of the same product."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(a, b):
    return a.float() @ b.float().transpose(-1, -2)


def _check(out, ref, tol=2e-2):
    err = (out.float() - ref).abs().max().item()
    scale = ref.abs().max().item() + 1e-6
    assert err / scale < tol, f"max err {err} vs scale {scale}"


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (256, 512, 256), (200, 600, 1600), (4096, 3072, 4096),
                                   (77, 88, 96), (1024, 1024, 8), (130, 264, 72)])
@pytest.mark.parametrize("a_mn,b_mn", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_gemm_layouts(M, N, K, a_mn, b_mn):
    from distdl_b200 import _native
    from distdl_b200.ops import gemm
    torch.manual_seed(0)
    dev = "cuda"
    # leading dimensions must be multiples of 8 elements: pad the storage
    def make(rows, cols, mn):
        if mn:
            ld = (rows + 7) // 8 * 8
            st = torch.randn(cols, ld, device=dev, dtype=torch.bfloat16)
            return st[:, :rows].t()
        ld = (cols + 7) // 8 * 8
        st = torch.randn(rows, ld, device=dev, dtype=torch.bfloat16)
        return st[:, :cols]
    a = make(M, K, a_mn)
    b = make(N, K, b_mn)
    out = gemm(a, b)
    torch.cuda.synchronize()
    assert _native.read_status()[0] == 0
    _check(out, _ref(a, b))


def test_gemm_bias_accumulate_fp32():
    from distdl_b200.ops import gemm
    torch.manual_seed(1)
    M, N, K = 512, 768, 320
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    out = gemm(a, b, bias=bias)
    _check(out, _ref(a, b) + bias.float())
    acc = torch.randn(M, N, device="cuda", dtype=torch.float32)
    ref = acc.clone() + _ref(a, b)
    gemm(a, b, out=acc, accumulate=True)
    _check(acc, ref, tol=1e-3)
    accb = torch.randn(M, N, device="cuda", dtype=torch.bfloat16)
    refb = accb.float() + _ref(a, b)
    gemm(a, b, out=accb, accumulate=True)
    _check(accb, refb)


def test_gemm_batched():
    from distdl_b200.ops import gemm
    torch.manual_seed(2)
    B, M, N, K = 5, 256, 384, 128
    a = torch.randn(B, M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(B, N, K, device="cuda", dtype=torch.bfloat16)
    out = gemm(a, b)
    _check(out, _ref(a, b))
    bt = torch.randn(B, K, N, device="cuda", dtype=torch.bfloat16)
    out = gemm(a, bt.transpose(1, 2))
    _check(out, a.float() @ bt.float())


def test_linear_autograd_matches_torch():
    from distdl_b200.ops import linear
    torch.manual_seed(3)
    x = torch.randn(4, 96, 256, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = (torch.randn(512, 256, device="cuda") * 0.05).to(torch.bfloat16).requires_grad_()
    b = torch.randn(512, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    y = linear(x, w, b)
    dy = torch.randn_like(y)
    y.backward(dy)
    xr = x.detach().float().requires_grad_()
    wr = w.detach().float().requires_grad_()
    br = b.detach().float().requires_grad_()
    yr = torch.nn.functional.linear(xr, wr, br)
    yr.backward(dy.float())
    _check(y, yr)
    _check(x.grad, xr.grad)
    _check(w.grad, wr.grad)
    _check(b.grad, br.grad)


@pytest.mark.parametrize("M,N,K", [(256, 512, 4096), (384, 256, 8192), (1024, 768, 1600), (512, 512, 14336)])
def test_gemm_error_bound_scales_with_the_contraction_length(M, N, K):
    """Element-wise bounds that a lost k-block cannot hide behind.  With fp32 output the only error is
    the accumulation's: a few fp32 roundings of sums of size sqrt(K), orders of magnitude below the
    sqrt(64) / sqrt(K) share of one 64-deep k-block.  With bf16 output every element is within one
    bf16 rounding of the exact value (plus the same accumulation term)."""
    from distdl_b200.ops import gemm
    torch.manual_seed(K)
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    ref = a.double() @ b.double().t()
    acc_term = 1e-4 * (K ** 0.5)                  # generous for fp32 accumulation in any order; one lost k-block is ~ 8
    out32 = gemm(a, b, out_dtype=torch.float32)
    err = (out32.double() - ref).abs().max().item()
    assert err < acc_term, (err, acc_term)
    out16 = gemm(a, b)
    bound = ref.abs() * 2.0 ** -8 + acc_term
    assert bool(((out16.double() - ref).abs() <= bound).all()), ((out16.double() - ref).abs() - bound).max().item()
    # the gradient layouts (dy @ w and dy^T @ x) under the same bound
    wg = gemm(a.t().contiguous().t(), b, out_dtype=torch.float32)          # A as a transposed (MN-major) view
    assert (wg.double() - ref).abs().max().item() < acc_term
    at = torch.randn(K, M, device="cuda", dtype=torch.bfloat16)      # MN-major operands, as in a weight gradient
    bt = torch.randn(K, N, device="cuda", dtype=torch.bfloat16)
    reft = at.double().t() @ bt.double()
    outt = gemm(at.t(), bt.t(), out_dtype=torch.float32)
    assert (outt.double() - reft).abs().max().item() < acc_term


@pytest.mark.parametrize("C,counts", [(384, (0, 1, 256, 257, 500)), (96, (0, 5, 96, 64, 33)), (1000, (1000, 512, 0, 64, 999))])
def test_batched_gemm_skips_zero_rows(C, counts):
    """Rows and terms that are known to be zero: the bits are those of the full product, for no live row, counts on
    and off the edges of tiles and k-blocks, and counts beyond the capacity; both output types."""
    from distdl_b200 import _native
    from distdl_b200.models.moe import batched_linear
    from distdl_b200.ops import gemm
    torch.manual_seed(3)
    E, d, f = len(counts), 136, 328
    rows = torch.tensor(counts, dtype=torch.int32, device="cuda")
    keep = (torch.arange(C, device="cuda")[None] < rows[:, None])[..., None]
    x = torch.where(keep, torch.randn(E, C, d, device="cuda"), torch.zeros((), device="cuda")).bfloat16()
    dy = torch.where(keep, torch.randn(E, C, f, device="cuda"), torch.zeros((), device="cuda")).bfloat16()
    w = torch.randn(E, f, d, device="cuda", dtype=torch.bfloat16)
    got, want = [], []
    for r, out in ((rows, got), (None, want)):
        a, b = x.clone().requires_grad_(), w.clone().requires_grad_()
        y = batched_linear(a, b, r)
        out += [y.detach(), *torch.autograd.grad(y, (a, b), dy), gemm(x, w, out_dtype=torch.float32, rows=r),
                gemm(dy.transpose(1, 2), x.transpose(1, 2), out_dtype=torch.float32, rows=r, bound_k=True) if r is not None
                else gemm(dy.transpose(1, 2), x.transpose(1, 2), out_dtype=torch.float32)]
    for g, v in zip(got, want):
        assert torch.equal(g, v)
    torch.cuda.synchronize()
    assert _native.read_status()[0] == 0


@pytest.mark.parametrize("M,N,K", [(1, 256, 8192), (33, 520, 6400), (128, 264, 14336), (129, 512, 8192), (200, 88, 6144),
                                   (300, 1000, 8192), (16, 8, 4096)])
@pytest.mark.parametrize("a_mn", [0, 1])
@pytest.mark.parametrize("b_mn", [0, 1])
def test_gemm_split_contraction(M, N, K, b_mn, a_mn):
    """Few tiles and a long contraction, both layouts of both operands: bias, both output types, accumulation, strided
    outputs; the same bits in every run, nothing written beside the output."""
    from distdl_b200 import _native
    from distdl_b200.ops import gemm
    assert _native.lib().dd_gemm_split(M, N, K) > 1
    torch.manual_seed(2)
    lead = (M + 7) // 8 * 8                                   # (a leading dimension that TMA can take)
    a = torch.randn(K, lead, device="cuda", dtype=torch.bfloat16)[:, :M].t() if a_mn else \
        torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(K, N, device="cuda", dtype=torch.bfloat16).t() if b_mn else \
        torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    bias = torch.randn(N, device="cuda")
    ref = _ref(a, b)
    for out in (torch.full((M, N + 8), 7.0, device="cuda", dtype=torch.bfloat16), torch.full((M, N + 4), 7.0, device="cuda"),
                torch.full((M, N + 1), 7.0, device="cuda")):
        view = out[:, :N]
        gemm(a, b, out=view, bias=bias)
        # bf16 results round once (2^-8); fp32 sums of K products in another order
        tol = 2 ** -8 if out.dtype == torch.bfloat16 else 2e-5
        _check(view, ref + bias, tol=tol)
        first = view.clone()
        gemm(a, b, out=view, bias=bias)
        assert torch.equal(view, first) and (out[:, N:] == 7.0).all()
        gemm(a, b, out=view, accumulate=True)
        _check(view, 2 * ref + bias, tol=2 * tol)
    torch.cuda.synchronize()
    assert _native.read_status()[0] == 0


@pytest.mark.parametrize("n_out,n_in,tokens", [(64, 512, 8192), (384, 256, 8192)])
@pytest.mark.parametrize("transposed", [False, True])
def test_weight_gradient_accumulates_over_a_split_contraction(n_out, n_in, tokens, transposed):
    """A small weight and many tokens: two micro-batches into the fp32 accumulator, stored either way."""
    from distdl_b200 import _native
    from distdl_b200.ops.gemm import weight_grad
    assert _native.lib().dd_gemm_split(*((n_in, n_out) if transposed else (n_out, n_in)), tokens) > 1
    torch.manual_seed(19)
    acc = torch.randn(*((n_in, n_out) if transposed else (n_out, n_in)), device="cuda")
    mg = acc.t() if transposed else acc
    want = mg.double()
    w = torch.empty(n_out, n_in, device="cuda", dtype=torch.bfloat16)
    w.main_grad = mg
    for _ in range(2):
        dy = torch.randn(tokens, n_out, device="cuda").bfloat16()
        x = torch.randn(tokens, n_in, device="cuda").bfloat16()
        want = want + dy.double().t() @ x.double()
        assert weight_grad(dy, x, w) is None
    assert (mg.double() - want).abs().max() < 1e-4 * tokens ** 0.5        # fp32 accumulation in any order
    torch.cuda.synchronize()
    assert _native.read_status()[0] == 0


@pytest.mark.parametrize("M,N,K", [(129, 8, 64), (257, 129, 72), (256, 128, 128), (4096, 1600, 136), (300, 392, 1024),
                                   (3000, 2048, 200), (1000, 4104, 64)])
@pytest.mark.parametrize("a_mn,b_mn", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_gemm_with_half_tiles(M, N, K, a_mn, b_mn):
    """Sizes whose waves make pairs of CTAs take 128 columns, with remainders in every direction and both majors.  A
    bf16 result is off by 2**-9 / sqrt(3) = 0.11 % of itself on average, 0.17 % at the lower end of a binade."""
    from distdl_b200 import _native
    from distdl_b200.ops import gemm
    torch.manual_seed(5)

    def make(rows, cols, mn):
        n, m = (cols, rows) if mn else (rows, cols)
        st = torch.randn(n, (m + 7) // 8 * 8, device="cuda", dtype=torch.bfloat16)[:, :m]
        return st.t() if mn else st
    a, b = make(M, K, a_mn), make(N, K, b_mn)
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    want = a.double() @ b.double().t() + bias.double()
    out = torch.full((M, N + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm(a, b, out=out[:, :N], bias=bias)
    assert (out[:, :N].double() - want).norm() < 2.5e-3 * want.norm()
    assert (out[:, N:] == 7).all()
    acc = torch.randn(M, N, device="cuda")
    before = acc.double()
    gemm(a, b, out=acc, accumulate=True)
    want = a.double() @ b.double().t() + before
    assert (acc.double() - want).norm() < 1e-5 * want.norm()
    assert _native.read_status()[0] == 0


@pytest.mark.parametrize("B,M,N,K", [(3, 257, 136, 72), (2, 300, 40, 200), (5, 129, 264, 64)])
@pytest.mark.parametrize("a_mn,b_mn", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_batched_gemm_with_half_tiles(B, M, N, K, a_mn, b_mn):
    """Batches whose tiles fit one wave take 128 columns: remainders in every direction, both majors (bounds as above)."""
    from distdl_b200 import _native
    from distdl_b200.ops import gemm
    torch.manual_seed(6)

    def make(rows, cols, mn):
        n, m = (cols, rows) if mn else (rows, cols)
        st = torch.randn(B, n, (m + 7) // 8 * 8, device="cuda", dtype=torch.bfloat16)[:, :, :m]
        return st.transpose(1, 2) if mn else st
    a, b = make(M, K, a_mn), make(N, K, b_mn)
    want = a.double() @ b.double().transpose(1, 2)
    out = torch.full((B, M, N + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm(a, b, out=out[:, :, :N])
    assert (out[:, :, :N].double() - want).norm() < 2.5e-3 * want.norm()
    assert (out[:, :, N:] == 7).all()
    acc = torch.randn(B, M, N, device="cuda")
    before = acc.double()
    gemm(a, b, out=acc, accumulate=True)
    assert (acc.double() - want - before).norm() < 1e-5 * (want + before).norm()
    assert _native.read_status()[0] == 0


@pytest.mark.parametrize("B,M,N,K,ctas", [
    (1, 257, 200, 4104, 2), (1, 512, 456, 4160, 4), (1, 1000, 520, 4168, 4), (3, 1288, 456, 4224, 6), (1, 2400, 200, 4160, 4),
    (3, 4300, 500, 4104, 18),        # 17 blocks: single ones before whole tiles, on either accumulator
    (1, 4300, 500, 4160, 8),         # the single ones in a last wave of their own, which has none beyond them
    (1, 6000, 5000, 4160, 0)])
@pytest.mark.parametrize("a_mn,b_mn", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_gemm_with_wide_tiles(B, M, N, K, ctas, a_mn, b_mn):
    """Contractions beyond 4096 take 512 x 256 per pair of CTAs: an odd number of 256-row blocks, a last wave in single
    blocks, remainders in every direction, both majors, few pairs and all.  bf16 results as above; fp32 sums of 16 terms, 264
    of them cut off at 2**-23, are off by less than 264 / 2 * 2**-23 = 1.6e-5."""
    from test_gemm_plan import WIDE, plan

    from distdl_b200 import _native
    from distdl_b200.ops import gemm
    torch.manual_seed(7)
    assert all(plan(M, N, K, B, flags, ctas)["kernel"] == WIDE for flags in (0, 1))

    def make(rows, cols, mn):
        n, m = (cols, rows) if mn else (rows, cols)
        st = torch.randn(B, n, (m + 7) // 8 * 8, device="cuda", dtype=torch.bfloat16)[:, :, :m]
        st = st.transpose(1, 2) if mn else st
        return st[0] if B == 1 else st
    a, b = make(M, K, a_mn), make(N, K, b_mn)
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    want = a.double() @ b.double().transpose(-1, -2)
    out = torch.full((*a.shape[:-1], N + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm(a, b, out=out[..., :N], bias=bias, max_ctas=ctas)
    assert (out[..., :N].double() - want - bias.double()).norm() < 2.5e-3 * want.norm()
    assert (out[..., N:] == 7).all()
    acc = torch.randn(*a.shape[:-1], N, device="cuda")
    before = acc.double()
    gemm(a, b, out=acc, accumulate=True, max_ctas=ctas)
    assert (acc.double() - want - before).norm() < 2e-5 * want.norm()
    bias = torch.randn(N, device="cuda")
    gemm(a, b, out=acc, bias=bias, max_ctas=ctas)
    assert (acc.double() - want - bias.double()).norm() < 2e-5 * want.norm()
    assert _native.read_status()[0] == 0


@pytest.mark.parametrize("B,M,N,K,ctas", [(1, 256, 640, 136, 4), (1, 513, 264, 200, 8), (1, 1000, 500, 72, 14),
                                          (3, 300, 256, 64, 10), (1, 2816, 2048, 64, 0), (1, 3000, 2048, 2048, 0)])
@pytest.mark.parametrize("a_mn,b_mn", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_gemm_whose_last_wave_is_taken_in_halves(B, M, N, K, ctas, a_mn, b_mn):
    """A last wave of no more than half as many tiles as pairs of CTAs: halves of 128 columns, some of them behind the
    matrix; bf16 and fp32 results (bounds as above)."""
    from distdl_b200 import _native
    from distdl_b200.ops import gemm
    torch.manual_seed(10)

    def make(rows, cols, mn):
        n, m = (cols, rows) if mn else (rows, cols)
        st = torch.randn(B, n, (m + 7) // 8 * 8, device="cuda", dtype=torch.bfloat16)[:, :, :m]
        st = st.transpose(1, 2) if mn else st
        return st[0] if B == 1 else st
    a, b = make(M, K, a_mn), make(N, K, b_mn)
    want = a.double() @ b.double().transpose(-1, -2)
    for pad in (8, 1):                                   # with TMA stores, and rows that do not start at 16 bytes
        out = torch.full((*a.shape[:-1], N + pad), 7.0, device="cuda", dtype=torch.bfloat16)
        gemm(a, b, out=out[..., :N], max_ctas=ctas)
        assert (out[..., :N].double() - want).norm() < 2.5e-3 * want.norm()
        assert (out[..., N:] == 7).all()
    acc = torch.randn(*a.shape[:-1], N, device="cuda")
    before = acc.double()
    gemm(a, b, out=acc, accumulate=True, max_ctas=ctas)
    assert (acc.double() - want - before).norm() < 1e-5 * want.norm()
    assert _native.read_status()[0] == 0


@pytest.mark.parametrize("B,M,N,K,ctas,parts", [
    (1, 33, 1000, 136, 0, 4), (1, 128, 264, 72, 3, 1), (1, 77, 1160, 200, 4, 4), (2, 20, 2312, 64, 4, 4), (1, 1, 520, 1600, 12, 4),
    (1, 20, 264, 136, 4, 2), (1, 128, 14336, 1600, 0, 2), (1, 33, 10240, 2048, 0, 2)])
@pytest.mark.parametrize("a_mn,b_mn", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_gemm_of_few_rows_in_parts_of_tiles(B, M, N, K, ctas, parts, a_mn, b_mn):
    """One row of tiles: quarters and halves of the only or of the last wave, some behind the matrix (bounds as above)."""
    from test_gemm_plan import SINGLE, plan

    from distdl_b200 import _native
    from distdl_b200.ops import gemm
    torch.manual_seed(11)
    p = plan(M, N, K, B, 0, ctas)
    assert (p["kernel"], p["parts"]) == (SINGLE, parts)

    def make(rows, cols, mn):
        n, m = (cols, rows) if mn else (rows, cols)
        st = torch.randn(B, n, (m + 7) // 8 * 8, device="cuda", dtype=torch.bfloat16)[:, :, :m]
        st = st.transpose(1, 2) if mn else st
        return st[0] if B == 1 else st
    a, b = make(M, K, a_mn), make(N, K, b_mn)
    want = a.double() @ b.double().transpose(-1, -2)
    out = torch.full((*a.shape[:-1], N + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm(a, b, out=out[..., :N], max_ctas=ctas)
    assert (out[..., :N].double() - want).norm() < 2.5e-3 * want.norm()
    assert (out[..., N:] == 7).all()
    acc = torch.randn(*a.shape[:-1], N, device="cuda")
    before = acc.double()
    gemm(a, b, out=acc, accumulate=True, max_ctas=ctas)
    assert (acc.double() - want - before).norm() < 1e-5 * want.norm()
    assert _native.read_status()[0] == 0


@pytest.mark.parametrize("C,K,N,kernel", [
    (1000, 4168, 2824, 1), (1000, 512, 2824, 3), (1000, 256, 2824, 3),      # 256-row tiles; eight k-blocks, four as the ring has
    (1000, 200, 2824, 3), (1000, 64, 2824, 3), (300, 1032, 14336, 3)])
@pytest.mark.parametrize("counts", [(0, 1, 256, 257), (512, 513, 768, 1000), (1000, 0, 0, 999), (0, 0, 0, 0)])
def test_wide_tiles_skip_zero_rows(counts, C, K, N, kernel):
    """Rows that are known to be zero, with tiles of 512 rows where the rule takes them: counts on and off the edges of blocks
    and tiles."""
    from test_gemm_plan import plan

    from distdl_b200 import _native
    from distdl_b200.ops import gemm
    torch.manual_seed(8)
    counts = [min(c, C) for c in counts + counts[::-1]]
    E = len(counts)
    assert plan(C, N, K, E, rows=1)["kernel"] == kernel
    rows = torch.tensor(counts, dtype=torch.int32, device="cuda")
    keep = (torch.arange(C, device="cuda")[None] < rows[:, None])[..., None]
    x = torch.where(keep, torch.randn(E, C, K, device="cuda"), torch.zeros((), device="cuda")).bfloat16()
    w = torch.randn(E, N, K, device="cuda", dtype=torch.bfloat16)
    for dt in (torch.bfloat16, torch.float32):
        out = torch.full((E, C, N), float("nan"), device="cuda", dtype=dt)
        assert torch.equal(gemm(x, w, out=out, rows=rows), gemm(x, w, out_dtype=dt))
    assert _native.read_status()[0] == 0


@pytest.mark.parametrize("M,N,K,kernel,group", [
    (2600, 2312, 64, 1, 4), (2312, 2600, 64, 1, 4), (2312, 2312, 5000, 1, 10), (4700, 5100, 4096, 1, 17),
    (5100, 4700, 4096, 1, -17), (4608, 9472, 4160, 3, 8), (5000, 4300, 4160, 3, -16)])
def test_gemm_tile_order_covers_every_tile(M, N, K, kernel, group):
    """Tiles by panels of rows and of columns, in one panel and in several, the last one narrower than the others, with
    tiles of 256 and of 512 rows."""
    from test_gemm_plan import plan

    from distdl_b200.ops import gemm
    torch.manual_seed(9)
    p = plan(M, N, K)
    assert (p["kernel"], p["group"]) == (kernel, group)
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    out = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    want = a.double() @ b.double().t()
    assert (gemm(a, b, out=out).double() - want).norm() < 2.5e-3 * want.norm()


def test_products_launched_ahead_are_ordered_on_streams_and_in_graphs():
    """A chain of products, each of the one before it, right behind library kernels that write its operands: on a stream of
    its own, and captured (twice the same bits as one kernel at a time)."""
    from distdl_b200.ops import gemm, rms_norm
    torch.manual_seed(12)
    x = torch.randn(2048, 1024, device="cuda", dtype=torch.bfloat16)
    ws = [torch.randn(1024, 1024, device="cuda", dtype=torch.bfloat16) / 32 for _ in range(4)]
    one = torch.ones(1024, device="cuda", dtype=torch.bfloat16)

    def chain(wait):
        y = x.clone()
        for i, w in enumerate(ws * 3):
            y = gemm(y, w if i % 2 else w.t().contiguous().t())
            wait()
            y = rms_norm(y, one) if i % 3 == 0 else y.mul(1.25)
            wait()
            y = gemm(y[:100], w, out=torch.zeros(2048, 1024, device="cuda", dtype=torch.bfloat16)[:100]) if i == 11 else y
            wait()
        return y

    want = chain(torch.cuda.synchronize)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        got = chain(lambda: None)
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = chain(lambda: None)
    for _ in range(3):
        got.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, want)


@pytest.mark.parametrize("M,N,K", [(128, 131072, 2048), (4096, 16384, 2048), (4096, 8192, 4160)])
def test_a_product_limited_to_some_sms_leaves_the_others_to_another_stream(M, N, K):
    """``max_ctas``: the product behind a limited one must not settle on the SMs that the limit leaves free, so that work of
    another stream ends while the limited one (milliseconds on four SMs) still runs.  One size for each kernel."""
    from distdl_b200.ops import gemm
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    c = torch.randn(2048, 512, device="cuda", dtype=torch.bfloat16)
    outs = [torch.empty(M, N, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    small = torch.empty(2048, 2048, device="cuda", dtype=torch.bfloat16)
    side = torch.cuda.Stream()
    start, end, other = (torch.cuda.Event(enable_timing=True) for _ in range(3))

    def both(record):
        if record:
            start.record()
        gemm(a, b, out=outs[0], max_ctas=4)
        gemm(a, b, out=outs[1])
        with torch.cuda.stream(side):
            gemm(c, c, out=small, max_ctas=64)
            if record:
                other.record()
        if record:
            end.record()
    for record in (False, True):
        torch.cuda.synchronize()
        both(record)
    torch.cuda.synchronize()
    assert start.elapsed_time(other) < 0.5 * start.elapsed_time(end)
    assert torch.equal(*outs)
