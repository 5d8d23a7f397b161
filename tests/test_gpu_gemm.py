"""tcgen05 GEMM (all operand layouts and output modes) against fp32 matmul of the same bf16 inputs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cu():
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    import easyllm_b200.ops.cuda as cu
    cu.lib()
    return cu


def _check(out, ref, K):
    """Two bounds: the largest element error (catches a single bad element) and the relative Frobenius error (a
    dropped k-slice or a misplaced tile moves it far above bf16 rounding noise, which sits near 1e-3)."""
    err = (out.float() - ref).abs().max().item()
    tol = 2e-2 * max(1.0, ref.abs().max().item()) if out.dtype == torch.bfloat16 else 1e-3 * (K ** 0.5)
    assert err <= tol, (err, tol)
    rel = ((out.float() - ref).norm() / ref.norm().clamp_min(1e-12)).item()
    assert rel <= (4e-3 if out.dtype == torch.bfloat16 else 1e-4), rel


SHAPES = [(128, 256, 64), (128, 128, 128), (200, 136, 72), (512, 768, 512), (1000, 520, 264), (4096, 4096, 1024)]


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_gemm_nt(cu, M, N, K):
    torch.manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    out = cu.gemm(a, b)
    torch.cuda.synchronize()
    cu.check_err_flag()
    _check(out, a.float() @ b.float().t(), K)


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_gemm_nt_bias_and_bn128(cu, M, N, K):
    torch.manual_seed(1)
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    ref = a.float() @ b.float().t()
    _check(cu.gemm(a, b, bias=bias), ref + bias.float(), K)
    _check(cu.gemm(a, b, bn=128), ref, K)
    cu.check_err_flag()


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_gemm_nn_dgrad_layout(cu, M, N, K):
    """dx = dy · W with W stored [K_red, N_out] (MN-major B)."""
    torch.manual_seed(2)
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(K, N, device="cuda", dtype=torch.bfloat16)
    out = cu.gemm(a, b, b_mn=True)
    cu.check_err_flag()
    _check(out, a.float() @ b.float(), K)


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_gemm_tn_wgrad_layout(cu, M, N, K):
    """dW = dyᵀ · x with both operands stored [K_red, rows] (MN-major A and B), fp32 out."""
    torch.manual_seed(3)
    a = torch.randn(K, M, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(K, N, device="cuda", dtype=torch.bfloat16)
    ref = a.float().t() @ b.float()
    out = cu.gemm(a, b, a_mn=True, b_mn=True, out_mode=2)
    _check(out, ref, K)
    acc = torch.ones(M, N, device="cuda")
    cu.gemm(a, b, out=acc, a_mn=True, b_mn=True, out_mode=1)
    _check(acc - 1, ref, K)
    out16 = cu.gemm(a, b, a_mn=True, b_mn=True)
    _check(out16, ref, K)
    cu.check_err_flag()


# (256,256), (384,320), (1000,520): under half a wave of tiles, every tile runs as two half-width units;
# (2304,1280): 45 whole tiles; (4096,4096): 256 tiles, the last 34 of them cut in two; (4096,9472): 592 whole tiles
PAIR_SHAPES = [(256, 256, 64), (384, 320, 192), (1000, 520, 264), (2304, 1280, 328), (4096, 4096, 1024),
               (4096, 9472, 256)]


@pytest.mark.parametrize("M,N,K", PAIR_SHAPES)
def test_gemm_pair_kernel_all_layouts(cu, M, N, K):
    """The CTA-pair kernel (tcgen05.mma.cta_group::2, one 256 x 256 tile per two-CTA cluster) forced on, against
    fp32 matmul: K-major / MN-major operands, bias, fp32 store and fp32 accumulate, ragged edges in M, N and K."""
    torch.manual_seed(M + N + K)
    bf = dict(device="cuda", dtype=torch.bfloat16)
    a, b = torch.randn(M, K, **bf), torch.randn(N, K, **bf)
    bias = torch.randn(N, **bf)
    ref = a.float() @ b.float().t()
    _check(cu.gemm(a, b, pair=True), ref, K)
    _check(cu.gemm(a, b, bias=bias, pair=True), ref + bias.float(), K)
    _check(cu.gemm(a, b, out_mode=2, pair=True), ref, K)
    bt, at = b.t().contiguous(), a.t().contiguous()            # [K, N], [K, M]
    _check(cu.gemm(a, bt, b_mn=True, pair=True), ref, K)
    _check(cu.gemm(at, bt, a_mn=True, b_mn=True, pair=True), ref, K)
    _check(cu.gemm(at, bt, a_mn=True, b_mn=True, out_mode=2, pair=True), ref, K)
    acc = torch.ones(M, N, device="cuda")
    cu.gemm(at, bt, out=acc, a_mn=True, b_mn=True, out_mode=1, pair=True)
    cu.gemm(at, bt, out=acc, a_mn=True, b_mn=True, out_mode=1, pair=True)
    _check(acc - 1, 2 * ref, K)
    torch.cuda.synchronize()
    cu.check_err_flag()
    # and the two kernels agree with each other much more closely than either does with the rounding bound
    one, two = cu.gemm(a, b, out_mode=2, pair=False), cu.gemm(a, b, out_mode=2, pair=True)
    assert (one - two).abs().max().item() <= 1e-4 * (K ** 0.5)
    # whole tiles in the last wave (tail halving off) give the same numbers as the half-width units
    cu.lib().ell_gemm_set_tail_split(0)
    try:
        whole = cu.gemm(a, b, out_mode=2, pair=True)
        whole_t = cu.gemm(at, bt, a_mn=True, b_mn=True, out_mode=2, pair=True)
    finally:
        cu.lib().ell_gemm_set_tail_split(1)
    assert (whole - two).abs().max().item() <= 1e-4 * (K ** 0.5)
    _check(whole_t, ref, K)
    torch.cuda.synchronize()
    cu.check_err_flag()


def test_linear_autograd_matches_torch(cu):
    from easyllm_b200 import ops
    torch.manual_seed(5)
    x = torch.randn(384, 512, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = (0.05 * torch.randn(768, 512, device="cuda")).to(torch.bfloat16).requires_grad_()
    b = torch.randn(768, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    dy = torch.randn(384, 768, device="cuda", dtype=torch.bfloat16)
    ops.set_gemm_backend("tcgen05")
    y = ops.linear(x, w, b)
    y.backward(dy)
    xf, wf, bf = x.detach().float().requires_grad_(), w.detach().float().requires_grad_(), b.detach().float().requires_grad_()
    yr = torch.nn.functional.linear(xf, wf, bf)
    yr.backward(dy.float())
    for got, want in ((y, yr), (x.grad, xf.grad), (w.grad, wf.grad), (b.grad, bf.grad)):
        assert (got.float() - want).abs().max().item() <= 3e-2 * max(1.0, want.abs().max().item())
    cu.check_err_flag()


@pytest.mark.parametrize("T,V,K,cut,start", [(256, 512, 256, 0, 0), (300, 1000, 128, 24, 0), (1024, 32000, 512, 0, 0),
                                             (128, 776, 64, 8, 776)])
def test_gemm_ce_epilogue_statistics(cu, T, V, K, cut, start):
    """LM-head GEMM with fused cross-entropy statistics against a plain fp32 log-softmax of the stored logits."""
    torch.manual_seed(T + V)
    x = torch.randn(T, K, device="cuda", dtype=torch.bfloat16)
    w = (torch.randn(V, K, device="cuda") * 0.2).to(torch.bfloat16)
    valid = V - cut
    tgt = torch.randint(start, start + valid, (T,), device="cuda")
    tgt[::7] = start + V + 5                      # targets owned by another vocabulary shard
    logits, parts = cu.gemm_ce(x, w, tgt, start, valid)
    torch.cuda.synchronize()
    cu.check_err_flag()
    want_logits = x.float() @ w.float().t()
    assert (logits.float() - want_logits).abs().max().item() < 2e-2 * max(1.0, want_logits.abs().max().item())
    lf = logits.float()[:, :valid]
    mx = lf.max(1).values
    se = torch.exp(lf - mx[:, None]).sum(1)
    loc = tgt - start
    hit = (loc >= 0) & (loc < valid)
    tl = torch.where(hit, lf.gather(1, loc.clamp(0, valid - 1)[:, None]).squeeze(1), torch.zeros_like(mx))
    torch.testing.assert_close(parts[:, 0], mx, rtol=0, atol=0)
    torch.testing.assert_close(parts[:, 1], se, rtol=2e-3, atol=1e-3)
    torch.testing.assert_close(parts[:, 2], tl, rtol=0, atol=0)
    # and against the stand-alone statistics kernel on the same stored logits
    ref_parts = cu.ce_fwd(logits, tgt, start, valid)
    torch.testing.assert_close(parts, ref_parts, rtol=2e-3, atol=1e-3)


def test_lm_head_ce_autograd_matches_unfused(cu):
    from easyllm_b200 import ops
    torch.manual_seed(5)
    T, V, K = 512, 2048, 256
    x = torch.randn(T, K, device="cuda", dtype=torch.bfloat16)
    w = (torch.randn(V, K, device="cuda") * 0.1).to(torch.bfloat16)
    tgt = torch.randint(0, V, (T,), device="cuda")
    outs = []
    for fused in (True, False):
        xx, ww = x.clone().requires_grad_(), w.clone().requires_grad_()
        if fused:
            loss = ops.lm_head_cross_entropy(xx, ww, tgt)
        else:
            loss = ops.vocab_parallel_cross_entropy(ops.linear(xx, ww), tgt, None, inplace_backward=True)
        loss.mean().backward()
        outs.append((loss.detach(), xx.grad.float(), ww.grad.float()))
    torch.cuda.synchronize()
    cu.check_err_flag()
    torch.testing.assert_close(outs[0][0], outs[1][0], rtol=1e-3, atol=1e-3)
    torch.testing.assert_close(outs[0][1], outs[1][1], rtol=2e-2, atol=1e-5)
    torch.testing.assert_close(outs[0][2], outs[1][2], rtol=2e-2, atol=1e-5)
    ref_loss = torch.nn.functional.cross_entropy(x.float() @ w.float().t(), tgt, reduction="none")
    torch.testing.assert_close(outs[0][0], ref_loss, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("split", [0, 1, 2, 4, 8])
@pytest.mark.parametrize("T,N,K", [(1, 8, 8), (1, 128, 512), (16, 136, 520), (17, 4096, 1024), (32, 127, 640), (33, 264, 576),
                                   (64, 11264, 512), (65, 256, 1032), (129, 384, 4096), (256, 1000, 768)])
def test_gemm_for_few_rows(cu, T, N, K, split):
    """Every width of the row tile and its remainders, weights in both orders, all outputs, rows inside wider ones; the split
    reduction has the precision of the tiled kernel or better, and the same bits every time."""
    if split > -(-K // 64):
        pytest.skip("fewer k-blocks than CTAs")
    torch.manual_seed(T * N + K)
    wide = torch.randn(T, K + 24, device="cuda", dtype=torch.bfloat16)
    x, w = wide[:, 8:8 + K], torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    ref = x.double() @ w.double().t()
    ld = N + 16
    out = torch.full((T, ld), 3.0, device="cuda", dtype=torch.bfloat16)
    cu.gemm_thin(x, w, out, bias, ldx=wide.shape[1], ldo=ld, split=split)
    _check(out[:, :N], (ref + bias.double()).float(), K)
    assert (out[:, N:] == 3.0).all()
    # fp32 sums of the tensor core: an ulp of the running sum for each 16 products (round towards zero)
    bound = max(1, K // 16) * 2.0 ** -23
    o32 = torch.empty(T, N, device="cuda")
    cu.gemm_thin(x, w, o32, ldx=wide.shape[1], out_mode=2, split=split)
    assert (o32.double() - ref).norm() <= bound * ref.norm()
    acc = torch.randn(T, N, device="cuda")
    want = acc.double() + ref
    cu.gemm_thin(x, w, acc, ldx=wide.shape[1], out_mode=1, split=split)
    assert (acc.double() - want).norm() <= bound * want.norm()
    again = torch.empty_like(o32)
    cu.gemm_thin(x, w, again, ldx=wide.shape[1], out_mode=2, split=split)
    assert torch.equal(o32, again)
    if N % 8 == 0:
        cu.gemm_thin(x, w.t().contiguous(), again, ldx=wide.shape[1], w_mn=True, out_mode=2, split=split)
        assert (again.double() - ref).norm() <= bound * ref.norm()
    cu.check_err_flag()


@pytest.mark.parametrize("T", [1, 16, 17, 100, 256])
@pytest.mark.parametrize("N,K", [(1024, 2816), (256, 1024), (2048, 512)])
def test_gemm_routes_agree(cu, T, N, K):
    """What ``gemm`` picks by size gives what the tiled kernel gives, for every form it takes."""
    torch.manual_seed(T + N)
    a, w = (torch.randn(*s, device="cuda", dtype=torch.bfloat16) for s in ((T, K), (N, K)))
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    wt = w.t().contiguous()
    for kw in ({}, {"bias": bias}, {"out_mode": 2}, {"b_mn": True}, {"b_mn": True, "out_mode": 2}):
        b = wt if kw.get("b_mn") else w
        _check(cu.gemm(a, b, **kw), cu.gemm(a, b, pair=False, **kw).float(), K)
    acc = torch.randn(T, N, device="cuda")
    want = cu.gemm(a, w, out=acc.clone(), out_mode=1, pair=False)
    _check(cu.gemm(a, w, out=acc, out_mode=1), want, K)
    cu.check_err_flag()


@pytest.mark.parametrize("M,F,K", [(256, 128, 64), (256, 1000, 72), (2049, 200, 520), (2304, 2824, 1024)])
@pytest.mark.parametrize("act,bias", [("silu", False), ("gelu_tanh", True)])
def test_gated_product(cu, M, F, K, act, bias):
    """One launch against the two it stands for in 64 bits: the result is rounded to bf16 once (2^-9 of itself), sums of K products
    in fp32 are off by at most K 2^-23 of the sum of magnitudes, which the activation (slope up to 1.13) passes on."""
    g = torch.Generator(device="cuda").manual_seed(M + F)
    x = torch.randn(M, 2 * K, device="cuda", generator=g).to(torch.bfloat16)[:, K:]          # rows of a wider tensor
    w = (torch.randn(2 * F, K, device="cuda", generator=g) * K ** -0.5).to(torch.bfloat16)
    b = torch.randn(2 * F, device="cuda", generator=g).to(torch.bfloat16) if bias else None
    y = cu.gemm_glu(x, w, b, act)
    cu.check_err_flag()
    z = x.double() @ w.double().t()
    size = x.double().abs() @ w.double().abs().t() * K * 2.0 ** -23
    if bias:
        z, size = z + b.double(), size + b.double().abs() * 2.0 ** -22
    a = torch.nn.functional.silu(z[:, :F]) if act == "silu" else torch.nn.functional.gelu(z[:, :F], approximate="tanh")
    want = a * z[:, F:]
    bound = want.abs() * 2.0 ** -8 + 1.2 * (size[:, :F] * z[:, F:].abs() + size[:, F:] * a.abs()) + 1e-6
    assert ((y.double() - want).abs() <= bound).all()


@pytest.mark.parametrize("T,N,K,split", [(16, 1024, 1024, 2), (128, 20000, 512, 4), (256, 4096, 1024, 8)])
def test_sums_that_never_arrive_end_in_an_error(cu, T, N, K, split):
    """One CTA of every cluster withholds its sums: the others' waits (2 ms here) run out, in the first exchange of a tile and in
    the second (128 rows and more have two), with tiles left to do and without.  The launch ends, reports it, and the next one is
    as ever."""
    from ctypes import c_int
    x, w = (torch.randn(*s, device="cuda", dtype=torch.bfloat16) for s in ((T, K), (N, K)))
    out = torch.empty(T, N, device="cuda")
    for mute in (0, split - 1):
        rc = cu.lib().ell_gemm_thin(cu._p(x), cu._p(w), cu._p(out), cu._p(None), *(c_int(i) for i in (T, N, K, K, K, N, 0, 2, split)),
                                    c_int(2000), c_int(mute), cu._p(cu.err_flag(x.device)), cu._stream())
        assert rc == 0
        with pytest.raises(cu.KernelError, match="gave up"):
            cu.check_err_flag()
        cu.gemm_thin(x, w, out, out_mode=2, split=split)
        cu.check_err_flag()
        _check(out, (x.double() @ w.double().t()).float(), K)


@pytest.mark.parametrize("N", [1, 33, 127, 1000, 18999])
def test_few_rows_of_a_weight_that_ends_within_a_warp(cu, N):
    """Unsplit reductions of 64 and 128 rows: the lanes past the last row of the weight store nothing, and the warp goes on to the
    next 16 columns, and to the next tile, together.  Sums of 64 products in fp32, rounded to bf16 once."""
    for T in (64, 100, 256):
        torch.manual_seed(N + T)
        x, w = (torch.randn(*s, device="cuda", dtype=torch.bfloat16) for s in ((T, 64), (N, 64)))
        out = torch.full((T, N + 8), 3.0, device="cuda", dtype=torch.bfloat16)
        cu.gemm_thin(x, w, out, ldo=N + 8, split=1)
        cu.check_err_flag()
        want, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
        assert ((out[:, :N].double() - want).abs() <= want.abs() * 2.0 ** -8 + size * 2.0 ** -17).all() and (out[:, N:] == 3.0).all()


@pytest.mark.parametrize("rows", [1, 16, 100, 256])
@pytest.mark.parametrize("N,K", [(2816, 1024), (1024, 2816)])
def test_forward_products_do_not_depend_on_the_other_rows(cu, rows, N, K):
    """The products that the tensor-parallel and the plain forward passes record: the bits of a row are those it has among 300."""
    from easyllm_b200 import ops
    torch.manual_seed(rows)
    x = torch.randn(300, K, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(N, K, device="cuda", dtype=torch.bfloat16).requires_grad_()
    many = ops.matmul_nt(x, w.detach())
    assert torch.equal(ops.matmul_nt(x[:rows].contiguous(), w.detach()), many[:rows])
    assert torch.equal(ops.linear(x[:rows], w).detach(), many[:rows])
    cu.check_err_flag()


@pytest.mark.parametrize("act", ["silu", "gelu_tanh"])
def test_gated_product_of_extreme_gates(cu, act):
    """Gates from -inf to inf, where the exponential over- and underflows: one product of a single term, so that gate and up are what
    is written here, against the activation in 64 bits (one rounding to bf16; results below 2^-126 may be 0)."""
    gates = [0.0, 1e-3, -1e-3, 1.0, -1.0, 5.0, -5.0, 20.0, -20.0, -60.0, 80.0, -80.0, 3e4, -3e4, 1e38, -1e38, float("inf"), float("-inf"), float("nan")]
    M, F, K = 256, 256, 64
    x, w = (torch.zeros(n, K, device="cuda", dtype=torch.bfloat16) for n in (M, 2 * F))
    g = torch.tensor(gates, device="cuda", dtype=torch.bfloat16)
    x[:, 0] = 1.0
    w[:len(gates), 0], w[F:, 0] = g, 2.0
    y = cu.gemm_glu(x, w, None, act)[:, :len(gates)].double()
    cu.check_err_flag()
    z = g.double()
    want = 2 * (torch.nn.functional.silu(z) if act == "silu" else torch.nn.functional.gelu(z, approximate="tanh"))
    ok = want.isfinite() & z.isfinite()
    assert ((y[:, ok] - want[ok]).abs() <= want[ok].abs() * 2.0 ** -8 + 2.0 ** -100).all()
    assert y[:, gates.index(float("inf"))].isinf().all() and y[:, -1].isnan().all()


def test_gated_product_of_rows_that_share_memory(cu):
    """An expanded row has no row stride that TMA takes: the two launches, which copy it first, give the result."""
    from easyllm_b200 import ops
    torch.manual_seed(0)
    w = torch.randn(1024, 128, device="cuda", dtype=torch.bfloat16)
    x = torch.randn(1, 128, device="cuda", dtype=torch.bfloat16)
    with torch.no_grad(), ops.serving():
        want = ops.glu_linear(x.repeat(256, 1), w[:512], w[512:])
        got = ops.glu_linear(x.expand(256, 128), w[:512], w[512:])
    cu.check_err_flag()
    assert (got - want).float().norm() <= 1e-2 * want.float().norm()
