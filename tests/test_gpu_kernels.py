"""sm_100a elementwise / reduction kernels against fp32 PyTorch statements of the same op."""
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


def _close(a, b, atol, rtol):
    assert torch.allclose(a.float(), b.float(), atol=atol, rtol=rtol), (a.float() - b.float()).abs().max().item()


@pytest.mark.parametrize("rows,cols", [(7, 256), (300, 4096), (1024, 5120), (33, 8192)])
def test_rmsnorm_fwd_bwd(cu, rows, cols):
    from easyllm_b200.ops import reference as ref
    torch.manual_seed(0)
    x = torch.randn(rows, cols, device="cuda", dtype=torch.bfloat16)
    res = torch.randn_like(x)
    w = (1 + 0.1 * torch.randn(cols, device="cuda")).to(torch.bfloat16)
    y, _, rstd = cu.rmsnorm_fwd(x, None, w, 1e-5)
    _close(y, ref.rmsnorm(x.float(), w.float(), 1e-5), 2e-2, 2e-2)
    y2, h, rstd2 = cu.rmsnorm_fwd(x, res, w, 1e-5)
    hr = (x.float() + res.float()).to(torch.bfloat16)
    assert torch.equal(h, hr)
    _close(y2, ref.rmsnorm(hr.float(), w.float(), 1e-5), 2e-2, 2e-2)
    # backward vs autograd of the fp32 statement
    dy = torch.randn_like(x)
    dres = torch.randn_like(x)
    hf = hr.float().requires_grad_()
    wf = w.float().requires_grad_()
    ref.rmsnorm(hf, wf, 1e-5).backward(dy.float())
    dh, dw = cu.rmsnorm_bwd(dy, h, w, rstd2, dres)
    _close(dh, hf.grad + dres.float(), 3e-2, 3e-2)
    _close(dw, wf.grad, 5e-2 * max(1.0, wf.grad.abs().max().item()), 3e-2)
    # accumulate mode adds onto an existing fp32 buffer
    acc = torch.ones(cols, device="cuda")
    cu.rmsnorm_bwd(dy, h, w, rstd2, None, dw_out=acc, accumulate=True)
    _close(acc - 1, wf.grad, 5e-2 * max(1.0, wf.grad.abs().max().item()), 3e-2)


@pytest.mark.parametrize("T,hq,hk,D", [(64, 4, 4, 128), (257, 8, 2, 128), (33, 4, 1, 64)])
def test_rope_packed(cu, T, hq, hk, D):
    from easyllm_b200.ops import reference as ref
    torch.manual_seed(1)
    W = (hq + 2 * hk) * D
    qkv = torch.randn(T, W, device="cuda", dtype=torch.bfloat16)
    pos = torch.randint(0, 500, (T,), device="cuda", dtype=torch.int32)
    cos, sin = ref.rope_tables(D, 512, device="cuda")
    q = qkv[:, :hq * D].reshape(T, hq, D).float()
    k = qkv[:, hq * D:(hq + hk) * D].reshape(T, hk, D).float()
    rq, rk = ref.rope(q, k, cos, sin, pos.long())
    v_before = qkv[:, (hq + hk) * D:].clone()
    orig = qkv.clone()
    cu.rope_(qkv, cos, sin, pos, hq + hk, D)
    _close(qkv[:, :hq * D].reshape(T, hq, D), rq, 2e-2, 2e-2)
    _close(qkv[:, hq * D:(hq + hk) * D].reshape(T, hk, D), rk, 2e-2, 2e-2)
    assert torch.equal(qkv[:, (hq + hk) * D:], v_before)
    cu.rope_(qkv, cos, sin, pos, hq + hk, D, backward=True)   # inverse rotation
    _close(qkv, orig, 3e-2, 3e-2)


@pytest.mark.parametrize("T,F", [(5, 64), (300, 11008), (128, 3456)])
def test_swiglu(cu, T, F):
    torch.manual_seed(2)
    gu = torch.randn(T, 2 * F, device="cuda", dtype=torch.bfloat16)
    out = cu.swiglu_fwd(gu)
    g, u = gu[:, :F].float().requires_grad_(), gu[:, F:].float().requires_grad_()
    r = torch.nn.functional.silu(g) * u
    _close(out, r, 2e-2, 2e-2)
    d = torch.randn(T, F, device="cuda", dtype=torch.bfloat16)
    r.backward(d.float())
    dgu = cu.swiglu_bwd(d, gu)
    _close(dgu[:, :F], g.grad, 3e-2, 3e-2)
    _close(dgu[:, F:], u.grad, 3e-2, 3e-2)


@pytest.mark.parametrize("n", [1000, 1 << 20, (1 << 20) + 3])
def test_adam_and_sumsq(cu, n):
    from easyllm_b200.ops import reference as ref
    torch.manual_seed(3)
    p = torch.randn(n, device="cuda"); g = torch.randn(n, device="cuda")
    m = torch.rand(n, device="cuda") * 0.1; v = torch.rand(n, device="cuda") * 0.01
    pr, mr, vr = p.clone(), m.clone(), v.clone()
    low = torch.empty(n, device="cuda", dtype=torch.bfloat16)
    scale = torch.tensor([0.5], device="cuda")
    cu.adam(p, g, m, v, low, 1e-3, 0.9, 0.95, 1e-8, 0.1, 7, True, 2.0, scale)
    ref.adam_step(pr, g, mr, vr, 1e-3, 0.9, 0.95, 1e-8, 0.1, 7, True, 1.0)
    _close(p, pr, 1e-6, 1e-5); _close(m, mr, 1e-6, 1e-5); _close(v, vr, 1e-7, 1e-5)
    assert torch.equal(low, p.to(torch.bfloat16))
    out = torch.zeros(1, device="cuda")
    cu.sumsq(g, out)
    _close(out, (g.double() ** 2).sum().float().view(1), 1e-2, 1e-4)


@pytest.mark.parametrize("T,V,valid", [(17, 1000, 1000), (256, 32000, 32000), (64, 38016, 38000)])
def test_cross_entropy(cu, T, V, valid):
    torch.manual_seed(4)
    logits = (3 * torch.randn(T, V, device="cuda")).to(torch.bfloat16)
    tgt = torch.randint(0, valid, (T,), device="cuda")
    parts = cu.ce_fwd(logits, tgt, 0, valid)
    lf = logits.float()[:, :valid].requires_grad_()
    ref_loss = torch.nn.functional.cross_entropy(lf, tgt, reduction="none")
    lse = torch.log(parts[:, 1]) + parts[:, 0]
    _close(lse - parts[:, 2], ref_loss, 2e-3, 2e-3)
    scale = torch.rand(T, device="cuda")
    (ref_loss * scale).sum().backward()
    work = logits.clone()
    cu.ce_bwd_(work, tgt, lse.contiguous(), scale, 0, valid)
    _close(work[:, :valid], lf.grad, 2e-3, 2e-2)
    if valid < V:
        assert work[:, valid:].abs().max().item() == 0
    # a shard that does not own the targets contributes target-logit 0
    parts2 = cu.ce_fwd(logits, tgt, V, valid)
    assert parts2[:, 2].abs().max().item() == 0


def test_accumulate_bf16_into_fp32(cu):
    x = torch.randn(100003, device="cuda").to(torch.bfloat16)
    acc = torch.ones(100003, device="cuda")
    cu.accum_bf16_to_f32(x, acc)
    _close(acc, 1 + x.float(), 1e-6, 1e-6)


def test_embedding_fwd_bwd(cu):
    from easyllm_b200 import ops
    torch.manual_seed(2)
    rows, h, T, start = 1000, 256, 4096, 3000
    w = torch.randn(rows, h, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    ids = torch.randint(start - 500, start + rows + 500, (4, T // 4), device="cuda")
    ids[0, :64] = start + 7                      # many duplicates: exercises the atomics
    out = ops.embedding(ids, w, start)
    mine = (ids >= start) & (ids < start + rows)
    want = torch.where(mine[..., None], w.detach()[(ids - start).clamp(0, rows - 1)], torch.zeros((), device="cuda", dtype=w.dtype))
    assert torch.equal(out, want)
    do = torch.randn_like(out)
    out.backward(do)
    ref = torch.zeros(rows, h, device="cuda")
    ref.index_add_(0, (ids - start)[mine], do.float()[mine])
    torch.testing.assert_close(w.grad.float(), ref, rtol=2e-2, atol=2e-2)
    # accumulation into an fp32 main_grad
    w2 = w.detach().clone().requires_grad_()
    w2.main_grad = torch.ones(rows, h, device="cuda")
    ops.embedding(ids, w2, start).backward(do)
    torch.testing.assert_close(w2.main_grad, ref + 1.0, rtol=1e-4, atol=1e-3)
    assert w2.grad is None
    torch.cuda.synchronize()
    cu.check_err_flag()


def test_bounded_wait_gives_up_and_reports(cu):
    """A wait on a flag that nothing sets (and on a barrier nobody arrives on) expires after its limit, the kernel
    returns with an error code the host reads, and the context stays usable."""
    import ctypes
    L = cu.lib()
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    waited = torch.zeros(1, dtype=torch.int64, device="cuda")
    err = cu.err_flag()
    rc = L.ell_bounded_wait_selftest(ctypes.c_void_p(flag.data_ptr()), ctypes.c_uint(1), ctypes.c_void_p(err.data_ptr()),
                                     ctypes.c_void_p(waited.data_ptr()), cu._stream())
    assert rc == 0
    torch.cuda.synchronize()
    assert 3.5e9 < int(waited) < 9e9, int(waited)          # two waits of 2 s each
    with pytest.raises(cu.KernelError):
        cu.check_err_flag()
    cu.check_err_flag()                                      # the error word was cleared by the read
    # the context is healthy: a tensor-core GEMM right after gives the right answer
    a = torch.randn(256, 128, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(256, 128, device="cuda", dtype=torch.bfloat16)
    torch.testing.assert_close(cu.gemm(a, b).float(), a.float() @ b.float().t(), rtol=2e-2, atol=2e-1)
    # success path: the flag is already at the wanted epoch, nothing is reported and nothing is waited for
    flag.fill_(7)
    rc = L.ell_bounded_wait_selftest(ctypes.c_void_p(flag.data_ptr()), ctypes.c_uint(7), ctypes.c_void_p(err.data_ptr()),
                                     ctypes.c_void_p(waited.data_ptr()), cu._stream())
    assert rc == 0
    torch.cuda.synchronize()
    assert int(waited) < 1e8
    cu.check_err_flag()


@pytest.mark.parametrize("rows,cols,res", [(64, 512, False), (300, 1024, True), (1000, 4096, True), (17, 8200, False)])
def test_layernorm_kernel_matches_fp32(cu, rows, cols, res):
    """Affine LayerNorm forward and backward (input, residual, weight and bias gradients) against F.layer_norm in
    fp32 on the same bf16 inputs."""
    from easyllm_b200 import ops
    torch.manual_seed(rows + cols)
    bf = dict(device="cuda", dtype=torch.bfloat16)
    x = (torch.randn(rows, cols, **bf) * 2 + 0.5).requires_grad_()
    r = torch.randn(rows, cols, **bf).requires_grad_() if res else None
    w = (1 + 0.1 * torch.randn(cols, **bf)).requires_grad_()
    b = (0.1 * torch.randn(cols, **bf)).requires_grad_()
    out = ops.layernorm(x, w, b, 1e-5, r)
    y, h = out if res else (out, None)
    dy = torch.randn_like(y)
    y.backward(dy)
    torch.cuda.synchronize()
    cu.check_err_flag()
    xf = x.detach().float().requires_grad_(); wf = w.detach().float().requires_grad_(); bf32 = b.detach().float().requires_grad_()
    rf = r.detach().float().requires_grad_() if res else None
    hf = (xf + rf).to(torch.bfloat16).float() if res else xf      # the kernel stores the sum in bf16 and normalises that
    yf = torch.nn.functional.layer_norm(hf, (cols,), wf, bf32, 1e-5)
    yf.backward(dy.float())
    assert (y.float() - yf).abs().max().item() < 4e-2
    assert (x.grad.float() - xf.grad).abs().max().item() < 4e-2 * max(1.0, xf.grad.abs().max().item())
    if res:
        assert torch.equal(x.grad, r.grad)
        assert (h.float() - (x.detach().float() + r.detach().float())).abs().max().item() < 4e-2
    for got, want in ((w.grad, wf.grad), (b.grad, bf32.grad)):
        assert ((got.float() - want).norm() / want.norm()).item() < 2e-2


def test_out_of_range_indices_are_reported_not_dereferenced(cu):
    """Bounds checks that are always on: a rotary position beyond the cos / sin tables and a token id beyond the
    embedding table set the device error word (the host raises at its next read) instead of reading past a buffer;
    the offending rows are left unrotated / zero."""
    from easyllm_b200.ops.reference import rope_tables
    torch.manual_seed(0)
    cos, sin = rope_tables(128, 64, device="cuda")                  # positions 0..63 only
    qkv = torch.randn(16, 3 * 128, device="cuda", dtype=torch.bfloat16)
    before = qkv.clone()
    pos = torch.arange(16, dtype=torch.int32, device="cuda")
    pos[5] = 4096                                                    # outside the tables
    cu.rope_(qkv, cos, sin, pos, 2, 128)
    torch.cuda.synchronize()
    with pytest.raises(cu.KernelError, match="code 32"):
        cu.check_err_flag()
    assert torch.equal(qkv[5], before[5]) and not torch.equal(qkv[4], before[4])
    w = torch.randn(100, 64, device="cuda", dtype=torch.bfloat16)
    ids = torch.tensor([1, 2, 250, 3], device="cuda")
    out = cu.embedding_fwd(ids, w, 0, 100)
    torch.cuda.synchronize()
    with pytest.raises(cu.KernelError, match="code 31"):
        cu.check_err_flag()
    assert torch.equal(out[2], torch.zeros_like(out[2])) and torch.equal(out[1], w[2])
    cu.check_err_flag()                                              # cleared


@pytest.mark.parametrize("rows", [1, 20, 100])
@pytest.mark.parametrize("capture", [False, True])
def test_chained_launches_keep_their_order(cu, rows, capture):
    """A run of dependent launches over three buffers that every launch reuses (matrix-vector, thin and tiled products, norm,
    GLU, accumulation), torch kernels, a copy and a forked stream in between: the result is that of the same launches with the
    GPU waited for after each."""
    import easyllm_b200.ops.cuda_infer as ci
    torch.manual_seed(rows)
    W, F = 1024, 2816
    w = [(torch.randn(n, k, device="cuda") * k ** -0.5).to(torch.bfloat16) for n, k in ((2 * F, W), (W, F), (W, W))]
    nw = torch.ones(W, device="cuda", dtype=torch.bfloat16)
    x0 = torch.randn(rows, W, device="cuda", dtype=torch.bfloat16)
    x, acc = torch.empty_like(x0), torch.empty(rows, W, device="cuda")
    side = torch.cuda.Stream()

    def chain(wait):
        x.copy_(x0)
        acc.zero_()
        for i in range(12):
            y = cu.rmsnorm_fwd(x, None, nw, 1e-5)[0]
            wait()
            h = ci.glu(ci.linear(y, w[0]), "silu")
            wait()
            ci.linear_add_(acc, h, w[1])
            wait()
            if i % 4 == 3:
                side.wait_stream(torch.cuda.current_stream())
                with torch.cuda.stream(side):
                    z = ci.linear(y, w[2])
                torch.cuda.current_stream().wait_stream(side)
                z.record_stream(torch.cuda.current_stream())
            else:
                z = ci.linear(y, w[2])
            wait()
            x.copy_(z)
            wait()
            x.add_(acc)
            wait()
        return x.clone(), acc.clone()

    want = chain(torch.cuda.synchronize)
    if capture:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = chain(lambda: None)
        for _ in range(3):
            graph.replay()
    else:
        got = chain(lambda: None)
    torch.cuda.synchronize()
    cu.check_err_flag()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("tokens,rows,cols,dtype", [(1, 8, 8, torch.int64), (37, 5, 264, torch.int32), (3001, 32000, 1024, torch.int64)])
@pytest.mark.parametrize("deterministic", [False, True])
def test_embedding_gradient_goes_to_main_grad(cu, tokens, rows, cols, dtype, deterministic):
    """Rows that come often, and a main_grad that already holds something; fp32 sums of n bf16 rows are within n 2^-24 of the
    sum of magnitudes.  Deterministic programs get F.embedding's own dense gradient."""
    from easyllm_b200.models.hf_models.modeling import TokenEmbedding
    torch.manual_seed(1)
    emb = TokenEmbedding(rows, cols, device="cuda", dtype=torch.bfloat16)
    ids = torch.randint(0, rows, (tokens,), device="cuda", dtype=dtype)
    before = torch.randn(rows, cols, device="cuda")
    emb.weight.main_grad = before.clone()
    dy = torch.randn(tokens, cols, device="cuda", dtype=torch.bfloat16)
    torch.use_deterministic_algorithms(deterministic)
    try:
        y = emb(ids)
        y.backward(dy)
    finally:
        torch.use_deterministic_algorithms(False)
    assert torch.equal(y, emb.weight[ids.long()])
    if deterministic:
        other = emb.weight.detach().clone().requires_grad_()
        torch.nn.functional.embedding(ids, other).backward(dy)
        assert torch.equal(emb.weight.grad, other.grad) and torch.equal(emb.weight.main_grad, before)
        return
    assert emb.weight.grad is None
    want, size = before.double(), before.double().abs()
    want.index_add_(0, ids.long(), dy.double())
    size.index_add_(0, ids.long(), dy.double().abs())
    assert ((emb.weight.main_grad.double() - want).abs() <= size * (tokens + 1) * 2.0 ** -24).all()


@pytest.mark.parametrize("tokens,rows,cols", [(1, 3, 8), (128, 200, 64), (129, 2, 64), (1024, 9, 64), (1025, 9, 64), (2000, 7, 1032), (4096, 300, 2048), (9000, 40, 64), (9000, 3000, 64)])
def test_embedding_gradient_repeats_itself(cu, tokens, rows, cols, monkeypatch):
    """Ids that come once and hundreds of times, within a block of tokens and over many, in one piece (up to 9000 tokens, three
    words of marks) and in several: the same bits every time, those of the sum in the order of the tokens in fp32."""
    from easyllm_b200 import ops
    if rows == 40:
        monkeypatch.setattr(cu, "ORDERED_TOKENS", 4200)
    torch.manual_seed(tokens)
    w = torch.nn.Parameter(torch.randn(rows, cols, device="cuda", dtype=torch.bfloat16))
    ids = torch.randint(0, rows, (tokens,), device="cuda")
    ids[tokens // 2:] = int(ids[0])
    dy = torch.randn(tokens, cols, device="cuda", dtype=torch.bfloat16)
    before = torch.randn(rows, cols, device="cuda")
    got = []
    for _ in range(4):
        w.main_grad = before.clone()
        ops.token_embedding(ids, w).backward(dy)
        got.append(w.main_grad)
    assert w.grad is None and all(torch.equal(got[0], g) for g in got[1:])
    for i in {int(ids[0]), int(ids[tokens // 3])}:
        want = before[i].clone()
        for first in range(0, tokens, cu.ORDERED_TOKENS):
            rows_of = (ids[first:first + cu.ORDERED_TOKENS] == i).nonzero().flatten() + first
            total = torch.zeros(cols, device="cuda")
            for t in rows_of.tolist():
                total += dy[t].float()
            want += total
        assert torch.equal(got[0][i], want)


def test_embedding_gradient_that_somebody_looks_at(cu):
    """torch.autograd.grad for the table, hooks on it and a recorded backward pass get the dense gradient; a gradient asked for
    another leaf alone changes nothing."""
    from easyllm_b200 import ops
    torch.manual_seed(0)
    w = torch.nn.Parameter(torch.randn(50, 64, device="cuda", dtype=torch.bfloat16))
    scale = torch.nn.Parameter(torch.ones(64, device="cuda", dtype=torch.bfloat16))
    ids, dy = torch.randint(0, 50, (30,), device="cuda"), torch.randn(30, 64, device="cuda", dtype=torch.bfloat16)
    want = torch.autograd.grad(torch.nn.functional.embedding(ids, w), w, dy)[0]
    w.main_grad = torch.zeros(50, 64, device="cuda")
    assert torch.equal(torch.autograd.grad(ops.token_embedding(ids, w), w, dy)[0], want)
    assert torch.equal(torch.autograd.grad(ops.token_embedding(ids, w), w, dy, create_graph=True)[0], want)
    torch.autograd.grad(ops.token_embedding(ids, w) * scale, scale, dy)
    assert not w.main_grad.any()
    for register in (w.register_hook, w.register_post_accumulate_grad_hook):
        seen = []
        handle = register(lambda g: seen.append(g.grad.clone() if g is w else g.clone()))
        ops.token_embedding(ids, w).backward(dy)
        handle.remove()
        assert torch.equal(seen[0], want) and not w.main_grad.any()
        w.grad = None
    ops.token_embedding(ids, w).backward(dy)
    assert w.grad is None and torch.allclose(w.main_grad, want.float(), atol=0.02, rtol=0.02)


@pytest.mark.parametrize("T,hq,hk,D", [(1, 1, 1, 16), (7, 8, 2, 128), (301, 5, 5, 80)])
def test_rope_append_is_rope_and_append(cu, T, hq, hk, D):
    """Bit for bit the two launches it stands for: rotated rows, and the cache rows of scattered places; other rows stay."""
    import easyllm_b200.ops.cuda_infer as ci
    from easyllm_b200.ops import reference as ref
    torch.manual_seed(T)
    cos, sin = ref.rope_tables(D, 512, device="cuda")
    qkv = torch.randn(T, (hq + 2 * hk) * D, device="cuda", dtype=torch.bfloat16)
    pos = torch.randint(0, 512, (T,), device="cuda", dtype=torch.int32)
    rows = torch.randperm(3 * T, device="cuda")[:T].to(torch.int32)
    length = torch.randint(1, 4, (T,), device="cuda", dtype=torch.int32)
    base = rows - length + 1 + 4
    caches = [[torch.full((3 * T + 4, hk, D), 7.0, device="cuda", dtype=torch.bfloat16) for _ in "kv"] for _ in range(2)]
    want = cu.rope_(qkv.clone(), cos, sin, pos, hq + hk, D)
    k, v = want[:, hq * D:(hq + hk) * D].view(T, hk, D), want[:, (hq + hk) * D:].view(T, hk, D)
    ci.kv_append(*caches[0], k, v, base, length)
    got = cu.rope_append_(qkv, cos, sin, pos, hq, hk, D, *caches[1], base, length)
    cu.check_err_flag()
    assert torch.equal(got, want) and all(torch.equal(a, b) for a, b in zip(*caches))
