"""tcgen05 flash attention (causal, GQA, packed documents) against fp32 exact attention."""
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


CASES = [  # T, Hq, Hk, cu_seqlens
    (128, 2, 2, None), (256, 4, 4, None), (300, 4, 2, None), (1024, 8, 1, None),
    (512, 4, 4, [0, 100, 101, 350, 512]), (777, 2, 1, [0, 128, 256, 640, 777]), (4096, 4, 4, None),
]


@pytest.mark.parametrize("T,Hq,Hk,cu_list", CASES)
def test_flash_fwd(cu, T, Hq, Hk, cu_list):
    from easyllm_b200.ops import reference as ref
    torch.manual_seed(T + Hq)
    W = (Hq + 2 * Hk) * 128
    qkv = torch.randn(T, W, device="cuda", dtype=torch.bfloat16)      # views into a packed buffer
    q = qkv[:, :Hq * 128].view(T, Hq, 128)
    k = qkv[:, Hq * 128:(Hq + Hk) * 128].view(T, Hk, 128)
    v = qkv[:, (Hq + Hk) * 128:].view(T, Hk, 128)
    cs = torch.tensor(cu_list, dtype=torch.int32, device="cuda") if cu_list else None
    rs = cu._row_start(cs, T, q.device)
    scale = 128 ** -0.5
    out, lse = cu.flash_attn_fwd(q, k, v, rs, scale)
    torch.cuda.synchronize()
    cu.check_err_flag()
    want = ref.attention_varlen(q.float(), k.float(), v.float(), cs, True, scale)
    err = (out.float() - want).abs().max().item()
    assert err < 2e-2, err
    # log-sum-exp of the first head against the exact one
    rep = Hq // Hk
    s = torch.einsum("td,sd->ts", q[:, 0].float(), k[:, 0].float()) * scale
    idx = torch.arange(T, device="cuda")
    mask = (idx[None, :] > idx[:, None]) | (idx[None, :] < rs[:, None])
    s = s.masked_fill(mask, float("-inf"))
    assert (torch.logsumexp(s, -1) - lse[0]).abs().max().item() < 2e-2


def test_flash_autograd_path(cu):
    from easyllm_b200 import ops
    from easyllm_b200.ops import reference as ref
    torch.manual_seed(0)
    T, H = 384, 2
    q = torch.randn(T, H, 128, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    k = torch.randn(T, H, 128, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    v = torch.randn(T, H, 128, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    ops.set_attention_backend("kernel")
    try:
        o = ops.flash_attention(q, k, v, None, T, True)
        do = torch.randn_like(o)
        o.backward(do)
    finally:
        ops.set_attention_backend("auto")
    qf, kf, vf = (t.detach().float().requires_grad_() for t in (q, k, v))
    of = ref.attention_varlen(qf, kf, vf, None, True)
    of.backward(do.float())
    for a, b in ((q.grad, qf.grad), (k.grad, kf.grad), (v.grad, vf.grad)):
        assert (a.float() - b).abs().max().item() < 5e-2 * max(1.0, b.abs().max().item())


BWD_CASES = [  # T, Hq, Hk, cu_seqlens
    (128, 1, 1, None), (256, 2, 2, None), (300, 4, 2, None), (1024, 8, 2, None),
    (512, 4, 4, [0, 100, 101, 350, 512]), (777, 2, 1, [0, 128, 256, 640, 777]), (2048, 2, 2, None),
]


@pytest.mark.parametrize("T,Hq,Hk,cu_list", BWD_CASES)
def test_flash_bwd_packed(cu, T, Hq, Hk, cu_list):
    """Backward kernel on views of a packed buffer, gradients written into one packed dQKV."""
    from easyllm_b200.ops import reference as ref
    torch.manual_seed(T * 7 + Hq)
    W = (Hq + 2 * Hk) * 128
    qkv = torch.randn(T, W, device="cuda", dtype=torch.bfloat16)
    q, k, v = cu._split_packed(qkv, Hq, Hk, 128)
    cs = torch.tensor(cu_list, dtype=torch.int32, device="cuda") if cu_list else None
    rs = cu._row_start(cs, T, q.device)
    scale = 128 ** -0.5
    out, lse = cu.flash_attn_fwd(q, k, v, rs, scale)
    do = torch.randn(T, Hq, 128, device="cuda", dtype=torch.bfloat16)
    dqkv = torch.full_like(qkv, float("nan"))
    dq, dk, dv = cu._split_packed(dqkv, Hq, Hk, 128)
    cu.flash_attn_bwd(do, q, k, v, out, lse, rs, scale, dq, dk, dv)
    torch.cuda.synchronize()
    cu.check_err_flag()
    assert torch.isfinite(dqkv.float()).all()
    qf, kf, vf = (t.detach().float().requires_grad_() for t in (q, k, v))
    of = ref.attention_varlen(qf, kf, vf, cs, True, scale)
    of.backward(do.float())
    for name, a, b in (("dq", dq, qf.grad), ("dk", dk, kf.grad), ("dv", dv, vf.grad)):
        err = (a.float() - b).abs().max().item()
        tol = 3e-2 * max(1.0, b.abs().max().item())
        assert err < tol, (name, err, tol)


def _exact(q, k, v, rs, scale, window, sink):
    T, H, i = q.shape[0], q.shape[1], torch.arange(q.shape[0], device=q.device)
    k, v = (t.repeat_interleave(H // k.shape[1], 1) for t in (k, v))
    seen = (i.view(1, -1) <= i.view(-1, 1)) & (i.view(1, -1) >= rs.view(-1, 1)) & (i.view(1, -1) > i.view(-1, 1) - (window or T))
    s = (torch.einsum("qhd,khd->hqk", q, k) * scale).masked_fill(~seen, float("-inf"))
    if sink is not None:
        s = torch.cat((s, sink.double().view(-1, 1, 1).expand(-1, T, 1)), 2)
    return torch.einsum("hqk,khd->qhd", torch.softmax(s, -1)[..., :T], v)


@pytest.mark.parametrize("lens,Hq,Hk,d,dv,window", [
    ([1], 1, 1, 128, 128, None), ([129], 3, 1, 128, 128, None), ([256, 1], 2, 2, 64, 128, None), ([90, 38, 500], 2, 1, 128, 72, None),
    ([300, 212, 1, 255], 150, 75, 64, 64, None), ([5] * 200, 3, 3, 40, 128, None), ([900], 2, 2, 128, 128, 70), ([1200, 30], 40, 8, 128, 128, 300)])
def test_attention_items_and_tiles(cu, lens, Hq, Hk, d, dv, window):
    """Borders of query tiles, second tiles without rows or with documents of their own, more items than CTAs, head sizes that
    fill no chunk.  Against 64 bits: scores are exact to fp32, P (2^-9) and the result (2^-9) are rounded to bf16 once each, so
    the relative error stays below 2 * 2^-9 / sqrt(3) where the roundings are independent, and below 2^-8 in any case."""
    torch.manual_seed(len(lens) + Hq)
    T = sum(lens)
    qkv = torch.randn(T, Hq * d + Hk * (d + dv), device="cuda", dtype=torch.bfloat16)
    q, k, v = qkv[:, :Hq * d].view(T, Hq, d), qkv[:, Hq * d:(Hq + Hk) * d].view(T, Hk, d), qkv[:, (Hq + Hk) * d:].view(T, Hk, dv)
    if qkv.stride(0) % 8:
        pytest.skip("rows of the packed buffer are not 16-byte aligned")
    starts = [sum(lens[:i]) for i in range(len(lens))]
    rs = torch.tensor([s for s, n in zip(starts, lens) for _ in range(n)], dtype=torch.int32, device="cuda")
    sink = torch.randn(Hq, device="cuda")
    out = cu.flash_attn_fwd(q, k, v, rs, d ** -0.5, sink=sink, window=window)[0]
    cu.check_err_flag()
    want = _exact(q.double(), k.double(), v.double(), rs, d ** -0.5, window, sink)
    assert ((out.double() - want).norm() / want.norm()).item() < 2.0 ** -8


@pytest.mark.parametrize("lens,Hq,Hk", [([1], 1, 1), ([127, 2], 2, 1), ([128, 128], 2, 2), ([33] * 20, 4, 2), ([300, 1, 84], 30, 30),
                                        ([500, 700], 16, 1)])
def test_attention_backward_against_64_bits(cu, lens, Hq, Hk):
    """Keys that end their document inside a query tile, items beyond the CTAs, query heads split over CTAs.  Each of dq, dk, dv takes
    two values rounded to bf16 into every product (P or dS, after P was rounded) and is rounded itself: at most 4 * 2^-9 / sqrt(3),
    with twice that for sums that cancel."""
    torch.manual_seed(len(lens) + Hq)
    T, scale = sum(lens), 128 ** -0.5
    qkv = torch.randn(T, (Hq + 2 * Hk) * 128, device="cuda", dtype=torch.bfloat16)
    q, k, v = cu._split_packed(qkv, Hq, Hk, 128)
    starts = [sum(lens[:i]) for i in range(len(lens))]
    rs = torch.tensor([s for s, n in zip(starts, lens) for _ in range(n)], dtype=torch.int32, device="cuda")
    out, lse = cu.flash_attn_fwd(q, k, v, rs, scale)
    do = torch.randn_like(out)
    grads = cu.flash_attn_bwd(do, q, k, v, out, lse, rs, scale)
    cu.check_err_flag()
    wide = [t.double().requires_grad_() for t in (q, k, v)]
    _exact(*wide, rs, scale, None, None).backward(do.double())
    for name, a, b in zip(("dq", "dk", "dv"), grads, wide):
        bound = 8 * 2.0 ** -9 / 3 ** 0.5 * max(b.grad.norm().item(), 1e-2 * do.double().norm().item())
        assert (a.double() - b.grad).norm().item() < bound, name


def test_attention_backward_of_results_on_no_16_byte_place(cu):
    """The row sums read the results 16 bytes at a time; a copy of them that starts elsewhere gives the same gradients."""
    torch.manual_seed(2)
    T, H = 70, 2
    q, k, v, do = (torch.randn(T, H, 128, device="cuda", dtype=torch.bfloat16) for _ in range(4))
    rs = torch.zeros(T, dtype=torch.int32, device="cuda")
    out, lse = cu.flash_attn_fwd(q, k, v, rs, 128 ** -0.5)
    moved = torch.empty(out.numel() + 4, device="cuda", dtype=torch.bfloat16)[4:].view_as(out).copy_(out)
    assert moved.data_ptr() % 16 == 8
    for a, b in zip(cu.flash_attn_bwd(do, q, k, v, out, lse, rs, 128 ** -0.5), cu.flash_attn_bwd(do, q, k, v, moved, lse, rs, 128 ** -0.5)):
        assert torch.equal(a, b)


def test_flash_packed_autograd_matches_library(cu):
    from easyllm_b200 import ops
    torch.manual_seed(3)
    T, Hq, Hk = 640, 4, 2
    cs = torch.tensor([0, 200, 640], dtype=torch.int32, device="cuda")
    base = torch.randn(T, (Hq + 2 * Hk) * 128, device="cuda", dtype=torch.bfloat16)
    do = torch.randn(T, Hq * 128, device="cuda", dtype=torch.bfloat16)
    grads = {}
    for which in ("kernel", "library"):
        cu.set_attention_backward(which)
        try:
            x = base.clone().requires_grad_()
            o = ops.flash_attention_packed(x, Hq, Hk, 128, cs, 440)
            o.backward(do)
            grads[which] = x.grad.float()
        finally:
            cu.set_attention_backward("kernel")
    torch.cuda.synchronize()
    cu.check_err_flag()
    ref_max = grads["library"].abs().max().item()
    assert (grads["kernel"] - grads["library"]).abs().max().item() < 3e-2 * max(1.0, ref_max)


def test_packed_attention_with_rope_matches_reference(cu):
    """RoPE folded into the packed attention op (in-place rotate, packed un-rotated gradient)."""
    from easyllm_b200 import ops
    from easyllm_b200.ops import reference as ref
    torch.manual_seed(11)
    T, Hq, Hk, D = 384, 4, 2, 128
    cos, sin = ref.rope_tables(D, T, device="cuda")
    pos = torch.arange(T, device="cuda")
    base = torch.randn(T, (Hq + 2 * Hk) * D, device="cuda", dtype=torch.bfloat16)
    do = torch.randn(T, Hq * D, device="cuda", dtype=torch.bfloat16)
    x = base.clone().requires_grad_()
    o = ops.flash_attention_packed(x * 1, Hq, Hk, D, None, T, rope=(cos, sin, pos))
    o.backward(do)
    torch.cuda.synchronize()
    cu.check_err_flag()
    xf = base.float().requires_grad_()
    q = xf[:, :Hq * D].view(T, Hq, D)
    k = xf[:, Hq * D:(Hq + Hk) * D].view(T, Hk, D)
    v = xf[:, (Hq + Hk) * D:].view(T, Hk, D)
    qr, kr = ref.rope(q, k, cos.float(), sin.float(), pos)
    of = ref.attention_varlen(qr, kr, v, None, True).reshape(T, Hq * D)
    of.backward(do.float())
    assert (o.float() - of).abs().max().item() < 3e-2
    assert (x.grad.float() - xf.grad).abs().max().item() < 3e-2 * max(1.0, xf.grad.abs().max().item())


@pytest.mark.parametrize("T,Hq,Hk,D,cu_list", [(384, 4, 4, 128, None), (640, 8, 2, 128, [0, 130, 300, 640]),
                                               (300, 4, 4, 64, None), (512, 4, 2, 64, [0, 100, 512]),
                                               (256, 2, 2, 96, None)])
@pytest.mark.parametrize("alibi", [False, True])
def test_attention_kernel_with_alibi_and_small_heads(cu, T, Hq, Hk, D, cu_list, alibi):
    """ALiBi slopes (the bias slope · (key − query) inside the kernel's softmax, forward and backward) and head
    dimensions below 128 (zero-padded to the kernel's 128 columns), forced onto the kernel path, against the fp32
    statement of the same attention; forward output and all three gradients."""
    from easyllm_b200 import ops
    from easyllm_b200.models.layers import alibi_slopes
    from easyllm_b200.ops import reference as ref
    torch.manual_seed(T + D + Hq)
    q, k, v = (torch.randn(T, h, D, device="cuda", dtype=torch.bfloat16, requires_grad=True) for h in (Hq, Hk, Hk))
    cs = torch.tensor(cu_list, dtype=torch.int32, device="cuda") if cu_list else None
    slopes = torch.tensor(alibi_slopes(Hq), dtype=torch.float32, device="cuda") if alibi else None
    ops.set_attention_backend("kernel")
    ops.set_strict(True)
    try:
        o = ops.flash_attention(q, k, v, cs, T, True, alibi_slopes=slopes)
        do = torch.randn_like(o)
        o.backward(do)
    finally:
        ops.set_attention_backend("auto")
        ops.set_strict(False)
    torch.cuda.synchronize()
    cu.check_err_flag()
    qf, kf, vf = (t.detach().float().requires_grad_() for t in (q, k, v))
    of = ref.attention_varlen(qf, kf, vf, cs, True, None, slopes)
    of.backward(do.float())
    assert (o.float() - of).abs().max().item() < 2e-2
    for a, b in ((q.grad, qf.grad), (k.grad, kf.grad), (v.grad, vf.grad)):
        assert (a.float() - b).abs().max().item() < 5e-2 * max(1.0, b.abs().max().item())
        assert ((a.float() - b).norm() / b.norm()).item() < 2e-2


def test_attention_dropout_is_rejected_with_the_fused_kernels_and_applied_on_the_eager_path():
    from easyllm_b200.models.config import update_model_cfg
    base = dict(num_layers=1, hidden_size=128, num_attention_heads=2, vocab_size=256, seq_length=32)
    with pytest.raises(ValueError, match="attention_dropout"):
        update_model_cfg(dict(base, transformer_layer_params={"attention_dropout": 0.1}))
    args = update_model_cfg(dict(base, transformer_layer_params={"attention_dropout": 0.1, "use_flash_attn": False}))
    assert args.attention_dropout == 0.1 and not args.use_flash_attn


def _rows_exact(q, k, v, base, length, scale, sink, slopes, window, gate):
    """``attention_rows`` in 64 bits, row by row."""
    T, H, _ = q.shape
    G = k.shape[1]
    out = []
    for t in range(T):
        lo = max(0, length[t] - window) if window else 0
        rows = slice(base[t] + lo, base[t] + length[t])
        kt, vt = (x[rows].double().repeat_interleave(H // G, 1) for x in (k, v))
        s = torch.einsum("hd,khd->hk", q[t].double(), kt) * scale
        if slopes is not None:
            s = s + slopes.double()[:, None] * torch.arange(lo - length[t] + 1, 1, device=q.device)
        if sink is not None:
            s = torch.cat((s, sink.double()[:, None]), 1)
        o = torch.einsum("hk,khd->hd", torch.softmax(s, -1)[:, :kt.shape[0]], vt)
        out.append(o if gate is None else o * torch.sigmoid(gate[t].double())[:, None])
    return torch.stack(out)


@pytest.mark.parametrize("extras", ["plain", "sink", "slopes", "window", "window gate"])
@pytest.mark.parametrize("H,G,d,dv", [(8, 2, 128, 128), (4, 4, 64, 96), (24, 1, 96, 48), (10, 2, 16, 128), (32, 2, 128, 64)])
@pytest.mark.parametrize("steps,past", [([1, 1, 1], [0, 700, 63]), ([3, 1], [5, 130]), ([65, 17, 200], [300, 0, 64]),
                                        ([1, 129], [1023, 1])])
def test_attention_over_cached_rows(steps, past, H, G, d, dv, extras):
    """Decoding and continued prompts: rows at the edges of units, tiles and ranges of keys, groups of query heads that do not
    fill a tile or need two.  The result is a 64-bit one rounded to bf16 (2^-9 / sqrt(3) relative, 1.65e-3 over many values):
    weights of 8 bits would add as much again."""
    from easyllm_b200.ops import infer as iops
    torch.manual_seed(sum(steps) + H * d)
    dev, cap = "cuda", 1280
    k, v = (torch.randn(len(steps) * cap, G, n, device=dev).bfloat16() for n in (d, dv))
    T = sum(steps)
    q = torch.randn(T, H, d + 8, device=dev).bfloat16().flatten(1)[:, :H * d].unflatten(1, (H, d))
    base = [i * cap for i, n in enumerate(steps) for _ in range(n)]
    length = [p + j + 1 for n, p in zip(steps, past) for j in range(n)]
    cu = torch.tensor([0] + steps, device=dev).cumsum(0).int()
    sink = torch.randn(H, device=dev) if "sink" in extras else None
    slopes = torch.rand(H, device=dev) * 0.2 if "slopes" in extras else None
    window = 77 if "window" in extras else None
    gate = torch.randn(T, H, device=dev).bfloat16() if "gate" in extras else None
    b, n = (torch.tensor(x, dtype=torch.int32, device=dev) for x in (base, length))
    want = _rows_exact(q, k, v, base, length, d ** -0.5, sink, slopes, window, gate)
    for kw in ({"cu_seqlens": cu, "max_q": max(steps)}, {"cu_seqlens": cu, "max_q": max(steps) + 70}, {}):
        for bound in (max(length), cap):
            o = iops.attention_rows(q, k, v, b, n, bound, d ** -0.5, sink, slopes, window, gate, **kw)
            assert (o.double() - want).norm() <= 1.9e-3 * want.norm()
            assert (o.double() - want).abs().max() <= 2.0 ** -8 * want.abs().max()


@pytest.mark.parametrize("steps,past,H,G", [([1] * 40, [63] * 40, 8, 1), ([1] * 40, [63] * 40, 8, 8), ([60, 60], [5, 130], 4, 2)])
def test_weights_of_cached_rows_keep_32_bits(steps, past, H, G):
    """Values +1 and -1 under pairs of keys that differ by a bf16 step in one place: the result is a sum of differences, some 2^-12, of
    weights.  Rounding the result to bf16 is 1.65e-3 over many values, the fp32 exponentials (1e-7 of a weight each) add 0.6e-3;
    weights of 16 bits, 2^-18 off at random, would add 1e-2."""
    from easyllm_b200.ops import infer as iops
    torch.manual_seed(H + G)
    dev, d, cap = "cuda", 64, 256
    q = torch.randn(sum(steps), H, d, device=dev).bfloat16()
    q[..., 0] *= 0.25
    k = torch.randn(len(steps) * cap, G, d, device=dev).bfloat16()
    k[1::2] = k[0::2]
    k[1::2, :, 0] *= 1 + 2.0 ** -7
    v = torch.ones(len(steps) * cap, G, d, device=dev).bfloat16()
    v[1::2] = -1
    base = [i * cap for i, n in enumerate(steps) for _ in range(n)]
    length = [p + j + 1 for n, p in zip(steps, past) for j in range(n)]
    b, n = (torch.tensor(x, dtype=torch.int32, device=dev) for x in (base, length))
    kw = {"cu_seqlens": torch.tensor([0] + steps, device=dev).cumsum(0).int(), "max_q": max(steps)} if max(steps) > 1 else {}
    pairs = n % 2 == 0                                   # rows that see whole pairs
    o = iops.attention_rows(q, k, v, b, n, max(length), d ** -0.5, **kw)[pairs].double()
    want = _rows_exact(q, k, v, base, length, d ** -0.5, None, None, None, None)[pairs]
    assert want.numel() > 0 and want.abs().mean() < 2.0 ** -9
    assert (o - want).norm() <= 2.4e-3 * want.norm()


def _parts(x):
    """fp64 ``x`` as three bf16 numbers, 24 bits of it."""
    out = []
    for _ in range(3):
        out.append(x.bfloat16())
        x = x - out[-1].double()
    return out


def _scores_of_keys(tokens, past, fill):
    """One head whose scores are the first places of the keys, for sequences that go on with ``tokens`` tokens after ``past``; the new
    tokens weigh nothing.  ``fill(i, k, v)``: the cached keys' scores and values of sequence i."""
    dev, d, n = "cuda", 64, len(past)
    cap = max(past) + tokens
    k, v = torch.zeros(n * cap, 1, d, device=dev).bfloat16(), torch.zeros(n * cap, 1, d, device=dev).bfloat16()
    q = torch.zeros(n * tokens, 1, d, device=dev).bfloat16()
    q[:, :, 0] = 1
    for i, p in enumerate(past):
        own = slice(i * cap, i * cap + p)
        fill(i, k[own, 0, 0], v[own, 0])
        if tokens > 1:
            k[i * cap + p:i * cap + p + tokens, 0, 0] = -300
    base = [i * cap for i in range(n) for _ in range(tokens)]
    length = [p + j + (tokens > 1) for p in past for j in range(tokens)]
    kw = {"cu_seqlens": torch.arange(0, n * tokens + 1, tokens, device=dev, dtype=torch.int32), "max_q": tokens} if tokens > 1 else {}
    return q, k, v, base, length, kw


@pytest.mark.parametrize("tokens", [1, 5, 17, 40])
def test_exponentials_of_cached_rows_keep_32_bits(tokens):
    """Two weights, 1 and e^-x, whose values 1 and -e^x (24 bits of it, in three keys) cancel: what is left is the error of the weight.
    expf is off by 2 units of 2^-23 at most; four products are cut, or rounded, at 2^-23 of the sum.  An exponential of base 2 of the
    rounded product x log2(e) would be off by up to 2^-18 ln 2 where that product is above 64."""
    from easyllm_b200.ops import infer as iops
    scores = [-40 - 30 * i / 64 for i in range(64)]        # the parts of e^-70 are no denormal numbers

    def fill(i, k, v):
        k[:] = torch.tensor([0] + [scores[i]] * 3, device=k.device)
        v[0] = 1
        for j, p in enumerate(_parts(-torch.exp(-k[1].double()))):
            v[1 + j] = p

    q, k, v, base, length, kw = _scores_of_keys(tokens, [4] * 64, fill)
    b, n = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in (base, length))
    o = iops.attention_rows(q, k, v, b, n, max(length), 1.0, **kw).double()
    want = _rows_exact(q, k, v, base, length, 1.0, None, None, None, None)
    assert want.abs().max() < 2.0 ** -23
    assert (o - want).abs().max() <= 6 * 2.0 ** -23


@pytest.mark.parametrize("tokens,sequences", [(33, 160), (128, 148), (40, 3)])
def test_sums_of_a_continued_prompt_round_every_tile(tokens, sequences):
    """3000 positive values and one that takes their sum away again: what is left is the error of the sum.  A tile of 64 keys is four
    products of the weights' first parts, each cut at 2^-23 of it, and is added to the sum with half of that; the weights are off by 2^-22
    at most.  Sums that stay in the tensor core's accumulators are cut 12 times a tile, 2e-5 over 47 tiles."""
    from easyllm_b200.ops import infer as iops
    torch.manual_seed(tokens)
    last = 3

    def fill(i, k, v):
        n = k.numel() - last
        k[:n] = -torch.rand(n, device=k.device)
        v[:n] = (torch.rand(n, v.shape[1], device=k.device) + 0.5).bfloat16()
        total = torch.exp(k[:n].double()) @ v[:n].double()
        for j, p in enumerate(_parts(-total)):
            v[n + j] = p
        sums.append((total, torch.exp(k.double()).sum()))

    sums = []
    q, k, v, base, length, kw = _scores_of_keys(tokens, [3000] * sequences, fill)
    b, n = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in (base, length))
    o = iops.attention_rows(q, k, v, b, n, max(length), 1.0, **kw).double()[::tokens, 0]
    want = _rows_exact(q[::tokens], k, v, base[::tokens], length[::tokens], 1.0, None, None, None, None)[:, 0]
    total, weights = torch.stack([t for t, _ in sums]), torch.stack([w for _, w in sums])
    off = ((o - want) * weights[:, None] / total).abs()
    assert off.max() <= (4 + 47 / 2 + 2) * 2.0 ** -23 and off.mean() <= 8 * 2.0 ** -23


@pytest.mark.parametrize("steps,past,H,G", [([1] * 3, [700, 63, 64], 8, 2), ([3, 4], [130, 20], 4, 1), ([65, 40], [300, 25], 8, 2), ([17], [15], 1, 1)])
def test_what_lies_behind_the_end_of_a_sequence_costs_nothing(steps, past, H, G):
    """Slots are used again: infinities and NaN that an earlier sequence left behind the end give the bits that zeros there give (rows that
    come out not finite are summed again key by key, in another order, in many times the time)."""
    from easyllm_b200.ops import infer as iops
    torch.manual_seed(sum(steps))
    dev, d, cap = "cuda", 128, 1024
    q = torch.randn(sum(steps), H, d, device=dev).bfloat16()
    k, v = (torch.randn(len(steps) * cap, G, d, device=dev).bfloat16() for _ in "kv")
    base = [i * cap for i, n in enumerate(steps) for _ in range(n)]
    length = [p + j + 1 for n, p in zip(steps, past) for j in range(n)]
    b, n = (torch.tensor(x, dtype=torch.int32, device=dev) for x in (base, length))
    kw = {"cu_seqlens": torch.tensor([0] + steps, device=dev).cumsum(0).int(), "max_q": max(steps)} if max(steps) > 1 else {}
    out = []
    for left in (0.0, float("nan"), float("inf")):
        for i, (new, p) in enumerate(zip(steps, past)):
            k[i * cap + p + new:(i + 1) * cap] = left
            v[i * cap + p + new:(i + 1) * cap] = left
        out.append(iops.attention_rows(q, k, v, b, n, max(length), d ** -0.5, **kw))
    assert bool(out[0].isfinite().all()) and torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])


@pytest.mark.parametrize("window", [None, 77])
@pytest.mark.parametrize("steps,past,H,G", [([1, 1], [700, 63], 8, 2), ([3, 4], [130, 20], 8, 2), ([65, 40], [300, 25], 8, 2), ([2, 20], [2500, 30], 4, 4)])
def test_values_that_are_not_finite_reach_the_rows_that_see_them(steps, past, H, G, window):
    """Infinities of both signs and NaN among the values and keys of cached and of later tokens: rows that do not see them (earlier
    tokens, windows that have moved on) have the finite result, rows that see an infinity have it with its sign."""
    from easyllm_b200.ops import infer as iops
    torch.manual_seed(sum(steps))
    dev, d, cap = "cuda", 64, 2560
    q = torch.randn(sum(steps), H, d, device=dev).bfloat16()
    k, v = (torch.randn(len(steps) * cap, G, d, device=dev).bfloat16() for _ in "kv")
    base = [i * cap for i, n in enumerate(steps) for _ in range(n)]
    length = [p + j + 1 for n, p in zip(steps, past) for j in range(n)]
    for i, (n, p) in enumerate(zip(steps, past)):
        last, mid, old = i * cap + p + n - 1, i * cap + p + n // 2, i * cap + p - 15
        v[last, 0, 0], v[last, G - 1, 3], v[last, 0, 5] = float("inf"), float("nan"), float("-inf")
        v[mid, 0, 9], v[old, G - 1, 7], v[i * cap + 2, 0, 11] = float("-inf"), float("inf"), float("inf")
    k[cap + past[1] + steps[1] - 1, G - 1, 4] = float("nan")
    b, n = (torch.tensor(x, dtype=torch.int32, device=dev) for x in (base, length))
    cu = torch.tensor([0] + steps, device=dev).cumsum(0).int()
    want = _rows_exact(q, k, v, base, length, d ** -0.5, None, None, window, None)
    fine = want.isfinite()
    assert 0 < int(fine.sum()) < fine.numel()
    for kw in ({"cu_seqlens": cu, "max_q": max(steps)}, {}):
        o = iops.attention_rows(q, k, v, b, n, max(length), d ** -0.5, window=window, **kw)
        assert torch.equal(o.isnan(), want.isnan()) and torch.equal(o.isinf(), want.isinf())
        assert bool((o[want.isinf()].double() == want[want.isinf()]).all())
        assert (o[fine].double() - want[fine]).norm() <= 1.9e-3 * want[fine].norm()


@pytest.mark.parametrize("offset,pad", [(0, 0), (2, 0), (0, 2)])
@pytest.mark.parametrize("tokens,past,H,G,d,dv", [(17, 47, 1, 1, 128, 128), (32, 0, 1, 1, 64, 64), (33, 31, 1, 1, 80, 16), (127, 65, 2, 2, 128, 64),
                                                  (43, 128, 3, 1, 128, 128), (42, 511, 3, 1, 32, 112), (9, 4000, 16, 1, 128, 128)])
def test_rows_of_a_continued_prompt_fill_tiles_to_their_edges(tokens, past, H, G, d, dv, offset, pad):
    """Groups of 32 rows and tiles of 128 that are filled, one short and one over, keys likewise; queries on 16-byte places and on none.
    Bounds as for the rows above."""
    from easyllm_b200.ops import infer as iops
    torch.manual_seed(tokens + d)
    dev, cap = "cuda", past + tokens + 3
    k, v = (torch.randn(2 * cap, G, n, device=dev).bfloat16() for n in (d, dv))
    ld = H * d + pad
    flat = torch.randn(offset + 2 * tokens * ld, device=dev).bfloat16()
    q = flat[offset:].view(2 * tokens, ld)[:, :H * d].unflatten(1, (H, d))
    assert q.data_ptr() % 16 == 2 * offset
    base, length = [0] * tokens + [cap] * tokens, [past + j + 1 for j in range(tokens)] * 2
    b, n = (torch.tensor(x, dtype=torch.int32, device=dev) for x in (base, length))
    cu = torch.tensor([0, tokens, 2 * tokens], dtype=torch.int32, device=dev)
    want = _rows_exact(q, k, v, base, length, d ** -0.5, None, None, None, None)
    o = iops.attention_rows(q, k, v, b, n, past + tokens, d ** -0.5, cu_seqlens=cu, max_q=tokens)
    assert (o.double() - want).norm() <= 1.9e-3 * want.norm()
    assert (o.double() - want).abs().max() <= 2.0 ** -8 * want.abs().max()


@pytest.mark.parametrize("hq,hk", [(5, 5), (6, 2)])
def test_heads_in_several_groups(cu, hq, hk):
    """So many tokens that the heads' CTAs come in several groups, the last one smaller: documents of 512 tokens alone (the same
    tiles, in one group) give the same bits."""
    torch.manual_seed(0)
    T, D, doc = (40960 if hq == hk else 81920), 128, 512
    q, k, v = (torch.randn(T, h, D, device="cuda", dtype=torch.bfloat16) for h in (hq, hk, hk))
    start = torch.arange(T, device="cuda", dtype=torch.int32) // doc * doc
    out, lse = cu.flash_attn_fwd(q, k, v, start, D ** -0.5)[:2]
    cu.check_err_flag()
    for a in (0, T // 2, T - 4 * doc):
        part = slice(a, a + 4 * doc)
        o, l = cu.flash_attn_fwd(q[part].contiguous(), k[part].contiguous(), v[part].contiguous(), start[:4 * doc].contiguous(),
                                 D ** -0.5)[:2]
        assert torch.equal(out[part], o) and torch.equal(lse[:, part], l)


@pytest.mark.parametrize("n,H,G,bound", [(1, 8, 2, 4000), (3, 4, 4, 100), (40, 8, 4, 4352), (148, 1, 1, 3000), (149, 1, 1, 3000)])
def test_ranges_of_decoding_rows(cu, n, H, G, bound):
    """Both sides of the rule for the number of key ranges, against the softmax in 64 bits.  Ranges are multiples of 64 keys: lengths one
    below, at and one above each of them, one key and the bound.  The result is rounded to bf16 (2^-8 of itself at most), weights and sums
    are off by 2^-18 of the weighted sum of magnitudes: a lost key (3000 keys: 1e-3, results of 0.03) shows."""
    import easyllm_b200.ops.cuda_infer as ci
    d = 64
    g = torch.Generator(device="cuda").manual_seed(n)
    cap = bound + 8
    k, v = (torch.randn(n * cap, G, d, device="cuda", generator=g).to(torch.bfloat16) for _ in "kv")
    q = torch.randn(n, H, d, device="cuda", generator=g).to(torch.bfloat16)
    base = torch.arange(n, device="cuda", dtype=torch.int32) * cap
    lengths = [1] + [x for m in range(64, bound + 1, 64) for x in (m - 1, m, m + 1) if x <= bound] + [bound]
    k64, v64 = k.double(), v.double()
    for first in range(0, len(lengths), n):
        now = (lengths[first:first + n] + [bound] * n)[:n]
        out = ci.attention_rows(q, k, v, base, torch.tensor(now, device="cuda", dtype=torch.int32), bound, d ** -0.5).double()
        for i, length in enumerate(now[:len(lengths) - first]):
            kk, vv = (t[i * cap:i * cap + length].repeat_interleave(H // G, 1) for t in (k64, v64))
            p = torch.softmax(torch.einsum("hd,khd->hk", q[i].double(), kk) * d ** -0.5, -1)
            want, size = torch.einsum("hk,khd->hd", p, vv), torch.einsum("hk,khd->hd", p, vv.abs())
            assert ((out[i] - want).abs() <= want.abs() * 2.0 ** -8 + size * 2.0 ** -18).all(), (i, length)


def test_sequence_borders_of_any_integer_type(cu):
    """Borders in 64 bits, and every other element of a tensor, are the borders they hold."""
    import easyllm_b200.ops.cuda_infer as ci
    torch.manual_seed(0)
    q, k, v = (torch.randn(n, 4, 64, device="cuda", dtype=torch.bfloat16) for n in (20, 40, 40))
    base, length = torch.zeros(20, dtype=torch.int32, device="cuda"), torch.arange(21, 41, dtype=torch.int32, device="cuda")
    borders = torch.tensor([0, 20], device="cuda")
    got = [ci.attention_rows(q, k, v, base, length, 40, 0.125, cu_seqlens=c, max_q=20)
           for c in (borders.int(), borders, torch.tensor([0, 7, 20, 7], device="cuda", dtype=torch.int32)[::2])]
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
