"""Each mechanism of the hybrid decoder layers alone, against its plain statement: on the CPU and, marked gpu, the
kernels in fp32 and bf16, with sizes that hit and miss their vector and tensor-core paths."""
import math

import pytest
import torch

import plain_pafodra as plain
from easyllm_b200.ops import infer as iops

DEVICES = ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)]
F32, BF16 = torch.float32, torch.bfloat16


def _device(name):
    if name == "cuda":
        if not torch.cuda.is_available():
            pytest.skip("no GPU")
        from easyllm_b200.ops import cuda
        cuda.lib()
    return torch.device(name)


def close(got, want, tol):
    d = (got.double().cpu() - want.double()).abs().max()
    assert d <= tol * max(1.0, float(want.abs().max())), float(d)


def rand(*shape, seed=0, scale=1.0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale


def meta_of(counts, dev, slots=None, start=None):
    cu = [0]
    for c in counts:
        cu.append(cu[-1] + c)

    def t(x):
        return torch.tensor(x, dtype=torch.int32, device=dev)
    m = {"cu_seqlens": t(cu), "max_seqlen": max(counts)}
    if slots is not None:
        m.update(seq_slot=t(slots), seq_pos0=t(start))
    return m


# ---- matrix products ---------------------------------------------------------------------------
@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("M,N,K", [(1, 5, 24), (1, 4096, 512), (3, 37, 50), (7, 264, 1032), (16, 1, 128), (70, 17, 64),
                                   (300, 520, 136), (33, 40, 20)])
def test_linear_forms(device, dtype, M, N, K):
    dev = _device(device)
    x, w, b = (t.to(dtype).to(dev) for t in (rand(M, K + 8, seed=1), rand(N, K, seed=2, scale=K ** -0.5), rand(N, seed=3)))
    want = x.double().cpu()[:, :K] @ w.double().cpu().t()
    tol = 2e-6 if dtype == F32 else 8e-3
    xs = x[:, :K]                                                  # a column slice of wider rows
    close(iops.linear(xs, w), want, tol)
    close(iops.linear(xs, w, b), want + b.double().cpu(), tol)
    close(iops.linear_f32(xs, w), want, 2e-6 if device == "cuda" or dtype == F32 else tol)
    close(iops.linear_act(xs, w, "tanh"), torch.tanh(want), tol)
    acc = rand(M, N, seed=4).to(dev)
    want_acc = rand(M, N, seed=4).double() + want
    assert iops.linear_add_(acc, xs.contiguous(), w) is acc
    close(acc, want_acc, 2e-6 if device == "cuda" or dtype == F32 else tol)
    ws = torch.stack([w, 2 * w, -w])
    xb = torch.stack([xs, xs + 1, xs])
    close(iops.linear_batch(xb, list(ws)), torch.stack([x_.double().cpu() @ w_.double().cpu().t() for x_, w_ in zip(xb, ws)]), tol)


def test_adjacent_parameters_alias_without_a_copy():
    ps = [torch.nn.Parameter(rand(n, 6, seed=n)) for n in (3, 5, 1)]
    before = torch.cat([p.detach() for p in ps])
    assert iops.fused_alias(ps) is None
    iops.make_adjacent_(ps)
    a = iops.fused_alias(ps)
    assert a is not None and torch.equal(a, before) and a.data_ptr() == ps[0].data_ptr()
    bs = [torch.nn.Parameter(rand(n, seed=n)) for n in (4, 2)]
    iops.make_adjacent_(bs)
    assert iops.fused_alias(bs).shape == (6,) and torch.equal(iops.fused(bs), torch.cat([b.detach() for b in bs]))


# ---- elementwise -------------------------------------------------------------------------------
@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("W", [8, 30, 264])
def test_norm_embedding_and_activations(device, dtype, W):
    dev = _device(device)
    tol = 1e-6 if dtype == F32 else 8e-3
    x, w, b, add = rand(9, W, scale=3.0), rand(W, seed=1), rand(W, seed=2), rand(W, seed=3).to(dtype)
    xd = x.clone().to(dev)
    y = iops.dynamic_tanh(xd, torch.tensor(0.7).to(dev), w.to(dev), b.to(dev), dtype, add.to(dev))
    close(y, plain.dynamic_tanh(x.double(), torch.tensor(0.7).double(), w.double(), b.double()), tol)
    close(xd, x + add.float(), 1e-6)                       # the stream gains the bias after its norm was taken
    table = rand(11, W, seed=4).to(dtype)
    ids = torch.tensor([3, 10, 0, 3])
    close(iops.embed_scaled(ids.to(dev), table.to(dev), 5.25), table[ids].double() * 5.25, 1e-6)
    gu = rand(9, 2 * W, seed=5, scale=2.0).to(dtype)
    g, u = gu.double()[:, :W], gu.double()[:, W:]
    close(iops.glu(gu.to(dev), "gelu_tanh"), plain.gelu_tanh(g) * u, tol)
    close(iops.glu(gu.to(dev), "silu"), plain.silu(g) * u, tol)
    z = rand(9, 3, seed=6)
    close(iops.relu2_scaled(gu.to(dev), z.to(dev)[:, 1]), plain.sigmoid(z.double()[:, 1:2]) * gu.double().clamp(min=0) ** 2, tol)


# ---- attention -----------------------------------------------------------------------------------
def _rows(counts, dev):
    """kv_base / kv_len / row_start of packed fresh sequences."""
    base, length, at = [], [], 0
    for c in counts:
        base += [at] * c
        length += list(range(1, c + 1))
        at += c
    return [torch.tensor(x, dtype=torch.int32, device=dev) for x in (base, length)]


def _attention(q, k, v, counts, scale, sink, dev, prefill):
    base, length = _rows(counts, dev)
    q, k, v = q.to(dev), k.to(dev), v.to(dev)
    sink = None if sink is None else sink.to(dev)
    if prefill:
        assert iops.prefill_kernel_ok(q, v)
        return iops.attention_prefill(q, k, v, base, scale, sink)
    return iops.attention_rows(q, k, v, base, length, max(counts), scale, sink)


@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("dtype,prefill", [(F32, False), (BF16, False), (BF16, True)])
@pytest.mark.parametrize("H,G,d,dv", [(4, 2, 16, 24), (3, 1, 64, 8), (6, 6, 96, 72), (2, 1, 128, 128), (24, 2, 40, 104)])
def test_sink_attention(device, dtype, prefill, H, G, d, dv):
    dev = _device(device)
    if prefill and device == "cpu":
        pytest.skip("the prefill kernel needs a GPU")
    counts = [1, 45, 2]
    T = sum(counts)
    q, k, v = rand(T, H, d, seed=1).to(dtype), rand(T, G, d, seed=2).to(dtype), rand(T, G, dv, seed=3).to(dtype)
    for sink in (rand(H, seed=4) * 2, None):
        got = _attention(q, k, v, counts, 0.37, sink, dev, prefill)
        want, at = [], 0
        for c in counts:
            part = slice(at, at + c)
            want.append(plain.sink_attention(q[part].double(), k[part].double(), v[part].double(), 0.37,
                                             None if sink is None else sink.double()))
            at += c
        close(got, torch.cat(want), 2e-6 if dtype == F32 else 2e-2)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,prefill", [(F32, False), (BF16, False), (BF16, True)])
@pytest.mark.parametrize("d,dv", [(64, 64), (96, 40), (128, 128)])
def test_far_keys_tile_edges_and_the_sink_stand_out(dtype, prefill, d, dv):
    """One key per query is the only one that scores: the first token, the neighbours of tile and range borders, the
    token itself.  Every other place reads almost nothing but the sink, so a wrong key, a key one place off, a lost
    first token or a sink that is left out (or counted twice) changes the value by its own size."""
    dev = _device("cuda")
    T, H, G = 1030, 4, 2
    targets = [0, 1, 63, 64, 127, 128, 129, 255, 256, 511, 512, 1023, 1024]
    gen = torch.Generator().manual_seed(0)
    code = torch.sign(torch.randn(T, d, generator=gen)) / math.sqrt(d)     # nearly orthogonal unit rows
    k = code.view(T, 1, d).repeat(1, G, 1)
    k[:, 1] = -k[:, 1]
    q = torch.zeros(T, H, d)
    v = torch.randn(T, G, dv, generator=gen)
    sink = torch.tensor([18.0, 20.0, 19.0, 21.0])
    hit = {}
    for i in range(T):
        seen = [t for t in targets if t <= i] + [i]
        hit[i] = [seen[(i + h) % len(seen)] for h in range(H)]
        for h in range(H):
            q[i, h] = k[hit[i][h], h // 2] * 20.0                          # score 20 at the target, about 20/sqrt(d) elsewhere
    q, k, v = q.to(dtype), k.to(dtype), v.to(dtype)
    got = _attention(q, k, v, [T], 1.0, sink, dev, prefill).double().cpu()
    s = torch.einsum("qhd,khd->hqk", q.double(), k.double().repeat_interleave(2, 1))
    s = s.masked_fill(torch.ones(T, T, dtype=torch.bool).triu(1), float("-inf"))
    p = torch.softmax(torch.cat((s, sink.double().view(H, 1, 1).expand(H, T, 1)), -1), -1)[..., :T]
    want = torch.einsum("hqk,khd->qhd", p, v.double().repeat_interleave(2, 1))
    assert max(float(p[h, i, hit[i][h]]) for i in (700, 1029) for h in range(H)) > 0.3
    close(got, want, 1e-5 if dtype == F32 else 2e-2)


@pytest.mark.parametrize("device", DEVICES)
def test_cache_rows_of_several_slots(device):
    """Keys and values go to their slot and position; queries of different sequences read their own rows only, with the
    far part of the cache left full of another sequence's keys."""
    dev = _device(device)
    G, H, d, dv, cap = 2, 4, 24, 16, 300
    kc, vc = rand(3, cap, G, d, seed=1).to(dev) * 9, rand(3, cap, G, dv, seed=2).to(dev) * 9
    ks, vs = rand(290, G, d, seed=3), rand(290, G, dv, seed=4)
    sink = rand(H, seed=5)
    n2, n0 = 151, 130
    for slot, rows, pos in ((2, range(0, 151), range(0, 151)), (0, range(151, 281), range(0, 130))):
        m = {"kv_base": torch.full((len(rows),), slot * cap, dtype=torch.int32, device=dev),
             "kv_len": torch.tensor([p + 1 for p in pos], dtype=torch.int32, device=dev)}
        iops.kv_append(kc, vc, ks[list(rows)].to(dev), vs[list(rows)].to(dev), m)
    q = rand(3, H, d, seed=6)
    base = torch.tensor([2 * cap, 0, 2 * cap], dtype=torch.int32, device=dev)
    length = torch.tensor([n2, n0, 64], dtype=torch.int32, device=dev)
    got = iops.attention_rows(q.to(dev), kc.view(-1, G, d), vc.view(-1, G, dv), base, length, cap, 0.5, sink.to(dev))
    for t, (a, n) in enumerate(((0, n2), (151, n0), (0, 64))):
        want = plain.sink_attention(torch.cat((torch.zeros(n - 1, H, d), q[t:t + 1])).double(), ks[a:a + n].double(),
                                    vs[a:a + n].double(), 0.5, sink.double())[-1]
        close(got[t], want, 2e-6)


# ---- recurrences -----------------------------------------------------------------------------------
CUTS = [[40], [1] * 40, [16, 17, 7], [2, 3, 33, 1, 1]]


@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("W", [20, 64, 1032])
def test_token_shift(device, dtype, W):
    dev = _device(device)
    h, mu = rand(40, W, seed=1).to(dtype), torch.rand(5, W, generator=torch.Generator().manual_seed(2))
    want = torch.stack([plain.token_shift(h.double(), m.double()) for m in mu])
    tol = 1e-6 if dtype == F32 else 2e-2
    close(iops.token_mix(h.to(dev), mu.to(dev), meta_of([40], dev), None), want, tol)
    for cuts in CUTS:
        tail, at, got = torch.full((3, W), 7.0, dtype=dtype, device=dev), 0, []
        for c in cuts:
            got.append(iops.token_mix(h[at:at + c].to(dev), mu.to(dev), meta_of([c], dev, [1], [at]), tail))
            at += c
        close(torch.cat(got, 1), want, tol)
        assert torch.equal(tail[1].cpu(), h[-1]) and bool((tail[[0, 2]] == 7).all())


def _scan_inputs(kind, H, G, d, dv, T, dtype):
    q, k, v = rand(T, G, d, seed=1), rand(T, G, d, seed=2, scale=d ** -0.5), rand(T, H, dv, seed=3)
    g = torch.exp(-torch.exp(rand(T, H, d, seed=4) - 3))
    if kind == "wkv":
        return q.to(dtype), k.to(dtype), v.to(dtype), g, rand(H, d, seed=5)
    return plain.unit(q) * d ** -0.5, plain.unit(k), v, g, torch.sigmoid(rand(T, H, seed=5))


def _scan(kind, ins, part, m, state, dev):
    a = [x[part].to(dev) for x in ins[:4]]
    if kind == "wkv":
        return iops.wkv_scan(*a, ins[4].to(dev), m, state)
    return iops.delta_scan(*a, ins[4][part].to(dev), m, state)


@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("kind,dtype", [("wkv", F32), ("wkv", BF16), ("delta", F32)])
@pytest.mark.parametrize("H,G,d,dv", [(2, 2, 32, 32), (4, 2, 20, 44), (2, 1, 128, 128), (1, 1, 200, 33), (3, 3, 64, 7)])
def test_scans(device, kind, dtype, H, G, d, dv):
    """A sequence in one piece, cut into steps, and beside others in a batch; the slot's old contents never show."""
    dev = _device(device)
    if kind == "wkv":
        G = H
    T = 40
    ins = _scan_inputs(kind, H, G, d, dv, T, dtype)
    which = [h // (H // G) for h in range(H)]
    qd, kd, vd, gd, ud = (x.double() for x in ins)
    want, S = (plain.wkv_recurrence(qd, kd, vd, gd, ud) if kind == "wkv"
               else plain.delta_recurrence(qd[:, which], kd[:, which], vd, gd, ud))
    tol = 4e-6
    close(_scan(kind, ins, slice(0, T), meta_of([T], dev), None, dev), want, tol)
    for cuts in CUTS:
        state = torch.full((3, H, dv, iops.padded_rows(d)), 5.0, device=dev)
        at, got = 0, []
        for c in cuts:
            got.append(_scan(kind, ins, slice(at, at + c), meta_of([c], dev, [2], [at]), state, dev))
            at += c
        close(torch.cat(got), want, tol)
        close(state[2][..., :d], S.transpose(1, 2), tol)
        assert bool((state[:2] == 5).all())
    # the same 40 tokens as three sequences of a batch, each in its own slot
    state = torch.full((4, H, dv, iops.padded_rows(d)), 5.0, device=dev)
    got = _scan(kind, ins, slice(0, T), meta_of([5, 1, 34], dev, [3, 0, 1], [0, 0, 0]), state, dev)
    at = 0
    for c, slot in ((5, 3), (1, 0), (34, 1)):
        p = slice(at, at + c)
        o, S = (plain.wkv_recurrence(qd[p], kd[p], vd[p], gd[p], ud) if kind == "wkv"
                else plain.delta_recurrence(qd[p][:, which], kd[p][:, which], vd[p], gd[p], ud[p]))
        close(got[p], o, tol)
        close(state[slot][..., :d], S.transpose(1, 2), tol)
        at += c


@pytest.mark.gpu
@pytest.mark.parametrize("kind,dtype", [("wkv", F32), ("wkv", BF16), ("delta", F32)])
@pytest.mark.parametrize("H,G,d,dv,counts", [(2, 2, 64, 64, [256]), (4, 2, 20, 48, [300, 1, 37]), (2, 1, 128, 128, [257, 16]),
                                             (1, 1, 100, 8, [15, 270, 273])])
def test_scans_in_chunks(kind, dtype, H, G, d, dv, counts):
    """Sequences long enough for chunks of 16 tokens, beside short ones and going on from a slot's state; decays between 0 and 1 with
    both ends among them.  Sums of up to 273 tokens in fp32: the tolerance of the other scans."""
    dev = _device("cuda")
    if kind == "wkv":
        G = H
    T = sum(counts)
    ins = list(_scan_inputs(kind, H, G, d, dv, 2 * T, dtype))
    ins[3][::7, :, ::3], ins[3][::5, :, 1::3] = 0.0, 1.0
    which = [h // (H // G) for h in range(H)]
    qd, kd, vd, gd, ud = (x.double() for x in ins)
    state = torch.full((5, H, dv, iops.padded_rows(d)), 5.0, device=dev)
    slots = [3, 0, 1][:len(counts)]
    done = [0] * len(counts)
    S = [None] * len(counts)
    for go in range(2):
        m = meta_of(counts, dev, slots, done)
        got = _scan(kind, ins, slice(go * T, (go + 1) * T), m, state, dev)
        at = go * T
        for i, c in enumerate(counts):
            p = slice(at, at + c)
            o, S[i] = (plain.wkv_recurrence(qd[p], kd[p], vd[p], gd[p], ud, S[i]) if kind == "wkv"
                       else plain.delta_recurrence(qd[p][:, which], kd[p][:, which], vd[p], gd[p], ud[p], S[i]))
            close(got[at - go * T:at - go * T + c], o, 4e-6)
            close(state[slots[i]][..., :d], S[i].transpose(1, 2), 4e-6)
            assert d % 32 == 0 or bool((state[slots[i]][..., d:] == 0).all())
            at, done[i] = at + c, done[i] + c
    assert bool((state[[2, 4]] == 5).all())


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["wkv", "delta"])
def test_a_chunk_does_not_look_ahead(kind):
    """A value that is not a number shows in its own column from its token on, not before it nor beside it."""
    dev = _device("cuda")
    T, t, j = 300, 133, 5
    ins = list(_scan_inputs(kind, 2, 2, 64, 32, T, F32))
    clean = _scan(kind, ins, slice(0, T), meta_of([T], dev), None, dev)
    ins[2] = ins[2].clone()
    ins[2][t, 1, j] = math.nan
    got = _scan(kind, ins, slice(0, T), meta_of([T], dev), None, dev)
    hit = torch.zeros_like(got, dtype=torch.bool)
    hit[t:, 1, j] = True
    assert torch.equal(got[~hit], clean[~hit]) and bool(got[t + 1:, 1, j].isnan().all())


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["wkv", "delta"])
def test_scans_in_rounds_of_chunks(kind, monkeypatch):
    """More tokens than the records of one round hold, against the kernels that go token by token."""
    from easyllm_b200.ops import cuda, cuda_infer
    dev = _device("cuda")
    H, T = 64, 5000 if kind == "delta" else 7500
    ins = _scan_inputs(kind, H, H, 128, 8, T, F32)
    need = cuda.lib().ell_scan_chunks_work(int(kind == "delta"), T, 2, T - 40, H, 128, 8)
    assert need * 4 < 520 << 20                        # the records of all chunks would take 550 MiB and more
    got = []
    for chunks in (True, False):
        if not chunks:
            monkeypatch.setattr(cuda_infer, "_scan_chunks", lambda *a: False)
        state = torch.zeros(2, H, 8, 128, device=dev)
        got.append((_scan(kind, ins, slice(0, T), meta_of([T - 40, 40], dev, [1, 0], [0, 0]), state, dev), state))
    cuda.check_err_flag()
    close(got[0][0], got[1][0].cpu(), 1e-5)
    close(got[0][1], got[1][1].cpu(), 1e-5)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["wkv", "delta"])
@pytest.mark.parametrize("d,T", [(64, 260), (128, 260), (128, 900)])
@pytest.mark.parametrize("decay", ["served", -3.0, 0.0])
def test_chunks_are_as_precise_as_tokens(kind, d, T, decay, monkeypatch):
    """The error of a scan in chunks against 64 bits is no larger than that of the scan token by token, from decays as a trained model
    has them to decays that forget in a few tokens: of the outputs always, of the state where it spans more than a few tokens (one
    rounding of a product is all of it otherwise)."""
    from easyllm_b200.ops import cuda_infer
    dev = _device("cuda")
    H = 4
    g = torch.Generator(dev).manual_seed(T + d)
    q, k, v, x = (torch.randn(T, H, d, device=dev, generator=g) for _ in range(4))
    rate = torch.rand(1, H, d, device=dev, generator=g) * 5 - 6 + 0.1 * x if decay == "served" else x + decay
    dec = torch.exp(-torch.exp(rate))
    if kind == "wkv":
        ins = [q.to(BF16), (k * d ** -0.5).to(BF16), v.to(BF16), dec, torch.randn(H, d, device=dev, generator=g)]
    else:
        ins = [plain.unit(q) * d ** -0.5, plain.unit(k), v, dec, torch.sigmoid(torch.randn(T, H, device=dev, generator=g))]
    qd, kd, vd, gd, ud = (t.double() for t in ins)
    S, want = torch.zeros(H, d, d, dtype=torch.float64, device=dev), torch.empty(T, H, d, dtype=torch.float64, device=dev)
    for t in range(T):                                      # [H, value column, key row]
        if kind == "wkv":
            kv = vd[t].unsqueeze(-1) * kd[t].unsqueeze(-2)
            want[t] = ((S + kv * ud.unsqueeze(-2)) * qd[t].unsqueeze(-2)).sum(-1)
            S = S * gd[t].unsqueeze(-2) + kv
        else:
            S = S * gd[t].unsqueeze(-2)
            e = ud[t].unsqueeze(-1) * (vd[t] - (S * kd[t].unsqueeze(-2)).sum(-1))
            S = S + e.unsqueeze(-1) * kd[t].unsqueeze(-2)
            want[t] = (S * qd[t].unsqueeze(-2)).sum(-1)
    off = []
    for chunks in (True, False):
        if not chunks:
            monkeypatch.setattr(cuda_infer, "_scan_chunks", lambda *a: False)
        state = torch.zeros(1, H, d, d, device=dev)
        o = _scan(kind, ins, slice(0, T), meta_of([T], dev, [0], [0]), state, dev)
        off.append(((o.double() - want).norm() / want.norm(), (state[0].double() - S).norm() / S.norm()))
    (o, s), (o_tokens, s_tokens) = off
    assert o <= 1.02 * o_tokens and (decay == 0.0 or s <= 1.02 * s_tokens), off


@pytest.mark.gpu
@pytest.mark.parametrize("kind,dtype,H,d,dv", [("wkv", BF16, 2, 64, 64), ("wkv", F32, 1, 100, 24), ("delta", F32, 2, 128, 40), ("delta", F32, 2, 36, 64)])
@pytest.mark.parametrize("bound", [None, 256, 257])
def test_scans_of_sequences_longer_than_their_bound(kind, dtype, H, d, dv, bound):
    """The scans need no bound of the sequences' lengths: one that is missing or too small (by whole chunks and by a few tokens)
    gives what the right one gives, going on from a slot's state."""
    dev = _device("cuda")
    counts = [300, 5, 260]
    T = sum(counts)
    ins = _scan_inputs(kind, H, H, d, dv, T, dtype)
    qd, kd, vd, gd, ud = (x.double() for x in ins)
    state = torch.zeros(3, H, dv, iops.padded_rows(d), device=dev)
    state[..., :d].normal_(generator=torch.Generator(dev).manual_seed(1))
    S0 = state.double().cpu()[..., :d].transpose(2, 3)
    m = meta_of(counts, dev, [2, 0, 1], [9, 9, 0])
    m["max_seqlen"] = bound
    if bound is None:
        del m["max_seqlen"]
    got = _scan(kind, ins, slice(0, T), m, state, dev)
    at = 0
    for i, c in enumerate(counts):
        p = slice(at, at + c)
        S = S0[[2, 0, 1][i]] if i < 2 else None
        o, S = (plain.wkv_recurrence if kind == "wkv" else plain.delta_recurrence)(qd[p], kd[p], vd[p], gd[p], ud if kind == "wkv" else ud[p], S)
        close(got[p], o, 4e-6)
        close(state[[2, 0, 1][i]][..., :d], S.transpose(1, 2), 4e-6)
        at += c
    assert bool((state[..., d:] == 0).all())


@pytest.mark.gpu
@pytest.mark.parametrize("kind,dtype,d", [("wkv", BF16, 64), ("wkv", F32, 128), ("delta", F32, 64), ("delta", F32, 128)])
@pytest.mark.parametrize("where", ["value", "state", "large", "key", "none"])
def test_infinities_in_a_scan_in_chunks(kind, dtype, d, where, monkeypatch):
    """An infinite value, state entry or key, and a finite value whose bf16 part is infinite, end where the scan token by token has
    them, with their sign; what is finite there is finite here."""
    from easyllm_b200.ops import cuda_infer
    dev = _device("cuda")
    H, dv, T, t = 2, 24, 300, 133
    ins = [x.clone() for x in _scan_inputs(kind, H, H, d, dv, T, dtype)]
    ins[0], ins[1] = ins[0].abs(), ins[1].abs()            # no infinities of both signs in a sum, which would be NaN anyway
    if kind == "wkv":
        ins[4] = ins[4].abs()
    first = torch.rand(1, H, dv, iops.padded_rows(d), device=dev)
    if where == "value":
        ins[2][t, 1, 5], ins[2][t + 60, 0, 17] = math.inf, -math.inf
    elif where == "large":
        ins[2][t, 1, 5] = torch.finfo(dtype).max
    elif where == "state":
        first[0, 1, 7, 3] = math.inf
    elif where == "key":
        ins[1][t, 1, 9] = math.inf
    got, kept = [], []
    for chunks in (True, False):
        if not chunks:
            monkeypatch.setattr(cuda_infer, "_scan_chunks", lambda *a: False)
        state = first.clone()
        got.append(_scan(kind, ins, slice(0, T), meta_of([T], dev, [0], [1]), state, dev))
        kept.append(state)
    assert where in ("none", "large") or not bool(got[1].isfinite().all())
    for a, b in (got, kept):
        fine = b.isfinite()
        assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isinf(), b.isinf()) and bool((a[b.isinf()] == b[b.isinf()]).all())
        rest = fine.clone()
        if where == "large":                               # a column of its own size
            rest[(slice(None), 1, 5) if b is got[1] else (0, 1, 5)] = False
        close(a[rest], b[rest].cpu(), 1e-5)
        assert bool(((a - b).abs()[fine & ~rest] <= 1e-5 * b.abs()[fine & ~rest].max()).all()) if bool((fine & ~rest).any()) else True


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n_seq", [1, 7, 61, 256, 1024, 5000])
@pytest.mark.parametrize("longest", [128, 300, 4096, 32768])
def test_records_of_a_scan_stay_within_their_limit(mode, n_seq, longest):
    """Host only: whatever the number and the lengths of the sequences, a scan's work space is 512 MiB at most, or it goes token by
    token and needs none; a single sequence of any length goes in chunks."""
    from easyllm_b200.ops import cuda
    for H, d, dv in ((16, 128, 128), (64, 128, 128), (64, 64, 64)):
        need = cuda.lib().ell_scan_chunks_work(mode, n_seq * longest, n_seq, longest, H, d, dv)
        assert 0 <= need * 4 <= 512 << 20
        assert n_seq > 1 or longest < 256 or need > 0


@pytest.mark.parametrize("counts,chunks", [([4096], True), ([512] * 8, True), ([128] + [16] * 60, False), ([256] + [32] * 60, False),
                                           ([300] * 20, True), ([2048] + [100] * 60, True), ([1024] + [16] * 30, True),
                                           ([260] + [1] * 63, False)])
def test_one_long_sequence_does_not_send_many_short_ones_through_chunks(counts, chunks):
    """Host only: which way a scan of the delta rule goes, 16 heads of 128 x 128."""
    from easyllm_b200.ops import cuda
    assert (cuda.lib().ell_scan_chunks_work(1, sum(counts), len(counts), max(counts), 16, 128, 128) > 0) == chunks


@pytest.mark.gpu
@pytest.mark.parametrize("kind,dtype", [("wkv", BF16), ("delta", F32)])
def test_records_of_every_sequence_are_found(kind, dtype):
    """Sequences of no token, of one and of many, in an order where the borders of records and of sequences fall apart: each has the
    result that it has alone."""
    dev = _device("cuda")
    counts = [1, 0, 257, 16, 15, 0, 0, 300, 33, 1, 1, 640, 17]
    T, H = sum(counts), 2
    ins = _scan_inputs(kind, H, H, 64, 32, T, dtype)
    state = torch.full((len(counts) + 1, H, 32, 64), 5.0, device=dev)
    slots = [(5 * i + 3) % len(counts) for i in range(len(counts))]
    got = _scan(kind, ins, slice(0, T), meta_of(counts, dev, slots, [0] * len(counts)), state, dev)
    at = 0
    for c, slot in zip(counts, slots):
        if c:
            one = torch.zeros(1, H, 32, 64, device=dev)
            part = [x[at:at + c] for x in ins[:4]] + [ins[4] if kind == "wkv" else ins[4][at:at + c]]
            want = _scan(kind, part, slice(0, c), meta_of([c], dev, [0], [0]), one, dev)
            close(got[at:at + c], want.cpu(), 4e-6)
            close(state[slot], one[0].cpu(), 4e-6)
        else:
            assert bool((state[slot] == 5).all())
        at += c


@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("kind", ["wkv", "delta"])
def test_state_is_carried_far(device, kind):
    """A value written at the first token with a decay of almost one is read 3000 tokens later."""
    dev = _device(device)
    T, d = (3000 if device == "cuda" else 300), 16
    k, q, v = torch.zeros(T, 1, d), torch.zeros(T, 1, d), torch.zeros(T, 1, 8)
    k[0, 0, 3], q[-1, 0, 3], v[0] = 1.0, 1.0, torch.arange(1.0, 9.0)
    g = torch.full((T, 1, d), 0.9999)
    extra = torch.zeros(1, d) if kind == "wkv" else torch.ones(T, 1)
    o = _scan(kind, (q, k, v, g, extra), slice(0, T), meta_of([T], dev), None, dev)
    close(o[-1, 0], torch.arange(1.0, 9.0).double() * 0.9999 ** (T - 2 if kind == "wkv" else T - 1), 1e-4)
    assert bool((o[:-1] == 0).all())


@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("H,G,d,dv,taps", [(4, 2, 32, 48, 4), (3, 1, 10, 14, 2), (2, 2, 128, 64, 1), (2, 1, 24, 130, 17)])
def test_delta_inputs(device, dtype, H, G, d, dv, taps):
    """Short convolution, unit heads, decays and step sizes, over cuts that fall inside the convolution's reach."""
    dev = _device(device)
    T, C = 40, 2 * G * d + H * dv
    x, w = rand(T, C, seed=1).to(dtype), rand(C, taps, seed=2)
    a, A_log, dt, b = rand(T, H * d, seed=3, scale=3.0), rand(H, seed=4) - 2, rand(H * d, seed=5), rand(T, H + 3, seed=6)
    y = plain.silu(plain.short_conv(x.double(), w.double()))
    want = (plain.unit(y[:, :G * d].view(T, G, d)) * d ** -0.5, plain.unit(y[:, G * d:2 * G * d].view(T, G, d)),
            y[:, 2 * G * d:].view(T, H, dv),
            torch.exp(-torch.exp(A_log.double())[:, None] * plain.softplus(a.double() + dt.double()).view(T, H, d)),
            plain.sigmoid(b.double()[:, :H]))
    convs = [torch.nn.Parameter(p.to(dev)) for p in w.split([G * d, G * d, H * dv])]
    for cuts in CUTS:
        tail = torch.full((3, C, taps - 1), 4.0, dtype=dtype, device=dev)
        at, got = 0, []
        for c in cuts:
            p = slice(at, at + c)
            got.append(iops.delta_inputs(x[p].to(dev), convs, a[p].to(dev), A_log.to(dev), dt.to(dev), b.to(dev)[p, :H], H, G,
                                         d, dv, meta_of([c], dev, [1], [at]), tail))
            at += c
        for g, e in zip(zip(*got), want):
            close(torch.cat(list(g)), e, 3e-6)
        if taps > 1:
            assert torch.equal(tail[1].cpu(), x[T - taps + 1:].t())


@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("H,dv", [(3, 20), (1, 64), (4, 129)])
def test_head_norm_and_gate(device, dtype, H, dv):
    dev = _device(device)
    o, gate = rand(7, H, dv, seed=1, scale=0.02), rand(7, H * dv, seed=2).to(dtype)
    for w, act, fn in ((rand(H * dv, seed=3), "silu", plain.silu), (rand(dv, seed=4), "sigmoid", plain.sigmoid)):
        want = plain.over_rms(o.double(), 1e-4) * (w.double().view(-1, dv))
        want = want.reshape(7, -1) * fn(gate.double())
        close(iops.head_norm_gate(o.to(dev), w.to(dev), gate.to(dev), act, 1e-4, dtype), want, 2e-6 if dtype == F32 else 8e-3)


# ---- mixture of experts ------------------------------------------------------------------------------
@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("T,E,top,W,F", [(1, 8, 2, 64, 48), (5, 3, 3, 30, 21), (300, 6, 2, 128, 72), (200, 40, 1, 64, 264),
                                         (130, 1, 1, 64, 136)])
def test_mixture_of_experts(device, dtype, T, E, top, W, F):
    """Few tokens (row kernels) and many (grouped GEMM), experts with no token and with more than a tile of them."""
    dev = _device(device)
    h, z = rand(T, W, seed=1).to(dtype), rand(T, E, seed=2, scale=2.0)
    if E == 6:
        z[:, 4] = -9.0                                     # nobody's expert
        z[:200, 1] = 9.0                                   # more than one tile
    up, down = rand(E, F, W, seed=3, scale=W ** -0.5).to(dtype), rand(E, W, F, seed=4, scale=F ** -0.5).to(dtype)
    s = plain.sigmoid(z.double())
    want = rand(T, W, seed=5).double()
    acc = want.float().to(dev)
    for t in range(T):
        for e in z[t].topk(top).indices.tolist():
            want[t] += torch.clamp(up[e].double() @ (s[t, e] * h[t].double()), min=0) ** 2 @ down[e].double().t()
    iops.moe_relu2_add_(acc, h.to(dev), z.to(dev), top, up.to(dev), down.to(dev))
    close(acc, want, 3e-6 if dtype == F32 else 2e-2)
