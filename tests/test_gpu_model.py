"""Flagship model on the GPU: kernel path vs the PyTorch (library) path on the same weights,
and the smoke entry point."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("no GPU")


def _run(backend, gemm, sd=None):
    from easyllm_b200 import ops
    from easyllm_b200.models import llama_custom
    ops.set_backend(backend)
    ops.set_gemm_backend(gemm)
    torch.manual_seed(0)
    m = llama_custom(num_layers=2, hidden_size=512, num_attention_heads=4, num_kv_attention_heads=2,
                     intermediate_size=1408, vocab_size=32000, bf16=True, seq_length=256,
                     checkpoint_activations=False)
    if sd is not None:
        m.load_state_dict(sd)
    g = torch.Generator().manual_seed(0)
    tok = torch.randint(0, 32000, (2, 256), generator=g).cuda()
    lab = torch.roll(tok, -1, 1)
    loss = m((tok, None, None), (lab, torch.ones_like(lab)))
    loss.backward()
    grads = {n: p.grad.float().clone() for n, p in m.named_parameters()}
    return loss.item(), grads, m.state_dict()


def test_kernel_path_matches_library_path():
    _need_gpu()
    from easyllm_b200 import ops
    try:
        l_ref, g_ref, sd = _run("torch", "cublas")
        l_k, g_k, _ = _run("b200", "tcgen05", sd)
    finally:
        ops.set_backend("b200"); ops.set_gemm_backend("tcgen05")
    assert abs(l_ref - l_k) < 3e-2, (l_ref, l_k)
    for n in g_ref:
        a, b = g_ref[n], g_k[n]
        denom = a.abs().max().item() + 1e-6
        assert (a - b).abs().max().item() / denom < 8e-2, n
    import easyllm_b200.ops.cuda as cu
    cu.check_err_flag()


def test_smoke_entry():
    _need_gpu()
    import __graft_entry__ as ge
    ge.smoke()


def test_hf_style_model_kernel_path_matches_library_path():
    """The generic HF-style decoder (llama / qwen-bias / GQA variants) through the sm_100a kernels vs the PyTorch path."""
    _need_gpu()
    from easyllm_b200 import ops
    from easyllm_b200.models.hf_models import CausalLM, HFArch
    import easyllm_b200.ops.cuda as cu
    for fam, extra in (("llama", {"num_key_value_heads": 2}), ("qwen", {})):
        torch.manual_seed(0)
        a = HFArch(family=fam, vocab_size=2048, hidden_size=512, intermediate_size=1408, num_hidden_layers=2,
                   num_attention_heads=4, qkv_bias=fam == "qwen", **extra)
        m = CausalLM(a, dtype=torch.bfloat16).cuda().train()
        ids = torch.randint(0, 2048, (2, 256), device="cuda")
        res = {}
        try:
            for backend, gemm in (("torch", "cublas"), ("b200", "tcgen05")):
                ops.set_backend(backend); ops.set_gemm_backend(gemm)
                m.zero_grad(set_to_none=True)
                out = m(input_ids=ids, labels=ids)
                out["loss"].backward()
                res[backend] = (float(out["loss"]), {n: p.grad.float().clone() for n, p in m.named_parameters()})
        finally:
            ops.set_backend("b200"); ops.set_gemm_backend("tcgen05")
        torch.cuda.synchronize()
        cu.check_err_flag()
        assert abs(res["torch"][0] - res["b200"][0]) < 3e-2, (fam, res["torch"][0], res["b200"][0])
        for n, g_ref in res["torch"][1].items():
            g_k = res["b200"][1][n]
            assert (g_ref - g_k).abs().max().item() / (g_ref.abs().max().item() + 1e-6) < 8e-2, (fam, n)
        # once the optimizer has moved the parameters into its flat buffer, q/k/v (and gate/up) are adjacent:
        # the fused projection aliases them and the wgrad GEMM accumulates into the adjacent fp32 main_grad views
        from easyllm_b200.optim import ZeroOptimizer
        opt = ZeroOptimizer(m.named_parameters(), lr=1e-4, stage=0)
        att = m.model.layers[0].self_attn if hasattr(m, "model") else None
        if att is not None:
            assert ops._adjacent_alias([att.q_proj.weight.detach(), att.k_proj.weight.detach(),
                                        att.v_proj.weight.detach()]) is not None
            assert ops._adjacent_alias([att.q_proj.weight.main_grad, att.k_proj.weight.main_grad,
                                        att.v_proj.weight.main_grad]) is not None
        opt.zero_grad()
        m(input_ids=ids, labels=ids)["loss"].backward()
        opt.accumulate_grads()
        torch.cuda.synchronize()
        cu.check_err_flag()
        for n, p in m.named_parameters():
            g_ref = res["torch"][1][n]
            assert (g_ref - p.main_grad.float()).abs().max().item() / (g_ref.abs().max().item() + 1e-6) < 8e-2, (fam, n)


def test_train_batch_refuses_a_step_after_a_kernel_gave_up_a_wait():
    """A fused kernel whose bounded wait expired writes the error word and leaves a partial result: the engine
    must raise before the optimizer update instead of training on it.  The word is set by hand here (no wait runs
    out, no kernel misbehaves)."""
    _need_gpu()
    from easyllm_b200.engine import PipelineEngine
    from easyllm_b200.models import llama_custom
    from easyllm_b200.optim import ZeroOptimizer
    from easyllm_b200.data.synthetic import synthetic_batches
    import easyllm_b200.ops.cuda as cu
    torch.manual_seed(0)
    m = llama_custom(num_layers=1, hidden_size=256, num_attention_heads=2, num_kv_attention_heads=2,
                     intermediate_size=512, vocab_size=1024, bf16=True, seq_length=128, checkpoint_activations=False)
    opt = ZeroOptimizer(m.named_parameters(), lr=1e-3, stage=1)
    eng = PipelineEngine(m, opt, None, {"train_micro_batch_size_per_gpu": 1, "gradient_accumulation_steps": 2,
                                        "bf16": {"enabled": True}})
    it = synthetic_batches(1024, 128, 1, seed=0)
    eng.train_batch(it)                                   # a clean step passes
    before = [p.detach().clone() for p in m.parameters()]
    cu.err_flag().fill_(5)                                # what a timed-out peer-flag wait would have written
    with pytest.raises(cu.KernelError):
        eng.train_batch(it)
    for p, q in zip(m.parameters(), before):              # the update was not applied
        assert torch.equal(p.detach(), q)
    opt.zero_grad()
    eng.train_batch(it)                                   # the word was cleared by the read: training goes on
    cu.check_err_flag()


def test_synchronizing_reads_do_not_grow_with_the_number_of_micro_batches():
    """A step may synchronise a few times (the gradient norm, the returned loss), but nothing per micro-batch: the
    batch is parsed on the host and the kernels range-check token ids themselves.  PyTorch's sync debug mode warns on
    every synchronising call; the count inside ``train_batch`` must be the same for 2 and for 6 micro-batches."""
    _need_gpu()
    import warnings
    from easyllm_b200.engine import PipelineEngine
    from easyllm_b200.models import llama_custom
    from easyllm_b200.optim import ZeroOptimizer
    from easyllm_b200.data.synthetic import synthetic_batches
    counts = []
    for accum in (2, 6):
        torch.manual_seed(0)
        m = llama_custom(num_layers=1, hidden_size=256, num_attention_heads=2, num_kv_attention_heads=2,
                         intermediate_size=512, vocab_size=1024, bf16=True, seq_length=128,
                         checkpoint_activations=False)
        opt = ZeroOptimizer(m.named_parameters(), lr=1e-3, stage=1, grad_clip=1.0)
        eng = PipelineEngine(m, opt, None, {"train_micro_batch_size_per_gpu": 1,
                                            "gradient_accumulation_steps": accum, "bf16": {"enabled": True}})
        it = synthetic_batches(1024, 128, 1, seed=0)
        eng.train_batch(it)                               # set-up work of the first step may synchronise
        torch.cuda.synchronize()
        torch.cuda.set_sync_debug_mode("warn")
        try:
            with warnings.catch_warnings(record=True) as seen:
                warnings.simplefilter("always")
                eng.train_batch(it)
        finally:
            torch.cuda.set_sync_debug_mode("default")
        counts.append(sum("synchroniz" in str(w.message).lower() for w in seen))
    assert counts[0] == counts[1], counts


@pytest.mark.parametrize("tokens", [5, 40, 256, 512])
@pytest.mark.parametrize("width,ff,kv", [(256, 704, 2), (1024, 2816, 8)])
def test_an_evaluation_gives_the_bits_of_the_recorded_pass(tokens, width, ff, kv):
    """One batch with gradients and without, before the model has served and after (which puts gate and up weights next to each
    other): the same logits and the same loss, bit for bit, at row counts of all the kernels that serving chooses between.  A step
    that serves the same tokens is near them."""
    from easyllm_b200.models.hf_models import CausalLM, arch_from_hf_config
    torch.manual_seed(tokens)
    cfg = {"model_type": "llama", "vocab_size": 512, "hidden_size": width, "intermediate_size": ff, "num_hidden_layers": 2,
           "num_attention_heads": width // 128, "num_key_value_heads": min(kv, width // 128), "rms_norm_eps": 1e-6,
           "max_position_embeddings": 1024}
    with torch.device("cuda"):
        model = CausalLM(arch_from_hf_config(cfg), dtype=torch.bfloat16)
    ids = torch.randint(0, 512, (1, tokens), device="cuda")
    for served in (False, True):
        if served:
            state = model.new_state(1, tokens)
            h, _ = model.step(state, [state.open()], [ids[0]])
            step = model.logits(h)
        recorded = model(ids)["logits"]
        assert recorded.requires_grad
        loss = model(ids, labels=ids)["loss"]
        with torch.no_grad():
            assert torch.equal(model(ids)["logits"], recorded) and torch.equal(model(ids, labels=ids)["loss"], loss)
    want = recorded.detach().float()[0]
    assert (step - want).norm() <= 2e-2 * want.norm()


def test_what_the_recorded_functions_refuse_is_refused_without_gradients():
    """vmap and forward-mode differentiation of an op, with gradients recorded and without: the functions refuse both, and so do the
    launches that skip them."""
    from easyllm_b200 import ops
    x = torch.randn(3, 16, 64, device="cuda", dtype=torch.bfloat16)
    w, nw = torch.randn(64, 64, device="cuda", dtype=torch.bfloat16), torch.ones(64, device="cuda", dtype=torch.bfloat16)
    for f in (lambda a: ops.linear(a, w), lambda a: ops.rmsnorm(a, nw), lambda a: ops.glu(a), lambda a: ops.linear_parts(a, (w, w))):
        for grad in (True, False):
            with torch.set_grad_enabled(grad):
                f(x[0])
                with pytest.raises(RuntimeError):
                    torch.func.vmap(f)(x)
                with pytest.raises(RuntimeError), torch.autograd.forward_ad.dual_level():
                    f(torch.autograd.forward_ad.make_dual(x[0], torch.ones_like(x[0])))


def _llama(width, heads, kv, ff, layers=2, **more):
    from easyllm_b200.models.hf_models import CausalLM, arch_from_hf_config
    cfg = {"model_type": "llama", "vocab_size": 512, "hidden_size": width, "intermediate_size": ff, "num_hidden_layers": layers,
           "num_attention_heads": heads, "num_key_value_heads": kv, **more}
    torch.manual_seed(0)
    with torch.device("cuda"):
        return CausalLM(arch_from_hf_config(cfg), dtype=torch.bfloat16).eval()


def _steps(model, monkeypatch, counts, natively, capacity=512):
    """Prompts that start, prompts that go on and one token each: everything that comes out or is kept, launches, and how many of the
    steps one call issued."""
    import easyllm_b200.ops.cuda as cu
    from easyllm_b200.ops import infer
    taken = []
    step = infer.decoder_step
    with monkeypatch.context() as m:
        m.setattr(infer, "decoder_step", lambda *a: taken.append(1) or step(*a))
        if not natively:
            m.setattr(infer, "decoder_step_ok", lambda *a: False)
        gen = torch.Generator().manual_seed(3)
        state = model.new_state(len(counts), capacity)
        slots = [state.open() for _ in counts]
        before, out = cu.LAUNCHES, []
        for n in (counts, counts, [1] * len(counts)):
            h, meta = model.step(state, slots, [torch.randint(0, 512, (c,), generator=gen).cuda() for c in n])
            out.append(model.logits(h[meta["last_rows"].cuda()]))
            out.append(h)
    cu.check_err_flag()
    return out + [t for c in state.layers for t in (c.k, c.v)], cu.LAUNCHES - before, len(taken)


# rows on both sides of the lines between the products: matrix-vector, few rows, single CTAs, CTA pairs (and the gated one)
@pytest.mark.parametrize("counts", [[1], [3, 2], [16], [17], [77], [200, 57], [256], [1999, 1, 130]])
@pytest.mark.parametrize("width,heads,kv,ff", [(1024, 8, 2, 2816), (256, 4, 4, 704), (768, 16, 16, 1024)])
def test_layers_of_a_step_issued_by_one_call_give_the_bits_of_the_modules(width, heads, kv, ff, counts, monkeypatch):
    _need_gpu()
    model = _llama(width, heads, kv, ff)
    a, la, na = _steps(model, monkeypatch, counts, True)
    b, lb, nb = _steps(model, monkeypatch, counts, False)
    assert (na, nb) == (3, 0) and la == lb
    assert all(torch.equal(x, y) for x, y in zip(a, b))


def test_a_changed_module_of_a_step_is_called(monkeypatch):
    """Hooks, replaced or adapted modules, biases, tables without rotation: the modules' own forward runs, with the same result."""
    _need_gpu()
    from torch import nn
    want = _steps(_llama(256, 4, 2, 512), monkeypatch, [9, 4], True)[0]

    def hooked(m, calls):
        m.model.layers[1].mlp.up_proj.register_forward_hook(lambda *_: calls.append(1))
        return m.model.layers[1].mlp

    def replaced(m, calls):
        class Own(nn.Linear):
            def forward(self, x):
                return super().forward(x)
        lin = m.model.layers[0].self_attn.o_proj
        lin.__class__ = Own

    def patched(m, calls):
        norm = m.model.layers[0].input_layernorm
        forward = norm.forward
        norm.forward = lambda *a: calls.append(1) or forward(*a)

    def everywhere(m, calls):
        handle = nn.modules.module.register_module_forward_hook(lambda *_: calls.append(1))
        handles.append(handle)

    handles = []
    for change, called in ((hooked, False), (replaced, False), (patched, True), (everywhere, True)):
        model, calls = _llama(256, 4, 2, 512), []
        change(model, calls)
        try:
            got, _, taken = _steps(model, monkeypatch, [9, 4], True)
        finally:
            for h in handles:
                h.remove()
        assert taken == 0 and bool(calls) == called, change
        assert all(torch.equal(x, y) for x, y in zip(got, want)), change
    for more in ({"attention_bias": True}, {"model_type": "baichuan2-13b"}):
        assert _steps(_llama(256, 4, 4, 512, **more), monkeypatch, [9, 4], True)[2] == 0
    with torch.no_grad():                            # weights apart: they are copied together for the call, as before
        model = _llama(256, 4, 2, 512)
        model.fuse_weights = lambda: None
        assert _steps(model, monkeypatch, [9, 4], True)[2] == 0


def _fewer_query_heads(m):
    from easyllm_b200.models.hf_models.modeling import Attention
    m.model.layers[1].self_attn = _like(m, Attention(m.arch, torch.bfloat16, {"heads": 2, "kv_heads": 2, "dim": 64, "vdim": 64}))


def _fewer_key_heads(m):
    from easyllm_b200.models.hf_models.modeling import Attention
    m.model.layers[0].self_attn = _like(m, Attention(m.arch, torch.bfloat16, {"heads": 4, "kv_heads": 1, "dim": 64, "vdim": 64}))


def _own_scale(m):
    from easyllm_b200.models.hf_models.modeling import Attention
    m.model.layers[1].self_attn = _like(m, Attention(m.arch, torch.bfloat16, {"heads": 4, "kv_heads": 2, "dim": 64, "vdim": 64, "scale": 0.5}))


def _sink(m):
    from easyllm_b200.models.hf_models.modeling import Attention
    m.model.layers[0].self_attn = _like(m, Attention(m.arch, torch.bfloat16, {"heads": 4, "kv_heads": 2, "dim": 64, "vdim": 64, "sink": True}))
    with torch.no_grad():
        m.model.layers[0].self_attn.sink.fill_(3.0)


def _scale_of_the_first(m):
    m.model.layers[0].self_attn.scale = 0.25


def _no_positions(m):
    m.model.layers[1].self_attn.slopes = torch.tensor([0.5, 0.25, 0.125, 0.0625])


def _narrower_feed_forward(m):
    import dataclasses
    from easyllm_b200.models.hf_models.modeling import MLP
    m.model.layers[1].mlp = _like(m, MLP(dataclasses.replace(m.arch, intermediate_size=256), torch.bfloat16))


def _like(m, part):
    part = part.to(m.lm_head.weight.device).eval()
    torch.manual_seed(5)
    part.apply(m._init)
    return part


_OTHER_LAYERS = [_fewer_query_heads, _fewer_key_heads, _own_scale, _sink, _scale_of_the_first, _no_positions, _narrower_feed_forward]


@pytest.mark.parametrize("change", _OTHER_LAYERS)
def test_a_layer_unlike_the_others_gives_the_result_of_its_modules(change, monkeypatch):
    _need_gpu()
    model = _llama(256, 4, 2, 512)
    change(model)
    got, _, taken = _steps(model, monkeypatch, [9, 4], True)
    want = _steps(model, monkeypatch, [9, 4], False)[0]
    assert taken == 0 and all(torch.equal(x, y) for x, y in zip(got, want))


@pytest.mark.parametrize("width,heads,ff", [(256, 4, 1004), (256, 4, 700), (132, 2, 704), (240, 10, 704)])
def test_sizes_that_the_kernels_do_not_take_are_served(width, heads, ff, monkeypatch):
    """Feed-forward widths, rows and heads that are no multiples of 8 or 16: no call for all layers, but an answer, near fp32's."""
    _need_gpu()
    model = _llama(width, heads, heads, ff)
    got, _, taken = _steps(model, monkeypatch, [9, 4], True)
    want = _steps(model.float(), monkeypatch, [9, 4], False)[0]
    assert taken == 0
    for x, y in zip(got[:6:2], want[:6:2]):          # logits: a dozen roundings to bf16 on the way, 2^-9 each
        assert (x.float() - y.float()).norm() <= 12 * 2.0 ** -9 * y.float().norm()


def test_a_refused_launch_on_pairs_is_repeated_without(monkeypatch):
    """The call comes back with the code of a refusal: the step is issued again on single CTAs, with a warning, and stays there."""
    _need_gpu()
    import easyllm_b200.ops.cuda as cu
    import easyllm_b200.ops.cuda_infer as ci
    model = _llama(512, 4, 2, 1024)
    cu.set_gemm_pair(False)
    try:
        want = _steps(model, monkeypatch, [256], True)[0]
        cu.set_gemm_pair(True)
        real = cu.lib()

        class Refusing:
            def __getattr__(self, name):
                return getattr(real, name)

            def ell_decoder_step(self, args, *rest):
                return ci._STEP_NO_PAIRS if args[len(args) - 3] else real.ell_decoder_step(args, *rest)

        monkeypatch.setattr(ci, "lib", lambda: Refusing())
        with pytest.warns(UserWarning, match="refused"):
            got = _steps(model, monkeypatch, [256], True)[0]
        assert not cu.gemm_pair_enabled()
        assert all(torch.equal(x, y) for x, y in zip(got, want))
    finally:
        cu.set_gemm_pair(True)


def test_a_refused_gated_launch_leaves_the_others_on_pairs(monkeypatch):
    """What the modules do: the plain product and the activation, and nothing is turned off."""
    _need_gpu()
    import easyllm_b200.ops.cuda as cu
    import easyllm_b200.ops.cuda_infer as ci
    model = _llama(512, 4, 2, 1024)
    with monkeypatch.context() as m:
        m.setattr(cu, "gemm_glu", lambda *a: None)
        want = _steps(model, monkeypatch, [256], False)[0]
    real = cu.lib()

    class Refusing:
        def __getattr__(self, name):
            return getattr(real, name)

        def ell_decoder_step(self, args, *rest):
            return ci._STEP_NOT_GATED if args[len(args) - 4] and args[len(args) - 3] else real.ell_decoder_step(args, *rest)

    monkeypatch.setattr(ci, "lib", lambda: Refusing())
    got = _steps(model, monkeypatch, [256], True)[0]
    assert cu.gemm_pair_enabled() and all(torch.equal(x, y) for x, y in zip(got, want))


def _train_layers(cfg, lens, natively, monkeypatch, change=None, freeze=(), drop=(), wrt=None, checkpointing=False):
    """One micro-batch through a model with an optimizer's fp32 gradient buffer: loss, gradients, launches and layers issued by one call."""
    import easyllm_b200.ops.cuda as cu
    from easyllm_b200.models.hf_models import CausalLM, arch_from_hf_config
    from easyllm_b200.ops import decoder
    from easyllm_b200.optim.zero import ZeroOptimizer
    torch.manual_seed(1)
    with torch.device("cuda"):
        model = CausalLM(arch_from_hf_config(cfg), dtype=torch.bfloat16).train()
    for name, p in model.named_parameters():
        p.requires_grad_(not any(f in name for f in freeze))
    opt = ZeroOptimizer([(n, p) for n, p in model.named_parameters() if p.requires_grad], lr=1e-4, stage=0)
    if change is not None:
        change(model)
    if checkpointing:
        model.gradient_checkpointing_enable()
    taken = []
    layer = decoder.train_layer
    with monkeypatch.context() as m:
        m.setattr(decoder, "train_layer", lambda *a: taken.append(1) or layer(*a))
        if not natively:
            m.setattr(decoder, "rows_ok", lambda x: False)
        gen, T, cu_seqlens = torch.Generator().manual_seed(2), sum(lens), torch.tensor([0] + lens).cumsum(0).int()
        opt.zero_grad()
        before = cu.LAUNCHES
        loss = model(input_ids=torch.randint(0, 512, (1, T), generator=gen), labels=torch.randint(0, 512, (1, T), generator=gen),
                     position_ids=torch.cat([torch.arange(n) for n in lens]).unsqueeze(0), cu_seqlens=cu_seqlens)["loss"]
        for p in drop:
            dict(model.named_parameters())[p].main_grad = None
        if wrt is not None:
            params = dict(model.named_parameters())
            torch.autograd.grad(loss, [params[n] for n in wrt], allow_unused=True)
        else:
            loss.backward()
            if not drop:                       # the optimizer adds gradients to the main_grad that it made
                opt.accumulate_grads()
    cu.check_err_flag()
    grads = {n: (p.grad.float() if p.grad is not None else p.main_grad if getattr(p, "main_grad", None) is not None else None)
             for n, p in model.named_parameters()}
    return loss.detach(), grads, cu.LAUNCHES - before, len(taken)


_TRAIN = {"model_type": "llama", "vocab_size": 512, "hidden_size": 512, "intermediate_size": 704, "num_hidden_layers": 3,
          "num_attention_heads": 4, "num_key_value_heads": 2}


def _same_gradients(a, b):
    """Equal bits where the layers' own kernels made them; what lies in front of the first layer gets one rounding to bf16 less."""
    for n in a:
        assert (a[n] is None) == (b[n] is None), n
        if a[n] is None:
            continue
        if "embed" in n:
            assert (a[n] - b[n]).norm() <= 2.0 ** -8 * b[n].norm()
        else:
            assert torch.equal(a[n], b[n]), n


@pytest.mark.parametrize("lens", [[1], [16], [5, 36], [200], [256], [257, 64], [2048, 3]])
@pytest.mark.parametrize("more", [{}, {"num_key_value_heads": 4, "intermediate_size": 1000}, {"model_type": "baichuan2-13b"}])
def test_layers_of_a_training_step_issued_by_one_call_give_the_bits_of_the_functions(lens, more, monkeypatch):
    _need_gpu()
    cfg = {**_TRAIN, **more}
    la, ga, na, ta = _train_layers(cfg, lens, True, monkeypatch)
    lb, gb, nb, tb = _train_layers(cfg, lens, False, monkeypatch)
    assert (ta, tb) == (3, 0) and na == nb
    assert torch.equal(la, lb)
    _same_gradients(ga, gb)


@pytest.mark.parametrize("kw,native", [
    ({"checkpointing": True}, 6),                                           # recomputed in the backward pass
    ({"freeze": ("layers.1.self_attn.q_proj",)}, 2),                        # a weight without a gradient: the layer's functions
    ({"freeze": ("embed_tokens",)}, 2),                                     # nothing in front of the first layer records
    ({"drop": ("model.layers.1.mlp.up_proj.weight", "model.layers.2.input_layernorm.weight")}, 3),   # gone between the passes
    ({"wrt": ("model.embed_tokens.weight",)}, 3),                           # no weight of a layer is asked for: no products for them
    ({"wrt": ("model.layers.1.mlp.down_proj.weight",)}, 3),
])
def test_layers_of_a_training_step_beside_the_usual_one(kw, native, monkeypatch):
    _need_gpu()
    la, ga, _, ta = _train_layers(_TRAIN, [40, 9], True, monkeypatch, **kw)
    lb, gb, _, tb = _train_layers(_TRAIN, [40, 9], False, monkeypatch, **kw)
    assert (ta, tb) == (native, 0)
    assert torch.equal(la, lb)
    if "drop" in kw:                                                        # bf16 gradients of autograd beside the fp32 ones
        for n in kw["drop"]:
            assert torch.equal(ga[n], gb[n]), n
    _same_gradients(ga, gb)


@pytest.mark.parametrize("cls,name", [("Attention", "forward"), ("Attention", "_attend"), ("MLP", "forward"), ("RMSNorm", "forward"),
                                      ("DecoderLayer", "__call__")])
def test_a_method_put_in_the_place_of_a_classes_own_is_called(cls, name, monkeypatch):
    _need_gpu()
    from easyllm_b200.models.hf_models import modeling
    want = _steps(_llama(256, 4, 2, 512), monkeypatch, [9, 4], False)[0]
    loss = _train_layers(_TRAIN, [33], False, monkeypatch)[0]
    own, calls = getattr(getattr(modeling, cls), name), []
    monkeypatch.setattr(getattr(modeling, cls), name, lambda *a, **k: calls.append(1) or own(*a, **k))
    got, _, taken = _steps(_llama(256, 4, 2, 512), monkeypatch, [9, 4], True)
    assert taken == 0 and calls and all(torch.equal(x, y) for x, y in zip(got, want))
    calls.clear()
    got, _, _, taken = _train_layers(_TRAIN, [33], True, monkeypatch)
    assert taken == 0 and torch.equal(got, loss)
    assert calls or name == "_attend"                # of cached rows only


@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("make", [lambda g: g.bfloat16(), lambda g: g.clone().t().contiguous().t()])
def test_a_gradient_buffer_that_a_product_is_not_added_to_is_refused(make, native, monkeypatch):
    _need_gpu()

    def other(m):
        w = m.model.layers[1].mlp.down_proj.weight
        w.main_grad = make(w.main_grad)

    with pytest.raises(ValueError):
        _train_layers(_TRAIN, [33], native, monkeypatch, change=other)


def test_a_changed_module_of_a_training_step_is_called(monkeypatch):
    _need_gpu()
    calls = []

    def hooked(m):
        m.model.layers[1].self_attn.o_proj.register_forward_hook(lambda *_: None)

    def patched(m):
        norm, forward = m.model.layers[0].post_attention_layernorm, m.model.layers[0].post_attention_layernorm.forward
        norm.forward = lambda *a: calls.append(1) or forward(*a)

    want = _train_layers(_TRAIN, [33], False, monkeypatch)
    for change in (hooked, patched):
        loss, grads, _, taken = _train_layers(_TRAIN, [33], True, monkeypatch, change=change)
        assert taken == 2 and torch.equal(loss, want[0])
        _same_gradients(grads, want[1])
    assert calls
    saved = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: saved.append(t.shape) or t.cpu(), lambda t: t.cuda()):
        loss, grads, _, taken = _train_layers(_TRAIN, [33], True, monkeypatch)
    assert taken == 3 and saved
    _same_gradients(grads, want[1])
