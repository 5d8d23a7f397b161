"""Rules that the kernel sources keep: what a kernel that starts while the one before ends may touch, and when; what is built
without approximate math."""
import glob
import os
import re

import pytest
import torch

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "easyllm_b200", "ops", "csrc")


def _kernels():
    """(file, kernel, names of its __restrict__ pointers, arguments of its wait or None) of all kernels."""
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for part in text.split("__global__")[1:]:
            head = re.search(r"(\w+)\s*\(((?:[^(){}]|\([^()]*\))*)\)\s*\{", part)
            if head is None:
                continue
            wait = re.search(r"chain_(?:enter|wait)\(([^)]*)\);", part[head.end():])
            out.append((os.path.basename(path), head.group(1), re.findall(r"\*\s*__restrict__\s+(\w+)", head.group(2)),
                        None if wait is None else re.findall(r"\w+", wait.group(1))))
    return out


def test_every_restricted_pointer_goes_through_the_wait():
    """A pointer that the wait does not get may be read, or written, before it: the compiler is free to take it that the wait
    leaves alone what only that pointer reaches."""
    waits = [k for k in _kernels() if k[3] is not None]
    assert len(waits) > 25
    for path, kernel, pointers, passed in waits:
        assert set(pointers) <= set(passed), (path, kernel, set(pointers) - set(passed))


def test_the_next_kernel_comes_in_after_the_allocation():
    """In a kernel that holds TMEM all threads meet between the allocation, which one warp makes and may wait for, and the call that
    lets the next kernel's CTAs in: they could take the TMEM that this kernel's CTA is still waiting for."""
    seen = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for part in text.split("__global__")[1:]:
            part = part.split("\n}\n")[0]
            alloc, let_in = re.search(r"tmem_alloc\w*(<[^>]*>)?\(", part), re.search(r"chain_(next|enter)\(", part)
            if alloc is not None and let_in is not None:
                seen += 1
                assert alloc.start() < let_in.start() and "__syncthreads();" in part[alloc.end():let_in.start()], (os.path.basename(path), part[:120])
    assert seen >= 3


def test_fast_math_sources_do_not_use_the_accurate_activations():
    """vec.cuh's activations are as accurate as the expf that the compiler's flags give them."""
    from easyllm_b200.ops import build
    for path in build.sources():
        base = os.path.splitext(os.path.basename(path))[0]
        if base not in build.ACCURATE_SOURCES:
            text = open(path).read()
            assert not any(f + "(" in text for f in ("silu_f", "sigmoid_f", "gelu_tanh_f")), base


def test_accurate_sources_use_no_approximate_exponential():
    from easyllm_b200.ops import build
    for base in build.ACCURATE_SOURCES:
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, base + ".cu")).read())
        assert not re.search(r"ex2_approx|ex2\.approx|__expf|__exp10f|exp2_poly|tanh\.approx", text), base


def test_attention_kernels_of_a_model_report_codes_of_their_own():
    """One word takes the code of the wait that ran out: within a model's attention kernels a code says which."""
    codes = {}
    for name in ("flash_attn", "flash_attn_bwd", "attn_rows"):
        for code in re.findall(r"k(?:Fa|Fb|Al|Af)Err\w* = (\d+)", open(os.path.join(CSRC, name + ".cu")).read()):
            assert codes.setdefault(code, name) == name and code not in ("1", "2", "3", "4", "5", "6", "15", "16", "31", "32", "41")
    assert len(codes) == 10


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 37, 300])
def test_operands_updated_in_place_keep_their_order(rows):
    """Dependent launches that read and write the same operands (rotation, rotation with append, dynamic tanh with its sum, decays,
    latent rows, sums of experts), each of which starts while the one before ends: the bits of the same launches with the GPU waited
    for after each."""
    import easyllm_b200.ops.cuda as cu
    import easyllm_b200.ops.cuda_infer as ci
    from easyllm_b200.ops import reference as ref
    torch.manual_seed(rows)
    dev, W, H, D, rank, rot, E, F = "cuda", 1024, 4, 64, 96, 32, 4, 64
    bf = dict(device=dev, dtype=torch.bfloat16)
    cos, sin = ref.rope_tables(D, 512, device=dev)
    lcos, lsin = (t.contiguous() for t in ref.rope_tables(rot, 512, device=dev))
    pos = torch.randint(0, 512, (rows,), device=dev, dtype=torch.int32)
    base, length = torch.arange(rows, device=dev, dtype=torch.int32) * 2, torch.ones(rows, device=dev, dtype=torch.int32)
    meta = {"position_ids": pos, "kv_base": base, "kv_len": length}
    qkv0, z0 = torch.randn(rows, 3 * H * D, **bf), torch.randn(rows, H * (D + rot) + rank + rot, **bf)
    x0, dec0 = torch.randn(rows, W, device=dev), torch.randn(rows, W, device=dev)
    ones, alpha, w0 = torch.ones(W, device=dev), torch.ones(1, device=dev), torch.zeros(W, device=dev)
    norm = torch.ones(rank, device=dev)
    up, down = torch.randn(E, F, W, **bf) * W ** -0.5, torch.randn(E, W, F, **bf) * F ** -0.5
    idx = torch.randint(0, E, (rows, 2), device=dev, dtype=torch.int32)
    wgt = torch.rand(rows, 2, device=dev)

    def chain(wait):
        qkv, z, x, dec = qkv0.clone(), z0.clone(), x0.clone(), dec0.clone()
        kc, vc, lat = torch.zeros(2 * rows, H, D, **bf), torch.zeros(2 * rows, H, D, **bf), torch.zeros(2 * rows, rank + rot, **bf)
        wait()
        for i in range(20):
            cu.rope_(qkv, cos, sin, pos, 2 * H, D, backward=bool(i & 1))
            wait()
            cu.rope_append_(qkv, cos, sin, pos, H, H, D, kc, vc, base, length)
            wait()
            ci.latent_inputs(z, H, D, rot, rank, norm, 1e-5, lcos, lsin, meta, lat)
            wait()
            y = ci.dynamic_tanh(x, alpha, ones, w0, torch.bfloat16, qkv[:, :W // 2].repeat(1, 2) if i == 0 else y)
            wait()
            ci._moe_add_(x, y, idx, wgt, up, down)
            wait()
            ci.wkv_decay_(dec, w0)
            wait()
            y = ci.dynamic_tanh(x, alpha, ones, dec[0].contiguous(), torch.bfloat16)
            wait()
        return qkv, z, x, dec, kc, vc, lat, y

    want = chain(torch.cuda.synchronize)
    for _ in range(3):
        got = chain(lambda: None)
        torch.cuda.synchronize()
        cu.check_err_flag()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
