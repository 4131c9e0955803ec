"""Parity of the memory-bound sm_100a kernels (through the C ABI) with the CPU oracle and with the
golden outputs of the reference's own kernels. NF4 and the dropout bits are compared bit for bit;
the floating-point ops use the reference's own tolerances (tests_local/ of the reference)."""

from types import SimpleNamespace

import pytest
import torch

from conftest import assert_close_rel_max, load_golden, rel_norm

pytestmark = pytest.mark.gpu

F16, F32, BF16 = torch.float16, torch.float32, torch.bfloat16
DEV = "cuda"


def _bits(t):
    return t.view(torch.int16) if t.element_size() == 2 else t.view(torch.int32)


# ----------------------------------------------------------------------------------- NF4
def _state_to_cuda(g):
    from oracle import nf4 as onf4

    nested = bool(g["nested"])
    inner = onf4.State(g["absmax2"], (g["absmax"].numel(),), g["code2"], g["blocksize2"],
                       F32) if nested else None
    return onf4.State(g["absmax"], tuple(g["shape"].tolist()), g["code"], g["blocksize"],
                      g["out"].dtype, offset=g["offset"] if nested else None, state2=inner)


@pytest.mark.parametrize("tag", ["a", "b", "c", "d"])
@pytest.mark.parametrize("dname", ["f16", "f32"])
def test_nf4_golden_bit_exact(tag, dname):
    from claudemaxing_b200.nf4 import dequantize_nf4

    g = load_golden(f"nf4_{tag}_{dname}")
    state = _state_to_cuda(g).to(DEV)
    out = dequantize_nf4(g["packed"].to(DEV), state)
    assert out.dtype == g["out"].dtype and out.shape == g["out"].shape
    assert torch.equal(_bits(out.cpu()), _bits(g["out"]))


@pytest.mark.parametrize("nested", [True, False])
@pytest.mark.parametrize("shape", [(1536, 1536), (256, 1536), (8960, 1536), (1536, 8960), (3, 64),
                                   (7, 34)])
def test_nf4_bit_exact_vs_oracle(shape, nested):
    # shapes of tests_local/test_nf4.py:27-29 plus one whose byte count is not a multiple of 16
    from claudemaxing_b200.nf4 import dequantize_nf4
    from oracle import nf4 as onf4

    gen = torch.Generator().manual_seed(shape[0] * 7 + nested)
    w = (torch.randn(*shape, generator=gen) * 0.05).half()
    w.view(-1)[:5] = torch.tensor([0.0, -0.0, 1e-7, 3.0, -2.5]).half()
    blocksize = 64 if shape != (7, 34) else 32
    packed, state = onf4.quantize_nf4(w, blocksize=blocksize, nested=nested)
    ref16 = onf4.dequantize_nf4(packed, state, F16)
    out16 = dequantize_nf4(packed.to(DEV), state.to(DEV))
    assert out16.dtype == F16 and out16.shape == ref16.shape
    assert torch.equal(_bits(out16.cpu()), _bits(ref16))
    out32 = dequantize_nf4(packed.to(DEV), state.to(DEV), F32)
    assert torch.equal(_bits(out32.cpu()), _bits(onf4.dequantize_nf4(packed, state, F32)))
    assert torch.equal(out32.half().cpu(), ref16)


@pytest.mark.parametrize("nested", [True, False])
@pytest.mark.parametrize("shape", [(1, 16), (33, 1000), (2, 4096 * 8 + 6)])
@pytest.mark.parametrize("shift", [0, 1])
def test_nf4_outputs_on_16_byte_boundaries_and_ragged_tails(shape, nested, shift):
    """An output that is 16- but not 32-byte aligned takes two stores per group; byte counts off a
    multiple of 8, and just over one CTA's share (8 KB), take the tail and the second CTA."""
    from claudemaxing_b200.nf4 import dequantize_nf4
    from oracle import nf4 as onf4

    gen = torch.Generator().manual_seed(shape[1])
    packed, state = onf4.quantize_nf4((torch.randn(*shape, generator=gen) * 0.05).half(), nested=nested)
    n = shape[0] * shape[1]
    for dtype in (F16, F32):
        step = 16 // torch.empty((), dtype=dtype).element_size() * shift
        buf = torch.full((n + step + 8,), 7.0, dtype=dtype, device=DEV)
        out = buf[step:step + n].view(shape)
        dequantize_nf4(packed.to(DEV), state.to(DEV), dtype, out=out)
        assert torch.equal(_bits(out.cpu()), _bits(onf4.dequantize_nf4(packed, state, dtype)))
        assert (buf[:step] == 7.0).all() and (buf[step + n:] == 7.0).all()


def test_nf4_quantiser_matches_oracle_and_roundtrip_is_idempotent():
    from claudemaxing_b200 import qlora
    from claudemaxing_b200.nf4 import dequantize_nf4
    from oracle import nf4 as onf4

    w = (torch.randn(512, 1536, generator=torch.Generator().manual_seed(3)) * 0.02).half()
    p_dev, s_dev = qlora.quantize_nf4(w.to(DEV))
    p_cpu, s_cpu = onf4.quantize_nf4(w)
    assert torch.equal(p_dev.cpu(), p_cpu)
    # the nested codes depend on mean(absmax), whose summation order differs between CPU and GPU
    assert abs(s_dev.offset.item() - s_cpu.offset.item()) < 1e-6
    assert (s_dev.absmax.cpu() != s_cpu.absmax).float().mean().item() < 0.01
    deq = dequantize_nf4(p_dev, s_dev)
    # quantising the dequantised weight again reproduces the same codes (a fixed point)
    p_again, _ = qlora.quantize_nf4(deq, nested=False)
    p_first, _ = qlora.quantize_nf4(w.to(DEV), nested=False)
    assert (p_again != p_first).float().mean().item() < 0.02


def test_nf4_batched_launch_is_bit_identical_to_single_launches():
    from claudemaxing_b200.nf4 import dequantize_nf4, dequantize_nf4_batch
    from oracle import nf4 as onf4

    shapes = [(1536, 1536), (256, 1536), (256, 1536), (1536, 1536), (8960, 1536), (8960, 1536),
              (1536, 8960), (3, 64), (7, 34)]  # one decoder layer + two odd ones: two launches
    weights = []
    for i, shape in enumerate(shapes):
        w = (torch.randn(*shape, generator=torch.Generator().manual_seed(i)) * 0.02).half()
        packed, state = onf4.quantize_nf4(w, blocksize=64)
        weights.append((packed.to(DEV), state.to(DEV)))
    batched = dequantize_nf4_batch(weights)
    for (packed, state), got in zip(weights, batched):
        assert torch.equal(_bits(got), _bits(dequantize_nf4(packed, state)))


def test_nf4_rejects_bad_arguments():
    from claudemaxing_b200 import _lib

    x = torch.zeros(64, dtype=torch.uint8, device=DEV)
    with pytest.raises(RuntimeError, match="blocksize"):
        _lib.call("soup_nf4_dequant", x.data_ptr(), x.data_ptr(), x.data_ptr(), None, None, None,
                  x.data_ptr(), 128, 48, 1, 0, _lib.F16, 0)


# ----------------------------------------------------------------------------------- RMSNorm
@pytest.mark.parametrize("tag", ["f16f32", "f16f16", "f32f32"])
def test_rmsnorm_golden(tag):
    from claudemaxing_b200.rmsnorm import rmsnorm

    g = load_golden(f"rmsnorm_{tag}")
    x = g["x"].to(DEV).requires_grad_(True)
    w = g["w"].to(DEV).requires_grad_(True)
    out = rmsnorm(x, w, 1e-6)
    out.backward(g["dy"].to(DEV))
    tol = 2e-3 if F16 in (g["x"].dtype, g["w"].dtype) else 1e-4
    assert out.dtype == g["out"].dtype
    assert_close_rel_max(out.detach().cpu(), g["out"], tol, "out")
    assert_close_rel_max(x.grad.cpu(), g["dx"], tol, "dx")
    assert_close_rel_max(w.grad.cpu(), g["dw"], 5e-3, "dw")


@pytest.mark.parametrize("shape", [(4, 512, 1536), (3, 77, 1001), (2, 1, 4096), (1, 3, 16384),
                                   (2, 33, 1288), (5, 7, 2048), (1, 19, 64), (3, 11, 3072)])
@pytest.mark.parametrize("dtypes", [(F16, F32), (F16, F16), (F32, F32), (BF16, BF16)])
@pytest.mark.parametrize("train_w", [False, True])
def test_rmsnorm_vs_oracle(shape, dtypes, train_w):
    from claudemaxing_b200.rmsnorm import rmsnorm
    from oracle import elementwise as ew

    xdt, wdt = dtypes
    gen = torch.Generator().manual_seed(1)
    x = (3 * torch.randn(*shape, generator=gen)).to(xdt)
    w = (1 + 0.5 * torch.randn(shape[-1], generator=gen)).to(wdt)
    dy = torch.randn(*shape, generator=gen).to(torch.promote_types(xdt, wdt))
    ref_out, ref_dx, ref_dw = ew.rmsnorm_fwd_bwd(x, w, dy, weight_grad=train_w)
    xd = x.to(DEV).requires_grad_(True)
    wd = w.to(DEV).requires_grad_(train_w)
    out = rmsnorm(xd, wd, 1e-6)
    out.backward(dy.to(DEV))
    tol = 1e-4 if dtypes == (F32, F32) else (2e-3 if BF16 not in dtypes else 1.6e-2)
    assert out.dtype == ref_out.dtype and xd.grad.dtype == xdt
    assert_close_rel_max(out.detach().cpu(), ref_out, tol, "out")
    assert_close_rel_max(xd.grad.cpu(), ref_dx, tol, "dx")
    if train_w:
        assert_close_rel_max(wd.grad.cpu(), ref_dw, 5 * tol, "dw")
    else:
        assert wd.grad is None


@pytest.mark.parametrize("cols", [256, 264, 512, 4088, 4096, 4104])
@pytest.mark.parametrize("rows", [1, 3, 4, 1783])   # 1783: three rows a step, a second step for some CTAs, a remainder
def test_rmsnorm_weight_gradient_at_the_edges_of_its_kernels(cols, rows):
    from claudemaxing_b200.rmsnorm import rmsnorm

    gen = torch.Generator().manual_seed(rows)
    x, dy = (torch.randn(rows, cols, generator=gen).half() for _ in range(2))
    w = (1 + 0.5 * torch.randn(cols, generator=gen)).half()
    norm = x.double() * (x.double().square().mean(-1, keepdim=True) + 1e-6).rsqrt()
    gn = dy.double() * w.double()
    want_dx = (gn - norm * (gn * norm).mean(-1, keepdim=True)) * (x.double().square().mean(-1, keepdim=True) + 1e-6).rsqrt()
    leaves = [t.to(DEV).requires_grad_() for t in (x, w)]
    rmsnorm(*leaves, 1e-6).backward(dy.to(DEV))
    # fp16: a rounding of dy * w and of the result each, half an ulp (4.9e-4) of their value
    assert_close_rel_max(leaves[0].grad.cpu(), want_dx.float(), 2e-3, "dx")
    assert_close_rel_max(leaves[1].grad.cpu(), (dy.double() * norm).sum(0).float(), 2e-3, "dw")
    again = [t.to(DEV).requires_grad_() for t in (x, w)]
    rmsnorm(*again, 1e-6).backward(dy.to(DEV))
    assert torch.equal(leaves[1].grad, again[1].grad)   # a fixed order of additions


@pytest.mark.parametrize("cols,last", [(264, 16384), (512, 16384), (520, 32768), (768, 32768)])
def test_rmsnorm_weight_gradient_of_many_narrow_fp32_rows(cols, last):
    """Up to `last` rows four CTAs an SM take a step of rows each, above them two CTAs of a row per warp, the faster
    way there: the partial sums tell which ran, and both agree with float64. Bounds: fp32 sums over a row and over
    all rows, against the largest value."""
    from claudemaxing_b200 import _lib

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for rows, ctas in ((last, 4 * sms), (last + 1, 2 * sms)):
        gen = torch.Generator(device=DEV).manual_seed(rows)
        x, dy = (torch.randn(rows, cols, generator=gen, device=DEV) for _ in range(2))
        w = 1 + 0.5 * torch.randn(cols, generator=gen, device=DEV)
        rstd = (x.square().mean(-1) + 1e-6).rsqrt()
        partials = _lib.lib().soup_rmsnorm_bwd_partials(rows, cols)
        part = torch.full((partials, cols), float("nan"), device=DEV)
        dx, dw = torch.empty_like(x), torch.empty_like(w)
        _lib.call("soup_rmsnorm_bwd", *map(_lib.ptr, (dy, x, w, rstd, dx, part, dw)), None, None, 0, rows, cols,
                  *[_lib.F32] * 4, 0, _lib.stream_of(x))
        assert part.isfinite().all(1).sum() == ctas
        norm, gn = x.double() * rstd.double()[:, None], dy.double() * w.double()
        want_dx = (gn - norm * (gn * norm).mean(-1, keepdim=True)) * rstd.double()[:, None]
        assert_close_rel_max(dx, want_dx.float(), 1e-5, "dx")
        assert_close_rel_max(dw, (dy.double() * norm).sum(0).float(), 1e-5, "dw")


def test_rmsnorm_fp16_copy_path_and_tiny_weights():
    # fp32 x, frozen fp32 w: forward leaves an fp16 copy for the next layers, backward uses it;
    # a 2e5 "massive activation" channel and tiny / zero weights (tests_local/test_rmsnorm.py:197-277)
    from claudemaxing_b200.rmsnorm import fp16_copy_of, rmsnorm
    from oracle import elementwise as ew

    gen = torch.Generator().manual_seed(2)
    x = torch.randn(2, 300, 1536, generator=gen)
    x[..., 7] = 2e5
    w = 1 + 0.5 * torch.randn(1536, generator=gen)
    w[3], w[50], w[900], w[1000] = 1e-5, -6.5e-6, 3e-4, 0.0
    dy = torch.randn(2, 300, 1536, generator=gen)
    x64, w64 = x.double().requires_grad_(True), w.double()
    ew.rmsnorm(x64, w64).backward(dy.double())
    xd = x.to(DEV).requires_grad_(True)
    wd = w.to(DEV)
    out = rmsnorm(xd, wd, 1e-6)
    low = fp16_copy_of(out)
    assert low is not None and low.dtype == F16 and torch.equal(low, out.detach().half())
    assert fp16_copy_of(out.detach().clone()) is None
    out.backward(dy.to(DEV))
    assert rel_norm(xd.grad.cpu(), x64.grad) < 1e-3
    out.detach().add_(1)  # a changed tensor (shared version counter) no longer has a copy
    assert fp16_copy_of(out) is None


# ----------------------------------------------------------------------------------- RoPE
@pytest.mark.parametrize("tag,tol", [("f16", 2e-3), ("f32", 1e-5)])
def test_rope_golden(tag, tol):
    from claudemaxing_b200.rope import rope

    g = load_golden(f"rope_{tag}")
    q = g["q"].to(DEV).requires_grad_(True)
    k = g["k"].to(DEV).requires_grad_(True)
    oq, ok = rope(q, k, g["cos"].to(DEV), g["sin"].to(DEV))
    torch.autograd.backward((oq, ok), (g["gq"].to(DEV), g["gk"].to(DEV)))
    for name, val in (("q_out", oq), ("k_out", ok), ("dq", q.grad), ("dk", k.grad)):
        assert_close_rel_max(val.detach().cpu(), g[name], tol, name)


@pytest.mark.parametrize("dims", [(4, 512, 12, 2, 128), (2, 37, 4, 4, 64), (1, 1, 2, 1, 128),
                                  (2, 5, 3, 1, 24)])
@pytest.mark.parametrize("dtype", [F32, F16])
@pytest.mark.parametrize("cos_batch_one", [False, True])
def test_rope_vs_oracle(dims, dtype, cos_batch_one):
    # shapes of tests_local/test_rope.py:28-31; q and k are transposed views, as in the model
    from claudemaxing_b200.rope import rope
    from oracle import elementwise as ew

    b, t, h, kv, d = dims
    gen = torch.Generator().manual_seed(0)
    q = torch.randn(b, t, h * d, generator=gen).to(dtype).view(b, t, h, d).transpose(1, 2)
    k = torch.randn(b, t, kv * d, generator=gen).to(dtype).view(b, t, kv, d).transpose(1, 2)
    cb = 1 if cos_batch_one else b
    pos = torch.arange(t, dtype=F32)[None].expand(cb, t)
    inv = 1.0 / (1e6 ** (torch.arange(0, d, 2, dtype=F32) / d))
    emb = torch.cat((pos[..., None] * inv,) * 2, -1)
    cos, sin = emb.cos().to(dtype), emb.sin().to(dtype)
    gq, gk = torch.randn(b, h, t, d, generator=gen).to(dtype), torch.randn(b, kv, t, d, generator=gen).to(dtype)
    ref = ew.rope_fwd_bwd(q, k, cos, sin, gq, gk)
    qd = q.to(DEV).requires_grad_(True)
    kd = k.to(DEV).requires_grad_(True)
    oq, ok = rope(qd, kd, cos.to(DEV), sin.to(DEV))
    assert oq.is_contiguous() and oq.shape == (b, h, t, d) and oq.dtype == dtype
    torch.autograd.backward((oq, ok), (gq.to(DEV), gk.to(DEV)))
    tol = 2e-3 if dtype == F16 else 1e-5
    for name, val, r in zip(("q", "k", "dq", "dk"), (oq, ok, qd.grad, kd.grad), ref):
        assert_close_rel_max(val.detach().cpu(), r, tol, name)


@pytest.mark.parametrize("heads", [(12, 2), (3, 2), (1, 1), (7, 0), (0, 5)])
@pytest.mark.parametrize("dtype", [F32, F16, BF16])
def test_rope_gradients_have_the_layout_of_their_inputs(heads, dtype):
    """Gradients of [b, h, t, d] outputs: heads that do and do not fill a thread's share, one of q and k
    alone; laid out as the projections q and k are views of, or as the contiguous tensors they are."""
    from claudemaxing_b200.rope import rope
    from oracle import elementwise as ew

    gen = torch.Generator().manual_seed(4)
    b, t, d = 2, 45, 128
    cos, sin = ew.rope_tables(torch.arange(t), d, dtype=dtype)
    rows = [torch.randn(b, t, max(h, 1) * d, generator=gen).to(dtype) for h in heads]
    grads = [torch.randn(b, max(h, 1), t, d, generator=gen).to(dtype) for h in heads]
    views = [x.view(b, t, -1, d).transpose(1, 2) for x in rows]
    want = ew.rope_fwd_bwd(*views, cos, sin, *grads)[2:]
    for contiguous in (False, True):
        leaves = [x.to(DEV).requires_grad_(h > 0) for x, h in zip(rows, heads)]
        inputs = [x.view(b, t, -1, d).transpose(1, 2) for x in leaves]
        if contiguous:
            inputs = [x.contiguous() for x in inputs]
        seen = [None, None]
        for i, x in enumerate(inputs):
            if x.requires_grad:
                x.register_hook(lambda g, i=i: seen.__setitem__(i, g.stride()))
        out = rope(*inputs, cos.to(DEV), sin.to(DEV))
        torch.autograd.backward(out, [g.to(DEV) for g in grads])
        for x, leaf, w, strides, h in zip(inputs, leaves, want, seen, heads):
            if h:
                assert strides == x.stride()
                assert_close_rel_max(leaf.grad.view(b, t, -1, d).transpose(1, 2).cpu(), w,
                                     {F32: 1e-5, F16: 2e-3, BF16: 1.6e-2}[dtype], "gradient")


def test_rope_packed_positions_restart_per_row():
    # benchmark config 3: one packed row of lengths {512,384,640,512}, positions restart at 0
    from claudemaxing_b200.rope import rope
    from oracle import elementwise as ew

    gen = torch.Generator().manual_seed(2)
    pos = torch.cat([torch.arange(n) for n in (512, 384, 640, 512)])
    cos, sin = ew.rope_tables(pos, 128, dtype=F16)
    q = torch.randn(1, 2048, 12 * 128, generator=gen).half().view(1, 2048, 12, 128).transpose(1, 2)
    k = torch.randn(1, 2048, 2 * 128, generator=gen).half().view(1, 2048, 2, 128).transpose(1, 2)
    rq, rk = ew.rope(q, k, cos, sin)
    oq, ok = rope(q.to(DEV), k.to(DEV), cos.to(DEV), sin.to(DEV))
    assert_close_rel_max(oq.cpu(), rq, 2e-3)
    assert_close_rel_max(ok.cpu(), rk, 2e-3)
    # rotation preserves the norm of every (x1, x2) pair up to rounding
    assert abs(oq.float().norm().item() / q.float().norm().item() - 1) < 1e-3


@pytest.mark.parametrize("dims", [(1280, 12, 2, 128), (37, 4, 4, 64), (5, 3, 1, 24)])
@pytest.mark.parametrize("with_term", [True, False])
def test_rope_of_a_sum_into_strided_outputs_is_the_chain_it_replaces(dims, with_term):
    """`rotate_into`: fp16 q (a column block of a wider projection output) + fp16 second term,
    fp32 tables, fp16 [tokens, heads, head_dim] outputs: bit-identical to what the per-op chain
    reaches (fp32 sum, rotation in fp32 through `rope`, one cast to fp16); and the transposed
    rotation written into column blocks of a wider gradient buffer."""
    from claudemaxing_b200.rope import rope, rotate_into

    t, h, kv, d = dims
    gen = torch.Generator().manual_seed(3)
    wide = torch.randn(t, (h + 2 * kv) * d, generator=gen).half().to(DEV)   # [q | k | v] columns
    term = torch.randn(1, t, h * d, generator=gen).half().to(DEV) if with_term else None
    pos = torch.arange(t, dtype=F32)[None]
    inv = 1.0 / (1e6 ** (torch.arange(0, d, 2, dtype=F32) / d))
    emb = torch.cat((pos[..., None] * inv,) * 2, -1)
    cos, sin = emb.cos().to(DEV), emb.sin().to(DEV)

    def heads_first(x, heads):
        return x.unflatten(-1, (heads, d)).unsqueeze(0).transpose(1, 2)

    q_in, k_in = heads_first(wide[:, :h * d], h), heads_first(wide[:, h * d:(h + kv) * d], kv)
    q_out = torch.empty(t, h, d, dtype=F16, device=DEV)
    k_out = torch.empty(t, kv, d, dtype=F16, device=DEV)
    rotate_into(q_in, None if term is None else heads_first(term[0], h), k_in, cos, sin,
                q_out.unsqueeze(0).transpose(1, 2), k_out.unsqueeze(0).transpose(1, 2))
    q_sum = q_in.float() if term is None else q_in.float() + heads_first(term[0], h).float()
    want_q, want_k = rope(q_sum, k_in.float(), cos, sin)
    assert torch.equal(q_out, want_q.half().transpose(1, 2)[0])
    assert torch.equal(k_out, want_k.half().transpose(1, 2)[0])
    # backward: fp16 gradients in, fp16 column blocks out; the chain casts the fp32 result once
    gq = torch.randn(t, h, d, generator=gen).half().to(DEV)
    gk = torch.randn(t, kv, d, generator=gen).half().to(DEV)
    buf = torch.full((t, (h + 2 * kv) * d), 7.0, dtype=F16, device=DEV)
    rotate_into(gq.unsqueeze(0).transpose(1, 2), None, gk.unsqueeze(0).transpose(1, 2), cos, sin,
                heads_first(buf[:, :h * d], h), heads_first(buf[:, h * d:(h + kv) * d], kv), backward=True)
    q_leaf = q_sum.clone().requires_grad_()
    k_leaf = k_in.float().clone().requires_grad_()
    oq, ok = rope(q_leaf, k_leaf, cos, sin)
    torch.autograd.backward((oq, ok), (gq.float().unsqueeze(0).transpose(1, 2), gk.float().unsqueeze(0).transpose(1, 2)))
    assert torch.equal(buf[:, :h * d], q_leaf.grad.half().transpose(1, 2)[0].reshape(t, h * d))
    assert torch.equal(buf[:, h * d:(h + kv) * d], k_leaf.grad.half().transpose(1, 2)[0].reshape(t, kv * d))
    assert (buf[:, (h + kv) * d:] == 7.0).all()    # the v block is not this kernel's to write


@pytest.mark.parametrize("dims", [(1280, 12, 2, 128), (37, 4, 4, 64), (5, 3, 1, 16), (1, 1, 1, 256)])
@pytest.mark.parametrize("with_terms", [True, False])
def test_qkv_split_and_rotation_is_the_rotation_and_the_sums_it_replaces(dims, with_terms):
    """`soup_qkv_rope_fwd` / `_bwd` against `rotate_into` and torch's sum and copy, bit for bit (the
    same fp32 operations and one rounding each), with a row pitch wider than the three blocks."""
    from claudemaxing_b200 import _lib
    from claudemaxing_b200.rope import rotate_into

    t, h, kv, d = dims
    gen = torch.Generator().manual_seed(4)
    cols, pitch = (h + 2 * kv) * d, (h + 2 * kv) * d + 8
    qkv = torch.randn(t, pitch, generator=gen).half().to(DEV)
    add_q = torch.randn(t, h * d, generator=gen).half().to(DEV) if with_terms else None
    add_v = torch.randn(t, kv * d, generator=gen).half().to(DEV) if with_terms else None
    emb = torch.randn(1, t, d, generator=gen) * 3
    cos, sin = emb.cos().to(DEV), emb.sin().to(DEV)

    def heads_first(x, heads):
        return x.unflatten(-1, (heads, d)).unsqueeze(0).transpose(1, 2)

    q, k, v = (torch.empty(t, heads, d, dtype=F16, device=DEV) for heads in (h, kv, kv))
    _lib.call("soup_qkv_rope_fwd", _lib.ptr(qkv), pitch, _lib.ptr(add_q), _lib.ptr(add_v), _lib.ptr(cos),
              _lib.ptr(sin), _lib.ptr(q), _lib.ptr(k), _lib.ptr(v), t, h, kv, d, _lib.stream_of(q))
    wq, wk = torch.empty_like(q), torch.empty_like(k)
    rotate_into(heads_first(qkv[:, :h * d], h), None if add_q is None else heads_first(add_q, h),
                heads_first(qkv[:, h * d:(h + kv) * d], kv), cos, sin,
                wq.unsqueeze(0).transpose(1, 2), wk.unsqueeze(0).transpose(1, 2))
    wv = qkv[:, (h + kv) * d:cols]
    assert torch.equal(q, wq) and torch.equal(k, wk)
    assert torch.equal(v.view(t, -1), wv if add_v is None else wv + add_v)
    dq, dk, dv = (torch.randn(t, heads, d, generator=gen).to(DEV) for heads in (h, kv, kv))
    got, want = torch.full((2, t, pitch), 7.0, dtype=F16, device=DEV)
    _lib.call("soup_qkv_rope_bwd", _lib.ptr(dq), _lib.ptr(dk), _lib.ptr(dv), _lib.ptr(cos), _lib.ptr(sin),
              _lib.ptr(got), pitch, t, h, kv, d, _lib.stream_of(dq))
    rotate_into(dq.unsqueeze(0).transpose(1, 2), None, dk.unsqueeze(0).transpose(1, 2), cos, sin,
                heads_first(want[:, :h * d], h), heads_first(want[:, h * d:(h + kv) * d], kv), backward=True)
    want[:, (h + kv) * d:cols] = dv.reshape(t, -1)
    assert torch.equal(got, want)


# From 148 row blocks of 16 on a CTA owns two of them: 2369 and 4609 rows leave the last one a single row of its first.
@pytest.mark.parametrize("rows", [1, 16, 33, 1280, 2369, 4609])
@pytest.mark.parametrize("hidden,outs", [(1536, (1536, 256)), (32, (16, 16)), (160, (48, 144))])
def test_lora_pair_backward_in_two_launches(rows, hidden, outs):
    """`soup_lora_pair_gain` / `soup_lora_pair_input` against the products they replace in float64, with
    fp16 roundings where those have them; ragged row blocks, strips that leave warps of a CTA idle, a
    row pitch of its own, sums added to what the buffers hold. Bounds: one fp16 ulp where a sum in
    another order rounds the other way (2^-10 of the value, 2^-10 of the largest), fp32 sums (1e-4)."""
    from claudemaxing_b200 import _lib

    gen = torch.Generator().manual_seed(rows + hidden)

    def rand(*shape, std=1.0):
        return (torch.randn(*shape, generator=gen) * std).half().to(DEV)

    pitch = outs[0] + 2 * outs[1]
    wide = rand(rows, pitch, std=0.1)
    g = (wide[:, :outs[0]], wide[:, outs[0] + outs[1]:])   # column blocks, on 16-byte boundaries
    a, a_pair = rand(2, rows, 16), rand(2, 16, hidden, std=0.05)
    b = tuple(rand(o, 16, std=0.05) for o in outs)
    x16 = rand(rows, hidden)
    keep = (torch.rand(2, rows * hidden, generator=gen) > 0.1).to(DEV)
    bits = (keep.view(2, -1, 8).to(torch.int32) << torch.arange(8, device=DEV, dtype=torch.int32)).sum(-1).to(torch.uint8)
    scales, alphas = (1 / 0.9, 1 / 0.8), (2.0, 0.5)
    gain = torch.empty(2, rows, 16, dtype=F16, device=DEV)
    db = [torch.ones(o, 16, device=DEV) for o in outs]
    da = [torch.ones(16, hidden, device=DEV) for _ in outs]
    dx = torch.full((rows, hidden), float("nan"), device=DEV)
    stream = _lib.stream_of(dx)
    _lib.call("soup_lora_pair_gain", _lib.ptr(g[0]), pitch, outs[0], _lib.ptr(g[1]), pitch, outs[1], _lib.ptr(a),
              _lib.ptr(b[0]), _lib.ptr(b[1]), _lib.ptr(gain), _lib.ptr(db[0]), _lib.ptr(db[1]), *alphas, rows, 16, stream)
    want_dx = torch.zeros(rows, hidden, dtype=torch.float64, device=DEV)
    for i in (0, 1):
        assert_close_rel_max(gain[i], (g[i].double() @ b[i].double()).float(), 2 ** -10, "gain")
        assert_close_rel_max(db[i], (1 + alphas[i] * (g[i].double().t() @ a[i].double())).float(), 1e-4, "dB")
    _lib.call("soup_lora_pair_input", _lib.ptr(x16), _lib.ptr(bits[0]), _lib.ptr(bits[1]), _lib.ptr(gain),
              _lib.ptr(a_pair), _lib.ptr(dx), _lib.ptr(da[0]), _lib.ptr(da[1]), *scales, rows, hidden, 16, stream)
    for i in (0, 1):
        k = keep[i].view(rows, hidden)
        xd = torch.where(k, x16.float() * scales[i], torch.zeros((), device=DEV)).half()
        want_dx += k * scales[i] * (gain[i].double() @ a_pair[i].double()).half().double()
        assert_close_rel_max(da[i], (1 + gain[i].double().t() @ xd.double()).float(), 1e-4, "dA")
    assert_close_rel_max(dx, want_dx.float(), 2 ** -10, "dx")


def _rows_of(kind, rows, out, gen):
    """An output gradient [1, rows, out]: a tensor of its own, a column block, one row broadcast over
    the tokens, or rows whose pitch is not a multiple of 16 bytes."""
    if kind == "broadcast":
        return (torch.randn(1, 1, out, generator=gen) * 0.1).half().to(DEV).expand(1, rows, out)
    wide = (torch.randn(1, rows, out + (3 if kind == "ragged" else 64), generator=gen) * 0.1).half().to(DEV)
    return wide[..., :out].contiguous() if kind in ("plain", "ordered") else wide[..., -out:] if kind == "block" else wide[..., :out]


@pytest.mark.parametrize("rank,rows,outs,kinds,launches", [
    (16, 80, (160, 48), ("plain", "plain"), 2),
    (16, 33, (160, 48), ("block", "plain"), 2),
    (16, 40, (160, 48), ("plain", "broadcast"), 0),   # a row pitch of zero
    (16, 40, (160, 48), ("ragged", "plain"), 0),
    (16, 40, (168, 48), ("plain", "plain"), 0),       # a width off the kernel's tiles
    (8, 40, (160, 48), ("plain", "plain"), 0),
    (16, 80, (160, 48), ("plain", "ordered"), 0),     # torch.use_deterministic_algorithms
])
def test_lora_pair_in_place_is_two_single_branches_whichever_way_its_backward_runs(
        rank, rows, outs, kinds, launches, monkeypatch):
    """The pair's backward adding into preset gradients against two LoRABranch nodes with the same
    dropout draws: through its two launches where they take the operands, through the products they
    replace otherwise. Bounds: an fp16 rank-r gradient that rounds the other way, 2^-10 of the largest
    value, in everything formed from it."""
    from claudemaxing_b200 import _lib
    from claudemaxing_b200.lora import LoRABranch, LoRABranchPair

    hidden, ps, scalings = 96, (0.1, 0.25), (2.0, 0.5)
    gen = torch.Generator().manual_seed(rank + rows)
    x = torch.randn(1, rows, hidden, generator=gen).to(DEV)
    x16 = x.half()
    weights = [(torch.randn(*shape, generator=gen) * 0.05).to(DEV)
               for out in outs for shape in ((rank, hidden), (out, rank))]
    preset = [torch.randn(w.shape, generator=gen).to(DEV) for w in weights]
    grads = [_rows_of(kind, rows, out, gen) for kind, out in zip(kinds, outs)]
    if "ordered" in kinds:   # the switch itself would refuse cuBLAS without a workspace setting
        monkeypatch.setattr(torch, "are_deterministic_algorithms_enabled", lambda: True)
    entry, made = _lib.call, []
    monkeypatch.setattr(_lib, "call", lambda name, *args: (made.append(name), entry(name, *args))[1])

    def run(pair):
        leaf = x.clone().requires_grad_()
        ws = [w.clone().requires_grad_() for w in weights]
        for w, g in zip(ws, preset):
            w.grad = g.clone()
        torch.cuda.manual_seed(5)
        b16s = [(ws[2 * i + 1].detach() * scalings[i]).half() for i in (0, 1)]
        if pair:
            monkeypatch.setattr(LoRABranch, "accumulate_in_place", True)
            a16_pair = torch.stack([ws[0].detach().half(), ws[2].detach().half()])
            out = LoRABranchPair.apply(leaf, x16, *ws, *ps, *scalings, a16_pair, *b16s)
        else:
            out = [LoRABranch.apply(leaf, x16, ws[2 * i], ws[2 * i + 1], ps[i], scalings[i],
                                    ws[2 * i].detach().half(), b16s[i], True) for i in (0, 1)]
        torch.autograd.backward(list(out), grads)
        monkeypatch.setattr(LoRABranch, "accumulate_in_place", False)
        return [*(t.detach() for t in out), leaf.grad, *(w.grad for w in ws)]

    want = run(False)
    made.clear()
    got = run(True)
    assert sum(name.startswith("soup_lora_pair") for name in made) == launches
    for name, a, b in zip(("out", "out", "dx", "dA", "dB", "dA", "dB"), got, want):
        assert_close_rel_max(a, b, 2 ** -10, name)


@pytest.mark.parametrize("cols", [8, 248, 256, 264, 4096, 4104])
@pytest.mark.parametrize("rows", [1, 5, 4000])
def test_rmsnorm_row_kernels_at_the_edges_of_their_shapes(rows, cols):
    """One CTA per row, four rows of one warp, and the ring kernels beside them (more than 4096 columns;
    many 16-bit rows): forward in fp32 and fp16 and the saved-output backward against float64. Bounds:
    fp32 sums of up to 4104 terms (1e-5); one rounding to fp16 after another (2^-10)."""
    import importlib

    from claudemaxing_b200 import _lib

    rms = importlib.import_module("claudemaxing_b200.rmsnorm")
    gen = torch.Generator().manual_seed(cols + rows)
    x = torch.randn(rows, cols, generator=gen).to(DEV)
    w = (torch.rand(cols, generator=gen) + 0.5).to(DEV)
    w[cols // 2] = 1e-5
    dy = torch.randn(rows, cols, generator=gen).to(DEV)

    def exact(t, weight):
        t = t.double()
        return t * torch.rsqrt(t.pow(2).mean(-1, keepdim=True) + 1e-6) * weight.double()

    out, rstd, low, slots, small = rms._forward_launch(x, w, 1e-6, F32, True)
    assert_close_rel_max(out, exact(x, w).float(), 1e-5)
    out16 = rms._forward_launch(x.half(), w.half(), 1e-6, F16, False)[0]
    assert_close_rel_max(out16.float(), exact(x.half(), w.half()).float(), 2 ** -10)
    dx = torch.empty_like(x)
    _lib.call("soup_rmsnorm_bwd", _lib.ptr(dy), _lib.ptr(low), _lib.ptr(w), _lib.ptr(rstd), _lib.ptr(dx), None,
              None, _lib.ptr(slots), _lib.ptr(small), small.shape[-1], rows, cols, _lib.F32, _lib.F16, _lib.F32,
              _lib.F32, 1, _lib.stream_of(dy))
    leaf = x.double().requires_grad_()
    exact(leaf, w).backward(dy.double())
    # the saved normalised values carry fp16's rounding
    assert_close_rel_max(dx, leaf.grad.float(), 2 ** -9)


@pytest.mark.parametrize("rows,cols", [(1280, 1536), (37, 256), (5, 4096)])
@pytest.mark.parametrize("with_residual", [True, False])
def test_rmsnorm_backward_with_the_residual_gradient_folded_in(rows, cols, with_residual):
    """`soup_rmsnorm_bwd_residual` = the saved-output RMSNorm backward, plus the residual branch's
    gradient, plus the fp16 copy of the sum: bit-identical to the backward kernel followed by
    torch's add and cast; and the autograd node `_NormResidual` gives the gradients of
    norm(h) and h + f(norm(h)) composed the plain way."""
    import importlib

    from claudemaxing_b200 import _lib

    rms = importlib.import_module("claudemaxing_b200.rmsnorm")
    block = importlib.import_module("claudemaxing_b200.decoder_block")
    gen = torch.Generator().manual_seed(8)
    h = torch.randn(1, rows, cols, generator=gen).to(DEV).requires_grad_()
    w = (torch.randn(cols, generator=gen) * 0.3 + 1.0).to(DEV)
    w[3] = 1e-5                                   # a tiny-|w| column goes through the side buffer
    dy = torch.randn(1, rows, cols, generator=gen).to(DEV)
    res = torch.randn(1, rows, cols, generator=gen).to(DEV) if with_residual else None
    out, rstd, low, slots, small = rms._forward_launch(h.detach().view(rows, cols), w, 1e-6, F32, True)
    plain = torch.empty(rows, cols, device=DEV)
    _lib.call("soup_rmsnorm_bwd", _lib.ptr(dy), _lib.ptr(low), _lib.ptr(w), _lib.ptr(rstd), _lib.ptr(plain),
              None, None, _lib.ptr(slots), _lib.ptr(small), small.shape[-1], rows, cols, _lib.F32,
              _lib.F16, _lib.F32, _lib.F32, 1, _lib.stream_of(dy))
    want = plain if res is None else plain + res.view(rows, cols)
    dx, dx16 = torch.empty(rows, cols, device=DEV), torch.empty(rows, cols, dtype=F16, device=DEV)
    try:
        _lib.call("soup_rmsnorm_bwd_residual", _lib.ptr(dy), _lib.ptr(low), _lib.ptr(w), _lib.ptr(rstd),
                  _lib.ptr(res), _lib.ptr(dx), _lib.ptr(dx16), _lib.ptr(slots), _lib.ptr(small),
                  small.shape[-1], rows, cols, _lib.stream_of(dy))
    except RuntimeError as err:     # rows too wide for the saved-output kernel: said so, not guessed
        assert cols > 1024 * 3 and "does not take the residual form" in str(err)
    else:
        assert cols <= 1024 * 3
        assert torch.equal(dx, want) and torch.equal(dx16, want.half())
    # the autograd node: y = norm(h) * 2 + h (a branch on the norm and the residual connection)
    x, h_res = block._NormResidual.apply(h, w, 1e-6)
    (x * 2.0 + h_res).backward(dy)
    h2 = h.detach().clone().requires_grad_()
    (rms.rmsnorm(h2, w, 1e-6) * 2.0 + h2).backward(dy)
    assert_close_rel_max(h.grad.cpu(), h2.grad.cpu(), 1e-5, "gradient through norm and residual")
    copy = block._GradCopies.take(h.grad)
    assert copy is None or torch.equal(copy.view_as(h.grad), h.grad.half())


# ----------------------------------------------------------------------------------- SwiGLU
@pytest.mark.parametrize("tag", ["f16", "f32", "mix", "noround"])
def test_swiglu_golden(tag):
    from claudemaxing_b200.swiglu_recompute import _silu_mul_bwd, _silu_mul_fwd

    g = load_golden(f"swiglu_{tag}")
    gate, up, dy = g["gate"].to(DEV), g["up"].to(DEV), g["dy"].to(DEV)
    out = torch.empty(gate.shape, dtype=g["out"].dtype, device=DEV)
    _silu_mul_fwd(gate, up, out, bool(g["round_silu"]))
    dg, du = torch.empty_like(gate), torch.empty_like(up)
    _silu_mul_bwd(dy, gate, up, dg, du, bool(g["round_silu"]))
    tol = 1e-4 if tag == "f32" else 2e-3
    assert_close_rel_max(out.cpu(), g["out"], tol, "out")
    assert_close_rel_max(dg.cpu(), g["dgate"], tol, "dgate")
    assert_close_rel_max(du.cpu(), g["dup"], tol, "dup")


@pytest.mark.parametrize("shape", [(4, 512, 8960), (3, 77, 1001), (1, 1, 8960), (5, 3)])
@pytest.mark.parametrize("dtypes", [(F16, F16), (F32, F32), (F16, F32), (F32, F16)])
@pytest.mark.parametrize("inplace", [False, True])
def test_swiglu_vs_oracle(shape, dtypes, inplace):
    from claudemaxing_b200.swiglu_recompute import swiglu_recompute
    from oracle import elementwise as ew

    gdt, udt = dtypes
    gen = torch.Generator().manual_seed(5)
    gate = torch.randn(*shape, generator=gen).to(gdt)
    up = torch.randn(*shape, generator=gen).to(udt)
    dy = torch.randn(*shape, generator=gen).to(torch.promote_types(gdt, udt))
    r_out, r_dg, r_du = ew.swiglu_fwd_bwd(gate, up, dy)
    g = gate.to(DEV).requires_grad_(True)
    u = up.to(DEV).requires_grad_(True)
    # inplace works on temporaries: feed clones whose storage backward may overwrite
    gi, ui = (g * 1, u * 1) if inplace else (g, u)
    out = swiglu_recompute(gi, ui, inplace)
    assert out.dtype == r_out.dtype
    out.backward(dy.to(DEV))
    tol = 1e-4 if dtypes == (F32, F32) else 2e-3
    assert_close_rel_max(out.detach().cpu(), r_out, tol, "out")
    assert_close_rel_max(g.grad.cpu(), r_dg, tol, "dgate")
    assert_close_rel_max(u.grad.cpu(), r_du, tol, "dup")
    if inplace:  # the gradients landed in the storage of the saved inputs
        assert gi.data_ptr() == g.grad.data_ptr() or torch.equal(gi.detach(), g.grad)
    else:
        assert torch.equal(g.detach().cpu(), gate) and torch.equal(u.detach().cpu(), up)


def test_swiglu_saves_exactly_gate_and_up_and_one_sided_grads():
    from claudemaxing_b200.swiglu_recompute import swiglu_recompute

    saved = []
    gate = torch.randn(64, 256, device=DEV, dtype=F16, requires_grad=True)
    up = torch.randn(64, 256, device=DEV, dtype=F16)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: saved.append(t) or t, lambda t: t):
        out = swiglu_recompute(gate, up)
    assert {t.data_ptr() for t in saved} == {gate.data_ptr(), up.data_ptr()}
    out.sum().backward()
    assert gate.grad is not None and up.grad is None


# ----------------------------------------------------------------------------------- dropout bits
def test_dropout_golden_bit_exact():
    from claudemaxing_b200.lora import _pack, _unpack

    g = load_golden("dropout")
    xd, bits = _pack(g["x"].to(DEV), g["mask"].to(DEV), g["scale"])
    assert torch.equal(bits.cpu(), g["bits"]) and torch.equal(_bits(xd.cpu()), _bits(g["xd"]))
    xd2, dx = _unpack(g["x16"].to(DEV), bits, g["g16"].to(DEV), g["scale"], F32)
    assert torch.equal(_bits(xd2.cpu()), _bits(g["xd2"])) and torch.equal(dx.cpu(), g["dx"])


@pytest.mark.parametrize("shape", [(3, 37, 64), (2048, 1536), (1, 8), (5, 24)])
@pytest.mark.parametrize("xdt", [F32, F16])
def test_dropout_bit_exact_vs_oracle(shape, xdt):
    from claudemaxing_b200.lora import _pack, _unpack
    from oracle import elementwise as ew

    gen = torch.Generator().manual_seed(9)
    x = torch.randn(*shape, generator=gen).to(xdt)
    mask = torch.rand(*shape, generator=gen) > 0.05
    scale = 1.0 / 0.95
    r_xd, r_bits = ew.dropout_pack(x, mask, scale)
    xd, bits = _pack(x.to(DEV), mask.to(DEV), scale)
    assert torch.equal(bits.cpu(), r_bits) and torch.equal(_bits(xd.cpu()), _bits(r_xd))
    g16 = torch.randn(*shape, generator=gen).half()
    r_xd2, r_dx = ew.dropout_unpack(x.half(), r_bits, g16, scale, F32)
    xd2, dx = _unpack(x.half().to(DEV), bits, g16.to(DEV), scale, F32)
    assert torch.equal(_bits(xd2.cpu()), _bits(r_xd2)) and torch.equal(dx.cpu(), r_dx)
    # pack -> unpack keeps the kept elements: unpacked bits give the mask back
    assert torch.equal((dx != 0).cpu() | (g16 == 0), mask | (g16 == 0))


def test_lora_branch_matches_plain_formula():
    # the branch against base-free peft math on the same dropout mask (same RNG stream)
    from claudemaxing_b200.lora import LoRABranch

    torch.manual_seed(0)
    x = torch.randn(4, 50, 256, device=DEV, requires_grad=True)
    a = torch.randn(16, 256, device=DEV, requires_grad=True) * 0.1
    b = torch.randn(64, 16, device=DEV, requires_grad=True) * 0.1
    a.retain_grad(), b.retain_grad()
    torch.manual_seed(123)
    out = LoRABranch.apply(x, x.detach().half(), a, b, 0.05, 2.0)
    g = torch.randn_like(out)
    out.backward(g)
    torch.manual_seed(123)
    x2 = x.detach().clone().requires_grad_(True)
    a2, b2 = a.detach().clone().requires_grad_(True), b.detach().clone().requires_grad_(True)
    xd = torch.nn.functional.dropout(x2, 0.05, True).half()
    ref = torch.nn.functional.linear(torch.nn.functional.linear(xd, a2.half()), b2.half()) * 2.0
    ref.backward(g)
    assert torch.equal(out, ref)
    assert rel_norm(x.grad.cpu(), x2.grad.cpu()) < 2e-3
    assert rel_norm(a.grad.cpu(), a2.grad.cpu()) < 5e-3
    assert rel_norm(b.grad.cpu(), b2.grad.cpu()) < 5e-3


@pytest.mark.parametrize("scaling", [2.0, 1.7])
def test_lora_branch_with_cast_scaled_weights_and_in_place_gradients(scaling, monkeypatch):
    """The branch given fp16 A and fp16(scaling * B) copies (no scaling pass over its output or
    the incoming gradient), adding its weight gradients into existing `.grad` tensors inside the
    GEMMs: the plain call's numbers (identical for a power-of-two scaling)."""
    from claudemaxing_b200.lora import LoRABranch

    torch.manual_seed(0)
    x = torch.randn(3, 40, 256, device=DEV)
    a = (torch.randn(16, 256, device=DEV) * 0.1).requires_grad_()
    b = (torch.randn(64, 16, device=DEV) * 0.1).requires_grad_()
    g = torch.randn(3, 40, 64, device=DEV).half()
    results = []
    for fast in (False, True):
        xx = x.clone().requires_grad_()
        a.grad, b.grad = torch.full_like(a, 0.5), torch.full_like(b, -0.25)   # something to add to
        kept = (a.grad, b.grad)
        monkeypatch.setattr(LoRABranch, "accumulate_in_place", fast)
        torch.manual_seed(7)
        extra = (a.detach().half(), (b.detach() * scaling).half(), True) if fast else ()
        out = LoRABranch.apply(xx, xx.detach().half(), a, b, 0.1, scaling, *extra)
        out.backward(g)
        assert (a.grad is kept[0] and b.grad is kept[1]) or not fast
        results.append((out.detach(), xx.grad, a.grad.clone(), b.grad.clone()))
    for name, plain, fast in zip(("out", "dx", "dA", "dB"), *results):
        if scaling == 2.0 and name in ("out", "dx"):
            assert torch.equal(plain, fast), name
        assert rel_norm(fast.float().cpu(), plain.float().cpu()) < 2e-3, name


# From 592 row blocks of 16 on a CTA owns two of them in the rank-16 gradient's launch (9473 rows: one row of the last
# CTA's first block), and a warp of the output's launch walks three row tiles (520 columns, 16391 rows).
@pytest.mark.parametrize("rows", [1, 15, 17, 1000, 9473, 16391])
@pytest.mark.parametrize("width,out", [(32, 8), (96, 40), (1568, 520)])
@pytest.mark.parametrize("scaling,given", [(2.0, False), (0.3, False), (0.3, True)])
def test_rank16_branch_at_the_edges_of_its_tiles(rows, width, out, scaling, given):
    """Against the products in float64 with fp16 roundings where those have them: row tiles, strips and
    chunks with remainders, a gradient row pitch of its own. Bounds: one fp16 ulp of the largest value per
    rounding that may go the other way (2^-10; two of them, the product and its scaling, in the output and in dx),
    fp32 sums (1e-4) of terms whose factors may round the other way."""
    from claudemaxing_b200.lora import LoRABranch

    gen = torch.Generator().manual_seed(rows + width)
    x = torch.randn(1, rows, width, generator=gen).to(DEV).requires_grad_()
    a, b = (((torch.randn(*shape, generator=gen) * 0.1).to(DEV)).requires_grad_() for shape in ((16, width), (out, 16)))
    g = torch.randn(1, rows, out + 8, generator=gen).half().to(DEV)[..., :out]
    a16, b16 = a.detach().half(), ((b.detach() * scaling) if given else b.detach()).half()
    torch.manual_seed(3)
    got = LoRABranch.apply(x, x.detach().half(), a, b, 0.1, scaling, *((a16, b16, True) if given else ()))
    got.backward(g)
    torch.manual_seed(3)
    mask = torch.native_dropout(x.detach(), 0.1, True)[1][0]
    keep = mask / 0.9
    f64 = lambda t: t.detach().double()
    once = lambda t: t.half().double()
    xd = once(mask * (x.detach()[0] * (1 / 0.9)))
    low = once(xd @ f64(a16).t())
    outer = 1.0 if given else scaling
    want = once(once(low @ f64(b16).t()) * outer)
    gs = once(f64(g[0]) * outer)
    gain = once(gs @ f64(b16))
    want_dx = once(gain @ f64(a16)) * keep.double()
    x16d = once(mask * (x.detach().half()[0].float() * (1 / 0.9)))
    assert_close_rel_max(got.detach()[0], want.half(), 2 ** -9, "out")
    assert_close_rel_max(x.grad[0], want_dx.float(), 2 ** -9, "dx")
    assert_close_rel_max(a.grad, (gain.t() @ x16d).float(), 2 ** -10, "dA")
    assert_close_rel_max(b.grad, (gs.t() @ low * (scaling if given else 1.0)).float(), 2 ** -10, "dB")


@pytest.mark.parametrize("extra", [0, 8])
def test_rank16_branch_at_the_widest_output_its_launches_take(extra):
    """2^24 columns run on the rank-16 launches, wider ones on the products. Both against the plain products (an fp16 ulp
    of the largest value, 2^-10)."""
    from claudemaxing_b200 import lora

    out, gen = (1 << 24) + extra, torch.Generator(device=DEV).manual_seed(extra)
    x = torch.randn(1, 1, 32, generator=gen, device=DEV)
    a = torch.randn(16, 32, generator=gen, device=DEV) * 0.1
    b = torch.randn(out, 16, generator=gen, device=DEV) * 0.1
    assert lora._rank16_covers(x, x.half(), [(a, b)]) == (extra == 0)
    torch.manual_seed(1)
    got = lora.LoRABranch.apply(x, x.half(), a, b, 0.1, 2.0)
    torch.manual_seed(1)
    dropped = torch.native_dropout(x, 0.1, True)[0].half()
    low = torch.nn.functional.linear(dropped, a.half())
    want = torch.nn.functional.linear(low, b.half()) * 2.0
    assert_close_rel_max(got, want, 2 ** -10, "out")


@pytest.mark.parametrize("pair", [False, True])
def test_lora_branch_frees_its_dropout_masks_before_its_outputs(pair):
    """The forward's peak: the bool masks (a byte an element) are gone before the products, whose outputs are the
    larger part here."""
    from claudemaxing_b200.lora import LoRABranch, LoRABranchPair

    rows, width, out = 4096, 256, 4096
    x = torch.randn(1, rows, width, device=DEV)
    x16 = x.half()
    a, b = (torch.randn(2, *shape, device=DEV) * 0.05 for shape in ((16, width), (out, 16)))
    a16, b16 = a.half(), b.half()
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    if pair:
        kept = LoRABranchPair.apply(x, x16, a[0], b[0], a[1], b[1], 0.1, 0.1, 1.0, 1.0, a16, b16[0], b16[1])
    else:
        kept = LoRABranch.apply(x, x16, a[0], b[0], 0.1, 1.0, a16[0], b16[0], True)
    n, branches = rows * width, 1 + pair
    # outputs, dropped input, its bits and the product with A; half a mask of room for rounded allocations
    want = branches * (2 * rows * out + 2 * n + n // 8 + 2 * rows * 16) + n // 2
    assert torch.cuda.max_memory_allocated() - before <= want
    del kept


def test_paired_lora_branches_are_the_two_single_branches():
    """LoRABranchPair (one packing launch, one batched product with A, one unpacking launch that
    sums the input gradients) against two LoRABranch calls with the same dropout draws: outputs
    and weight gradients per adapter and the summed input gradient, bit for bit."""
    from claudemaxing_b200.lora import LoRABranch, LoRABranchPair

    torch.manual_seed(0)
    x = torch.randn(1, 80, 256, device=DEV)
    weights = [(torch.randn(16, 256, device=DEV) * 0.1).requires_grad_(),
               (torch.randn(96, 16, device=DEV) * 0.1).requires_grad_(),
               (torch.randn(16, 256, device=DEV) * 0.1).requires_grad_(),
               (torch.randn(32, 16, device=DEV) * 0.1).requires_grad_()]
    g1, g2 = torch.randn(1, 80, 96, device=DEV).half(), torch.randn(1, 80, 32, device=DEV).half()
    a16 = torch.stack([weights[0].detach().half(), weights[2].detach().half()])
    b1, b2 = (weights[1].detach() * 2.0).half(), (weights[3].detach() * 2.0).half()
    results = []
    for paired in (False, True):
        xx = x.clone().requires_grad_()
        for w in weights:
            w.grad = None
        torch.manual_seed(5)
        if paired:
            o1, o2 = LoRABranchPair.apply(xx, xx.detach().half(), *weights, 0.1, 0.1, 2.0, 2.0, a16, b1, b2)
        else:
            o1 = LoRABranch.apply(xx, xx.detach().half(), weights[0], weights[1], 0.1, 2.0, a16[0], b1, True)
            o2 = LoRABranch.apply(xx, xx.detach().half(), weights[2], weights[3], 0.1, 2.0, a16[1], b2, True)
        torch.autograd.backward((o1, o2), (g1, g2))
        results.append([o1.detach(), o2.detach(), xx.grad] + [w.grad.clone() for w in weights])
    for name, single, pair in zip(("out1", "out2", "dx", "dA1", "dB1", "dA2", "dB2"), *results):
        assert torch.equal(single, pair), name


def test_paired_lora_branches_of_many_elements_go_through_the_products(monkeypatch):
    """Backward on either side of `lora.ONE_BY_ONE`: adapter by adapter up to it, the products of both beyond, with
    the same numbers. Bounds: an fp16 rank-16 gradient or product that rounds the other way, 2^-10 of the largest
    value each."""
    import importlib

    lora = importlib.import_module("claudemaxing_b200.lora")
    names = []
    real = lora._lib.call
    monkeypatch.setattr(lora._lib, "call", lambda name, *args: (names.append(name), real(name, *args))[1])
    hidden, outs = 4096, (256, 64)
    most = lora.ONE_BY_ONE
    for rows, one_by_one in ((most // hidden, True), (most // hidden + 1, False)):
        gen = torch.Generator(device=DEV).manual_seed(rows)
        rand = lambda *shape, std=1.0: torch.randn(*shape, generator=gen, device=DEV) * std
        x = rand(1, rows, hidden)
        ws = [rand(*shape, std=0.05) for shape in ((16, hidden), (outs[0], 16), (16, hidden), (outs[1], 16))]
        grads = [rand(1, rows, o, std=0.1).half() for o in outs]
        results = []
        for limit, expected in ((most, one_by_one), (0 if one_by_one else 1 << 40, not one_by_one)):
            monkeypatch.setattr(lora, "ONE_BY_ONE", limit)
            torch.manual_seed(9)
            leaves = [t.clone().requires_grad_() for t in (x, *ws)]
            a16 = torch.stack([ws[0], ws[2]]).half()
            out = lora.LoRABranchPair.apply(leaves[0], x.half(), *leaves[1:], 0.1, 0.25, 1.0, 1.0, a16, ws[1].half(),
                                            ws[3].half())
            del names[:]
            results.append(torch.autograd.grad(out, leaves, grads))
            assert ("soup_lora_branch_bwd" in names) == expected
        for name, first, second in zip(("dx", "dA1", "dB1", "dA2", "dB2"), *results):
            assert_close_rel_max(first, second, 2 ** -9, name)


@pytest.mark.parametrize("rows", [1, 127, 129, 257, 700, 2560])
@pytest.mark.parametrize("hidden,inter", [(8, 8), (72, 200), (520, 1096), (1536, 2048)])
def test_mlp_products_with_their_elementwise_passes(rows, hidden, inter):
    """`soup_mlp_fwd` / `soup_mlp_bwd`: row tiles, column tiles and K blocks with remainders, one and two K
    splits (2560 x 1536 has 60 tiles, the others fewer), several tiles a CTA pair; gate and up alone. Each result
    against float64 from the kernels' own operands of that step. Bounds: one fp16 ulp of the largest value (2^-10) where a sum rounds the other way, two where the
    gradient of the activation does before the gradients are formed, 2e-5 for fp32 sums of fp16 products."""
    from claudemaxing_b200 import _lib

    gen = torch.Generator(device=DEV).manual_seed(rows + inter)

    def rand(*shape, std=1.0, dtype=F16):
        return (torch.randn(*shape, generator=gen, device=DEV) * std).to(dtype)

    x, dy = rand(rows, hidden), rand(rows, hidden)
    wg, wu, wd = (rand(*shape, std=hidden ** -0.5) for shape in ((inter, hidden), (inter, hidden), (hidden, inter)))
    residual = rand(rows, hidden, dtype=F32)
    P, stream = _lib.ptr, _lib.stream_of(x)
    results = []
    for _ in range(2):
        gate, up, act, d_gate, d_up = (torch.full((rows, inter), float("nan"), dtype=F16, device=DEV) for _ in range(5))
        out, dx = (torch.full((rows, hidden), float("nan"), device=DEV) for _ in range(2))
        _lib.call("soup_mlp_fwd", P(x), P(residual), P(wg), P(wu), P(wd), P(gate), P(up), P(act), P(out), rows, hidden,
                  inter, stream)
        _lib.call("soup_mlp_bwd", P(dy), P(gate), P(up), P(wg), P(wu), P(wd), P(d_gate), P(d_up), P(dx), rows, hidden,
                  inter, stream)
        results.append((gate, up, act, out, d_gate, d_up, dx))
    gate2, up2 = torch.empty_like(gate), torch.empty_like(up)
    _lib.call("soup_mlp_fwd", P(x), None, P(wg), P(wu), None, P(gate2), P(up2), None, None, rows, hidden, inter, stream)
    _lib.check_device_status()
    for first, second in (*zip(*results), (gate2, gate), (up2, up)):
        assert torch.equal(first, second)
    f64 = lambda t: t.double()
    g, u = f64(gate), f64(up)
    sig = torch.sigmoid(g)
    d_act = (f64(dy) @ f64(wd)).half().double()
    for name, got, want, bound in (
            ("gate", gate, f64(x) @ f64(wg).t(), 2 ** -10), ("up", up, f64(x) @ f64(wu).t(), 2 ** -10),
            ("act", act, g * sig * u, 2 ** -10), ("out", out, f64(residual) + f64(act) @ f64(wd).t(), 2e-5),
            ("d_up", d_up, d_act * g * sig, 2 ** -9),
            ("d_gate", d_gate, d_act * u * sig * (1 + g * (1 - sig)), 2 ** -9),
            ("dx", dx, f64(d_gate) @ f64(wg) + f64(d_up) @ f64(wu), 2e-5)):
        assert_close_rel_max(got.float(), want.float(), bound, name)


@pytest.mark.parametrize("rows,hidden,inter,forward,backward", [
    (1472, 1536, 3072, 1, 1),
    (6464, 1536, 1024, 1, 0),
    (4416, 512, 2048, 0, 1),
    (257, 72, 200, 0, 0),
])
def test_gated_mlp_node_on_its_launches(rows, hidden, inter, forward, backward, monkeypatch):
    """The fused block's MLP node where the launches pay in both directions, in one and in none: the entries it calls,
    the numbers of the library's products, and the same bits whether gate and up are kept or formed again and
    overwritten by their gradients. Bounds: gate, up and the activation's gradient may round the other way, 2^-10 of
    their value each, in sums over them: 2^-9 of the largest."""
    import importlib

    block = importlib.import_module("claudemaxing_b200.decoder_block")
    gen = torch.Generator(device=DEV).manual_seed(rows)
    rand = lambda *shape, std=1.0: torch.randn(*shape, generator=gen, device=DEV) * std
    weights = [rand(*shape, std=hidden ** -0.5).half() for shape in ((inter, hidden), (inter, hidden), (hidden, inter))]
    x, residual, dy = (rand(1, rows, hidden) for _ in range(3))
    names = []
    real = block._lib.call
    monkeypatch.setattr(block._lib, "call", lambda name, *args: (names.append(name), real(name, *args))[1])

    def run(keep):
        del names[:]
        gate, up, down = (SimpleNamespace(dequantized=lambda dtype, w=w: w) for w in weights)
        leaves = [x.clone().requires_grad_(), residual.clone().requires_grad_()]
        out = block._GatedMLPAddResidual.apply(leaves[0], leaves[0].detach().half(), leaves[1],
                                               SimpleNamespace(gate=gate, up=up, down=down, keep_products=keep))
        out.backward(dy)
        return out.detach(), leaves[0].grad, leaves[1].grad

    kept = run(True)
    assert (names.count("soup_mlp_fwd"), names.count("soup_mlp_bwd")) == (forward, backward)
    again = run(False)
    assert (names.count("soup_mlp_fwd"), names.count("soup_mlp_bwd")) == (2 * forward, backward)
    block._lib.check_device_status()
    for first, second in zip(kept, again):
        assert torch.equal(first, second)
    monkeypatch.setattr(block, "_mlp_kernels_cover", lambda *a: False)
    for name, got, want in zip(("out", "dx", "dresidual"), kept, run(True)):
        assert_close_rel_max(got, want, 2 ** -9, name)
    assert "soup_mlp_fwd" not in names and "soup_mlp_bwd" not in names


def test_ops_refuse_cpu_tensors():
    from claudemaxing_b200.rmsnorm import rmsnorm
    from claudemaxing_b200.swiglu_recompute import swiglu_recompute

    with pytest.raises(RuntimeError, match="CUDA"):
        rmsnorm(torch.randn(4, 64), torch.ones(64), 1e-6)
    with pytest.raises(RuntimeError, match="CUDA"):
        swiglu_recompute(torch.randn(4, 64), torch.randn(4, 64))


# ------------------------------------------------------------------------- bounded waits
def test_a_wait_that_nothing_completes_runs_out_and_reports():
    """Failure detection on the device: the kernels' waits give up after their limit, record a
    code and return; the context stays usable (no trap, no hang)."""
    import ctypes

    from claudemaxing_b200 import _lib

    gave_up, status = ctypes.c_int(-1), ctypes.c_int(-1)
    _lib.call("soup_wait_selftest", 2_000_000, ctypes.byref(gave_up), ctypes.byref(status),
              torch.cuda.current_stream().cuda_stream)
    assert gave_up.value == 1 and status.value == 99
    # the device still works
    x = torch.arange(8, device=DEV).sum().item()
    assert x == 28
    # the code reached the device's sticky status word, where the host-side check finds it: the
    # package raises instead of handing out results of a step whose kernels gave up
    row = ctypes.c_int(-1)
    _lib.call("soup_row_status", ctypes.byref(row), torch.cuda.current_stream().cuda_stream)
    assert row.value == 99
    with pytest.raises(RuntimeError, match="device status 99"):
        _lib.check_device_status()
    _lib.check_device_status()          # cleared by the failing check: healthy again
    assert _lib.device_status() == 0


def test_device_status_stays_clear_after_a_healthy_step():
    from claudemaxing_b200 import _lib, fused_head_loss

    _lib.device_status(clear=True)
    gen = torch.Generator().manual_seed(3)
    h = torch.randn(300, 256, generator=gen).half().to(DEV).requires_grad_(True)
    w = (torch.randn(5000, 256, generator=gen) * 0.05).half().to(DEV)
    t = torch.randint(0, 5000, (300,), generator=gen).to(DEV)
    loss, _ = fused_head_loss(h[None], w, None, target=t[None])
    loss.backward()
    _lib.check_device_status()
