"""The packed row's attention kernels (csrc/attention.cu) through the C ABI: forward output and
log-sum-exp, and the three gradients, against the float64 oracle (oracle/attention.py), on the
reference's golden vectors, at the shapes of the reference's own attention test with its
criterion (tests_local/test_attention.py:45-50, :85-97: the error against fp32 must stay within
three times the error of torch's fp16 SDPA on the same inputs), and on the edge cases of the
packed layout (empty and one-token segments, segments that end inside a tile, strided q/k/v)."""

import pytest
import torch

from conftest import assert_close_rel_max, rel_norm

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _cu(lens):
    return torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32)


def _forward(q, k, v, cu, scale=None):
    """(out, lse) of the forward kernel on [N, h, 128] fp16 views (any row pitch)."""
    from claudemaxing_b200 import _lib

    n, hq, d = q.shape
    scale = d ** -0.5 if scale is None else scale
    out = torch.full((n, hq, d), float("nan"), dtype=torch.float16, device=DEV)
    lse = torch.full((hq, n), float("nan"), dtype=torch.float32, device=DEV)
    cu = cu.to(DEV)
    _lib.call("soup_attn_fwd", _lib.ptr(q), _lib.ptr(k), _lib.ptr(v), _lib.ptr(cu), _lib.ptr(out),
              _lib.ptr(lse), n, cu.numel() - 1, hq, k.shape[1], d, q.stride(0), k.stride(0),
              v.stride(0), float(scale), _lib.stream_of(q))
    _lib.check_device_status()
    return out, lse


def _run(q, k, v, cu, grad, scale=None):
    """(out, lse, dq, dk, dv) of the kernels on [N, h, 128] fp16 views (any row pitch)."""
    from claudemaxing_b200 import _lib
    from claudemaxing_b200.attention import attention_gradients

    out, lse = _forward(q, k, v, cu, scale)
    scale = q.shape[2] ** -0.5 if scale is None else scale
    cu = cu.to(DEV)
    dq, dk, dv = attention_gradients(q, k, v, out, lse, grad, cu, scale)
    _lib.check_device_status()
    return out, lse, dq, dk, dv


@pytest.mark.parametrize("tag", ["a", "b"])
def test_attention_kernels_on_the_reference_kernels_golden_vectors(tag):
    from test_oracle_golden import _packed_attention_case

    _, q, k, v, cu, grad, want = _packed_attention_case(tag)
    out, _, dq, dk, dv = _run(q.to(DEV), k.to(DEV), v.to(DEV), cu, grad.to(DEV))
    for name, got in (("out", out), ("dq", dq), ("dk", dk), ("dv", dv)):
        assert_close_rel_max(got.float().cpu(), want[name].float(), 4e-3, name)


@pytest.mark.parametrize("hq,hk,lens", [
    (12, 2, [128, 128]),
    (12, 2, [200, 150, 77, 1]),
    (12, 2, [512, 300, 129]),
    (4, 4, [70]),
    (12, 2, [300, 0, 280, 296, 292, 112]),
    (6, 1, [1000, 3]),
    (4, 2, [40] * 100 + [3]),        # more than 64 segments: the plain tile order
    (2, 1, [2500]),                  # twenty key tiles: many turns of every barrier
    (12, 2, [2500, 700, 1]),         # long walks, one head per forward CTA
    (12, 2, [3500, 700, 1]),         # long enough for two
    (3, 1, [129, 255]),              # an odd group: one head per CTA whatever the size
])
def test_attention_kernels_against_fp32_with_the_fp16_sdpa_error_as_the_bar(hq, hk, lens):
    from oracle import attention as oat

    from claudemaxing_b200.attention import mask_of_segments

    torch.manual_seed(0)
    n, d = sum(lens), 128
    cu = _cu(lens)
    q, k, v = (torch.randn(n, h, d, device=DEV).half() for h in (hq, hk, hk))
    grad = torch.randn(n, hq, d, device=DEV).half()
    out, lse, dq, dk, dv = _run(q, k, v, cu, grad)
    want_out, want_lse = oat.segment_attention(q.cpu(), k.cpu(), v.cpu(), cu)
    want = (want_out,) + oat.segment_attention_backward(q.cpu(), k.cpu(), v.cpu(), cu, grad.cpu())
    # the bar: torch's fp16 SDPA with the mask on the same inputs
    leaves = [t.clone().requires_grad_() for t in (q, k, v)]
    ref = torch.nn.functional.scaled_dot_product_attention(
        leaves[0].transpose(0, 1)[None], leaves[1].transpose(0, 1)[None], leaves[2].transpose(0, 1)[None],
        attn_mask=mask_of_segments(cu.to(DEV), n), enable_gqa=hq != hk)[0].transpose(0, 1)
    ref.backward(grad)
    bar = (ref.detach(),) + tuple(t.grad for t in leaves)
    for name, got, exact, lib in zip(("out", "dq", "dk", "dv"), (out, dq, dk, dv), want, bar):
        assert torch.isfinite(got).all(), name
        err, allowed = rel_norm(got.float().cpu(), exact.float()), rel_norm(lib.float().cpu(), exact.float())
        assert err <= 3 * allowed + 1e-4, (name, err, allowed)
    assert dk.dtype == dv.dtype == torch.float32 and dq.dtype == torch.float16
    assert (lse.double().cpu() - want_lse).abs().max() < 2e-3


@pytest.mark.parametrize("hq,hk,lens", [(4, 2, [700, 130]), (12, 2, [2600, 520]), (12, 2, [4100, 520])])
def test_attention_forward_when_the_row_maximum_keeps_growing(hq, hk, lens):
    """Scores that grow along the keys, then fall: every row's accumulator is rescaled, some rows of a
    warp earlier than others. One and two heads per CTA. P is rounded to fp16 relative to the row's
    maximum so far, 2^-11 an element: the bound of the plain cases."""
    from oracle import attention as oat

    torch.manual_seed(2)
    n, d = sum(lens), 128
    q, k, v = (torch.randn(n, h, d, device=DEV) for h in (hq, hk, hk))
    ramp = torch.cat([torch.cat([torch.linspace(0.05, 8, L - L // 4), torch.linspace(8, 0.5, L // 4)]) for L in lens])
    k = (k * ramp.to(DEV)[:, None, None]).half()
    q, v = q.half(), v.half()
    grad = torch.randn(n, hq, d, device=DEV).half()
    cu = _cu(lens)
    out, lse, dq, dk, dv = _run(q, k, v, cu, grad)
    want_out, want_lse = oat.segment_attention(q.cpu(), k.cpu(), v.cpu(), cu)
    want = (want_out,) + oat.segment_attention_backward(q.cpu(), k.cpu(), v.cpu(), cu, grad.cpu())
    for name, got, exact in zip(("out", "dq", "dk", "dv"), (out, dq, dk, dv), want):
        assert rel_norm(got.float().cpu(), exact.float()) < 2e-3, name
    assert (lse.double().cpu() - want_lse).abs().max() < 2e-3


@pytest.mark.parametrize("scale", [0.0, -0.05])
@pytest.mark.parametrize("hq,hk,lens", [(4, 2, [300, 130]), (12, 2, [4100, 520])])
def test_attention_with_a_scale_of_zero_or_less(hq, hk, lens, scale):
    """Every visible key weighs the same, or the smaller scores more; hidden keys weigh nothing either way.
    One and two heads per CTA; bounds of the plain cases."""
    from oracle import attention as oat

    gen = torch.Generator().manual_seed(12)
    q, k, v, grad = (torch.randn(sum(lens), h, 128, generator=gen).half() for h in (hq, hk, hk, hq))
    cu = _cu(lens)
    got = _run(q.to(DEV), k.to(DEV), v.to(DEV), cu, grad.to(DEV), scale=scale)
    out, lse = oat.segment_attention(q, k, v, cu, scale)
    want = (out, lse) + oat.segment_attention_backward(q, k, v, cu, grad, scale)
    for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), got, want):
        if scale == 0.0 and name in ("dq", "dk"):
            assert (a == 0).all(), name
        else:
            assert rel_norm(a.float().cpu(), b.float()) < 2e-3, name


def test_attention_gradients_are_reproducible_when_torch_is_told_to_be():
    """torch.use_deterministic_algorithms: no sums in any order; the gradients of several key tiles and
    a group of heads come out the same twice, and within the two kernels' fp16 rounding of the others."""
    from claudemaxing_b200.attention import SegmentAttention

    gen = torch.Generator().manual_seed(6)
    lens = [700, 333]
    q, k, v = (torch.randn(sum(lens), h, 128, generator=gen).half().to(DEV).requires_grad_() for h in (12, 2, 2))
    grad = torch.randn(q.shape, generator=gen).half().to(DEV)
    cu = _cu(lens).to(DEV)

    def gradients():
        return torch.autograd.grad(SegmentAttention.apply(q, k, v, cu, max(lens), 128 ** -0.5), (q, k, v), grad)

    own = gradients()
    torch.use_deterministic_algorithms(True)
    try:
        first, second = gradients(), gradients()
    finally:
        torch.use_deterministic_algorithms(False)
    for name, a, b, c in zip("qkv", first, second, own):
        assert torch.equal(a, b), name
        assert rel_norm(a.float(), c.float()) < 2e-3, name


@pytest.mark.parametrize("hq,hk,lens", [(4, 2, [700, 130]), (12, 2, [4100, 520])])
@pytest.mark.parametrize("case", ["far", "masked", "mixed"])
def test_attention_forward_at_scores_far_from_zero_and_at_minus_infinity(hq, hk, lens, case):
    """One and two heads per CTA. "far": scores up to 1e9, where every row attends to one key; "mixed":
    every other row's are small, so a warp holds both kinds; "masked": keys whose scores are -inf, a
    whole key tile and two keys of the next, in front of finite ones. An fp32 sum of 128 products is
    within 2^-17 of their magnitudes' sum, about twice the largest score here: the log-sum-exp's bound,
    and far under the gap of the two largest scores (asserted), so that a far row is one key's value."""
    from oracle import attention as oat

    gen = torch.Generator().manual_seed(8)
    n, d = sum(lens), 128
    q, k, v = (torch.randn(n, h, d, generator=gen) for h in (hq, hk, hk))
    rows = torch.arange(n)
    far = rows >= 0 if case == "far" else rows % 2 == 0 if case == "mixed" else rows < 0
    q[far] *= 12000
    if case != "masked":
        k *= 12000
        q[~far] /= 12000
    else:
        q[..., 0] = q[..., 0].abs() + 0.1
        k[:130, :, 0] = float("-inf")
    q, k, v = q.clamp(-6e4, 6e4).half(), (k if case == "masked" else k.clamp(-6e4, 6e4)).half(), v.half()
    cu = _cu(lens)
    q_d, k_d, v_d = q.to(DEV), k.to(DEV), v.to(DEV)
    out, lse = _forward(q_d, k_d, v_d, cu)
    want, want_lse = oat.segment_attention(q, k, v, cu)
    if case == "masked":      # the first 130 rows see nothing else
        assert torch.isfinite(out[130:]).all()
        assert rel_norm(out[130:].float().cpu(), want[130:].float()) < 2e-3
        assert (lse[:, 130:].double().cpu() - want_lse[:, 130:]).abs().max() < 2e-3
        return
    gap = torch.full((hq, n), float("inf"), dtype=torch.float64)
    for b, e in zip(cu.tolist(), cu.tolist()[1:]):
        z = torch.einsum("qhd,khd->hqk", q_d[b:e].double(), k_d[b:e].double().repeat_interleave(hq // hk, 1))
        z.masked_fill_(~torch.ones(e - b, e - b, dtype=torch.bool, device=DEV).tril(), float("-inf"))
        two = z.topk(2, -1).values.cpu()
        gap[:, b:e] = two[..., 0] - two[..., 1]
    clear = (gap > 1e5) | ~far          # of ten thousand rows one has two keys that close
    assert clear.double().mean() > 0.99
    keep = clear.t()[..., None]
    assert rel_norm(out.float().cpu() * keep, want.float() * keep) < 2e-3
    error = (lse.double().cpu() - want_lse).abs()
    assert (error <= 2e-3 + 2.0 ** -16 * want_lse.abs()).all()


def test_attention_kernels_read_q_k_v_as_column_blocks_and_leave_other_rows_alone():
    """q, k and v as column blocks of one wider matrix (row pitch larger than heads x 128), and
    segments that do not cover the last tokens: those rows of out are not written, those of the
    gradients are zero."""
    from oracle import attention as oat

    torch.manual_seed(1)
    lens, spare = [130, 61], 9
    n_seg, hq, hk, d = sum(lens), 4, 2, 128
    n = n_seg + spare
    wide = torch.randn(n, (hq + 2 * hk) * d, device=DEV).half()
    q = wide[:, :hq * d].unflatten(-1, (hq, d))
    k = wide[:, hq * d:(hq + hk) * d].unflatten(-1, (hk, d))
    v = wide[:, (hq + hk) * d:].unflatten(-1, (hk, d))
    grad = torch.randn(n, hq, d, device=DEV).half()
    out, _, dq, dk, dv = _run(q, k, v, _cu(lens), grad, scale=0.11)
    want_out, _ = oat.segment_attention(q.cpu(), k.cpu(), v.cpu(), _cu(lens), 0.11)
    want = oat.segment_attention_backward(q.cpu(), k.cpu(), v.cpu(), _cu(lens), grad.cpu(), 0.11)
    assert_close_rel_max(out[:n_seg].float().cpu(), want_out[:n_seg].float(), 4e-3, "out")
    for name, got, exact in zip(("dq", "dk", "dv"), (dq[:n_seg], dk[:n_seg], dv[:n_seg]), want):
        assert_close_rel_max(got.float().cpu(), exact[:n_seg].float(), 4e-3, name)
    assert torch.isnan(out[n_seg:].float()).all()             # never touched
    for got in (dq, dk, dv):
        assert (got[n_seg:] == 0).all()                       # cleared, nothing added


def test_attention_kernels_refuse_what_they_do_not_cover():
    from claudemaxing_b200 import _lib

    q = torch.zeros(8, 2, 64, dtype=torch.float16, device=DEV)
    cu = torch.tensor([0, 8], dtype=torch.int32, device=DEV)
    out, lse = torch.empty_like(q), torch.empty(2, 8, device=DEV)
    with pytest.raises(RuntimeError, match="head_dim must be 128"):
        _lib.call("soup_attn_fwd", _lib.ptr(q), _lib.ptr(q), _lib.ptr(q), _lib.ptr(cu), _lib.ptr(out),
                  _lib.ptr(lse), 8, 1, 2, 2, 64, 128, 128, 128, 0.125, _lib.stream_of(q))
    q = torch.zeros(8, 3, 128, dtype=torch.float16, device=DEV)
    with pytest.raises(RuntimeError, match="multiple of key heads"):
        _lib.call("soup_attn_fwd", _lib.ptr(q), _lib.ptr(q), _lib.ptr(q), _lib.ptr(cu), _lib.ptr(q),
                  _lib.ptr(lse), 8, 1, 3, 2, 128, 384, 384, 384, 0.1, _lib.stream_of(q))


@pytest.mark.parametrize("pitch", [0, 64])
def test_gradients_pass_through_the_views_of_a_decoder_block(pitch):
    """[1, heads, tokens, 128] views of token-major rows (dense, or column blocks of a wider matrix): the
    numbers of the [tokens, heads, 128] form, and no gradient of another layout that views would copy."""
    from claudemaxing_b200.attention import SegmentAttention, segment_attention

    gen = torch.Generator().manual_seed(8)
    lens, heads = [130, 1, 77], (4, 2, 2)
    n = sum(lens)
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32).to(DEV)
    wide = [torch.randn(n, h * 128 + pitch, generator=gen).half().to(DEV) for h in heads]
    grad = torch.randn(1, n, heads[0], 128, generator=gen).half().to(DEV)
    flat = [w[:, :h * 128].unflatten(1, (h, 128)).detach().requires_grad_() for w, h in zip(wide, heads)]
    want = SegmentAttention.apply(*flat, cu, max(lens), 0.1)
    want.backward(grad[0])
    leaves = [w[:, :h * 128].unflatten(1, (h, 128)).detach().requires_grad_() for w, h in zip(wide, heads)]
    views = [x.unsqueeze(0).transpose(1, 2) for x in leaves]
    seen = []
    for x in views:
        x.register_hook(lambda g: seen.append(g.transpose(1, 2)[0].is_contiguous()))
    out = segment_attention(*views, cu, max(lens), 0.1)
    assert out.shape == (1, n, heads[0], 128) and torch.equal(out[0], want) and not out._is_view()
    out.backward(grad)
    assert seen == [True] * 3
    for x, w in zip(leaves, flat):   # sums of up to two tiles in any order
        assert (x.grad.float() - w.grad.float()).abs().max() <= 2e-3 * w.grad.float().abs().max()


def test_saved_tensors_may_come_back_as_contiguous_copies():
    """Under a saved-tensor hook the gradients are those without one (with pinned memory `save_on_cpu` brings back
    contiguous copies)."""
    from claudemaxing_b200.attention import segment_attention

    gen = torch.Generator().manual_seed(11)
    lens, heads = [130, 1, 77], (4, 2, 2)
    n = sum(lens)
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32).to(DEV)
    rows = [torch.randn(n, h, 128, generator=gen).half().to(DEV).requires_grad_() for h in heads]
    grad = torch.randn(1, n, heads[0], 128, generator=gen).half().to(DEV)

    def gradients():
        out = segment_attention(*(x.unsqueeze(0).transpose(1, 2) for x in rows), cu, max(lens), 0.1)
        return torch.autograd.grad(out, rows, grad)

    want = gradients()
    with torch.autograd.graph.save_on_cpu(pin_memory=True):
        got = gradients()
    for x, w in zip(got, want):   # sums of up to two tiles in any order
        assert (x.float() - w.float()).abs().max() <= 2e-3 * w.float().abs().max()


@pytest.mark.parametrize("heads,hq,hk,lens", [
    (2, 12, 2, [513] * 19 + [1, 129, 0]),        # several units an SM, walks of up to five tiles
    (3, 12, 2, [130] * 70),                      # more than 64 segments, walks of two tiles, one row in the last
    (2, 4, 2, [40] * 200),                       # walks of one tile: every step begins another head
    (4, 16, 4, [257] * 40),
])
def test_backward_of_several_heads_per_cta(heads, hq, hk, lens):
    """A CTA that walks its key/value tile for one head after another: gradients of every head against float64.
    Bound: fp16 P, dS and dO o O's rounding, as in the other tests here, 4e-3 of the largest."""
    import ctypes

    from claudemaxing_b200 import _lib
    from oracle.attention import segment_attention_backward

    n = sum(lens)
    plan = ctypes.c_int()
    _lib.call("soup_attn_plan", n, len(lens), hq, hk, None, ctypes.byref(plan))
    assert plan.value == heads
    gen = torch.Generator().manual_seed(heads)
    q, k, v, g = (torch.randn(n, h, 128, generator=gen).half() for h in (hq, hk, hk, hq))
    _, _, dq, dk, dv = _run(q.to(DEV), k.to(DEV), v.to(DEV), _cu(lens), g.to(DEV))
    want = segment_attention_backward(q, k, v, _cu(lens), g)
    for name, got, w in zip(("dq", "dk", "dv"), (dq, dk, dv), want):
        assert_close_rel_max(got.float().cpu(), w.float(), 4e-3, name)


@pytest.mark.parametrize("plain,bounded,hq,hk,lens", [
    (3, 1, 12, 2, [4096] + [20] * 100),          # more than 64 segments
    (2, 1, 12, 2, [20] * 10 + [2000] + [20] * 10),
    (3, 2, 12, 2, [512] * 2 + [64] * 30),
    (2, 3, 12, 2, [512] * 16),
])
def test_backward_planned_for_the_longest_segment(plain, bounded, hq, hk, lens):
    """One long segment among short ones has its heads apart (a CTA that walked three of them one after another would
    be the launch's end): the plan with the bound, and the same gradients. Bound: sums of up to 32 tiles in any
    order, in fp32, rounded to fp16."""
    import ctypes

    from claudemaxing_b200 import _lib
    from claudemaxing_b200.attention import SegmentAttention, attention_gradients

    n, longest = sum(lens), max(lens)
    heads = ctypes.c_int()
    for bound, want in ((0, plain), (longest, bounded)):
        _lib.call("soup_attn_plan_bounded", n, len(lens), bound, hq, hk, None, ctypes.byref(heads))
        assert heads.value == want
    gen = torch.Generator().manual_seed(len(lens))
    q, k, v, g = (torch.randn(n, h, 128, generator=gen).half().to(DEV) for h in (hq, hk, hk, hq))
    cu = _cu(lens).to(DEV)
    out, lse = _forward(q, k, v, cu)
    scale = 128 ** -0.5
    apart = attention_gradients(q, k, v, out, lse, g, cu, scale)
    together = attention_gradients(q, k, v, out, lse, g, cu, scale, longest)
    leaves = [t.clone().requires_grad_() for t in (q, k, v)]
    SegmentAttention.apply(*leaves, cu, longest, scale).backward(g)
    _lib.check_device_status()
    for a, b, leaf in zip(apart, together, leaves):
        largest = a.float().abs().max()
        assert (a.float() - b.float()).abs().max() <= 1e-3 * largest
        assert (leaf.grad.float() - b.float()).abs().max() <= 1e-3 * largest
