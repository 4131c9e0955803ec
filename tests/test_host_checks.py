"""What the Python side refuses before a launch reads or writes anything, on CPU tensors with the
launches replaced by a recorder, and the plans the library makes on the host."""

import ctypes
from types import SimpleNamespace

import pytest
import torch

from claudemaxing_b200 import _lib
from claudemaxing_b200 import decoder_block as D
from claudemaxing_b200 import lm_head_loss as L


@pytest.fixture
def launches(monkeypatch):
    """The entry points that were called, in order; none of them runs."""
    made = []
    monkeypatch.setattr(_lib, "call", lambda name, *args: made.append((name, args)))
    monkeypatch.setattr(_lib, "require_cuda", lambda *tensors: None)
    monkeypatch.setattr(_lib, "stream_of", lambda t: None)
    return made


def test_a_cpu_tensor_has_no_stream(monkeypatch):
    """A launch whose operands nobody else has checked ends here, not on a stream with host pointers."""
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda index: 0, raising=False)
    with pytest.raises(ValueError, match="cpu"):
        _lib.stream_of(torch.zeros(2))


@pytest.mark.parametrize("targets", [7, 9, 12])
@pytest.mark.parametrize("grad", [True, False])
def test_head_refuses_a_target_of_another_length_than_the_hidden_states(launches, targets, grad):
    hidden = torch.randn(1, 8, 64).half().requires_grad_(grad)
    weight = torch.randn(300, 64).half()
    target = torch.zeros(1, targets, dtype=torch.int64)
    with pytest.raises(RuntimeError, match="targets for 8 rows"):
        L.fused_head_loss(hidden, weight, None, target=target)
    with pytest.raises(RuntimeError, match="targets for 8 rows"):
        L.head_partial(hidden.detach()[0], weight, target.reshape(-1), want_grad=grad)
    with pytest.raises(RuntimeError, match="targets for 8 rows"):
        L.head_finish(L.HeadState(8, "cpu"), target.reshape(-1), weight)
    assert not launches
    L.fused_head_loss(hidden, weight, None, target=torch.zeros(1, 8, dtype=torch.int64))
    assert [name for name, _ in launches] == ["soup_lmhead_ce", "soup_lmhead_finish", "soup_lmhead_totals"]


def test_head_gradient_of_several_losses_is_refused(launches):
    """A divisor of several elements makes a loss of several; its gradient is no single factor."""
    def loss_of(divisor):
        hidden = torch.randn(1, 8, 64).half().requires_grad_()
        return L.fused_head_loss(hidden, torch.randn(300, 64).half(), None, num_items_in_batch=divisor,
                                 target=torch.zeros(1, 8, dtype=torch.int64))[0]

    several = loss_of(torch.tensor([2.0, 4.0]))
    assert several.shape == (2,)
    with pytest.raises(RuntimeError, match="one loss"):
        several.sum().backward()
    assert "soup_lmhead_backward" not in [name for name, _ in launches]
    for divisor in (None, 3, torch.tensor([2.0]), torch.tensor(2.0)):
        loss_of(divisor).sum().backward()
    assert [name for name, _ in launches].count("soup_lmhead_backward") == 4


def _head_plan(rows, columns, chunk_tiles=0):
    """(rows per block, column tiles of the first chunk, of a later one); without a device the library
    plans for 148 SMs."""
    out = [ctypes.c_int64() for _ in range(3)]
    _lib.lib().soup_lmhead_plan(rows, columns, chunk_tiles, *(ctypes.byref(x) for x in out))
    return tuple(x.value for x in out)


@pytest.mark.parametrize("columns", [300, 32000, 50257, 151936])
def test_head_rounds_no_more_of_the_vocabulary_twice_than_37_tiles(columns):
    """The first chunk's probabilities are rounded against their tile's maximum and again after the merge."""
    for rows in (1, 24, 128, 256, 257, 512, 600, 1168, 2048, 4096, 8192):
        first = _head_plan(rows, columns)[1]
        assert 1 <= first <= 37, rows


def test_head_row_block_follows_the_waves_a_chunk_may_have(monkeypatch):
    """Rows per block: twice the column tiles of so many waves of 74 pairs at eight row tiles, over the
    shard's tiles (594 at full width, 75 of eight ranks), in multiples of 2048 up to 8192."""
    def blocks():
        return [_head_plan(65536, columns)[0] for columns in (151936, 37984, 18992)]

    assert blocks() == [4096, 6144, 8192]
    monkeypatch.setenv("SOUP_LMHEAD_WAVES", "4")
    assert blocks() == [4096, 4096, 6144]
    monkeypatch.setenv("SOUP_LMHEAD_WAVES", "16")
    assert blocks() == [4096, 8192, 8192]


@pytest.mark.parametrize("rows", [1, 128, 1168, 2048, 8192])
def test_head_workspace_holds_no_more_probabilities_than_a_chunk_has(launches, rows):
    """bf16 probabilities of the largest chunk with the gradient, none without; a call is handed the
    workspace of its own kind."""
    block, first, later = _head_plan(rows, 151936)
    assert later == max(first, -(-(594 - first) // -(-(594 - first) // later)))   # equal chunks, none larger
    lib = _lib.lib()
    full = lib.soup_lmhead_workspace_bytes(rows, 64, 151936, 0)
    forward = lib.soup_lmhead_forward_workspace_bytes(rows, 64, 151936, 0)
    assert full - forward == -(-block * later * 512 // 1024) * 1024
    assert forward <= block * (later * 16 + 4) + 4096
    hidden, weight = torch.zeros(rows, 64).half(), torch.zeros(300, 64).half()
    for grad in (True, False):
        L.head_partial(hidden, weight, torch.zeros(rows, dtype=torch.int64), want_grad=grad,
                       w_bf16=weight.bfloat16())
        _, args = launches.pop()
        wanted = lib.soup_lmhead_workspace_bytes if grad else lib.soup_lmhead_forward_workspace_bytes
        assert args[13] == wanted(rows, 64, 300, 0)


def test_nf4_batch_takes_one_offset_per_weight(launches, monkeypatch):
    from types import SimpleNamespace

    from claudemaxing_b200 import nf4

    def weight(offset):
        second = SimpleNamespace(code=torch.zeros(256), absmax=torch.zeros(1), blocksize=256)
        state = SimpleNamespace(shape=(2, 64), dtype=torch.float16, nested=True, blocksize=64, code=torch.zeros(16),
                                absmax=torch.zeros(2, dtype=torch.uint8), state2=second, offset=offset)
        return torch.zeros(64, dtype=torch.uint8), state

    for offset in (torch.tensor(0.5), torch.tensor([0.5]), 0.5, torch.tensor(0.5, dtype=torch.float64)):
        assert nf4.dequantize_nf4_batch([weight(offset)])[0].shape == (2, 64)
    with pytest.raises(RuntimeError):
        nf4.dequantize_nf4_batch([weight(torch.tensor([0.5, 0.25]))])
    assert [name for name, _ in launches] == ["soup_nf4_dequant_batch"] * 4


class _Projection:
    def __init__(self, out_features, weight):
        self.out_features, self.group, self._weight = out_features, self, weight

    def stacked(self, bases, dtype):
        return self._weight


class _Plan:
    head_dim = 16

    def __init__(self, heads, kv_heads, hidden):
        weight = torch.randn((heads + 2 * kv_heads) * 16, hidden).half()
        self.q, self.k, self.v = (_Projection(h * 16, weight) for h in (heads, kv_heads, kv_heads))

    @staticmethod
    def qkv_bias(device):
        return None


def _qkv(lora_q_width=64, lora_v_width=32, tables=((1, 5, 16), (1, 5, 16))):
    x = torch.randn(1, 5, 32, requires_grad=True)
    lora_q, lora_v = (torch.randn(1, 5, width).half() for width in (lora_q_width, lora_v_width))
    cos, sin = (torch.randn(*shape) for shape in tables)
    return D._QKVRope.apply(x, x.detach().half(), lora_q, lora_v, cos, sin, _Plan(4, 2, 32)), cos, sin


def test_qkv_split_reads_adapter_terms_and_tables_of_its_own_shape_and_device_only(launches, monkeypatch):
    """The launch takes bare pointers: an adapter term narrower than its projection is refused, tables
    of another shape go to the rotation that reads their strides, and every tensor that is read has
    been checked to be on the device."""
    checked = []
    monkeypatch.setattr(_lib, "require_cuda", lambda *tensors: checked.extend(tensors))
    (q, k, v), cos, sin = _qkv()
    assert [name for name, _ in launches] == ["soup_qkv_rope_fwd"]
    assert any(t is cos for t in checked) and any(t is sin for t in checked)
    assert q.shape == (5, 4, 16) and k.shape == v.shape == (5, 2, 16)
    for width in (dict(lora_q_width=48), dict(lora_v_width=16), dict(lora_q_width=80)):
        with pytest.raises(RuntimeError, match="invalid for input of size"):
            _qkv(**width)
    launches.clear()
    _qkv(tables=((1, 5, 16), (1, 5, 8)))
    assert [name for name, _ in launches] == ["soup_rope_sum"]


def test_mlp_kernels_take_operands_of_one_device_only():
    """A launch reaches one device: operands of two go to the library's products, which refuse them."""
    rows = torch.zeros(2944, 768, dtype=torch.float16)
    weights = [torch.zeros(*shape, dtype=torch.float16) for shape in ((3072, 768), (3072, 768), (768, 3072))]
    residual = torch.zeros(2944, 768)
    away = torch.device("meta")
    assert D._mlp_kernels_cover(rows, weights, False, residual)
    assert not D._mlp_kernels_cover(rows, weights, False, residual.to(away))
    for i in range(3):
        mixed = [w.to(away) if i == j else w for j, w in enumerate(weights)]
        assert not D._mlp_kernels_cover(rows, mixed, False, residual)


def test_mlp_residual_is_as_wide_as_the_output(launches):
    """As many elements in rows of another width: the library's product refuses them, no launch is made."""
    weights = [torch.zeros(*shape, dtype=torch.float16) for shape in ((3072, 768), (3072, 768), (768, 3072))]
    gate, up, down = (SimpleNamespace(dequantized=lambda dtype, w=w: w) for w in weights)
    plan = SimpleNamespace(gate=gate, up=up, down=down, keep_products=True)
    x = torch.zeros(1, 2944, 768)
    D._GatedMLPAddResidual.apply(x, x.half(), torch.zeros(1, 2944, 768), plan)
    assert [name for name, _ in launches] == ["soup_mlp_fwd"]
    del launches[:]
    with pytest.raises(RuntimeError):
        D._GatedMLPAddResidual.apply(x, x.half(), torch.zeros(1, 1472, 1536), plan)
    assert not any(args[8] is not None for name, args in launches if name == "soup_mlp_fwd")   # no output


@pytest.mark.parametrize("longest,entry", [(4096, "soup_attn_bwd_bounded"), (0, "soup_attn_bwd")])
def test_segment_attention_backward_knows_the_longest_segment(launches, longest, entry):
    """The bound reaches the launch where it changes its plan (12 query heads, 2 key heads, a long segment among
    a hundred short ones)."""
    from claudemaxing_b200 import attention as A

    n, cu = 6096, torch.tensor([0, 4096] + [4096 + 20 * (i + 1) for i in range(100)], dtype=torch.int32)
    q, k, v = (torch.zeros(n, h, 128, dtype=torch.float16, requires_grad=True) for h in (12, 2, 2))
    A.SegmentAttention.apply(q, k, v, cu, longest, 0.1).backward(torch.zeros(n, 12, 128, dtype=torch.float16))
    name, args = launches[-1]
    assert name == entry and args[12:14] == (n, 101)
    if longest:
        assert args[14] == longest


@pytest.mark.parametrize("hidden,inter,slower,faster", [
    (1536, 8960, [512, 896, 1152], [1280, 1408, 3072, 4608, 16384]),
    (2048, 11008, [512, 1280], [1024, 2048, 3072, 8192]),
    (3584, 18944, [768, 896], [1280, 2304, 8192]),
    (4096, 14336, [896, 1152], [2048, 8192]),
    (5120, 27648, [896, 1024], [1280, 4096]),
    (8192, 28672, [512, 1152], [1280, 4096]),
])
def test_mlp_launches_pay_where_both_directions_measured_faster(hidden, inter, slower, faster):
    pays = _lib.lib().soup_mlp_pays
    for backward in (0, 1):
        assert [pays(rows, hidden, inter, backward) for rows in slower] == [0] * len(slower)
        assert [pays(rows, hidden, inter, backward) for rows in faster] == [1] * len(faster)
