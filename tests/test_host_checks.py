"""What the Python side refuses before a launch reads or writes anything, on CPU tensors with the
launches replaced by a recorder."""

import pytest
import torch

from claudemaxing_b200 import _lib
from claudemaxing_b200 import lm_head_loss as L


@pytest.fixture
def launches(monkeypatch):
    """The entry points that were called, in order; none of them runs."""
    made = []
    monkeypatch.setattr(_lib, "call", lambda name, *args: made.append((name, args)))
    monkeypatch.setattr(_lib, "require_cuda", lambda *tensors: None)
    monkeypatch.setattr(_lib, "stream_of", lambda t: None)
    return made


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
