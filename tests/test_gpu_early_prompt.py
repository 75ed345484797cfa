"""Short RWKV-5/6 prompts: which sums they get follows from the state's content, not from how it is passed."""
import pytest
import torch

from chatrwkv_b200 import synth
from tests.golden.make_golden import TOY

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [2, 9, 100, 511, 512, 600])
@pytest.mark.parametrize("name", ["v4", "v5", "v6"])
def test_no_state_and_a_zero_state_are_the_same_prompt(name, T):
    from chatrwkv_b200.model import RWKV
    model = RWKV(synth.make_checkpoint(**TOY[name]), "cuda fp16i8", verbose=False)
    ids = synth.make_tokens(T, TOY[name]["vocab"], T)
    l0, s0 = model.forward(ids, None, full_output=True)
    l1, s1 = model.forward(ids, [t.clone() for t in model._zero_state()], full_output=True)
    assert torch.equal(l0, l1)
    assert all(torch.equal(a, b) for a, b in zip(s0, s1))


@pytest.mark.parametrize("name", ["v5", "v6"])
def test_initial_state_is_recognised(name):
    from chatrwkv_b200.model import RWKV
    model = RWKV(synth.make_checkpoint(**TOY[name]), "cuda fp16i8", verbose=False)
    assert model._is_initial(model._zero_state())
    _, state = model.forward([5], None)
    state = [t.clone() for t in state]
    assert not model._is_initial(state)
    zeroed = [t.zero_() for t in state]
    assert model._is_initial(zeroed)
