"""RWKV-5/6 prompts through the grouped launches (mixes, r / k / v / g, group norm + gate, head) against the oracle and against
the separate launches: prompts past EARLY_PROMPT, a second chunk on a carried state, and short prompts with the rule off."""
import copy

import pytest
import torch

from chatrwkv_b200 import ops, synth
from oracle import rwkv_oracle as orc
from tests.golden.make_golden import TOY

pytestmark = pytest.mark.gpu
TOL = 2e-2                                                   # logits, as in the other comparisons with the oracle


@pytest.mark.parametrize("chunks", [(520,), (40, 25), (1, 30)])
@pytest.mark.parametrize("name", ["v5", "v6"])
def test_prompts_on_the_grouped_launches(name, chunks, monkeypatch):
    from chatrwkv_b200.model import RWKV
    ck = synth.make_checkpoint(**TOY[name])
    model = RWKV(copy.deepcopy(ck), "cuda fp16i8", verbose=False)
    model.EARLY_PROMPT = 0
    oracle = orc.OracleRWKV(ck, atype=torch.float16)
    launched = []
    batch = ops.mm8_seq_batch
    monkeypatch.setattr(ops, "mm8_seq_batch", lambda *a: launched.append(batch(*a)) or launched[-1])
    state = ostate = sstate = None
    for k, T in enumerate(chunks):
        ids = synth.make_tokens(T, TOY[name]["vocab"], 31 * k + T)
        logits, state = model.forward(ids, state, full_output=True)
        state = [t.clone() for t in state]
        if T > 1:
            assert launched and all(launched)
        with monkeypatch.context() as m:                     # the separate launches on the same input
            m.setattr(ops, "mm8_seq_batch", lambda *a: False)
            slogits, sstate = model.forward(ids, sstate, full_output=True)
            sstate = [t.clone() for t in sstate]
        lo, ostate = oracle.forward(ids, ostate, full_output=True)
        lo = lo.reshape(-1, lo.shape[-1])
        for got in (logits, slogits):
            assert (got.reshape(lo.shape).cpu() - lo).abs().max().item() < TOL
    for a, b in zip(state, sstate):
        assert (a.float() - b.float()).abs().max().item() <= 2e-2 * max(1.0, b.float().abs().max().item())
