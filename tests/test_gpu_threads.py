"""Prompts of one model from several threads, each on a stream of its own, give what they give one after the other."""
import threading

import pytest
import torch

from chatrwkv_b200 import synth
from tests.golden.make_golden import TOY

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["v4", "v5", "v6"])
def test_threads_on_their_own_streams(name):
    from chatrwkv_b200.model import RWKV
    model = RWKV(synth.make_checkpoint(**TOY[name]), "cuda fp16i8", verbose=False)
    V = TOY[name]["vocab"]
    # a short prompt, a ragged chunk on its state, and one past the length from which an empty state changes kernels
    jobs = [[synth.make_tokens(n + k, V, 10 * n + k) for n in (600, 37, 9)] for k in range(4)]

    def one(job):
        out, state = [], None
        for ids in job:
            logits, state = model.forward(ids, state)
            out.append([logits.clone()] + [t.clone() for t in state])
        return out
    want = [one(job) for job in jobs]
    torch.cuda.synchronize()
    got, errors = [[] for _ in jobs], []

    def work(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(5):
                    got[k].append(one(jobs[k]))
                torch.cuda.current_stream().synchronize()
        except Exception as e:                               # (an assertion in a thread would be lost)
            errors.append(e)
    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for k, w in enumerate(want):
        for g in got[k]:
            for a, b in zip(g, w):
                assert all(torch.equal(x, y) for x, y in zip(a, b)), k
