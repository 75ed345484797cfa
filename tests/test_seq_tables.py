"""The tables of the grouped prompt launches (RWKV._seq_group): host logic, run without a GPU on a stub of the launch."""
import threading
import time

import pytest
import torch

from chatrwkv_b200 import _lib, ops
from chatrwkv_b200.model import RWKV

N, M = 32, 16


@pytest.fixture
def model():
    m = RWKV.__new__(RWKV)
    m._world, m._seq_tables, m._mm = 1, {}, {}
    m.w = {"ln.weight": torch.ones(N, dtype=torch.float16), "ln.bias": torch.zeros(N, dtype=torch.float16)}
    for name in ("r", "k"):
        m.w["mix_" + name] = torch.rand(N).half()
        m.w[name] = torch.zeros((N, M), dtype=torch.uint8)
        for s, n in (("_mx", M), ("_rx", M), ("_my", N), ("_ry", N)):
            m.w[name + s] = torch.zeros(n, dtype=torch.float16)
    return m


def _group(model, x, sx):
    return model._ln_mix_group(x, sx, False, [("r", _lib.EPI_SIGMOID), ("k", _lib.EPI_STORE)], 0, ("ln.weight", "ln.bias"),
                               ["mix_r", "mix_k"])


def test_threads_launch_with_their_own_pointers(model, monkeypatch):
    """Calls that overlap in time (the launch lets other threads run) never see each other's activations."""
    mine, wrong = threading.local(), []

    def launch(arr, n, T, D, device):
        for _ in range(3):
            x, sx = mine.now
            if any(q.x != x.data_ptr() for q in arr) or arr[0].sx != sx.data_ptr():
                wrong.append(T)
            time.sleep(0)
        return True
    monkeypatch.setattr(ops, "mm8_seq_batch", launch)

    def work(T):
        for _ in range(200):
            mine.now = torch.zeros((T, N), dtype=torch.float16), torch.zeros(N, dtype=torch.float16)
            outs, _ = _group(model, *mine.now)
            assert [tuple(o.shape) for o in outs] == [(T, M)] * 2
    threads = [threading.Thread(target=work, args=(T,)) for T in (3, 5, 9, 17)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_replaced_norms_and_mixes_are_seen(model, monkeypatch):
    """An entry of `model.w` that a program replaces after the first prompt: the next launch reads the new tensor (the old one's
    memory may be gone)."""
    seen = []

    def launch(arr, n, T, D, device):
        seen.append([arr[0].ln_w, arr[0].ln_b] + [q.mix for q in arr])
        return True
    monkeypatch.setattr(ops, "mm8_seq_batch", launch)
    x, sx = torch.zeros((4, N), dtype=torch.float16), torch.zeros(N, dtype=torch.float16)
    keep = []
    for _ in range(2):
        _group(model, x, sx)
        names = ("ln.weight", "ln.bias", "mix_r", "mix_k")
        assert seen[-1] == [model.w[k].data_ptr() for k in names]
        for k in names:
            keep.append(model.w[k])
            model.w[k] = model.w[k].clone()


def test_batched_rwkv4_step_refuses_states_that_are_not_fp32(monkeypatch):
    """The recurrence inside the operand pass reads and writes fp32: a program that stores its sessions in fp16 gets an error."""
    m = RWKV.__new__(RWKV)
    m._world, m._seq_tables, m._mm, m.args = 1, {}, {}, None
    bb, att = "blocks.0.", "blocks.0.att."
    m.w = {bb + "ln1.weight": torch.ones(N).half(), bb + "ln1.bias": torch.zeros(N).half(), att + "time_decay": torch.zeros(N),
           att + "time_first": torch.zeros(N)}
    for n in ("k", "v", "r"):
        m.w[att + "time_mix_" + n] = torch.rand(N).half()
    for n in ("receptance", "key", "value", "output"):
        m.w[att + n + ".weight"] = torch.zeros((N, N), dtype=torch.uint8)
        for s in ("_mx", "_rx", "_my", "_ry"):
            m.w[att + n + ".weight" + s] = torch.zeros(N, dtype=torch.float16)
    monkeypatch.setattr(ops, "mm8_seq_batch", lambda *a: True)
    x, sx = torch.zeros((3, N), dtype=torch.float16), torch.zeros((3, N), dtype=torch.float16)
    f32 = [torch.zeros(3, N) for _ in range(3)]
    m._att_seq_v4(x, [sx] + f32 + [sx], 0, rows=True)
    for i in range(3):
        bad = list(f32)
        bad[i] = bad[i].half()
        with pytest.raises(_lib.RwkvB200Error, match="fp32"):
            m._att_seq_v4(x, [sx] + bad + [sx], 0, rows=True)


@pytest.mark.parametrize("rows", [False, True])
def test_rwkv56_states_that_are_not_fp32_are_refused(rows):
    m = RWKV.__new__(RWKV)
    x, sx = torch.zeros((3, N), dtype=torch.float16), torch.zeros(N, dtype=torch.float16)
    with pytest.raises(_lib.RwkvB200Error, match="fp32"):
        m._att_seq_v56(x, [sx, torch.zeros((2, 16, 16), dtype=torch.float16)], 0, rows=rows)
