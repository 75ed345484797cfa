"""rwkv_mm8_seq_batch (grouped matmuls with the prologues in the operand pass) and rwkv_wkv56_one_rows against the separate
calls they replace, at row lengths on both sides of the preparation's forms."""
import pytest
import torch

from tests.util import packed_case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from chatrwkv_b200 import ops as o
    return o


def _table(mats, N, kind, **common):
    from chatrwkv_b200 import _lib
    arr = (_lib.Mm8SeqProblem * len(mats))()
    for q, (wq, mx, rx, my, ry) in zip(arr, mats):
        q.w, q.w_stride, q.M = wq.data_ptr(), wq.stride(0), wq.shape[1]
        q.mx, q.rx, q.my, q.ry = mx.data_ptr(), rx.data_ptr(), my.data_ptr(), ry.data_ptr()
        q.epilogue, q.out_scale, q.kind = _lib.EPI_STORE, 1.0, kind
        for k, v in common.items():
            setattr(q, k, v)
    return arr


def _close(got, want):
    # The prologue's sums run in another order: a value may fall one fp16 step (2^-10 of itself at most) the other way before
    # the matmul.  Were every value to, the dot product would move by 2^-10 of its root mean square (rms below); single results
    # by a few times that, and by their own store's rounding of values several times the root mean square: 8 times in all.
    rms = want.float().pow(2).mean().sqrt()
    assert torch.isfinite(got).all() and (got.float() - want.float()).abs().max() <= 2 ** -7 * rms
    assert (got.float() - want.float()).pow(2).mean().sqrt() <= 2 ** -10 * rms


# forms of the operand pass: E = 4 / 8 / 16 channels a thread by the row length with few rows, 256, 512 and 1024 threads with many
@pytest.mark.parametrize("T,N", [(2, 300), (16, 768), (40, 4096), (5, 5120), (120, 8064), (300, 1024), (310, 4100), (170, 8200), (4, 16000)])
@pytest.mark.parametrize("mode,rows", [(0, True), (0, False), (1, False), (2, True)])
def test_layer_norm_mix(ops, T, N, mode, rows):
    from chatrwkv_b200 import _lib
    from chatrwkv_b200._lib import check, lib
    g = torch.Generator(device="cuda").manual_seed(T + N + mode)
    h = lambda *s: torch.randn(*s, generator=g, device="cuda").half()
    mats = [packed_case(N, M, seed=M)[1] for M in ((264, 128, 40, 16) if mode == 0 and rows else (264, 128) if mode != 2 else (264,))]
    x, sx, lw, lb = h(T, N), (h(T, N) if rows else h(N)), h(N), h(N)
    mix = [torch.rand(N, generator=g, device="cuda").half() for _ in mats]
    xx, ns = torch.empty(T, N, dtype=torch.float16, device="cuda"), torch.empty(N, dtype=torch.float16, device="cuda")
    arr = _table(mats, N, _lib.PRO_LN_MIX, mode=mode, x=x.data_ptr(), x_stride=N, ln_w=lw.data_ptr(), ln_b=lb.data_ptr())
    ys = [torch.empty(T, m[0].shape[1], dtype=torch.float16, device="cuda") for m in mats]
    for q, y, m in zip(arr, ys, mix):
        q.y, q.y_stride = y.data_ptr(), y.stride(0)
        if mode != 2:
            q.mix = m.data_ptr()
    arr[0].xx_out, arr[0].xx_stride, arr[0].new_state = xx.data_ptr(), N, ns.data_ptr()
    if mode != 2:
        arr[0].sx, arr[0].sx_stride = sx.data_ptr(), (N if rows else 0)
    assert ops.mm8_seq_batch(arr, len(mats), T, N, x.device)
    outs = [torch.empty_like(x) for _ in mats]
    xx2 = torch.empty_like(x)
    if N > 8192:                                             # past rwkv_ln_mix's rows: torch, one fp16 rounding per operation
        xx2 = torch.nn.functional.layer_norm(x.float(), (N,), lw.float(), lb.float(), 1e-5).half()
        prev = sx if rows else torch.cat((sx[None], xx2[:-1]))
        outs = [xx2 * m + prev * (1 - m) if mode == 0 else xx2 + (prev - xx2) * m for m in mix] if mode != 2 else []
    else:
        ptrs = lambda ts: (__import__("ctypes").c_void_p * len(ts))(*[t.data_ptr() for t in ts])
        check(lib().rwkv_ln_mix_rows(T, N, x.data_ptr(), N, sx.data_ptr() if mode != 2 else None, N if rows and mode != 2 else 0,
                                     lw.data_ptr(), lb.data_ptr(), 0 if mode == 2 else mode, 0 if mode == 2 else len(mats), ptrs(mix), 0,
                                     ptrs(outs), N, xx2.data_ptr(), N, None, torch.cuda.current_stream().cuda_stream), "ln_mix")
    if mode == 2:
        outs = [xx2]
    torch.cuda.synchronize()
    assert (xx.float() - xx2.float()).abs().max() <= 2 ** -10 * xx2.abs().max().float()
    assert torch.equal(ns, xx[-1])
    for y, o, m in zip(ys, outs, mats):
        want = torch.empty_like(y)
        torch.ops.rwkv.mm8_seq(T, N, y.shape[1], o, *m, want)
        _close(y, want)


@pytest.mark.parametrize("T,N", [(3, 320), (16, 4096), (9, 5120), (2, 512), (310, 1024), (300, 4096), (300, 8192), (3, 8320), (5, 10240)])
def test_wkv4_step_and_group_norm_gate(ops, T, N):
    from chatrwkv_b200 import _lib
    from chatrwkv_b200._lib import check, lib
    g = torch.Generator(device="cuda").manual_seed(T + N)
    f = lambda *s: torch.randn(*s, generator=g, device="cuda")
    mat = packed_case(N, 200, seed=N)[1]
    y, want = (torch.empty(T, 200, dtype=torch.float16, device="cuda") for _ in range(2))
    r, k, v, td, tf = f(T, N).sigmoid().half(), f(T, N).half(), f(T, N).half(), -f(N).exp(), f(N)
    st = [f(T, N), f(T, N).abs() + 1, f(T, N)]
    st2 = [t.clone() for t in st]
    arr = _table([mat], N, _lib.PRO_WKV4, x=r.data_ptr(), x_stride=N, k=k.data_ptr(), v=v.data_ptr(), t_decay=td.data_ptr(),
                 t_first=tf.data_ptr(), aa=st[0].data_ptr(), bb=st[1].data_ptr(), pp=st[2].data_ptr(), y=y.data_ptr(), y_stride=200)
    assert ops.mm8_seq_batch(arr, 1, T, N, y.device)
    o = torch.empty_like(r)
    ops.wkv4_seq(td, tf, k.view(T, 1, N), v.view(T, 1, N), o.view(T, 1, N), *st2, r=r.view(T, 1, N))
    torch.ops.rwkv.mm8_seq(T, N, 200, o, *mat, want)
    _close(y, want)
    for a, b in zip(st, st2):
        torch.testing.assert_close(a, b, rtol=1e-6, atol=1e-6)
    for head in [h for h in (16, 32, 64, 128) if N % h == 0]:
        x, gate, lw, lb = f(T, N), f(T, N).half(), f(N), f(N)
        gate[T // 2, 5] = 3000.0                             # an outlier channel: the row takes a fourth digit
        arr = _table([mat], N, _lib.PRO_GN_GATE, x=x.data_ptr(), x_stride=N, gate=gate.data_ptr(), gate_stride=N, head=head, eps=64e-5,
                     ln_w=lw.data_ptr(), ln_b=lb.data_ptr(), y=y.data_ptr(), y_stride=200)
        assert ops.mm8_seq_batch(arr, 1, T, N, y.device)
        check(lib().rwkv_v56_seq_gn_gate(T, N // head, head, x.data_ptr(), lw.data_ptr(), lb.data_ptr(), gate.data_ptr(), o.data_ptr(),
                                         64e-5, torch.cuda.current_stream().cuda_stream), "gn_gate")
        torch.ops.rwkv.mm8_seq(T, N, 200, o, *mat, want)
        _close(y, want)


@pytest.mark.parametrize("per_row", [0, 1])
@pytest.mark.parametrize("B,H,N", [(1, 3, 64), (5, 2, 32), (3, 4, 128)])
def test_wkv56_rows_equal_single_sequences(ops, B, H, N, per_row):
    from chatrwkv_b200._lib import check, lib
    g = torch.Generator(device="cuda").manual_seed(B * N)
    f = lambda *s: torch.randn(*s, generator=g, device="cuda")
    r, k, v, gate = (f(B, H * N).half() for _ in range(4))
    w, u, lw, lb = f(B if per_row else 1, H * N).sigmoid(), f(H * N), f(H * N), f(H * N)
    S = f(B, H, N, N)
    out, S2 = torch.empty_like(r), S.clone()
    st = torch.cuda.current_stream().cuda_stream
    check(lib().rwkv_wkv56_one_rows(B, H, N, r.data_ptr(), k.data_ptr(), v.data_ptr(), w.data_ptr(), per_row, u.data_ptr(), S2.data_ptr(),
                                    S2.data_ptr(), lw.data_ptr(), lb.data_ptr(), gate.data_ptr(), out.data_ptr(), st), "rows")
    for b in range(B):
        o, s = torch.empty_like(out[b]), torch.empty_like(S[b])
        check(lib().rwkv_wkv56_one(H, N, r[b].data_ptr(), k[b].data_ptr(), v[b].data_ptr(), w[b if per_row else 0].data_ptr(), u.data_ptr(),
                                   S[b].data_ptr(), s.data_ptr(), lw.data_ptr(), lb.data_ptr(), gate[b].data_ptr(), o.data_ptr(), st), "one")
        torch.cuda.synchronize()
        assert torch.equal(out[b], o) and torch.equal(S2[b], s)
