"""Small-batch recurrences (weights and the step hand-off inside one cluster of 1 to 16 CTAs) at the edges of their
tiles: against fp32 step-by-step maths and bit for bit over repeats and batch shards."""
import ctypes

import pytest
import torch

from fastlstm_b200 import _lib
from test_gpu_recurrence import TD, _bwd, _cmp, _desc, _fwd, _torch_bwd, _torch_fwd

pytestmark = pytest.mark.gpu

# (T, B, H): one CTA with 1, 3 and 8 unit groups; several chunks; clusters of 3, 4, 6, 8 with whole and partial last
# CTAs; K split over two warps (11 to 16 CTAs, K steps in odd halves); weights partly in shared memory; batches of
# one row, one row past a chunk, chunks shared by replicas
SHAPES = [(5, 3, 8), (4, 9, 24), (9, 1300, 64), (3, 1, 64), (5, 33, 72), (6, 270, 128), (4, 17, 136), (7, 120, 200),
          (5, 360, 256), (1, 9, 256), (6, 8, 264), (4, 57, 288), (5, 100, 384), (3, 40, 448), (6, 110, 512), (2, 1, 512),
          (4, 15, 520), (3, 50, 640), (4, 9, 768),
          # as many chunks a cluster as the dispatch gives them: 4 and 3
          (4, 480, 256), (4, 224, 320), (3, 168, 448)]


def _plan(d, phase):
    buf = ctypes.create_string_buffer(512)
    assert _lib.load().blstm_plan_detail(d, phase, buf, 512) == 0
    return buf.value.decode()


@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
@pytest.mark.parametrize("shape", SHAPES)
def test_small_batch_recurrences_against_fp32_maths(dtype, shape):
    lib, (T, B, H), dt = _lib.load(), shape, TD[dtype]
    g = torch.Generator(device="cuda").manual_seed(B * 31 + H)
    r = lambda *s, std=1.0: (torch.randn(*s, generator=g, device="cuda") * std).to(dt)
    pre, h0, c0 = r(T, B, 4 * H), r(B, H, std=0.3), r(B, H, std=0.3)
    dout, dh_n, dc_n = r(T, B, H), r(B, H), r(B, H)
    Wh = ((torch.rand(4 * H, H, generator=g, device="cuda") * 2 - 1) / H ** 0.5).to(dt)
    d = _desc(dtype, T, B, H)
    assert "small-batch" in _plan(d, 0)
    ifgo, out, cell = _fwd(lib, d, pre, Wh, h0, c0)
    rg, ro, rc = _torch_fwd(pre, Wh, h0, c0)
    tol = 4e-3 if dtype == "fp16" else 3e-2
    _cmp("ifgo", ifgo, rg, tol * 4)
    _cmp("out", out[1:], ro, tol)
    _cmp("cell", cell[1:], rc, tol * 2)
    infer = _fwd(lib, _desc(dtype, T, B, H, _lib.FLAG_INFERENCE), pre, Wh, h0, c0)
    assert torch.equal(infer[1], out) and torch.equal(infer[2][T], cell[T]) and torch.equal(infer[0], pre)
    n = (B + 1) // 2                                   # a shard of the rows sums in the same order
    part = _fwd(lib, _desc(dtype, T, n, H), pre[:, :n].contiguous(), Wh, h0[:n].contiguous(), c0[:n].contiguous())
    assert torch.equal(part[1], out[:, :n]) and torch.equal(part[2][1:], cell[1:, :n])
    if H > 640:
        return
    assert "small-batch" in _plan(d, 1)
    got = _bwd(lib, d, dout, dh_n, dc_n, ifgo, cell, Wh)
    wg, wh, wc = _torch_bwd(dout, dh_n, dc_n, ifgo, cell, Wh)
    tol = 6e-3 if dtype == "fp16" else 4e-2
    for name, a, b in (("d_ifgo", got[0], wg), ("dh0", got[1][None], wh[None]), ("dc0", got[2][None], wc[None])):
        _cmp(name, a, b, tol * max(float(b.float().abs().max()), 1.0))
    assert torch.allclose(got[3], got[0].float().sum(dim=(0, 1)), rtol=1e-4, atol=1e-3 * T * B ** 0.5)
    again = _bwd(lib, d, dout, dh_n, dc_n, ifgo, cell, Wh)
    assert all(torch.equal(a, b) for a, b in zip(got, again))


@pytest.mark.parametrize("phase", ["fwd", "bwd"])
@pytest.mark.parametrize("shape", [(5, 9, 256), (5, 40, 512)])
def test_small_batch_recurrences_give_up_with_a_status_when_nothing_arrives(phase, shape):
    """With the arrivals suppressed every wait runs out (20 ms), the blocks leave together and the next launch works."""
    lib, (T, B, H) = _lib.load(), shape
    z = lambda *s: torch.zeros(*s, device="cuda", dtype=torch.bfloat16)
    s = torch.cuda.current_stream().cuda_stream
    ph = _lib.PHASE_FWD if phase == "fwd" else _lib.PHASE_BWD
    ifgo, out, cell, Wh, dg, dh0, dc0 = (z(T, B, 4 * H), z(T + 1, B, H), z(T + 1, B, H), z(4 * H, H), z(T, B, 4 * H), z(B, H), z(B, H))
    for flags, want in ((_lib.FLAG_TEST_NO_ARRIVE, _lib.E_WAIT_TIMEOUT), (0, 0)):
        d = _lib.Desc(_lib.BF16, T, B, H, H, flags, 20000, 0)
        assert "small-batch" in _plan(d, ph)
        n = lib.blstm_workspace_bytes(d, ph)
        ws = torch.zeros(n, dtype=torch.uint8, device="cuda")
        if phase == "fwd":
            rc = lib.blstm_fwd_recurrence(d, ifgo.data_ptr(), Wh.data_ptr(), out.data_ptr(), cell.data_ptr(), ws.data_ptr(), n, s)
        else:
            rc = lib.blstm_bwd_recurrence(d, out.data_ptr(), None, None, ifgo.data_ptr(), cell.data_ptr(), Wh.data_ptr(),
                                          dg.data_ptr(), dh0.data_ptr(), dc0.data_ptr(), None, ws.data_ptr(), n, s)
        assert rc == 0 and lib.blstm_read_status(ws.data_ptr(), None, s) == want


# fp32: one CTA, clusters of 2 to 14; rows per chunk 1, 2, 4, 8; several chunks; hidden sizes that are no multiple of anything
F32_SHAPES = [(5, 3, 7), (4, 300, 32), (6, 40, 33), (3, 600, 64), (5, 1, 100), (4, 45, 128), (5, 44, 257), (3, 9, 200),
              (4, 100, 320), (1, 5, 96), (6, 130, 160)]


@pytest.mark.parametrize("shape", F32_SHAPES)
def test_fp32_cluster_recurrences_against_fp64_maths(shape):
    lib, (T, B, H) = _lib.load(), shape
    g = torch.Generator(device="cuda").manual_seed(B * 17 + H)
    r = lambda *s, std=1.0: torch.randn(*s, generator=g, device="cuda") * std
    pre, h0, c0 = r(T, B, 4 * H), r(B, H, std=0.3), r(B, H, std=0.3)
    dout, dh_n, dc_n = r(T, B, H), r(B, H), r(B, H)
    Wh = (torch.rand(4 * H, H, generator=g, device="cuda") * 2 - 1) / H ** 0.5
    d = _lib.Desc(_lib.F32, T, B, H, H, 0, 0, 0)
    ifgo, out, cell = _fwd(lib, d, pre, Wh, h0, c0)
    W, h, c = Wh.double(), h0.double(), c0.double()
    for t in range(T):
        a = pre[t].double() + h @ W.T
        i, f, gg, o = a.split(H, dim=1)
        c = torch.sigmoid(f) * c + torch.sigmoid(i) * torch.tanh(gg)
        h = torch.sigmoid(o) * torch.tanh(c)
        for name, got, want in (("ifgo", ifgo[t], a), ("out", out[t + 1], h), ("cell", cell[t + 1], c)):
            assert float((got - want).abs().max()) <= 1e-5 * max(1.0, float(want.abs().max())), (name, t)
    infer = _fwd(lib, _lib.Desc(_lib.F32, T, B, H, H, _lib.FLAG_INFERENCE, 0, 0), pre, Wh, h0, c0)
    assert torch.equal(infer[1], out) and torch.equal(infer[2][T], cell[T]) and torch.equal(infer[0], pre)
    n = (B + 1) // 2
    part = _fwd(lib, _lib.Desc(_lib.F32, T, n, H, H, 0, 0, 0), pre[:, :n].contiguous(), Wh, h0[:n].contiguous(), c0[:n].contiguous())
    assert torch.equal(part[1], out[:, :n])
    dg, dh0, dc0, db = _bwd(lib, d, dout, dh_n, dc_n, ifgo, cell, Wh)
    dh, dc, want_db = dh_n.double(), dc_n.double(), 0
    for t in reversed(range(T)):
        pi, pf, pg, po = ifgo[t].double().split(H, dim=1)
        si, sf, so, tg, tc = torch.sigmoid(pi), torch.sigmoid(pf), torch.sigmoid(po), torch.tanh(pg), torch.tanh(cell[t + 1].double())
        dh = dout[t].double() + dh
        dc = dc + dh * so * (1 - tc * tc)
        q = torch.cat([dc * tg * si * (1 - si), dc * cell[t].double() * sf * (1 - sf), dc * si * (1 - tg * tg),
                       dh * tc * so * (1 - so)], dim=1)
        assert float((dg[t] - q).abs().max()) <= 1e-5 * max(1.0, float(q.abs().max())), t
        dc, dh, want_db = dc * sf, q @ W, want_db + q.sum(0)
    for got, want in ((dh0, dh), (dc0, dc), (db, want_db)):
        assert float((got - want).abs().max()) <= 1e-5 * max(1.0, float(want.abs().max()))
    again = _bwd(lib, d, dout, dh_n, dc_n, ifgo, cell, Wh)
    assert all(torch.equal(a, b) for a, b in zip((dg, dh0, dc0, db), again))


# (T, B, I, H): partial tiles in M, N and K, rows that allow 16-byte copies and rows that do not, K split and not
@pytest.mark.parametrize("shape", [(3, 5, 1, 3), (1, 64, 16, 16), (40, 33, 123, 65), (64, 16, 128, 128), (10, 100, 257, 40)])
def test_fp32_gemms_against_fp64_matmul(shape):
    lib, (T, B, I, H) = _lib.load(), shape
    g = torch.Generator(device="cuda").manual_seed(T + I)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, Wx, bx, bh, dg, out = r(T, B, I), r(4 * H, I), r(4 * H), r(4 * H), r(T, B, 4 * H), r(T + 1, B, H)
    d = _lib.Desc(_lib.F32, T, B, I, H, 0, 0, 0)
    s = torch.cuda.current_stream().cuda_stream
    n = lib.blstm_workspace_bytes(d, _lib.PHASE_BWD)
    ws = torch.zeros(n, dtype=torch.uint8, device="cuda")
    new = lambda *sh: torch.full(sh, float("nan"), device="cuda")
    ifgo, dx, dWx, dWh = new(T * B, 4 * H), new(T * B, I), new(4 * H, I), new(4 * H, H)
    _lib.check(lib.blstm_input_projection(d, x.data_ptr(), Wx.data_ptr(), bx.data_ptr(), bh.data_ptr(), ifgo.data_ptr(), s))
    _lib.check(lib.blstm_dgrad_input(d, dg.data_ptr(), Wx.data_ptr(), dx.data_ptr(), ws.data_ptr(), n, s))
    _lib.check(lib.blstm_wgrad(d, dg.data_ptr(), x.data_ptr(), out.data_ptr(), dWx.data_ptr(), dWh.data_ptr(), ws.data_ptr(), n, s))
    X, D, O = x.double().view(T * B, I), dg.double().view(T * B, -1), out[:-1].double().reshape(T * B, H)
    for got, want in ((ifgo, X @ Wx.double().T + bx.double() + bh.double()), (dx, D @ Wx.double()), (dWx, D.T @ X), (dWh, D.T @ O)):
        assert float((got - want).norm() / want.norm()) <= 1e-6


# one row; a partial n-tile; the most rows; sizes the 16-byte accesses do not take (fp32); K in partial blocks of 32
@pytest.mark.parametrize("dtype,B,I,H", [("bf16", 1, 512, 512), ("fp16", 9, 40, 72), ("bf16", 64, 136, 8), ("fp16", 33, 8, 1024),
                                         ("fp32", 1, 16, 64), ("fp32", 7, 123, 65), ("fp32", 64, 200, 400), ("fp32", 2, 3, 5)])
@pytest.mark.parametrize("states", [False, True])
def test_single_timestep_kernel_against_fp64_maths(dtype, B, I, H, states):
    lib = _lib.load()
    dt = {"fp32": torch.float32, **TD}[dtype]
    g = torch.Generator(device="cuda").manual_seed(B + I + H)
    r = lambda *s, std=1.0: (torch.randn(*s, generator=g, device="cuda") * std).to(dt)
    x, Wx, Wh, bx, bh = r(1, B, I), r(4 * H, I, std=I ** -0.5), r(4 * H, H, std=H ** -0.5), r(4 * H, std=0.1), r(4 * H, std=0.1)
    h0, c0 = (r(B, H, std=0.3), r(B, H, std=0.3)) if states else (None, None)
    p = lambda t: None if t is None else t.data_ptr()
    s = torch.cuda.current_stream().cuda_stream
    res = []
    for flags in (0, _lib.FLAG_INFERENCE):
        d = _lib.Desc(_lib.DTYPE_CODE[dtype], 1, B, I, H, flags, 0, 0)
        assert lib.blstm_plan_name(d, _lib.PHASE_FWD_OP) == b"step"
        out, cell, ifgo = (torch.full(sh, float("nan"), device="cuda", dtype=dt) for sh in ((2, B, H), (2, B, H), (1, B, 4 * H)))
        n = lib.blstm_workspace_bytes(d, 0)
        ws = torch.ones(n, dtype=torch.uint8, device="cuda")
        _lib.check(lib.blstm_fwd(d, p(x), p(h0), p(c0), p(Wx), p(Wh), p(bx), p(bh), p(out), p(cell), p(ifgo) if not flags else None,
                                 p(ws), n, s))
        assert lib.blstm_read_status(ws.data_ptr(), None, s) == 0
        res.append((out, cell, ifgo))
    z = torch.zeros(B, H, device="cuda", dtype=torch.float64)
    hp, cp = (z, z) if h0 is None else (h0.double(), c0.double())
    a = x[0].double() @ Wx.double().T + hp @ Wh.double().T + bx.double() + bh.double()
    i, f, gg, o = a.split(H, dim=1)
    c = torch.sigmoid(f) * cp + torch.sigmoid(i) * torch.tanh(gg)
    h = torch.sigmoid(o) * torch.tanh(c)
    tol = {"fp32": 1e-5, "fp16": 3e-3, "bf16": 2e-2}[dtype]
    out, cell, ifgo = res[0]
    for got, want in ((out[0], hp), (cell[0], cp), (out[1], h), (cell[1], c), (ifgo[0], a)):
        assert float((got.double() - want).abs().max()) <= tol * max(1.0, float(want.abs().max()))
    assert torch.equal(res[1][0], out) and torch.equal(res[1][1], cell)


def test_mailbox_hears_of_a_wait_that_ran_out():
    """Launches of a thread that has set a mailbox also leave a device-side error there (no fault: suppressed arrivals)."""
    lib = _lib.load()
    T, B, H = 4, 9, 256
    z = lambda *s: torch.zeros(*s, device="cuda", dtype=torch.bfloat16)
    ifgo, out, cell, Wh = z(T, B, 4 * H), z(T + 1, B, H), z(T + 1, B, H), z(4 * H, H)
    mail = torch.zeros(4, dtype=torch.int32).pin_memory()
    s = torch.cuda.current_stream().cuda_stream
    d = _lib.Desc(_lib.BF16, T, B, H, H, _lib.FLAG_TEST_NO_ARRIVE, 20000, 0)
    n = lib.blstm_workspace_bytes(d, 0)
    ws = torch.zeros(n, dtype=torch.uint8, device="cuda")
    lib.blstm_set_mailbox(mail.data_ptr())
    try:
        assert lib.blstm_fwd_recurrence(d, ifgo.data_ptr(), Wh.data_ptr(), out.data_ptr(), cell.data_ptr(), ws.data_ptr(), n, s) == 0
    finally:
        lib.blstm_set_mailbox(None)
    torch.cuda.synchronize()
    assert mail[1] == _lib.E_WAIT_TIMEOUT and mail[2] >= 1


@pytest.mark.parametrize("G,R,C,R2,C2", [(4, 65, 123, 128, 128), (4, 128, 128, 65, 123), (1, 40, 33, 40, 64), (3, 7, 8, 7, 8), (1, 5, 3, 5, 3)])
@pytest.mark.parametrize("src,dst", [("fp32", "fp32"), ("fp32", "bf16"), ("fp16", "fp16"), ("bf16", "fp32")])
def test_repack_pads_crops_and_converts(G, R, C, R2, C2, src, dst):
    import ctypes
    lib = _lib.load()
    ty = {"fp32": torch.float32, **TD}
    a = torch.randn(G, R, C, device="cuda").to(ty[src])
    b = torch.full((G, R2, C2), float("nan"), device="cuda", dtype=ty[dst])

    class Item(ctypes.Structure):
        _fields_ = [("src", ctypes.c_void_p), ("dst", ctypes.c_void_p), ("sd", ctypes.c_int32), ("dd", ctypes.c_int32),
                    ("groups", ctypes.c_int64), ("r", ctypes.c_int32), ("c", ctypes.c_int32), ("r2", ctypes.c_int32), ("c2", ctypes.c_int32)]
    items = (Item * 1)(Item(a.data_ptr(), b.data_ptr(), _lib.DTYPE_CODE[src], _lib.DTYPE_CODE[dst], G, R, C, R2, C2))
    _lib.check(lib.blstm_repack(items, 1, torch.cuda.current_stream().cuda_stream))
    want = torch.zeros(G, R2, C2, device="cuda", dtype=ty[dst])
    r, c = min(R, R2), min(C, C2)
    want[:, :r, :c] = a[:, :r, :c].to(ty[dst])
    assert torch.equal(b, want)


@pytest.mark.parametrize("lengths,C", [([1], 1), ([4, 9, 1, 6, 9, 2], 12), ([33] * 5, 8), ([70, 2, 41, 70], 130)])
@pytest.mark.parametrize("dtype", ["fp32", "bf16"])
def test_packed_row_maps_and_gathers(lengths, C, dtype):
    """The maps between packed rows and the padded grid, forwards and turned, and the gathers they drive, against
    torch's packing; each map's inverse carries the gradient."""
    from torch.nn.utils.rnn import pack_padded_sequence
    host = _lib.host()
    ty = {"fp32": torch.float32, **TD}[dtype]
    T, B = max(lengths), len(lengths)
    x = torch.randn(T, B, C).to(ty)
    turned_x = torch.zeros_like(x)
    for b, n in enumerate(lengths):
        x[n:, b] = 0
        turned_x[:n, b] = x[:n, b].flip(0)
    seq = pack_padded_sequence(x.cuda(), torch.tensor(lengths), enforce_sorted=False)
    padded, turned, rev, inv_last, last, packed, packed_t = host.packed_maps(seq.batch_sizes, seq.unsorted_indices, seq.data)
    data = seq.data.clone().requires_grad_(True)
    a = host.gather_rows(data, padded, packed, [T, B])
    b = host.gather_rows(data, turned, packed_t, [T, B])
    assert torch.equal(a.cpu(), x) and torch.equal(b.cpu(), turned_x)
    assert torch.equal(host.gather_rows(a, packed, padded, [data.shape[0]]), data)
    assert torch.equal(host.gather_rows(b, packed_t, turned, [data.shape[0]]), data)
    assert torch.equal(host.gather_rows(a, rev, rev, [T, B]).cpu(), turned_x)
    h = host.gather_rows(a, last, inv_last, [B])
    assert torch.equal(h.cpu(), torch.stack([x[n - 1, i] for i, n in enumerate(lengths)]))
    h.sum().backward()
    want = pack_padded_sequence(torch.stack([torch.arange(T) == n - 1 for n in lengths], 1)[:, :, None].expand(T, B, C).to(ty),
                                torch.tensor(lengths), enforce_sorted=False).data
    assert torch.equal(data.grad.cpu(), want)


@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("T,B,H", [(48, 3, 40), (64, 32, 128), (50, 17, 320)])
def test_directions_side_by_side_match_nn_lstm(T, B, H, packed):
    """Both directions at once, each on half of the device, against torch.nn.LSTM in float64 - twice, so that the
    second pass reuses the first one's memory on both streams."""
    import fastlstm_b200 as F
    from torch.nn.utils.rnn import pack_padded_sequence
    torch.manual_seed(T + H)
    ref = torch.nn.LSTM(24, H, num_layers=2, bidirectional=True).double()
    m = F.FastLSTM(24, H, num_layers=2, bidirectional=True, device="cuda", dtype=torch.bfloat16)
    with torch.no_grad():
        for p in ref.parameters():
            p.copy_(p.bfloat16().double())
    m.load_state_dict({k: v.bfloat16() for k, v in ref.state_dict().items()})
    lengths = torch.randint(1, T + 1, (B,))
    lengths[B // 2] = T
    for seed in range(2):
        x = torch.randn(T, B, 24).bfloat16()
        res = []
        for mod, xi in ((m, x.cuda().requires_grad_(True)), (ref, x.double().requires_grad_(True))):
            mod.zero_grad()
            out, (hn, cn) = mod(pack_padded_sequence(xi, lengths, enforce_sorted=False) if packed else xi)
            out = out.data if packed else out
            (out.float().square().sum() + hn.float().sum()).backward()
            res.append([t.detach().double().cpu() for t in (out, hn, cn, xi.grad, *(p.grad for p in mod.parameters()))])
        for i, (a, b) in enumerate(zip(*res)):
            assert (a - b).norm() <= 2e-2 * b.norm() + 1e-6, i
    F.check_status()


@pytest.mark.parametrize("packed", [False, True])
def test_directions_side_by_side_when_nothing_but_the_weights_needs_a_gradient(packed):
    """No input gradient, no kept states: the last holders of what the directions share are nodes of the backward pass.
    Passes on different batches back to back, nothing waited for in between, give bit for bit the gradients of each
    batch on its own."""
    import fastlstm_b200 as F
    from torch.nn.utils.rnn import pack_padded_sequence
    torch.manual_seed(3)
    T, B, H = 64, 24, 128
    m = F.FastLSTM(24, H, num_layers=2, bidirectional=True, device="cuda", dtype=torch.bfloat16)
    xs, lens = [torch.randn(T, B, 24, device="cuda").bfloat16() for _ in range(6)], [torch.randint(1, T + 1, (B,)) for _ in range(6)]
    for n in lens:
        n[0] = T

    def grads(k):
        m.zero_grad()
        out = m(pack_padded_sequence(xs[k], lens[k], enforce_sorted=False) if packed else xs[k])[0]
        out = out.data if packed else out
        torch.autograd.backward([out], [torch.ones_like(out)])
        return [p.grad for p in m.parameters()]
    alone = []
    for k in range(6):
        alone.append([g.clone() for g in grads(k)])
        torch.cuda.synchronize()
    for _ in range(3):
        for g, want in zip([grads(k) for k in range(6)], alone):
            assert all(torch.equal(a, b) for a, b in zip(g, want))
    F.check_status()


@pytest.mark.parametrize("T,B,H,P,states", [(2, 1, 33, 7, True), (40, 9, 96, 32, True), (30, 64, 512, 128, False)])
def test_projected_layer_matches_nn_lstm(T, B, H, P, states):
    """The projected layer as an ordinary one with the recurrent weights W_hh W_hr."""
    import fastlstm_b200 as F
    torch.manual_seed(H)
    ref = torch.nn.LSTM(20, H, proj_size=P).double()
    with torch.no_grad():
        for p in ref.parameters():
            p.copy_(p.half().double())
    m = F.FastLSTM(20, H, proj_size=P, device="cuda", dtype=torch.float16)
    m.load_state_dict({k: v.half() for k, v in ref.state_dict().items()})
    x, h0, c0 = (torch.randn(*s).half() * 0.5 for s in ((T, B, 20), (1, B, P), (1, B, H)))
    res = []
    for mod, cast in ((m, lambda t: t.cuda().requires_grad_(True)), (ref, lambda t: t.double().requires_grad_(True))):
        xi, hi, ci = cast(x), cast(h0), cast(c0)
        out, (hn, cn) = mod(xi, (hi, ci)) if states else mod(xi)
        (out.float().square().sum() + hn.float().sum() + cn.float().sum()).backward()
        grads = [xi.grad] + ([hi.grad, ci.grad] if states else []) + [p.grad for p in mod.parameters()]
        res.append([t.detach().double().cpu() for t in (out, hn, cn, *grads)])
    for i, (a, b) in enumerate(zip(*res)):
        assert (a - b).norm() <= 1e-2 * b.norm() + 1e-6, i
    F.check_status()
