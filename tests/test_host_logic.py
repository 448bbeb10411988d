"""Host-side behaviour of the module that needs no GPU."""
import glob
import os
import re

import pytest
import torch
import torch.nn as nn

from fastlstm_b200 import FastLSTM, lstm_persistent_fwd


def test_init_matches_nn_lstm_rng_order():
    # same check as the reference's tests/test_lstm.py:116-129
    torch.manual_seed(123)
    m1 = FastLSTM(8, 3, num_layers=2)
    torch.manual_seed(123)
    m2 = nn.LSTM(8, 3, num_layers=2)
    names = [n for n, _ in m1.named_parameters()]
    assert names == [n for n, _ in m2.named_parameters()]
    for n, p in m1.named_parameters():
        torch.testing.assert_close(p, getattr(m2, n))


def test_state_dict_interchange_and_no_bias():
    m1 = FastLSTM(5, 4, num_layers=2, bias=False)
    m2 = nn.LSTM(5, 4, num_layers=2, bias=False)
    m1.load_state_dict(m2.state_dict())
    m2.load_state_dict(m1.state_dict())
    assert all("bias" not in n for n, _ in m1.named_parameters())


def test_cpu_tensors_are_rejected_loudly():
    m = FastLSTM(4, 4)
    with pytest.raises(ValueError, match="CUDA"):
        m(torch.randn(3, 2, 4))
    with pytest.raises(ValueError):
        lstm_persistent_fwd(torch.randn(3, 2, 4), None, None, torch.randn(16, 4), None,
                            torch.randn(16, 4), None)


def test_unknown_version_rejected():
    with pytest.raises(ValueError):
        FastLSTM(4, 4, version="graph")


def test_bidirectional_parameters_match_nn_lstm_and_options_are_validated():
    m = FastLSTM(12, 8, num_layers=2, bidirectional=True, dropout=0.25)
    ref = nn.LSTM(12, 8, num_layers=2, bidirectional=True, dropout=0.25)
    assert [(n, tuple(p.shape)) for n, p in m.named_parameters()] == \
           [(n, tuple(p.shape)) for n, p in ref.named_parameters()]
    m.load_state_dict(ref.state_dict())
    ref.load_state_dict(m.state_dict())
    with pytest.raises(ValueError):
        FastLSTM(4, 4, proj_size=4)           # like nn.LSTM: smaller than hidden_size
    with pytest.raises(ValueError):
        FastLSTM(4, 4, dropout=1.5)


class _TorchLayer:
    """Stand-in for PersistentLSTMfn on CPU: the same call signature, plain differentiable torch ops."""

    @staticmethod
    def apply(x, h0, c0, Wx, bx, Wh, bh, inference=None, sink=None, want_cells=False):
        T, B, _ = x.shape
        H = Wh.shape[1]
        h = x.new_zeros(B, H) if h0 is None else h0
        c = x.new_zeros(B, H) if c0 is None else c0
        outs, cells = [], []
        for t in range(T):
            a = x[t] @ Wx.T + h @ Wh.T + (0 if bx is None else bx + bh)
            i, f, g, o = a.split(H, dim=1)
            c = torch.sigmoid(f) * c + torch.sigmoid(i) * torch.tanh(g)
            h = torch.sigmoid(o) * torch.tanh(c)
            outs.append(h)
            cells.append(c)
        out = torch.stack(outs)
        res = (out, out[-1], cells[-1])
        return res + (torch.stack(cells).detach(),) if want_cells else res


@pytest.mark.parametrize("bidirectional", [False, True])
def test_packed_sequence_plumbing_matches_nn_lstm(monkeypatch, bidirectional):
    """PackedSequence in, PackedSequence out, states at every sequence's own last step, the reverse
    direction from every sequence's own end, gradients through the packed output and h_n - checked on
    CPU with a torch stand-in for the CUDA layer against torch.nn.LSTM."""
    import fastlstm_b200.lstm as mod
    from torch.nn.utils.rnn import pack_padded_sequence
    monkeypatch.setattr(mod, "PersistentLSTMfn", _TorchLayer)
    torch.manual_seed(4)
    I, H, L = 5, 6, 2
    ref = torch.nn.LSTM(I, H, num_layers=L, bidirectional=bidirectional).double()
    m = mod.FastLSTM(I, H, num_layers=L, bidirectional=bidirectional, dtype=torch.float64)
    m.load_state_dict(ref.state_dict())
    lengths = torch.tensor([3, 7, 1, 5])
    x = torch.randn(7, 4, I, dtype=torch.float64)
    nd = 2 if bidirectional else 1
    h0, c0 = torch.randn(L * nd, 4, H, dtype=torch.float64), torch.randn(L * nd, 4, H, dtype=torch.float64)
    results = []
    for net in (ref, m):
        xi = x.clone().requires_grad_()
        out, (hn, cn) = net(pack_padded_sequence(xi, lengths, enforce_sorted=False), (h0, c0))
        (out.data.square().sum() + hn.sum()).backward()
        results.append((out, hn, cn, xi.grad, [p.grad.clone() for p in net.parameters()]))
        net.zero_grad()
    (o1, h1, c1, g1, p1), (o2, h2, c2, g2, p2) = results
    assert torch.equal(o1.batch_sizes, o2.batch_sizes) and torch.equal(o1.sorted_indices, o2.sorted_indices)
    for a, b in ((o1.data, o2.data), (h1, h2), (c1, c2), (g1, g2)):
        torch.testing.assert_close(a, b, rtol=1e-9, atol=1e-10)
    for a, b in zip(p1, p2):
        torch.testing.assert_close(a, b, rtol=1e-9, atol=1e-10)


def test_persistent_plans_fit_the_device_for_a_sweep_of_shapes():
    """Every tensor-core plan must be launchable on a 148-SM part: the forward grid within the SM count,
    the backward grid within the 33 clusters of four that can be resident at once, shared memory
    within the 227 KB a CTA may have.  (Geometry only: nothing is launched.)"""
    import re
    from fastlstm_b200 import plan_detail
    seen = set()
    for H in (64, 128, 192, 256, 320, 384, 512, 640, 768, 1024, 1280, 1536, 2048):
        for B in (1, 32, 100, 128, 129, 256, 400, 512, 640, 1024, 1300, 2048, 2304, 4096, 4800, 8192):
            for phase in ("fwd", "bwd"):
                s = plan_detail(torch.bfloat16, 8, B, H, H, phase)
                assert s.startswith("sm100"), (B, H, phase, s)
                grid = int(re.search(r"grid=(\d+)", s).group(1))
                assert grid <= (132 if phase == "bwd" else 148), (B, H, phase, s)
                if phase == "bwd":
                    assert grid % 4 == 0, s
                m = re.search(r"smem=(\d+)", s)
                if m:
                    assert int(m.group(1)) <= 232448, (B, H, phase, s)
                seen.add(re.sub(r"grid=\d+|smem=\d+", "", s))
    assert len(seen) > 20      # the sweep meets many different plans


@pytest.mark.parametrize("bidirectional", [False, True])
def test_proj_size_plumbing_matches_nn_lstm(monkeypatch, bidirectional):
    """nn.LSTM's output projection (proj_size): parameter names, shapes and order, the stepwise layer with
    the projected state zero-padded to the cell's width, initial states of the projected width, packed
    input - checked on CPU with a torch stand-in for the CUDA cell against torch.nn.LSTM."""
    import fastlstm_b200.lstm as mod
    from torch.nn.utils.rnn import pack_padded_sequence
    monkeypatch.setattr(mod, "PersistentLSTMfn", _TorchLayer)
    torch.manual_seed(7)
    I, H, P, L = 5, 8, 3, 2
    ref = torch.nn.LSTM(I, H, num_layers=L, bidirectional=bidirectional, proj_size=P).double()
    m = mod.FastLSTM(I, H, num_layers=L, bidirectional=bidirectional, proj_size=P, dtype=torch.float64)
    assert [n for n, _ in m.named_parameters()] == [n for n, _ in ref.named_parameters()]
    assert [tuple(p.shape) for p in m.parameters()] == [tuple(p.shape) for p in ref.parameters()]
    m.load_state_dict(ref.state_dict())
    nd = 2 if bidirectional else 1
    x = torch.randn(6, 4, I, dtype=torch.float64)
    h0, c0 = torch.randn(L * nd, 4, P, dtype=torch.float64), torch.randn(L * nd, 4, H, dtype=torch.float64)
    for packed in (False, True):
        results = []
        for net in (ref, m):
            xi = x.clone().requires_grad_()
            inp = pack_padded_sequence(xi, torch.tensor([6, 2, 5, 1]), enforce_sorted=False) if packed else xi
            out, (hn, cn) = net(inp, (h0, c0))
            data = out.data if packed else out
            (data.square().sum() + hn.sum() + (0 if packed else cn.sum())).backward()
            results.append((data, hn, cn, xi.grad, [p.grad.clone() for p in net.parameters()]))
            net.zero_grad()
        (o1, h1, c1, g1, p1), (o2, h2, c2, g2, p2) = results
        assert o2.shape[-1] == P * nd and h2.shape == (L * nd, 4, P) and c2.shape == (L * nd, 4, H)
        for a, b in ((o1, o2), (h1, h2), (c1, c2), (g1, g2)):
            torch.testing.assert_close(a, b, rtol=1e-9, atol=1e-10)
        for a, b in zip(p1, p2):
            torch.testing.assert_close(a, b, rtol=1e-9, atol=1e-10)
    # without initial states, and the constructor's checks
    out, (hn, cn) = m(x)
    ro, (rh, rc) = ref(x)
    torch.testing.assert_close(out, ro, rtol=1e-9, atol=1e-10)
    with pytest.raises(ValueError):
        mod.FastLSTM(I, H, proj_size=H)
    with pytest.raises(ValueError):
        mod.FastLSTM(I, H, proj_size=-1)


def test_every_hand_off_through_global_memory_is_a_release():
    # what a CTA counts in on a global counter other SMs read behind ld.acquire.gpu: without a release on this side nothing
    # orders the data before the count, whatever was waited for locally
    import fastlstm_b200
    counted = 0
    for path in glob.glob(os.path.join(os.path.dirname(fastlstm_b200.__file__), "csrc", "*.cu*")):
        with open(path) as f:
            code = re.sub(r"//.*", "", f.read())
        assert not re.search(r"\b(red|atom)\.(async\.)?relaxed", code), path
        for call in re.findall(r"(\w+)\(&p\.flags\[", code):
            assert call in ("red_release_gpu_add", "wait_flag_ge", "ld_acquire_gpu"), (path, call)
            counted += call == "red_release_gpu_add"
    assert counted >= 7


def test_signals_to_the_cluster_carry_the_reads_before_them():
    # a CTA that says its reads are done lets a peer overwrite what was read: a relaxed arrival needs a fence in front, and the
    # peer an acquire at cluster scope
    import fastlstm_b200
    relaxed = waits = 0
    for path in glob.glob(os.path.join(os.path.dirname(fastlstm_b200.__file__), "csrc", "*.cu")):
        with open(path) as f:
            code = re.sub(r"//.*", "", f.read())
        for before in re.findall(r"((?:.*\n){3}).*mbar_arrive_remote_relaxed\(", code):
            assert "fence_acq_rel_cluster();" in before, path
            relaxed += 1
        for wait in re.findall(r"(\w+)\(&?(?:consumed|rdy)\b.*?, wc\)", code):
            assert wait == "mbar_wait_cluster", (path, wait)
            waits += 1
    assert relaxed >= 2 and waits >= 3


def test_the_lanes_that_fetch_come_behind_the_lane_that_acquired():
    # one lane acquires a hand-off counter, others issue the loads: the shuffle that hands its finding on orders no memory
    import fastlstm_b200
    found = 0
    for path in glob.glob(os.path.join(os.path.dirname(fastlstm_b200.__file__), "csrc", "*.cu")):
        with open(path) as f:
            code = re.sub(r"//.*", "", f.read())
        for follows in re.findall(r"seen = __shfl_sync\(0xffffffffu, seen, 0\);\s*(\S+)", code):
            assert follows == "__syncwarp();", path
            found += 1
    assert found >= 4


@pytest.mark.parametrize("packed", [False, True])
def test_memory_that_two_streams_share_is_not_reused_under_a_queued_read(monkeypatch, packed):
    """The directions of a layer on two streams (fakes; the operators by plain torch): what the side stream reads of the main
    stream's memory is recorded there - backward's last holder may be a node on either - and the side stream comes behind
    the main stream's last read of what it has made."""
    import contextlib
    from torch.nn.utils import parametrize
    from torch.nn.utils.rnn import pack_padded_sequence
    from fastlstm_b200 import _lib, lstm
    log, made_on, recorded, reads = [], {}, set(), []
    key = lambda t: t.untyped_storage().data_ptr()

    class Stream:
        stream_id = device_index = device_type = 0

        def __init__(self, name):
            self.name = name

        def wait_stream(self, other):
            log.append((self.name, "waits for", other.name))
    main, side, now = Stream("main"), Stream("side"), []
    now.append(main)

    @contextlib.contextmanager
    def on(stream):
        now.append(stream)
        yield
        now.pop()

    keep = []

    def op(out, *used):                    # an operator of the current stream
        reads.extend((now[-1].name, t) for t in used if t is not None)
        for t in out:
            made_on[key(t)] = now[-1].name
            keep.append(t)
        return out

    class Host:
        def packed_maps(self, batch_sizes, rank, data):
            T, B = batch_sizes.numel(), int(batch_sizes[0])
            maps = torch.zeros(4 * T * B + B + 2 * data.shape[0], dtype=torch.long)
            op([maps])
            return list(maps.split([T * B] * 4 + [B] + [data.shape[0]] * 2))

        def gather_rows(self, src, idx, inv, lead):
            return op([src.reshape(-1, src.shape[-1])[idx].view(*lead, -1).clone()], src, idx, inv)[0]

    def layer(x, h0, c0, Wx, bx, Wh, bh, inference, want_cells=False, **_):
        out, cells = x @ Wx.t()[:, :Wh.shape[1]], x @ Wx.t()[:, -Wh.shape[1]:]
        h, c = out[-1].clone(), cells[-1].clone()
        op([out, cells, h, c], x, Wx, Wh, bx, bh)
        return (out, h, c) + ((cells,) if want_cells else ())

    class Twice(nn.Module):
        def forward(self, w):
            return 2 * w
    m = FastLSTM(6, 4, num_layers=2, bidirectional=True)
    parametrize.register_parametrization(m, "weight_ih_l0_reverse", Twice())
    params = {key(p) for p in m.parameters()}
    monkeypatch.setattr(_lib, "host", lambda: Host())
    monkeypatch.setattr(lstm, "_layer", layer)
    monkeypatch.setattr(lstm, "_shares_device", lambda *a: True)
    monkeypatch.setattr(lstm, "_side_stream", lambda d: side)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda d=None: now[-1])
    monkeypatch.setattr(torch.cuda, "stream", on)
    monkeypatch.setattr(torch.Tensor, "is_cuda", True)
    monkeypatch.setattr(torch.Tensor, "record_stream", lambda t, s: recorded.add((key(t), s.name)))
    for name in ("cat", "stack"):
        f = getattr(torch, name)
        monkeypatch.setattr(torch, name, lambda ts, dim=0, f=f, name=name: log.append(("main", name)) or f(ts, dim=dim))
    x = torch.randn(5, 3, 6)
    if packed:
        m._forward_packed_rows(pack_padded_sequence(x, [5, 4, 2]), None)
    else:
        m._forward_padded(x, None, None)
    shared = [t for who, t in reads if who == "side" and made_on.get(key(t), "main") == "main" and key(t) not in params]
    assert len(shared) >= (8 if packed else 3)
    for t in shared:
        assert (key(t), "side") in recorded, t.shape
    assert log[-1] == ("side", "waits for", "main") and ("main", "waits for", "side") in log
    last = max(i for i, e in enumerate(log) if e[0] == "main" and e[1] in ("cat", "stack"))
    assert log.index(("main", "waits for", "side")) < last < len(log) - 1
    # every layer's concatenation too, before the next layer's work may free what it read
    for i, e in enumerate(log):
        if e == ("main", "cat"):
            assert ("side", "waits for", "main") in log[i + 1:i + 4]


def test_how_a_layer_runs_does_not_hang_on_the_words_of_a_plan(monkeypatch):
    # plan_detail is text for people; the family behind it is what the host arranges launches by
    from fastlstm_b200 import _lib, lstm
    cases = [(dt, T, B, H) for dt in (torch.float16, torch.bfloat16, torch.float32) for T in (8, 64, 256)
             for B in (8, 64, 512, 1500, 4096) for H in (64, 128, 192, 320, 512, 576, 1088)]
    words = {"small-batch": _lib.FAMILY_SMALL_BATCH, "resident weights": _lib.FAMILY_RESIDENT, "TI=": _lib.FAMILY_BATCH_TILES, "generic": _lib.FAMILY_GENERIC}
    seen = set()
    for dt, T, B, H in cases:
        if dt == torch.float32:
            continue
        for phase in ("fwd", "bwd"):
            for half in (False, True):
                want = next(f for w, f in words.items() if w in lstm.plan_detail(dt, T, B, H, H, phase, half))
                assert lstm._family(dt, T, B, H, H, phase, half) == want
                seen.add(want)
    assert len(seen) == 4

    def ways():
        lstm._shares_device.cache_clear()
        lstm._wavefront_pays.cache_clear()
        return [(lstm._shares_device(dt, T, B, H, H), lstm._wavefront_pays(dt, T, B, H, True), lstm._wavefront_pays(dt, T, B, H, False))
                for dt, T, B, H in cases]
    before = ways()
    monkeypatch.setattr(lstm, "plan_detail", lambda *a, **k: "reworded")
    assert ways() == before and len(set(before)) > 2


def test_small_batch_kernels_where_they_measured_faster():
    # hidden size -> most rows (forward, backward) that the small-batch recurrences get: 15 clusters of 8 CTAs at 256, 7 of 16
    # above, eight rows a chunk.  At 512 a batch of 256 and its halves stay in the same backward kernel.
    from fastlstm_b200 import _lib, lstm
    for H, most in {192: (960, 960), 256: (480, 720), 384: (168, 224), 512: (112, 280), 576: (56, 112)}.items():
        for phase, n in zip(("fwd", "bwd"), most):
            for B in (8, n // 2, n, n + 1):
                small = lstm._family(torch.bfloat16, 64, B, H, H, phase) == _lib.FAMILY_SMALL_BATCH
                assert small == (B <= n), (H, B, phase)
    # (a size that only the CUDA-core kernels would take instead)
    assert lstm._family(torch.bfloat16, 64, 1100, 200, 200, "bwd") == _lib.FAMILY_SMALL_BATCH


def test_plans_without_a_device_are_those_of_a_b200():
    # 22 clusters of six CTAs are resident at once on 148 SMs, so the largest backward plan fits over six
    from fastlstm_b200 import plan_detail
    s = plan_detail(torch.bfloat16, 8, 32, 2048, 2048, "bwd")
    assert "resident weights cluster=6 " in s and "grid=96 " in s, s
    # a second issuer is worth a CTA more a cluster where the rows of a group stay within 32, and only there
    for H, B, want in ((1728, 32, "cluster=6"), (1728, 17, "cluster=6"), (1408, 64, "cluster=5"), (1408, 96, "cluster=4"), (1664, 32, "cluster=5")):
        s = plan_detail(torch.bfloat16, 8, B, H, H, "bwd")
        assert want in s and ("issuers=2" in s) == (B != 96), (H, B, s)


def test_wavefront_where_it_measured_faster():
    from fastlstm_b200 import lstm
    bf = torch.bfloat16
    for grad, T, B, H, want in ((True, 256, 968, 192, True), (True, 128, 768, 384, True), (True, 64, 768, 384, False),
                                (True, 256, 392, 576, False), (True, 256, 512, 512, False), (True, 256, 32, 256, False),
                                (False, 256, 64, 64, False), (False, 256, 64, 256, False), (False, 128, 64, 512, False),
                                (False, 128, 128, 512, True), (False, 64, 128, 512, False), (False, 128, 1000, 192, True),
                                # (long sequences of few rows: the clusters of two layers fit beside each other)
                                (False, 1024, 64, 64, True), (False, 256, 8, 256, True), (False, 128, 8, 256, False),
                                (False, 1024, 64, 192, False), (False, 1024, 1000, 64, False), (False, 1024, 100, 512, False),
                                (False, 256, 200, 320, True), (False, 256, 400, 256, False)):
        assert lstm._wavefront_pays(bf, T, B, H, grad) == want, (grad, T, B, H)
        if H <= 512 and B > 8:
            # ... and it is what the module asks before it runs, and the benchmark before it reports
            x = type("OnGpu", (), dict(is_cuda=True, shape=(T, B, H), dtype=bf))
            m = FastLSTM(H, H, num_layers=2, device="meta", dtype=bf)
            assert bool(m._wavefront(x, None, None, grad)) == want


def _ring_faults(lanes, start, step, S2, n_kg, items=3):
    """Walks every interleaving of the producer's lanes, the copies' landing, the issuer and the MMAs' completion over one ring of
    S2 stages whose fills are told by the parities of `full` and `empty`; returns what goes wrong first, or None.  An item is n_kg
    groups, the lanes meet behind each; lane l issues groups start(l, pos), start + step, ..."""
    total = items * n_kg
    plan = []                                        # per lane and item: the fills (numbers 0.. in ring order) that it issues
    for l in lanes:
        plan.append([[it * n_kg + kg for kg in range(start(l, it * n_kg % S2), n_kg, step)] for it in range(items)])
    # state: item, each lane's position in it; fills armed / landed per stage; fills the issuer has taken / whose MMAs are done
    first = (0, (0,) * len(lanes), ((-1, True),) * S2, 0, 0)
    seen, todo = {first}, [first]
    while todo:
        item, at, stages, taken, done = todo.pop()
        moves = []
        for i, p in enumerate(plan):
            if item < items and at[i] < len(p[item]):
                fill = p[item][at[i]]
                st, turn = fill % S2, fill // S2
                consumed = len(range(st, done, S2))  # phases of empty[st] that are over
                if (consumed & 1) != ((turn & 1) ^ 1):          # the lane's wait for that parity returns
                    if consumed != turn:
                        return f"lane {lanes[i]} fills stage {st} for the {turn + 1}. time after {consumed} of its fills were consumed"
                    if not stages[st][1]:
                        return f"stage {st} armed twice"
                    moves.append((item, at[:i] + (at[i] + 1,) + at[i + 1:], stages[:st] + ((fill, False),) + stages[st + 1:], taken, done))
        if item < items and all(a == len(p[item]) for a, p in zip(at, plan)):
            moves.append((item + 1, (0,) * len(lanes), stages, taken, done))
        for st, (fill, landed) in enumerate(stages):
            if not landed:
                moves.append((item, at, stages[:st] + ((fill, True),) + stages[st + 1:], taken, done))
        if taken < total:
            st, turn = taken % S2, taken // S2
            fill, landed = stages[st]
            full = (fill // S2 if not landed else fill // S2 + 1) if fill >= 0 else 0      # phases of full[st] that are over
            if (full & 1) != (turn & 1):
                if fill != taken or not landed:
                    return f"the issuer takes fill {fill} of stage {st} for fill {taken}"
                moves.append((item, at, stages, taken + 1, done))
        if done < taken:
            moves.append((item, at, stages, taken, done + 1))
        if not moves and done < total:
            return f"nothing moves after {done} of {total} fills"
        for m in moves:
            if m not in seen:
                seen.add(m)
                todo.append(m)
    return None


def test_the_stages_of_the_backward_ring_are_filled_in_turn():
    # Which lanes fill the ring of `tiles_kernel`, and with which groups of K chunks, is read from the source; how many stages and
    # groups there are comes from every plan that batches of a few hundred to some thousand rows get.
    import fastlstm_b200
    from fastlstm_b200 import plan_detail
    with open(os.path.join(os.path.dirname(fastlstm_b200.__file__), "csrc", "sm100_resident_tiles.cu")) as f:
        code = re.sub(r"//.*", "", f.read())
    two, first = re.search(r"const int two = ([^;]+);.*?if \(lane <= two\) \{\s*for \(int kg = ([^;]+); kg < n_kg; kg \+= 1 \+ two\)", code, re.S).groups()
    two = two.replace("&&", "and").replace("||", "or")
    rings = set()
    for H in range(256, 1025, 64):
        for B in range(64, 8193, 32):
            for half in (False, True):
                s = plan_detail(torch.bfloat16, 8, B, H, H, "bwd", half)
                m = re.search(r" n=(\d+) .* chunks=(\d+) .*stages=(\d+) chunks_per_stage=(\d+)", s)
                if m and "tiles=" in s and "rows_per_tile" not in s:
                    rings.add((int(m.group(3)) // 2, -(-int(m.group(2)) // int(m.group(4))), int(m.group(1))))
    assert len(rings) >= 6 and any(S2 == 1 and n_kg > 1 for S2, n_kg, _ in rings), rings
    for S2, n_kg, N in sorted(rings):
        of = int(eval(two, {}, {"S2": S2, "N": N, "n_kg": n_kg}))
        fault = _ring_faults(list(range(1 + of)), lambda lane, pos: eval(first, {}, {"lane": lane, "pos": pos, "two": of}), 1 + of, S2, n_kg)
        assert fault is None, (S2, n_kg, fault)


def test_two_lanes_cannot_share_a_stage():
    # (what the walk above has to find: two lanes dealt the groups of a one-stage ring in turn tell their fills by one parity)
    deal = lambda lane, pos: (lane + pos) & 1
    assert _ring_faults([0, 1], deal, 2, 1, 2) is not None
    assert _ring_faults([0, 1], deal, 2, 2, 4) is None and _ring_faults([0], lambda lane, pos: 0, 1, 1, 2) is None


def test_stages_of_the_backward_ring_where_they_measured_faster():
    # 64-row tiles: eight groups of CTAs at H = 448 and 512, eleven at 320 and 384, sixteen at 256
    from fastlstm_b200 import plan_detail
    for H, groups, long_from in ((256, 16, 4), (320, 11, 9), (384, 11, 9), (448, 8, 5), (512, 8, 5)):
        for tiles in range(4, 9):
            s = plan_detail(torch.bfloat16, 8, 64 * groups * tiles, H, H, "bwd")
            want = "stages=2 chunks_per_stage=4 " if tiles >= long_from else "stages=4 chunks_per_stage=2 "
            assert f"tiles={tiles} " in s and "n=64 " in s and want in s, (H, tiles, s)


def test_no_wavefront_where_half_of_the_device_takes_several_tiles_in_turn():
    # without gradients, resident weights: two tiles of rows a group of CTAs on half of the device, or the layers stay one after the
    # other with their cell states in 32 bits throughout
    from fastlstm_b200 import lstm, plan_detail
    bf = torch.bfloat16
    for H in range(256, 1025, 64):
        most = 64 * (74 // (H // 32))
        for B in (most, most + 1, min(most + 97, 1024 if H <= 256 else 768 if H <= 384 else 512 if H <= 576 else 256)):
            two = B <= most
            assert ("rows_per_tile" in plan_detail(bf, 64, B, H, H, "fwd", True)) == two, (H, B)
            for T in (128, 256, 1024):
                assert lstm._wavefront_pays(bf, T, B, H, False) == two, (T, B, H)
    for B, H in ((704, 256), (512, 512), (257, 512), (224, 768), (256, 832), (130, 896), (256, 1024)):
        assert not lstm._wavefront_pays(bf, 256, B, H, False)


def test_backward_of_832_units_leaves_groups_of_two_tiles_to_the_other_kernel():
    from fastlstm_b200 import _lib, lstm
    for H, B, family in ((832, 257, _lib.FAMILY_BATCH_TILES), (832, 352, _lib.FAMILY_BATCH_TILES), (832, 353, _lib.FAMILY_RESIDENT),
                         (832, 512, _lib.FAMILY_RESIDENT), (896, 289, _lib.FAMILY_RESIDENT), (768, 481, _lib.FAMILY_RESIDENT),
                         (448, 800, _lib.FAMILY_RESIDENT)):
        assert lstm._family(torch.bfloat16, 64, B, H, H, "bwd") == family, (H, B)


def test_plans_behind_the_tests_of_several_tiles():
    # what tests/test_gpu_resident.py means to run: tiles of the fullest group, rows of a tile
    from fastlstm_b200 import plan_detail
    for phase, cases in (("fwd", ((289, 1024, 3, 32), (1023, 1024, 8, 32), (1700, 512, 6, 32), (2300, 256, 4, 32), (2849, 768, 15, 32), (2913, 768, 16, 32),
                                  (400, 832, 3, 32), (600, 960, 5, 32))),
                         ("bwd", ((300, 1024, 3, 32), (1023, 1024, 8, 32), (1024, 512, 4, 32), (1990, 896, 16, 32), (521, 832, 5, 32), (600, 768, 4, 32),
                                  (700, 960, 6, 32), (1400, 384, 4, 32), (4200, 320, 6, 64), (5632, 384, 8, 64), (3000, 448, 6, 64), (4096, 448, 8, 64),
                                  (2048, 512, 4, 64), (3072, 512, 6, 64), (4096, 512, 8, 64), (8192, 256, 8, 64)))):
        for B, H, tiles, rows in cases:
            s = plan_detail(torch.bfloat16, 8, B, H, H, phase)
            assert f" tiles={tiles} " in s and f" n={rows} " in s, (phase, B, H, s)
