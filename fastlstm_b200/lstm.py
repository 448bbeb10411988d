"""Host side of the B200 LSTM layer: the reference's module surface over the C ABI.

Mirrors oleicht/FastLSTM `fastlstm/lstm.py`:

  lstm_persistent_fwd   <- fastlstm/lstm.py:31-146
  lstm_persistent_bwd   <- fastlstm/lstm.py:236-334
  Wgrad                 <- fastlstm/lstm.py:494-501
  PersistentLSTMfn      <- fastlstm/lstm.py:504-538
  FastLSTM              <- fastlstm/lstm.py:586-698

Differences (all additions): `bias` and `batch_first` constructor arguments,
gradients through the returned (h_n, c_n), fp32 weight/bias gradients, fp32
matmuls stay fp32 (the reference flips the global TF32 switch on import,
fastlstm/lstm.py:15-19; this module does not).  PyTorch is used for device
memory, streams and autograd only; every device computation goes through
libfastlstm_b200.so and there is no fallback path.  What a call does on the
host - checks, buffers, the C ABI calls - is csrc/host.cpp.
"""
from __future__ import annotations

import contextlib
import functools
import os

import torch
import torch.nn as nn

from . import _lib

_DTYPE_CODE = {torch.float32: _lib.F32, torch.float16: _lib.F16, torch.bfloat16: _lib.BF16}

_FORCE_GENERIC = os.environ.get("FASTLSTM_B200_FORCE_GENERIC", "0") == "1"
_WAIT_LIMIT_US = int(os.environ.get("FASTLSTM_B200_WAIT_LIMIT_US", "0"))


def _desc(dtype, T, B, I, H, flags=0):
    if dtype not in _DTYPE_CODE:
        raise ValueError(f"unsupported dtype {dtype}; expected float32, float16 or bfloat16")
    if _FORCE_GENERIC:
        flags |= _lib.FLAG_FORCE_GENERIC
    return _lib.Desc(_DTYPE_CODE[dtype], T, B, I, H, flags, _WAIT_LIMIT_US, 0)


def check_status(wait: bool = True):
    """Raise if any finished launch recorded a device-side error (a bounded wait
    that ran out).  With wait=True, first waits for all outstanding launches.  (Launches write such an
    error to mapped host memory; every operator call looks there too.)"""
    _lib.host().check_status(bool(wait))


def _profiled(name):
    """record_function while a profiler runs, nothing otherwise (entering one costs 5 us either way)."""
    prof = torch.autograd.profiler
    return prof.record_function(name) if prof._is_profiler_enabled else contextlib.nullcontext()


_PHASES = {"fwd": _lib.PHASE_FWD, "bwd": _lib.PHASE_BWD, "fwd_op": _lib.PHASE_FWD_OP}


def plan_name(dtype, T, B, I, H, phase="fwd"):
    """Kernel family ("generic" / "sm100", for phase "fwd_op" also "fused") the library picks for this
    problem.  Phases: "fwd" / "bwd" = the recurrences, "fwd_op" = the whole forward operator."""
    d = _desc(dtype, T, B, I, H)
    return _lib.load().blstm_plan_name(d, _PHASES[phase]).decode()


def _family(dtype, T, B, I, H, phase, half_device=False):
    """Which kernels (_lib.FAMILY_*) the library picks for this problem, on half of the SMs where half_device."""
    return _lib.load().blstm_plan_family(_desc(dtype, T, B, I, H, _lib.FLAG_HALF_DEVICE if half_device else 0), _PHASES[phase])


def plan_detail(dtype, T, B, I, H, phase="fwd", half_device=False):
    """One-line description of the launch geometry the library picks for this problem (on half of the SMs)."""
    import ctypes
    d = _desc(dtype, T, B, I, H, _lib.FLAG_HALF_DEVICE if half_device else 0)
    buf = ctypes.create_string_buffer(512)
    _lib.check(_lib.load().blstm_plan_detail(d, _PHASES[phase], buf, 512), "blstm_plan_detail")
    return buf.value.decode()


# ---------------------------------------------------------------------------
# Operator functions (same names and argument meaning as the reference)
# ---------------------------------------------------------------------------
def lstm_persistent_fwd(x, h0, c0, Wx, bx, Wh, bh, inference=False, half_device=False):
    """Forward of one layer.  x [T,B,I]; h0,c0 [B,H] or None; Wx [4H,I]; Wh [4H,H];
    bx,bh [4H] or None.  Returns (out[T+1,B,H], cell[T+1,B,H], ifgo[T,B,4H]);
    slot 0 of out/cell is the initial state.  (fastlstm/lstm.py:31-146)
    inference=True: nothing is saved for backward - ifgo and cell[1..T-1] are left unwritten
    (cell[T] is still c_n), which halves the bytes each step moves.
    half_device=True: the recurrence is planned for half of the SMs (two layers side by side)."""
    if x.dim() == 2:
        x = x[None]
    return _lib.host().fwd(x, h0, c0, Wx, bx, Wh, bh, bool(inference), bool(half_device))


def lstm_persistent_bwd(dh, dc_n, dh_n, x, h, cell, ifgo, Wx, Wh, need_dx=True, wgrads=None, half_device=False):
    """Backward of one layer.  dh [T,B,H] gradient of out[1:]; dc_n, dh_n [B,H]
    (or None) gradients of the final states; h = out[T+1,B,H] from forward.
    Returns (d_x, dh_0, dc_0, dWx, dbx, dWh, dbh); weight and bias gradients are
    fp32, dbx is dbh.  (fastlstm/lstm.py:236-334)
    wgrads: optional flat fp32 tensor of 4H*(I+H+1) elements laid out dWx | dWh | db that the
    kernels write into (a data-parallel gradient bucket); allocated here when None."""
    return _lib.host().bwd(dh.contiguous(), dc_n, dh_n, x, h, cell, ifgo, Wx, Wh, bool(need_dx), wgrads, bool(half_device))


def Wgrad(d_ifgo, x, h):
    """(dbx, dbh, dWx, dWh) from d_ifgo [T,B,4H], x [T,B,I], h = out[T+1,B,H].
    (fastlstm/lstm.py:494-501; fp32 results, no transpose copy)"""
    return _lib.host().wgrad(d_ifgo, x, h)


# ---------------------------------------------------------------------------
# Ragged 16-bit shapes on the tensor-core kernels: TMA wants 16-byte row pitches (I % 8 == 0) and the
# tcgen05 recurrences hidden sizes in multiples of 64 (small batches: of 8).  Other shapes are zero-padded on the host: a padded
# hidden unit has zero weights, bias and state, so its pre-activations are 0, its cell and output stay
# exactly 0 and it feeds nothing into the real units; padded input columns meet zero weights.  The
# padded copies cost a few small kernels per call - far less than the CUDA-core kernels they replace.
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=1024)
def _padded_sizes(dtype, I, H, T=1, B=None):
    """(Ip, Hp) when the layer should run zero-padded on the tensor-core kernels, else None.  With a
    batch size: hidden sizes in multiples of 8 where the small-batch recurrences take them."""
    if dtype not in (torch.float16, torch.bfloat16) or _FORCE_GENERIC:
        return None
    if max(I, H) <= 64 and T <= 12:           # tiny sizes have the fused kernel
        return None
    Ip, Hp = -(-I // 8) * 8, -(-H // 8) * 8
    if Ip == I and H % 64 == 0:
        return None
    if B is None or any(plan_name(dtype, T, B, Ip, Hp, phase) != "sm100" for phase in ("fwd", "bwd")):
        Hp = -(-H // 64) * 64
    if (Ip, Hp) == (I, H) or Hp > 2048:
        return None
    return Ip, Hp


def _pad_last(t, n):
    return t if t is None or t.shape[-1] == n else torch.nn.functional.pad(t, (0, n - t.shape[-1]))


def _pad_gates(W, H, Hp, cols=None):
    """[4H, K] (or [4H]) -> [4Hp, cols or K]: every gate's block padded with zero rows (and columns)."""
    if W is None:
        return None
    if W.dim() == 1:
        return torch.nn.functional.pad(W.view(4, H), (0, Hp - H)).reshape(4 * Hp)
    K = W.shape[1]
    cols = K if cols is None else cols
    return torch.nn.functional.pad(W.view(4, H, K), (0, cols - K, 0, Hp - H)).reshape(4 * Hp, cols)


def _unpad_gates(G, H, Hp, cols=None):
    """inverse of _pad_gates for gradients: [4Hp, Kp] -> [4H, cols]."""
    if G.dim() == 1:
        return G.view(4, Hp)[:, :H].reshape(4 * H)
    cols = G.shape[1] if cols is None else cols
    return G.view(4, Hp, G.shape[1])[:, :H, :cols].reshape(4 * H, cols)


class PersistentLSTMfn(torch.autograd.Function):
    """autograd Function of one layer (fastlstm/lstm.py:504-538).

    forward(x, h_0, c_0, Wx, bx, Wh, bh) -> (out[T,B,H], h_n[B,H], c_n[B,H]);
    unlike the reference, h_n and c_n are flat outputs and differentiable."""

    @staticmethod
    def forward(ctx, x, h_0, c_0, Wx, bx, Wh, bh, inference=None, sink=None, want_cells=False):
        if torch.is_autocast_enabled("cuda"):
            target = torch.get_autocast_dtype("cuda")
            x, Wx, Wh = x.to(target), Wx.to(target), Wh.to(target)
            bx = None if bx is None else bx.to(target)
            bh = None if bh is None else bh.to(target)
            h_0 = None if h_0 is None else h_0.to(target)
            c_0 = None if c_0 is None else c_0.to(target)
        x = x.contiguous()
        I, H = x.shape[-1], Wh.shape[1]
        ctx.pad = _padded_sizes(x.dtype, I, H, x.shape[0], x.shape[1])
        ctx.sizes = (I, H)
        if ctx.pad is not None:
            Ip, Hp = ctx.pad
            x = _pad_last(x, Ip)
            Wx, Wh = _pad_gates(Wx, H, Hp, Ip), _pad_gates(Wh, H, Hp, Hp)
            bx, bh = _pad_gates(bx, H, Hp), _pad_gates(bh, H, Hp)
            h_0, c_0 = _pad_last(h_0, Hp), _pad_last(c_0, Hp)
        # Grad mode is always off inside Function.forward and needs_input_grad mirrors requires_grad
        # whatever the grad mode, so the caller (persistent_lstm / FastLSTM.forward) decides whether
        # anything has to be saved; a bare apply() with the reference's seven arguments saves unless
        # no input requires a gradient.
        if inference is None:
            inference = not any(ctx.needs_input_grad)
        ctx.inference = bool(inference)
        ctx.sink = sink
        with _profiled("fastlstm_b200::fwd"):
            out, cell, ifgo = lstm_persistent_fwd(
                x, None if h_0 is None else h_0.contiguous(), None if c_0 is None else c_0.contiguous(),
                Wx.contiguous(), bx, Wh.contiguous(), bh, inference=inference)
        ctx.h0_is_none = h_0 is None
        ctx.has_bias = (bx is not None, bh is not None)
        ctx.save_for_backward(x, out, cell, ifgo, Wx, Wh)
        ctx.want_cells = bool(want_cells)
        res = (out[1:, :, :H], out[-1, :, :H], cell[-1, :, :H]) if ctx.pad is not None else (out[1:], out[-1], cell[-1])
        if want_cells:
            # cell states of every step, for callers that need c at a step other than the last (packed
            # sequences of different lengths); no gradient flows back through this output
            cells = cell[1:, :, :H] if ctx.pad is not None else cell[1:]
            ctx.mark_non_differentiable(cells)
            return res + (cells,)
        return res

    @staticmethod
    def backward(ctx, d_out, d_hn, d_cn, *_):
        if ctx.inference:
            raise RuntimeError("this forward ran in inference mode (nothing was saved); backward is not possible")
        x, out, cell, ifgo, Wx, Wh = ctx.saved_tensors
        T, B, H = out.shape[0] - 1, out.shape[1], out.shape[2]
        if d_out is None:
            d_out = torch.zeros((T, B, H), device=x.device, dtype=x.dtype)
        d_out = d_out.to(x.dtype)
        d_hn = None if d_hn is None else d_hn.to(x.dtype)
        d_cn = None if d_cn is None else d_cn.to(x.dtype)
        if ctx.pad is not None:
            d_out, d_hn, d_cn = _pad_last(d_out, H), _pad_last(d_hn, H), _pad_last(d_cn, H)   # H is the padded size here
        d_out = d_out.contiguous()
        d_hn = None if d_hn is None else d_hn.contiguous()
        d_cn = None if d_cn is None else d_cn.contiguous()
        with _profiled("fastlstm_b200::bwd"):
            d_x, dh_0, dc_0, dWx, dbx, dWh, dbh = lstm_persistent_bwd(
                d_out, d_cn, d_hn, x, out, cell, ifgo, Wx.contiguous(), Wh.contiguous(),
                need_dx=ctx.needs_input_grad[0],
                wgrads=None if (ctx.sink is None or ctx.pad is not None) else ctx.sink.buffer)
        if ctx.pad is not None:
            I0, H0 = ctx.sizes
            d_x = None if d_x is None else d_x[..., :I0]
            dh_0, dc_0 = dh_0[:, :H0], dc_0[:, :H0]
            dWx, dWh = _unpad_gates(dWx, H0, H, I0), _unpad_gates(dWh, H0, H, H0)
            dbx = dbh = _unpad_gates(dbx, H0, H)
        if ctx.h0_is_none:
            dh_0 = dc_0 = None
        if ctx.sink is not None and ctx.pad is not None:
            # padded layer: the kernels wrote padded gradients, the bucket takes the unpadded ones
            n1, n2 = dWx.numel(), dWx.numel() + dWh.numel()
            ctx.sink.buffer[:n1].copy_(dWx.reshape(-1))
            ctx.sink.buffer[n1:n2].copy_(dWh.reshape(-1))
            ctx.sink.buffer[n2:].copy_(dbx)
        if ctx.sink is not None:
            # the fp32 gradients went straight into the caller's bucket segment: autograd sees none
            # (it would round them to the parameter dtype), the bucket hands them to p.grad later
            ctx.sink.filled()
            return (d_x, dh_0, dc_0, None, None, None, None, None, None, None)
        return (d_x, dh_0, dc_0, dWx, dbx if ctx.has_bias[0] else None, dWh,
                dbh if ctx.has_bias[1] else None, None, None, None)


def _layer(x, h0, c0, Wx, bx, Wh, bh, inference, stacked=False, want_cells=False, main=None):
    """One layer on the GPU, as PersistentLSTMfn computes it (same casts, padding and gradients), with the
    conversions in one launch and the autograd node in the host extension.  stacked: the final states come as
    tensors [1,B,H] of their own.  want_cells: also the cell states of every step (no gradient).  main: planned
    for half of the device, another layer runs beside it; the stream that the gradients will be used on."""
    host = _lib.host()
    if (h0 is None) != (c0 is None):
        raise ValueError("h0 and c0 must both be given or both be None")
    to = torch.get_autocast_dtype("cuda") if torch.is_autocast_enabled("cuda") else None
    T, B, I = x.shape
    H = Wh.shape[1]
    Ip, Hp = _padded_sizes(x.dtype if to is None else to, I, H, T, B) or (0, 0)
    xp, h0p, c0p, Wxp, bxp, Whp, bhp = host.prepare(x, h0, c0, Wx, bx, Wh, bh, to, Ip, Hp)
    with _profiled("fastlstm_b200::fwd"):
        out, cell, ifgo = lstm_persistent_fwd(xp, h0p, c0p, Wxp, bxp, Whp, bhp, inference=inference, half_device=main is not None)
    if not inference:
        on = None if main is None else (main.stream_id, main.device_index, main.device_type)
        res = host.attach(x, h0, c0, Wx, bx, Wh, bh, xp, Wxp, Whp, out, cell, ifgo, stacked, on)
    else:
        res = out[1:, :, :H], out[-1, :, :H], cell[-1, :, :H]
        if stacked:
            res = res[0], res[1][None].clone(), res[2][None].clone()
    return res + (cell[1:, :, :H],) if want_cells else res


@functools.lru_cache(maxsize=1024)
def _shares_device(dtype, T, B, I, H):
    """True when two launches of this layer's recurrences can run side by side to advantage: clusters that wait
    for nothing outside themselves, and enough steps to pay for the streams (some 30 us of host time)."""
    Ip, Hp = _padded_sizes(dtype, I, H, T, B) or (I, H)
    return T >= 48 and all(_family(dtype, T, B, Ip, Hp, phase) == _lib.FAMILY_SMALL_BATCH for phase in ("fwd", "bwd"))


@functools.lru_cache(maxsize=1024)
def _wavefront_pays(dtype, T, B, H, grad):
    """Whether a stack that could run as a wavefront should.  Two layers, ms layer after layer / as a wavefront (B200):

    Without gradients the small-batch recurrences have SMs to spare only while a layer's clusters fit beside the other's
    with no more rows to work through in turn; the launches of a wavefront then take some 0.45 ms of the host
    (B=64, H=64: T=256 0.33 / 0.42, T=512 0.59 / 0.50, T=1024 1.10 / 0.83; B=16, H=128: T=256 0.38 / 0.42, T=512 0.69 / 0.57; B=8,
    H=512: T=128 0.47 / 0.45, T=512 1.61 / 1.16; but B=64, H=192: T=1024 1.58 / 1.70, B=1000, H=64: 1.37 / 1.78).  Where a cluster has
    four chunks in turn, from H = 384 on three, and half of the device would have resident weights, 32 rows to a group of H / 32 CTAs at
    most, these win (T=256: B=200, H=320 1.50 / 1.30; B=130, H=448 1.50 / 1.37; B=150, H=384 1.33 / 1.33, T=512 2.57 / 2.41; but
    B=400, H=256, 48 rows, 1.32 / 1.59; B=100, H=512, two chunks, 1.26 / 1.37).
    Resident weights gain from 128 steps on where half of the device holds them with two tiles of rows, 64 to a group of H / 32 CTAs at most
    (T=128 and 256: B=128, H=512 0.81 / 0.65 and 1.56 / 1.17; B=448, H=320 0.90 / 0.82 and 1.75 / 1.53; B=128, H=1024 1.09 / 1.05 and 2.13 / 1.91), the kernels
    with several 128-row tiles always (T=128, B=1000, H=192: 1.31 / 1.05).  With three or four tiles a group on half of the device the
    layers stay one after the other, where the cell state is held in 32 bits over the whole sequence: as a wavefront the error of the
    output against 64 bits grows by 0.06 to 0.3 % (bf16 and fp16, T=512 and T=128).  It would gain at some of these sizes and lose at
    others (T=128 and 256: B=704, H=256 1.10 / 0.90 and 2.14 / 1.65; B=512, H=512 1.25 / 1.20 and 2.45 / 2.23; B=256, H=768
    1.27 / 1.18 and 2.48 / 2.19; but B=288, H=512 0.93 / 0.97 and 1.80 / 1.80; B=256, H=832 1.33 / 1.37 and 2.60 / 2.56; B=130, H=896
    1.03 / 1.16 and 1.98 / 2.14; B=256, H=1024 1.51 / 1.70 and 3.01 / 3.19).

    A training step's launches for every chunk cost more, so not where both directions stay on the chip (T=256, B=512, H=512
    6.4 / 6.8; T=256, B=32, H=256 1.25 / 1.8) nor for few steps (T=64, B=712, H=320: 1.78 / 1.95, T=128: 3.27 / 3.3, T=256:
    6.30 / 6.00; B=768, H=384: 2.18 / 2.22, 4.10 / 3.88, 7.97 / 7.15; B=968, H=192: 1.78 / 1.82, T=96: 2.54 / 2.33, T=256 6.33 / 5.37), and not at H=576, where half
    of the device gives backward four tiles a CTA (B=392: T=128 4.13 / 4.64, T=256 8.02 / 8.55, T=512 15.8 / 16.4)."""
    on_chip = (_lib.FAMILY_RESIDENT, _lib.FAMILY_SMALL_BATCH)
    fwd = _family(dtype, T, B, H, H, "fwd")
    if grad:
        return T >= (96 if H < 320 else 128) and H <= 384 and not (fwd in on_chip and _family(dtype, T, B, H, H, "bwd") in on_chip)
    if fwd == _lib.FAMILY_BATCH_TILES:
        return True
    half = _family(dtype, T, B, H, H, "fwd", True)
    if fwd == _lib.FAMILY_RESIDENT:
        return T >= 128 and half in on_chip and B <= 64 * (74 // (H // 32))
    lib, whole, part = _lib.load(), _desc(dtype, T, B, H, H), _desc(dtype, T, B, H, H, _lib.FLAG_HALF_DEVICE)
    turns = lib.blstm_plan_turns(whole, _lib.PHASE_FWD)
    if half == _lib.FAMILY_SMALL_BATCH:
        return (T >= (128 if H >= 512 else 192) and T * (H + 64) >= 65536
                and turns == lib.blstm_plan_turns(part, _lib.PHASE_FWD) and lib.blstm_plan_beside(part, _lib.PHASE_FWD) >= 2)
    long_enough = T >= 128 if turns >= 4 else turns == 3 and H >= 384 and T >= 256
    return half == _lib.FAMILY_RESIDENT and long_enough and B <= 32 * (74 // (H // 32))


class _Beside:
    """Runs the second direction of a layer on the side stream beside the first.  Entering makes the side stream wait for
    everything so far, join() makes the current stream wait for the side stream, and release(), behind the readers of what
    the side stream has made, the side stream for them: it may get that memory back before they have run.  The other way
    round the last holder of a tensor can be a backward node of the side stream, so what that stream reads of the current
    one's memory - the input, row maps, weights that are not parameters - is recorded with the allocator, and so are the
    gradients its nodes hand out (LayerState in csrc/host.cpp).  A no-op where `on` is false."""

    def __init__(self, device, on, *reads):
        self.main = torch.cuda.current_stream(device) if on else None
        self.side = _side_stream(device) if on else None
        if on:
            for t in reads:
                if t is not None and not isinstance(t, nn.Parameter):     # (parameters outlive the graph)
                    t.record_stream(self.side)
            self.side.wait_stream(self.main)

    def stream(self, d):
        return torch.cuda.stream(self.side) if d and self.side is not None else contextlib.nullcontext()

    def join(self):
        if self.side is not None:
            self.main.wait_stream(self.side)

    def release(self):
        if self.side is not None:
            self.side.wait_stream(self.main)


_side_streams = {}


def _side_stream(device):
    """One extra stream per device for the layer wavefront (created once, reused)."""
    key = torch.device(device).index if torch.device(device).index is not None else torch.cuda.current_device()
    if key not in _side_streams:
        _side_streams[key] = torch.cuda.Stream(device=key)
    return _side_streams[key]


class WavefrontLSTMfn(torch.autograd.Function):
    """A unidirectional stack of layers as ONE autograd node that runs the layers as a wavefront over
    time chunks: layer l works on chunk k while layer l-1 works on chunk k+1, on two streams, each
    recurrence planned for half of the SMs (the reference runs the layers one after the other,
    fastlstm/lstm.py:685-696, and lists the wavefront as missing, README.md:94).  It pays when a
    layer alone cannot fill the GPU: few batch tiles, every CTA with one tile, every step one
    hand-off chain.  A chunk is an ordinary call of the layer operators with the previous chunk's
    final state as its initial state (the cell state crosses a chunk boundary in the storage dtype).

    forward(x[T,B,I], n_chunks, sinks, inference, h0, c0, *params) with params = (Wx, bx, Wh, bh) per
    layer, h0/c0 [L,B,H] or None  ->  (out[T,B,H], h_n[L,B,H], c_n[L,B,H]).  inference=True: nothing is
    saved for backward and the recurrences skip the stores only backward needs."""

    @staticmethod
    def forward(ctx, x, n_chunks, sinks, inference, h0, c0, *params):
        L = len(params) // 4
        T = x.shape[0]
        x = x.contiguous()
        bounds = [(T * k) // n_chunks for k in range(n_chunks + 1)]
        chunks = [(bounds[k], bounds[k + 1]) for k in range(n_chunks) if bounds[k + 1] > bounds[k]]
        NC = len(chunks)
        main = torch.cuda.current_stream(x.device)
        streams = [main, _side_stream(x.device)]
        streams[1].wait_stream(main)
        saved = [[None] * NC for _ in range(L)]
        done = [[None] * NC for _ in range(L)]
        with _profiled("fastlstm_b200::wavefront_fwd"):
            for diag in range(NC + L - 1):
                for l in range(L):
                    k = diag - l
                    if k < 0 or k >= NC:
                        continue
                    Wx, bx, Wh, bh = params[4 * l:4 * l + 4]
                    st = streams[l % 2]
                    if l > 0:
                        st.wait_event(done[l - 1][k])
                    with torch.cuda.stream(st):
                        t0, t1 = chunks[k]
                        xc = x[t0:t1] if l == 0 else saved[l - 1][k][1][1:]
                        if k == 0:
                            hp = None if h0 is None else h0[l].contiguous()
                            cp = None if c0 is None else c0[l].contiguous()
                        else:
                            hp, cp = saved[l][k - 1][1][-1], saved[l][k - 1][2][-1]
                        out, cell, ifgo = lstm_persistent_fwd(xc, hp, cp, Wx.contiguous(), bx, Wh.contiguous(), bh,
                                                              inference=bool(inference), half_device=True)
                        saved[l][k] = (xc, out, cell, None if inference else ifgo)
                        done[l][k] = torch.cuda.Event()
                        done[l][k].record(st)
            main.wait_stream(streams[1])
            top = saved[L - 1]
            y = torch.cat([top[k][1][1:] for k in range(NC)], dim=0) if NC > 1 else top[0][1][1:].clone()
            h_n = torch.stack([saved[l][NC - 1][1][-1] for l in range(L)])
            c_n = torch.stack([saved[l][NC - 1][2][-1] for l in range(L)])
            # (the side stream may get its memory back before the reads above have run)
            streams[1].wait_stream(main)
        ctx.inference = bool(inference)
        if not inference:
            ctx.saved = saved
            ctx.params = params
            ctx.sinks = sinks
            ctx.chunks = chunks
            ctx.had_state = h0 is not None
        return y, h_n, c_n

    @staticmethod
    def backward(ctx, d_out, d_hn, d_cn):
        if ctx.inference:
            raise RuntimeError("this forward ran in inference mode (nothing was saved); backward is not possible")
        saved, params, chunks, sinks = ctx.saved, ctx.params, ctx.chunks, ctx.sinks
        L, NC = len(saved), len(chunks)
        x0 = saved[0][0][0]
        dt, dev = x0.dtype, x0.device
        B, H = saved[0][0][1].shape[1], saved[0][0][1].shape[2]
        main = torch.cuda.current_stream(dev)
        streams = [main, _side_stream(dev)]
        streams[1].wait_stream(main)
        d_out = None if d_out is None else d_out.to(dt).contiguous()
        d_hn = None if d_hn is None else d_hn.to(dt).contiguous()
        d_cn = None if d_cn is None else d_cn.to(dt).contiguous()
        need_dx0 = ctx.needs_input_grad[0]
        dx = [[None] * NC for _ in range(L)]
        carry = [[None] * NC for _ in range(L)]
        done = [[None] * NC for _ in range(L)]
        acc = [None] * L
        with _profiled("fastlstm_b200::wavefront_bwd"):
            for diag in range(NC + L - 1):
                for li in range(L):
                    l = L - 1 - li
                    k = NC - 1 - (diag - li)
                    if k < 0 or k >= NC:
                        continue
                    Wx, bx, Wh, bh = params[4 * l:4 * l + 4]
                    st = streams[l % 2]
                    if l < L - 1:
                        st.wait_event(done[l + 1][k])
                    with torch.cuda.stream(st):
                        xc, out, cell, ifgo = saved[l][k]
                        t0, t1 = chunks[k]
                        if l == L - 1:
                            dh = d_out[t0:t1] if d_out is not None else torch.zeros((t1 - t0, B, H), device=dev, dtype=dt)
                        else:
                            dh = dx[l + 1][k]
                        if k == NC - 1:
                            dh_n = None if d_hn is None else d_hn[l]
                            dc_n = None if d_cn is None else d_cn[l]
                        else:
                            dh_n, dc_n = carry[l][k + 1]
                        I = xc.shape[-1]
                        first = acc[l] is None
                        buf = torch.empty(4 * H * (I + H + 1), device=dev, dtype=torch.float32)
                        d_x, dh_0, dc_0, _, _, _, _ = lstm_persistent_bwd(
                            dh, dc_n, dh_n, xc, out, cell, ifgo, Wx.contiguous(), Wh.contiguous(),
                            need_dx=(l > 0 or need_dx0), wgrads=buf, half_device=True)
                        if first:
                            acc[l] = buf
                        else:
                            acc[l].add_(buf)
                        dx[l][k], carry[l][k] = d_x, (dh_0, dc_0)
                        if k == 0 and sinks is not None:
                            # the layer's fp32 gradients go straight into its bucket segment, whose
                            # all-reduce starts here, beside the backward of the layers below
                            sinks[l].buffer.copy_(acc[l])
                            sinks[l].filled()
                        done[l][k] = torch.cuda.Event()
                        done[l][k].record(st)
            main.wait_stream(streams[1])
            d_x = None
            if need_dx0:
                d_x = torch.cat(dx[0], dim=0) if NC > 1 else dx[0][0]
            dh0 = dc0 = None
            if ctx.had_state:
                dh0 = torch.stack([carry[l][0][0] for l in range(L)])
                dc0 = torch.stack([carry[l][0][1] for l in range(L)])
            streams[1].wait_stream(main)
            for l in range(1, L, 2):
                acc[l].record_stream(main)       # (the parameters' gradients are used there)
        grads = []
        for l in range(L):
            Wx, bx, Wh, bh = params[4 * l:4 * l + 4]
            if sinks is not None:
                grads += [None, None, None, None]
                continue
            I = Wx.shape[1]
            dWx = acc[l][:4 * H * I].view(4 * H, I)
            dWh = acc[l][4 * H * I:4 * H * (I + H)].view(4 * H, H)
            db = acc[l][4 * H * (I + H):]
            grads += [dWx, db if bx is not None else None, dWh, db if bh is not None else None]
        return (d_x, None, None, None, dh0, dc0, *grads)


def _nothing_to_save(*tensors):
    """True when no backward can follow this forward: grad mode is off, or no input requires one."""
    return not (torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in tensors))


def persistent_lstm(x, h_0, c_0, Wx, bx, Wh, bh):
    """Reference-shaped call: returns (out, (h_n, c_n)) like PersistentLSTMfn.apply
    does in fastlstm/lstm.py:522."""
    inference = _nothing_to_save(x, h_0, c_0, Wx, bx, Wh, bh)
    out, h_n, c_n = PersistentLSTMfn.apply(x, h_0, c_0, Wx, bx, Wh, bh, inference, None)
    return out, (h_n, c_n)


class FastLSTM(nn.Module):
    """nn.LSTM-style stacked LSTM on the B200 kernels (fastlstm/lstm.py:586-698).

    Parameters have nn.LSTM's names, shapes, registration order, init distribution and RNG order
    (weight_ih_l{k}[_reverse], weight_hh_l{k}[_reverse], bias_ih_l{k}[_reverse],
    bias_hh_l{k}[_reverse]), so state dicts are interchangeable with torch.nn.LSTM.  `version` is
    accepted for source compatibility; only "persistent" exists here.

    Beyond the reference (which lists them as missing, README.md:92-93): `bidirectional` runs the
    same kernels on the time-reversed input and concatenates the two directions' outputs
    (states are ordered layer-major, direction-minor, like nn.LSTM); `dropout` is applied to
    the outputs of every layer but the last while training; a `PackedSequence` input gives a
    `PackedSequence` output and the states at every sequence's own last step.  `proj_size` > 0 adds
    nn.LSTM's output projection (`weight_hr_l{k}`: h_t = W_hr (o * tanh(c_t)), recurrent weights
    [4H, proj_size])."""

    def __init__(self, input_size, hidden_size, num_layers=1, *, bias=True, batch_first=False,
                 version="persistent", device=None, dtype=None, dropout=0.0, bidirectional=False,
                 proj_size=0):
        # Everything after num_layers is keyword-only: the reference's positional order continues with
        # (version, device, dtype), nn.LSTM's with (bias, batch_first, dropout, ...); a positional call
        # written for either would silently bind the wrong option here, so it raises TypeError instead.
        super().__init__()
        if not isinstance(bias, bool) or not isinstance(batch_first, bool):
            raise TypeError("bias and batch_first must be bool")
        if version != "persistent":
            raise ValueError(f"Not implemented: {version} (only 'persistent' exists)")
        if not isinstance(proj_size, int) or proj_size < 0:
            raise ValueError("proj_size should be a positive integer or zero to disable projections")
        if proj_size >= hidden_size:
            raise ValueError("proj_size has to be a positive integer, smaller than hidden_size")
        if not 0.0 <= float(dropout) <= 1.0:
            raise ValueError("dropout should be a number in range [0, 1]")
        self.input_size, self.hidden_size, self.num_layers = input_size, hidden_size, num_layers
        self.bias, self.batch_first, self.version = bias, batch_first, version
        self.dropout, self.bidirectional = float(dropout), bool(bidirectional)
        self.num_directions = 2 if bidirectional else 1
        self.proj_size = proj_size
        self._sinks = None            # per (layer, direction) gradient sinks of a GradBucket, or None
        self._names = {(layer, d): tuple(f"{n}_l{layer}{sfx}" for n in ("weight_ih", "bias_ih", "weight_hh", "bias_hh"))
                       for layer in range(num_layers) for d, sfx in enumerate(self._suffixes())}
        k = 1.0 / hidden_size ** 0.5
        fk = dict(device=device, dtype=dtype)

        def u(*shape):
            return nn.Parameter(torch.rand(*shape, **fk) * 2 * k - k)

        out_size = proj_size if proj_size > 0 else hidden_size       # width of h (and of a layer's output)
        for layer in range(num_layers):
            in_l = input_size if layer == 0 else out_size * self.num_directions
            for sfx in self._suffixes():
                setattr(self, f"weight_ih_l{layer}{sfx}", u(4 * hidden_size, in_l))
                setattr(self, f"weight_hh_l{layer}{sfx}", u(4 * hidden_size, out_size))
                if bias:
                    setattr(self, f"bias_ih_l{layer}{sfx}", u(4 * hidden_size))
                    setattr(self, f"bias_hh_l{layer}{sfx}", u(4 * hidden_size))
                if proj_size > 0:
                    setattr(self, f"weight_hr_l{layer}{sfx}", u(proj_size, hidden_size))

    def _suffixes(self):
        return ("", "_reverse") if self.bidirectional else ("",)

    def layer_params(self, layer, reverse=False):
        own = self._parameters           # (a reparametrised weight is an attribute instead)
        return tuple(own[n] if n in own else getattr(self, n, None) for n in self._names[layer, int(reverse)])

    def _projected_layer(self, x_d, h0, c0, Wx, bx, Wh, bh, Whr, inference):
        """One direction of one layer with an output projection (nn.LSTM's proj_size).  With m_t = o * tanh(c_t)
        and h_t = W_hr m_t the recurrent term W_hh h_t is (W_hh W_hr) m_t: the unprojected state m is an ordinary
        layer of width H with the recurrent weights W_hh W_hr, the projection of all steps one product behind it.
        A given h_0 enters as further input columns (weights W_hh) that are zero but at the first step.  Returns
        (out [T,B,P], h_n [B,P], c_n [B,H]).  (Step by step, one launch of the cell and a product per step, a
        training step of 60 steps of 32 rows at H = 512 took 31 ms, this way 0.5.)"""
        T, B = x_d.shape[0], x_d.shape[1]
        m0 = None
        if h0 is not None:
            first = torch.cat([h0[None].to(x_d.dtype), x_d.new_zeros(T - 1, B, self.proj_size)]) if T > 1 else h0[None].to(x_d.dtype)
            x_d, Wx = torch.cat([x_d, first], dim=-1), torch.cat([Wx, Wh], dim=-1)
            m0 = x_d.new_zeros(B, self.hidden_size)
        W = Wh @ Whr
        if x_d.is_cuda:
            m, _, c_n = _layer(x_d, m0, c0, Wx, bx, W, bh, inference)
        else:
            m, _, c_n = PersistentLSTMfn.apply(x_d, m0, c0, Wx, bx, W, bh, inference, None)
        out = m @ Whr.t()
        return out, out[-1], c_n

    def _projected_steps(self, x_d, h0, c0, Wx, bx, Wh, bh, Whr, inference):
        """The same as T single-step calls of the cell (the operator with T = 1; the projected state is zero-padded
        to the cell's width and `Wh` [4H,P] to [4H,H], which is exact) with the projection in between, for packed
        input: every step's cell state is differentiable.  Returns (out [T,B,P], cells [T,B,H], h_n [B,P],
        c_n [B,H])."""
        T, B = x_d.shape[0], x_d.shape[1]
        H, P = self.hidden_size, self.proj_size
        pad = torch.nn.functional.pad
        Wh_wide = pad(Wh, (0, H - P))
        h = x_d.new_zeros(B, P) if h0 is None else h0
        c = c0
        outs, cells = [], []
        for t in range(T):
            o, _, c = PersistentLSTMfn.apply(x_d[t:t + 1], pad(h, (0, H - P)), c, Wx, bx, Wh_wide, bh, inference, None)
            h = o[0] @ Whr.t()
            outs.append(h)
            cells.append(c)
        return torch.stack(outs), torch.stack(cells), h, c

    def forward(self, x, h_c_0=None):
        if isinstance(x, torch.nn.utils.rnn.PackedSequence):
            return self._forward_packed(x, h_c_0)
        if x.dim() != 3:
            raise ValueError("expected a 3-D input [T,B,I] (or [B,T,I] with batch_first)")
        if not torch.is_grad_enabled():
            res = self._forward_inference(x, h_c_0)
            if res is not None:
                return res
        if self.batch_first:
            x = x.transpose(0, 1)
        return self._forward_padded(x, h_c_0, None)

    def _forward_inference(self, x, h_c_0):
        """Grad mode off, one direction, nothing to convert or pad: the layers without autograd nodes; a single
        timestep, where the host is what takes the time, in one call of the host extension.  None when the
        general path has to run."""
        if (self.num_directions != 1 or self.proj_size > 0 or not x.is_cuda or torch.is_autocast_enabled("cuda")
                or (self.dropout > 0.0 and self.training and self.num_layers > 1)):
            return None
        L, H, dt = self.num_layers, self.hidden_size, x.dtype
        T, B = (x.shape[1], x.shape[0]) if self.batch_first else (x.shape[0], x.shape[1])
        if T > 1 and (self._wavefront(x.transpose(0, 1) if self.batch_first else x, h_c_0, None, False)
                      or any(_padded_sizes(dt, n, H, T, B) is not None for n in {x.shape[2], H})):
            return None
        if T == 1 and dt != torch.float32 and (H % 8 or x.shape[2] % 8):
            return None
        h0 = c0 = None
        if h_c_0 is not None:
            h0, c0 = h_c_0
            if not (torch.is_tensor(h0) and torch.is_tensor(c0) and h0.dim() == 3 and c0.dim() == 3
                    and h0.shape[0] == L and c0.shape[0] == L and h0.dtype == dt and c0.dtype == dt):
                return None
        params = []
        for layer in range(L):
            params += self.layer_params(layer)
        if any(p is not None and p.dtype != dt for p in params):
            return None
        if T == 1:
            out, h_n, c_n = _lib.host().infer(x, h0, c0, params, self.batch_first)
            return out, (h_n, c_n)
        x = (x.transpose(0, 1) if self.batch_first else x).contiguous()
        h_n, c_n = [], []
        for layer in range(L):
            Wx, bx, Wh, bh = params[4 * layer:4 * layer + 4]
            out, cell, _ = lstm_persistent_fwd(x, None if h0 is None else h0[layer].contiguous(),
                                               None if c0 is None else c0[layer].contiguous(),
                                               Wx.contiguous(), bx, Wh.contiguous(), bh, inference=True)
            x = out[1:]
            h_n.append(out[-1])
            c_n.append(cell[-1])
        return x.transpose(0, 1) if self.batch_first else x, (torch.stack(h_n), torch.stack(c_n))

    def _forward_packed(self, seq, h_c_0):
        """PackedSequence input (torch.nn.LSTM's convention; the reference lists it as missing,
        README.md:92-93).  The sequences are padded to the longest, every layer runs over all T steps
        (steps past a sequence's end compute values nobody reads - the recurrence is causal), the
        final states are read at each sequence's own last step, and the output is packed again with
        the input's ordering.  The reverse direction of a bidirectional layer walks every sequence
        from its own end.  Gradients flow through the packed output and h_n; c_n of sequences shorter
        than the longest carries no gradient."""
        from torch.nn.utils.rnn import PackedSequence, pack_padded_sequence, pad_packed_sequence
        if seq.data.is_cuda and self.proj_size == 0 and self._sinks is None:
            return self._forward_packed_rows(seq, h_c_0)
        x, lengths = pad_packed_sequence(seq, batch_first=False)          # [T,B,I], original batch order
        out, states = self._forward_padded(x, h_c_0, lengths.to(x.device))
        if seq.sorted_indices is not None:
            out, lengths = out.index_select(1, seq.sorted_indices), lengths[seq.sorted_indices.cpu()]
        data = pack_padded_sequence(out, lengths, enforce_sorted=True).data
        return PackedSequence(data, seq.batch_sizes, seq.sorted_indices, seq.unsorted_indices), states

    def _forward_packed_rows(self, seq, h_c_0):
        """_forward_packed on the GPU: row gathers between the packed rows and the padded [T,B] grid, one kernel
        each whatever T, with gathers as gradients.  The reverse direction reads its input turned and leaves its
        output so; steps past a sequence's end are never read, so nothing masks them."""
        from torch.nn.utils.rnn import PackedSequence
        host = _lib.host()
        nd, data = self.num_directions, seq.data
        T, B = seq.batch_sizes.numel(), int(seq.batch_sizes[0])
        padded, turned, rev, inv_last, last, packed, packed_t = host.packed_maps(seq.batch_sizes, seq.unsorted_indices, data)
        h_0, c_0 = self._initial_states(h_c_0)
        h_n, c_n, x = [], [], None
        dt = torch.get_autocast_dtype("cuda") if torch.is_autocast_enabled("cuda") else data.dtype
        for layer in range(self.num_layers):
            outs, top = [], layer == self.num_layers - 1
            half = nd == 2 and _shares_device(dt, T, B, (data if x is None else x).shape[-1], self.hidden_size)
            if x is None:
                xs = [host.gather_rows(data, *maps, [T, B]) for maps in ((padded, packed), (turned, packed_t))[:nd]]
            else:
                xs = [x] if nd == 1 else [x, host.gather_rows(x, rev, rev, [T, B])]
            params = [self.layer_params(layer, reverse=(d == 1)) for d in range(nd)]
            beside = _Beside(data.device, half, xs[-1], turned, *params[-1])        # (the maps are views of one tensor)
            for d, x_d in enumerate(xs):
                Wx, bx, Wh, bh = params[d]
                hl, cl = h_0[layer * nd + d], c_0[layer * nd + d]
                with beside.stream(d):
                    inference = _nothing_to_save(x_d, hl, cl, Wx, bx, Wh, bh)
                    o, _, _, cells = _layer(x_d, hl, cl, Wx, bx, Wh, bh, inference, want_cells=True, main=beside.main)
                    h_n.append(host.gather_rows(o, last, inv_last, [B]))       # states at each sequence's own last step
                    c_n.append(host.gather_rows(cells, last, inv_last, [B]))
                    if top:
                        o = host.gather_rows(o, packed_t if d else packed, turned if d else padded, [data.shape[0]])
                    elif d:
                        o = host.gather_rows(o, rev, rev, [T, B])
                outs.append(o)
            beside.join()
            x = outs[0] if nd == 1 else torch.cat(outs, dim=-1)
            if top:
                states = torch.stack(h_n), torch.stack(c_n)
            beside.release()
            if self.dropout > 0.0 and self.training and not top:
                x = torch.nn.functional.dropout(x, self.dropout, True)
        return PackedSequence(x, seq.batch_sizes, seq.sorted_indices, seq.unsorted_indices), states

    def _initial_states(self, h_c_0):
        """One (h_0, c_0) per layer and direction, or Nones."""
        n = self.num_layers * self.num_directions
        if h_c_0 is None:
            return [None] * n, [None] * n
        h_0, c_0 = h_c_0
        if h_0 is None or c_0 is None:
            raise ValueError("h_c_0 must be a pair (h_0, c_0) of [num_layers * num_directions, B, H] "
                             "tensors or None")
        if len(h_0) != n or len(c_0) != n:
            raise ValueError(f"expected {n} initial states, got {len(h_0)} / {len(c_0)}")
        return h_0, c_0

    def _wavefront_chunks(self, x, h_c_0, lengths):
        """Number of time chunks for the layer wavefront, or 0 when the stack runs layer after layer.
        The wavefront needs two or more layers of one direction on the tensor-core kernels and pays
        when a layer alone leaves the GPU latency bound: every CTA has a single batch tile on the
        whole device and at most two on half of it."""
        if (x.shape[0] < 64 or self.num_layers < 2 or self.num_directions != 1 or self.proj_size > 0 or lengths is not None
                or (self.dropout > 0.0 and self.training) or not x.is_cuda
                or x.dtype not in (torch.float16, torch.bfloat16) or torch.is_autocast_enabled("cuda")):
            return 0
        T, B, I = x.shape
        H = self.hidden_size
        if H % 64 != 0 or H > 1024 or I % 8 != 0 or os.environ.get("FASTLSTM_B200_WAVEFRONT", "1") == "0":
            return 0
        if any(p.dtype != x.dtype for p in self.parameters()):
            return 0
        sms = 148
        tiles, ctas_per_tile = -(-B // 128), H // 16
        if ctas_per_tile > sms // 2:          # (a single tile's CTAs must fit on half of the SMs)
            return 0
        if tiles > sms // ctas_per_tile or tiles > 2 * ((sms // 2) // ctas_per_tile):
            return 0
        return max(1, min(int(os.environ.get("FASTLSTM_B200_WAVEFRONT_CHUNKS", "4")), T // 16))

    def _wavefront(self, x, h_c_0, lengths, grad):
        """Number of time chunks that this call runs as a wavefront over, or 0."""
        n = self._wavefront_chunks(x, h_c_0, lengths)
        return n if n and _wavefront_pays(x.dtype, x.shape[0], x.shape[1], self.hidden_size, grad) else 0

    def _forward_wavefront(self, x, h_c_0, n_chunks):
        h0 = c0 = None
        if h_c_0 is not None:
            h0, c0 = h_c_0
            if h0 is None or c0 is None:
                raise ValueError("h_c_0 must be a pair (h_0, c_0) of [num_layers, B, H] tensors or None")
            h0 = torch.stack(list(h0)) if not torch.is_tensor(h0) else h0
            c0 = torch.stack(list(c0)) if not torch.is_tensor(c0) else c0
            if h0.shape[0] != self.num_layers or c0.shape[0] != self.num_layers:
                raise ValueError(f"expected {self.num_layers} initial states, got {h0.shape[0]} / {c0.shape[0]}")
            h0, c0 = h0.to(x.dtype), c0.to(x.dtype)
        params = []
        for layer in range(self.num_layers):
            params += list(self.layer_params(layer))
        inference = _nothing_to_save(x, h0, c0, *params)
        out, h_n, c_n = WavefrontLSTMfn.apply(x, n_chunks, self._sinks, inference, h0, c0, *params)
        if self.batch_first:
            out = out.transpose(0, 1)
        return out, (h_n, c_n)

    def _forward_padded(self, x, h_c_0, lengths):
        """x [T,B,I]; lengths: None, or the [B] valid lengths (device tensor) of padded sequences."""
        n_chunks = self._wavefront(x, h_c_0, lengths, torch.is_grad_enabled())
        if n_chunks:
            return self._forward_wavefront(x, h_c_0, n_chunks)
        nd = self.num_directions
        T, B = x.shape[0], x.shape[1]
        if lengths is not None:
            steps = torch.arange(T, device=x.device)[:, None]                       # [T,1]
            valid = steps < lengths[None, :]                                         # [T,B]
            # per-sequence time reversal (identity past the end) and the index of the last valid step
            rev = torch.where(valid, lengths[None, :] - 1 - steps, steps)            # [T,B]
            last = (lengths - 1).clamp(min=0)                                        # [B]

            def reverse_time(t):
                return t.gather(0, rev[:, :, None].expand(-1, -1, t.shape[2]))

            def at_last(t):                                                          # [T,B,H] -> [B,H]
                return t.gather(0, last[None, :, None].expand(1, -1, t.shape[2]))[0]
        h_0, c_0 = self._initial_states(h_c_0)
        h_n, c_n = [], []
        single = (self.num_layers * nd == 1 and self.proj_size == 0 and lengths is None and self._sinks is None and x.is_cuda)
        dt = torch.get_autocast_dtype("cuda") if torch.is_autocast_enabled("cuda") else x.dtype
        for layer in range(self.num_layers):
            outs = []
            half = (nd == 2 and x.is_cuda and lengths is None and self._sinks is None and self.proj_size == 0
                    and _shares_device(dt, T, B, x.shape[2], self.hidden_size))
            turned = x.flip(0) if half else x
            params = [self.layer_params(layer, reverse=(d == 1)) for d in range(nd)]
            beside = _Beside(x.device, half, turned, *params[-1])
            for d in range(nd):
                Wx, bx, Wh, bh = params[d]
                if half:
                    hl, cl = h_0[layer * nd + d], c_0[layer * nd + d]
                    x_d = turned if d else x
                    with beside.stream(d):
                        inference = _nothing_to_save(x_d, hl, cl, Wx, bx, Wh, bh)
                        o, h_i, c_i = _layer(x_d, hl, cl, Wx, bx, Wh, bh, inference, main=beside.main)
                        outs.append(o.flip(0) if d else o)
                    h_n.append(h_i)
                    c_n.append(c_i)
                    continue
                # the reverse direction walks t = T-1 .. 0 (every sequence from its own end when packed)
                x_d = x if d == 0 else (x.flip(0) if lengths is None else reverse_time(x))
                hl, cl = h_0[layer * nd + d], c_0[layer * nd + d]
                inference = _nothing_to_save(x_d, hl, cl, Wx, bx, Wh, bh)
                sink = None if self._sinks is None else self._sinks[layer * nd + d]
                if self.proj_size > 0:
                    Whr = getattr(self, f"weight_hr_l{layer}{'_reverse' if d == 1 else ''}")
                    if hl is not None and cl is None or hl is None and cl is not None:
                        raise ValueError("h_0 and c_0 must both be given or both be None")
                    if lengths is None:
                        o, h_i, c_i = self._projected_layer(x_d, hl, cl, Wx, bx, Wh, bh, Whr, inference)
                    else:
                        cl_ = x_d.new_zeros(B, self.hidden_size) if cl is None else cl
                        o, cells, _, _ = self._projected_steps(x_d, hl, cl_, Wx, bx, Wh, bh, Whr, inference)
                        h_i, c_i = at_last(o), at_last(cells)
                        o = o * valid[:, :, None].to(o.dtype)
                elif lengths is None and sink is None and x_d.is_cuda:
                    o, h_i, c_i = _layer(x_d, hl, cl, Wx, bx, Wh, bh, inference, single)
                elif lengths is None:
                    o, h_i, c_i = PersistentLSTMfn.apply(x_d, hl, cl, Wx, bx, Wh, bh, inference, sink)
                else:
                    o, _, _, cells = PersistentLSTMfn.apply(x_d, hl, cl, Wx, bx, Wh, bh, inference, sink, True)
                    h_i, c_i = at_last(o), at_last(cells)      # states at each sequence's own last step
                    o = o * valid[:, :, None].to(o.dtype)      # steps past the end read as zeros
                outs.append(o if d == 0 else (o.flip(0) if lengths is None else reverse_time(o)))
                h_n.append(h_i)
                c_n.append(c_i)
            beside.join()
            x = outs[0] if nd == 1 else torch.cat(outs, dim=-1)
            if layer == self.num_layers - 1:
                # (a single layer has made the stacked tensors itself)
                states = (h_n[0], c_n[0]) if single else (torch.stack(h_n), torch.stack(c_n))
            beside.release()
            if self.dropout > 0.0 and self.training and layer < self.num_layers - 1:
                x = torch.nn.functional.dropout(x, self.dropout, True)
        if self.batch_first and lengths is None:
            x = x.transpose(0, 1)
        return x, states
