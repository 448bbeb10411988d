"""Recurrences whose weights stay on the chip (large hidden sizes) against the fp32 step-by-step evaluation."""
import ctypes

import pytest
import torch

from fastlstm_b200 import _lib
from test_gpu_recurrence import TD, _bwd, _cmp, _desc, _fwd, _torch_bwd, _torch_fwd

pytestmark = pytest.mark.gpu

# N = 16 and 32; one row, ragged rows and groups; half an M tile in backward (H % 128 == 64); K split over 1 and 2 (forward),
# 4 (one issuer too), 5 and 6 (the same) CTAs backward; weights that fit tensor memory and weights that do not
SHAPES = [(4, 1, 768), (3, 65, 704), (5, 100, 768), (3, 250, 768), (4, 256, 1024), (2, 130, 960), (3, 33, 1088), (3, 64, 1536),
          (4, 32, 2048), (3, 17, 1984), (2, 9, 2048), (3, 29, 1728), (3, 61, 1408), (3, 90, 1408),
          # several tiles of 64 rows a group in backward: four, five and eight, a partial last tile, half an M tile, odd numbers of K chunks
          (3, 1600, 512), (3, 4096, 512), (5, 2300, 448), (3, 3210, 320), (3, 4000, 256), (1, 2047, 512)]


@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
@pytest.mark.parametrize("shape", SHAPES)
def test_resident_recurrences_against_fp32_maths(dtype, shape):
    lib = _lib.load()
    T, B, H = shape
    dt = TD[dtype]
    g = torch.Generator(device="cuda").manual_seed(B + H)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    d = _desc(dtype, T, B, H)
    Wh = ((torch.rand(4 * H, H, generator=g, device="cuda") * 2 - 1) / H ** 0.5).to(dt)
    pre, h0, c0 = rnd(T, B, 4 * H).to(dt), (rnd(B, H) * 0.3).to(dt), rnd(B, H).to(dt)
    ifgo, out, cell = _fwd(lib, d, pre, Wh, h0, c0)
    want = _torch_fwd(pre, Wh, h0, c0)
    tol = 8e-3 if dtype == "bf16" else 2e-3
    _cmp("ifgo", ifgo, want[0], 4 * tol)
    _cmp("out", out[1:], want[1], tol)
    _cmp("cell", cell[1:], want[2], 2 * tol)
    again = _fwd(lib, d, pre, Wh, h0, c0)
    assert torch.equal(out, again[1]) and torch.equal(ifgo, again[0])
    ifgo, cell, dout = rnd(T, B, 4 * H).to(dt), (rnd(T + 1, B, H) * 0.7).to(dt), rnd(T, B, H).to(dt)
    dh, dc = rnd(B, H).to(dt), rnd(B, H).to(dt)
    got = _bwd(lib, d, dout, dh, dc, ifgo, cell, Wh)
    for name, a, b in zip(("d_ifgo", "dh0", "dc0", "db"), got, _torch_bwd(dout, dh, dc, ifgo, cell, Wh)):
        _cmp(name, a, b, (1e-2 if dtype == "bf16" else 3e-3) * float(b.abs().max()))
    assert all(torch.equal(a, b) for a, b in zip(got, _bwd(lib, d, dout, dh, dc, ifgo, cell, Wh)))


# Where a group of rows becomes two tiles: 16 and 17 rows, a last group whose second tile has no rows, tiles of 16 rows with one
# issuer and with two, of 32 rows, K in two parts forward, enough steps for the tiles to take turns
@pytest.mark.parametrize("shape", [(9, 64, 1024), (9, 65, 1024), (9, 17, 2048), (9, 32, 2048), (9, 100, 768), (9, 257, 512), (9, 250, 768)])
def test_tiles_that_take_turns(shape):
    test_resident_recurrences_against_fp32_maths("bf16", shape)
    test_resident_recurrences_against_fp32_maths("fp16", shape)


# One tile of up to 32 rows a group, backward up to H = 448: a full group, ragged ones, 24 rows, half an M tile, an odd number of K chunks
@pytest.mark.parametrize("shape", [(9, 352, 320), (5, 289, 320), (9, 350, 384), (4, 264, 384), (9, 255, 448)])
def test_one_tile_of_32_rows_backward(shape):
    lib = _lib.load()
    buf = ctypes.create_string_buffer(512)
    _lib.check(lib.blstm_plan_detail(_desc("bf16", *shape), _lib.PHASE_BWD, buf, 512))
    assert b"tiles=1 " in buf.value and b"n=32 " in buf.value, buf.value
    test_resident_recurrences_against_fp32_maths("bf16", shape)
    test_resident_recurrences_against_fp32_maths("fp16", shape)


@pytest.mark.parametrize("phase", [0, 1])
@pytest.mark.parametrize("B,H", [(32, 1024), (32, 1536), (2048, 512)])
def test_resident_recurrences_give_up_with_a_status_when_nothing_arrives(phase, B, H):
    lib = _lib.load()
    T = 3
    z = lambda *s: torch.zeros(*s, device="cuda", dtype=torch.bfloat16)
    d = _lib.Desc(_lib.BF16, T, B, H, H, _lib.FLAG_TEST_NO_ARRIVE, 20000, 0)
    n = lib.blstm_workspace_bytes(d, phase)
    ws, s = torch.zeros(n, dtype=torch.uint8, device="cuda"), torch.cuda.current_stream().cuda_stream
    ifgo, Wh, out, cell, c = z(T, B, 4 * H), z(4 * H, H), z(T + 1, B, H), z(T + 1, B, H), z(2, B, H)
    if phase == 0:
        rc = lib.blstm_fwd_recurrence(d, ifgo.data_ptr(), Wh.data_ptr(), out.data_ptr(), cell.data_ptr(), ws.data_ptr(), n, s)
    else:
        rc = lib.blstm_bwd_recurrence(d, out.data_ptr(), None, None, ifgo.data_ptr(), cell.data_ptr(), Wh.data_ptr(), z(T, B, 4 * H).data_ptr(),
                                      c[0].data_ptr(), c[1].data_ptr(), None, ws.data_ptr(), n, s)
    assert rc == 0
    assert lib.blstm_read_status(ws.data_ptr(), None, s) == _lib.E_WAIT_TIMEOUT


# Several 32-row tiles per group, forward: three, four, six, eight (all of tensor memory and of shared memory taken), fifteen and
# sixteen, groups with one tile less, a last tile of one row, weights past tensor memory, an odd number of K chunks
@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
@pytest.mark.parametrize("shape", [(9, 289, 1024), (6, 1023, 1024), (3, 1700, 512), (4, 2300, 256), (3, 2849, 768), (3, 2913, 768), (5, 400, 832), (1, 600, 960)])
def test_forward_tiles_against_fp32_maths(dtype, shape):
    lib = _lib.load()
    T, B, H = shape
    dt = TD[dtype]
    g = torch.Generator(device="cuda").manual_seed(B + H)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    d = _desc(dtype, T, B, H)
    Wh = ((torch.rand(4 * H, H, generator=g, device="cuda") * 2 - 1) / H ** 0.5).to(dt)
    pre, h0, c0 = rnd(T, B, 4 * H).to(dt), (rnd(B, H) * 0.3).to(dt), rnd(B, H).to(dt)
    ifgo, out, cell = _fwd(lib, d, pre, Wh, h0, c0)
    want = _torch_fwd(pre, Wh, h0, c0)
    tol = 8e-3 if dtype == "bf16" else 2e-3          # as above
    _cmp("ifgo", ifgo, want[0], 4 * tol)
    _cmp("out", out[1:], want[1], tol)
    _cmp("cell", cell[1:], want[2], 2 * tol)
    again = _fwd(lib, d, pre, Wh, h0, c0)
    assert torch.equal(out, again[1]) and torch.equal(ifgo, again[0]) and torch.equal(cell, again[2])
    # without gradients: outputs and the last cell state only
    inf = _fwd(lib, _desc(dtype, T, B, H, _lib.FLAG_INFERENCE), pre, Wh, h0, c0)
    assert torch.equal(out, inf[1]) and torch.equal(cell[T], inf[2][T])


# Several 32-row tiles per group, backward: three, four, eight (with weights in shared memory) and sixteen, groups with one tile less,
# half an M tile, K chunks that do not divide into stages
@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
@pytest.mark.parametrize("shape", [(5, 300, 1024), (4, 1023, 1024), (5, 1024, 512), (3, 1990, 896), (5, 521, 832), (4, 600, 768), (1, 700, 960), (4, 1400, 384)])
def test_backward_tiles_against_fp32_maths(dtype, shape):
    lib = _lib.load()
    T, B, H = shape
    dt = TD[dtype]
    g = torch.Generator(device="cuda").manual_seed(B + H)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    d = _desc(dtype, T, B, H)
    Wh = ((torch.rand(4 * H, H, generator=g, device="cuda") * 2 - 1) / H ** 0.5).to(dt)
    ifgo, cell, dout = rnd(T, B, 4 * H).to(dt), (rnd(T + 1, B, H) * 0.7).to(dt), rnd(T, B, H).to(dt)
    dh, dc = rnd(B, H).to(dt), rnd(B, H).to(dt)
    got = _bwd(lib, d, dout, dh, dc, ifgo, cell, Wh)
    for name, a, b in zip(("d_ifgo", "dh0", "dc0", "db"), got, _torch_bwd(dout, dh, dc, ifgo, cell, Wh)):
        _cmp(name, a, b, (1e-2 if dtype == "bf16" else 3e-3) * float(b.abs().max()))          # as above
    assert all(torch.equal(a, b) for a, b in zip(got, _bwd(lib, d, dout, dh, dc, ifgo, cell, Wh)))


# 64-row tiles through every ring that the plans give, enough steps for each stage to be filled many times: two stages of two chunks (H = 320
# and 384; four tiles at 512), one of four with a shorter last one (448) and without (512), one that holds an item's chunks (256)
@pytest.mark.parametrize("shape", [(30, 4200, 320), (30, 5632, 384), (30, 3000, 448), (30, 4096, 448), (30, 2048, 512), (30, 3072, 512),
                                   (30, 4096, 512), (30, 8192, 256)])
def test_backward_ring_over_many_steps(shape):
    # (errors do not add up over the steps: what a step carries on in dh shrinks with the gates' derivatives, and dc is held in fp32)
    test_backward_tiles_against_fp32_maths("bf16", shape)
    test_backward_tiles_against_fp32_maths("fp16", shape)


def test_backward_tiles_give_up_with_a_status_when_nothing_arrives():
    test_resident_recurrences_give_up_with_a_status_when_nothing_arrives(1, 600, 1024)


def test_forward_tiles_give_up_with_a_status_when_nothing_arrives():
    test_resident_recurrences_give_up_with_a_status_when_nothing_arrives(0, 1024, 512)


@pytest.mark.parametrize("B,H", [(16, 64), (40, 512), (64, 1024), (200, 512)])
def test_bias_grad_for_every_backward_plan(B, H):
    lib = _lib.load()
    T = 7
    d = _desc("bf16", T, B, H)
    dg, db = torch.randn(T, B, 4 * H, device="cuda").bfloat16(), torch.empty(4 * H, device="cuda")
    n = lib.blstm_workspace_bytes(d, _lib.PHASE_BWD)
    ws = torch.zeros(n, dtype=torch.uint8, device="cuda")
    _lib.check(lib.blstm_bias_grad(d, dg.data_ptr(), db.data_ptr(), ws.data_ptr(), n, torch.cuda.current_stream().cuda_stream))
    want = dg.double().sum((0, 1))
    assert float((db.double() - want).abs().max()) <= 1e-4 * float(want.abs().max())
