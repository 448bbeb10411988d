"""The work that users of the LSTM layer have it do, as cases that can be timed and compared.

A case is one call of `FastLSTM` as a program makes it: a streaming step, a sequence without gradients, or a training
step (forward and backward, gradients of the input, the initial states and every parameter).  Values follow the
benchmark's distributions: x and upstream gradients N(0,1), weights U(-1/sqrt(H), 1/sqrt(H)), initial states zero or
small."""
import math

import torch

from fastlstm_b200 import FastLSTM

TYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}

DEFAULTS = {"train": True, "dtype": "bf16", "layers": 1, "batch_first": False, "bidirectional": False, "packed": False,
            "autocast": False, "proj": 0, "state": 0.0, "state_grads": False}


def _case(name=None, **given):
    c = dict(DEFAULTS, **given)
    return c if name is None else dict(c, name=name)


def listed():
    return [
        # A stream of one user: one new timestep, the state of the last one handed back in.  Latency and launches.
        _case("stream_step", train=False, layers=2, steps=1, batch=1, inputs=512, hidden=512, state=0.1),
        # The latency floor of the reference's benchmark grid: the smallest hidden size and batch, a long sequence.
        _case("infer_small", train=False, dtype="fp16", steps=1024, batch=4, inputs=64, hidden=64),
        # Benchmark workload c2: small hidden size, a long sequence, forward only.
        _case("infer_c2", train=False, dtype="fp16", steps=1024, batch=64, inputs=256, hidden=256),
        # Benchmark workload c1: the fp32 user with nn.LSTM's batch_first and gradients through the final states.
        _case("train_c1_fp32", dtype="fp32", steps=64, batch=16, inputs=128, hidden=128, batch_first=True, state=0.1,
              state_grads=True),
        # The test grid's ragged fp32 stack: no size is a multiple of anything.
        _case("train_ragged_fp32", dtype="fp32", layers=2, steps=100, batch=44, inputs=123, hidden=257),
        # Tagging and speech encoders: sequences of different lengths, both directions, an odd batch.
        _case("train_packed_bidir", layers=2, steps=150, batch=37, inputs=80, hidden=320, bidirectional=True, packed=True),
        # Speech models with nn.LSTM's output projection.
        _case("train_proj", dtype="fp16", steps=60, batch=32, inputs=80, hidden=512, proj=128),
        # fp32 master weights under autocast, the usual mixed-precision training loop.
        _case("train_autocast", autocast=True, steps=256, batch=256, inputs=768, hidden=768),
        # Benchmark workload c3: the mid-size training step.
        _case("train_c3", dtype="fp16", steps=512, batch=256, inputs=1024, hidden=1024, state=0.01),
        # Benchmark workload c4: a large hidden size with a small batch.
        _case("train_c4", steps=1024, batch=32, inputs=2048, hidden=2048),
        # One of eight data-parallel shards of benchmark workload c5.
        _case("train_c5_shard", layers=2, steps=256, batch=512, inputs=512, hidden=512),
        # Benchmark workload c5 on one GPU: the largest.
        _case("train_c5", layers=2, steps=256, batch=4096, inputs=512, hidden=512),
    ]


def _spread(rng, lo, hi):
    """A whole number of [lo, hi], even over the logarithm."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _hidden(rng, lo, hi):
    """Hidden sizes: most models round them to 64 or 8, some do not."""
    h = _spread(rng, lo, hi)
    unit = rng.choice((64, 64, 8, 1))
    return max(lo, min(hi, -(-h // unit) * unit))


#: how often each kind of use is drawn
KINDS = (("stream", 2), ("infer", 3), ("train", 5), ("train_fp32", 2), ("packed", 1), ("proj", 1), ("autocast", 1))


def draw(rng):
    kind = rng.choice([k for k, n in KINDS for _ in range(n)])
    half = rng.choice(("fp16", "bf16"))
    if kind == "stream":
        dtype = rng.choice(("fp32", "fp16", "bf16"))
        h = _hidden(rng, 64, 512 if dtype == "fp32" else 1024)
        c = _case(train=False, dtype=dtype, layers=rng.choice((1, 2, 3)), steps=1, batch=_spread(rng, 1, 64),
                  inputs=rng.choice((h, _spread(rng, 16, 512))), hidden=h, state=0.1)
    elif kind == "infer":
        h = _hidden(rng, 32, 1024)
        c = _case(train=False, dtype=half, layers=rng.choice((1, 1, 2)), steps=_spread(rng, 16, 1024),
                  batch=_spread(rng, 1, 512), inputs=rng.choice((h, _spread(rng, 16, 512))), hidden=h,
                  batch_first=rng.random() < 0.5)
    elif kind == "train_fp32":
        c = _case(dtype="fp32", layers=rng.choice((1, 2)), steps=_spread(rng, 10, 100), batch=_spread(rng, 4, 100),
                  inputs=_spread(rng, 16, 256), hidden=_hidden(rng, 16, 320), batch_first=rng.random() < 0.5,
                  state=rng.choice((0.0, 0.1)))
        c["state_grads"] = c["state"] > 0
    elif kind == "packed":
        c = _case(dtype=half, layers=rng.choice((1, 2)), steps=_spread(rng, 16, 200), batch=_spread(rng, 4, 128),
                  inputs=_spread(rng, 40, 512), hidden=_hidden(rng, 64, 512), bidirectional=rng.random() < 0.7, packed=True)
    elif kind == "proj":
        h = _hidden(rng, 64, 512)
        c = _case(dtype=rng.choice((half, "fp32")), steps=_spread(rng, 8, 60), batch=_spread(rng, 4, 64),
                  inputs=_spread(rng, 40, 256), hidden=h, proj=rng.choice((h // 4, h // 2)))
    else:
        h = _hidden(rng, 64, 2048)
        c = _case(dtype=half, layers=rng.choice((1, 2)), steps=_spread(rng, 16, 1024), batch=_spread(rng, 4, 4096),
                  inputs=rng.choice((h, _spread(rng, 16, 1024))), hidden=h, autocast=kind == "autocast",
                  bidirectional=rng.random() < 0.15, state=rng.choice((0.0, 0.0, 0.01)))
        most = work(listed()[-1])["flops"] / 2          # no larger than the largest listed case
        while work(c)["flops"] > most or c["steps"] * c["layers"] > 1024:
            c["steps"], c["batch"] = max(1, c["steps"] // 2), max(1, c["batch"] * 3 // 4)
    return c


def prepare(case, seed):
    dt = TYPES[case["dtype"]]
    T, B, L = case["steps"], case["batch"], case["layers"]
    nd = 2 if case["bidirectional"] else 1
    torch.manual_seed(seed)
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, std=1.0, dtype=dt):
        return (torch.randn(*shape, generator=g, device="cuda") * std).to(dtype)

    held = torch.float32 if case["autocast"] else dt             # what the program keeps its parameters and inputs in
    module = FastLSTM(case["inputs"], case["hidden"], num_layers=L, batch_first=case["batch_first"], device="cuda",
                      dtype=held, bidirectional=case["bidirectional"], proj_size=case["proj"])
    module.train(case["train"])
    width = case["proj"] or case["hidden"]
    shape = (lambda n: (B, T, n)) if case["batch_first"] else (lambda n: (T, B, n))
    s = {"case": case, "module": module, "x": normal(*shape(case["inputs"]), dtype=held), "hc": None, "grads": None}
    if case["packed"]:
        # from T down to a third of it, in an order of the seed's
        lengths = T - torch.arange(B) * (T - max(1, T // 3)) // B
        lengths = lengths[torch.randperm(B, generator=torch.Generator().manual_seed(seed))]
        s["lengths"] = lengths
    if case["state"] > 0:
        s["hc"] = (normal(L * nd, B, width, std=case["state"], dtype=held),
                   normal(L * nd, B, case["hidden"], std=case["state"], dtype=held))
    if case["train"]:
        rows = int(s["lengths"].sum()) if case["packed"] else None
        s["grads"] = [normal(rows, nd * width) if case["packed"] else normal(*shape(nd * width))]
        if case["state_grads"]:
            s["grads"] += [normal(L * nd, B, width), normal(L * nd, B, case["hidden"])]
            for t in s["hc"]:
                t.requires_grad_()
        s["x"].requires_grad_()
    return s


def run(s):
    case, module = s["case"], s["module"]
    if not case["train"]:
        with torch.no_grad():
            out, (h, c) = module(s["x"], s["hc"])
        return [out, h, c]
    leaves = [s["x"], *module.parameters(), *(s["hc"] if case["state_grads"] else ())]
    for t in leaves:
        t.grad = None
    x = s["x"]
    if case["packed"]:
        x = torch.nn.utils.rnn.pack_padded_sequence(x, s["lengths"], enforce_sorted=False)
    with torch.autocast("cuda", dtype=TYPES[case["dtype"]], enabled=case["autocast"]):
        out, (h, c) = module(x, s["hc"])
    data = out.data if case["packed"] else out
    torch.autograd.backward([data, h, c] if case["state_grads"] else [data], s["grads"])
    return [data.detach(), h.detach(), c.detach(), *(t.grad for t in leaves)]


def work(case):
    """Bytes: the input, the parameters and the output once, and for training the saved gates and cell states (written and
    read), the upstream gradient, and the gradients of input and parameters.  Flops: the contractions."""
    T, B, H = case["steps"], case["batch"], case["hidden"]
    nd, P = (2 if case["bidirectional"] else 1), case["proj"]
    width = P or H
    e = 4 if case["dtype"] == "fp32" else 2
    held = 4 if case["autocast"] or e == 4 else 2
    flops = params = 0
    width_in = case["inputs"]
    for _ in range(case["layers"]):
        params += nd * (4 * H * (width_in + width + 2) + P * H)
        flops += nd * T * B * 2 * (4 * H * (width_in + width) + P * H)
        width_in = nd * width
    states = case["layers"] * nd * B * (width + H)
    rows = T * B
    bytes_ = held * (rows * case["inputs"] + params) + e * (rows * nd * width + states * (2 if case["state"] else 1))
    if case["train"]:
        flops *= 3
        bytes_ += held * (rows * case["inputs"] + params) + e * rows * nd * width
        bytes_ += 2 * e * case["layers"] * nd * rows * 5 * H
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """16-bit: what rounding states and gate gradients to the storage type at every step adds up to; fp32: sums of a few
    thousand terms in another order."""
    return {"rel": {"fp32": 1e-5, "fp16": 3e-3, "bf16": 1e-2}[case["dtype"]]}
