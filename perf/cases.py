"""The work a user has this framework do, as measurable cases.

Four public entry points are covered: the `LSTM` module (training steps and evaluation), the `Engine` handle
(inference), the `StreamingLSTM` operator on pinned host tensors, and the v1 C interface.  `listed()` names twelve
cases, `draw()` gives further ones of the same ranges:

    kind    "train"   LSTM module: forward, then backward to x, h0, c0 and every parameter
            "eval"    LSTM module under no_grad
            "infer"   Engine(training=False).forward, weights set once
            "stream"  StreamingLSTM on pinned fp16 host tensors, forward and backward
            "v1"      lstm_forward of the C interface on fp32 device tensors
    dtype   "f32", "f16", "bf16" (arithmetic type; stream and v1 always compute in f16)
    layers, batch, input_size, hidden_size, steps (time steps), recompute (checkpoint interval, 0 = full gate cache)
"""
import ctypes
import math

import torch

from flashlstm_poc_b200 import _lib
from flashlstm_poc_b200.engine import Engine
from flashlstm_poc_b200.lstm import LSTM
from flashlstm_poc_b200.streaming_lstm import StreamingLSTM

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}


def _case(name, kind, dtype, layers, batch, input_size, hidden_size, steps, recompute=0):
    case = {"kind": kind, "dtype": dtype, "layers": layers, "batch": batch, "input_size": input_size,
            "hidden_size": hidden_size, "steps": steps, "recompute": recompute}
    return dict(case, name=name) if name else case


def listed():
    return [
        # one time step of one sequence through two layers, states carried by the caller: token-by-token generation
        _case("decode_f16_l2_h1024_b1_t1", "infer", "f16", 2, 1, 1024, 1024, 1),
        # a short chunk of a few live sequences through a small stack: streaming recognition, evaluation of small models
        _case("eval_bf16_l3_h320_b16_t20", "eval", "bf16", 3, 16, 80, 320, 20),
        # the fp32 configuration of the benchmark: small models, and training where 16 bits do not suffice
        _case("train_f32_h256_b32_t128", "train", "f32", 1, 32, 256, 256, 128),
        # sizes that are no multiple of any tile: sequence models are often trained with such widths and short windows
        _case("train_f16_l2_h650_b20_t35", "train", "f16", 2, 20, 650, 650, 35),
        # feature sequences of an odd batch into a mid-sized stack
        _case("train_bf16_l3_i200_h512_b37_t150", "train", "bf16", 3, 37, 200, 512, 150),
        # the one-GPU fp16 configuration of the benchmark
        _case("train_f16_h1024_b64_t512", "train", "f16", 1, 64, 1024, 1024, 512),
        # one GPU's eighth of the benchmark's batch-sharded configuration
        _case("train_bf16_l2_h2048_b32_t1024", "train", "bf16", 2, 32, 2048, 2048, 1024),
        # that configuration whole on one GPU: the largest case
        _case("train_bf16_l2_h2048_b256_t1024", "train", "bf16", 2, 256, 2048, 2048, 1024),
        # four layers trained with activation checkpoints instead of a full gate cache
        _case("train_bf16_l4_h1024_b256_t256_r32", "train", "bf16", 4, 256, 1024, 1024, 256, 32),
        # the benchmark's inference configuration: weights far larger than shared memory
        _case("infer_f16_h4096_b8_t2048", "infer", "f16", 1, 8, 4096, 4096, 2048),
        # the streaming operator: x, y, dy, dx and the checkpoints in pinned host memory
        _case("stream_f16_h1024_b64_t512_r32", "stream", "f16", 1, 64, 1024, 1024, 512, 32),
        # the v1 C interface at the batch and width of the sequence-length sweep
        _case("v1_h1024_b32_t512", "v1", "f16", 1, 32, 1024, 1024, 512),
    ]


_LARGEST = 1.06e14  # operations of the largest listed case (training, 2 layers, H = 2048, B = 256, T = 1024)


def draw(rng):
    def spread(lo, hi):  # whole numbers, evenly over their logarithm
        return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    kind = rng.choices(["train", "eval", "infer", "stream", "v1"], [10, 2, 4, 2, 2])[0]
    dtype = rng.choices(["f32", "f16", "bf16"], [2, 4, 4])[0] if kind in ("train", "eval", "infer") else "f16"
    hidden = spread(32, 1024 if dtype == "f32" else 2048 if kind == "train" else 4096 if kind == "infer" else 1536)
    ragged = rng.random() < 0.3
    if not ragged:  # most models have round widths
        hidden = max(64, (hidden + 32) // 64 * 64)
    width = hidden if rng.random() < 0.5 else spread(16, 2048)
    if not ragged and width != hidden:
        width = (width + 7) // 8 * 8
    layers = 1 if kind in ("stream", "v1") else rng.choice([1, 1, 2, 2, 3, 4])
    batch = spread(1, {"train": 512, "eval": 64, "infer": 64, "stream": 128, "v1": 64}[kind])
    steps = spread(1, 2048 if kind == "infer" else 1024)
    if kind == "infer" and rng.random() < 0.4:
        steps = spread(1, 16)  # generation step by step, or a few steps at a time
    if kind in ("train", "eval"):
        steps = max(8, steps)
    steps = max(1, min(steps, 2048 // layers))
    recompute = 0
    if kind == "stream":
        recompute = min(steps, rng.choice([1, 8, 32]))
    elif kind == "train" and dtype != "f32" and not ragged and rng.random() < 0.15:
        recompute = min(steps, rng.choice([16, 32, 64]))
    case = _case(None, kind, dtype, layers, batch, width, hidden, steps, recompute)
    # no dearer than the largest listed case; fp32 and ragged shapes run at the rates of the ordinary cores
    most = 5e11 if dtype == "f32" or ragged else _LARGEST
    while work(case)["flops"] > most and (case["steps"] > 8 or case["batch"] > 1):
        if case["steps"] > 8:
            case["steps"] = max(8, case["steps"] * 3 // 4)
        else:
            case["batch"] = max(1, case["batch"] * 3 // 4)
    case["recompute"] = min(case["recompute"], case["steps"])
    return case


class _V1:
    """The v1 C interface as a ctypes caller holds it: one handle with packed weights."""

    class Buffers(ctypes.Structure):
        _fields_ = [("impl", ctypes.c_void_p)]

    def __init__(self, steps, batch, input_size, hidden_size, w_ih, w_hh):
        self.lib = ctypes.CDLL(_lib.LIB_PATH)
        sizes, ptr = [ctypes.c_size_t] * 4, ctypes.c_void_p
        self.lib.lstm_create_buffers.argtypes = [ctypes.c_int, *sizes, ctypes.c_int, ctypes.POINTER(self.Buffers)]
        self.lib.lstm_pack_weights.argtypes = [ctypes.c_int, ptr, ptr, *sizes[:2], ctypes.POINTER(self.Buffers)]
        self.lib.lstm_forward.argtypes = [ptr] * 8 + sizes + [ctypes.POINTER(self.Buffers), ctypes.c_int]
        self.lib.lstm_destroy_buffers.argtypes = [ctypes.POINTER(self.Buffers)]
        self.sizes = (steps, batch, input_size, hidden_size)
        self.buffers = self.Buffers()
        self._ok(self.lib.lstm_create_buffers(0, *self.sizes, 0, ctypes.byref(self.buffers)))
        torch.cuda.current_stream().synchronize()
        self._ok(self.lib.lstm_pack_weights(0, w_ih.data_ptr(), w_hh.data_ptr(), input_size, hidden_size,
                                            ctypes.byref(self.buffers)))

    @staticmethod
    def _ok(code):
        if code != 0:
            raise RuntimeError(f"v1 call failed with code {code}")

    def forward(self, *tensors):
        self._ok(self.lib.lstm_forward(*(t.data_ptr() for t in tensors), *self.sizes, ctypes.byref(self.buffers), 0))

    def __del__(self):
        if self.buffers.impl:
            self.lib.lstm_destroy_buffers(ctypes.byref(self.buffers))


def prepare(case, seed):
    kind, dtype = case["kind"], DTYPES[case["dtype"]]
    L, B, I, H, T = (case[k] for k in ("layers", "batch", "input_size", "hidden_size", "steps"))
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, std=1.0, kind_of=dtype):
        return torch.randn(shape, generator=gen, device="cuda").mul_(std).to(kind_of)

    def parameter(*shape):  # torch.nn.LSTM's initial distribution
        bound = 1.0 / math.sqrt(H)
        return torch.empty(shape, device="cuda").uniform_(-bound, bound, generator=gen)

    params = []
    for layer in range(L):
        width = I if layer == 0 else H
        params += [parameter(4 * H, width), parameter(4 * H, H), parameter(4 * H), parameter(4 * H)]
    state = {"kind": kind, "recompute": case["recompute"]}
    if kind in ("train", "eval"):
        model = LSTM(I, H, L, dtype=dtype, recompute_interval=case["recompute"] if kind == "train" else 0)
        with torch.no_grad():
            for p, value in zip(model.parameters(), params):
                p.copy_(value)
        state.update(model=model, params=list(model.parameters()), x=normal(T, B, I),
                     h0=normal(L, B, H, std=0.1), c0=normal(L, B, H, std=0.1))
        if kind == "train":
            for name in ("x", "h0", "c0"):
                state[name].requires_grad_(True)
            state["dy"] = normal(T, B, H)
    elif kind == "infer":
        engine = Engine(case["dtype"], L, B, I, H, T, training=False)
        for layer in range(L):
            engine.set_weights(layer, *params[4 * layer:4 * layer + 4])
        state.update(engine=engine, x=normal(T, B, I), h0=normal(L, B, H, std=0.1), c0=normal(L, B, H, std=0.1))
    elif kind == "stream":
        model = StreamingLSTM(I, H)
        with torch.no_grad():
            for p, value in zip(model.parameters(), params):
                p.copy_(value)
        state.update(model=model, params=list(model.parameters()), x=normal(T, B, I).cpu().pin_memory(),
                     dy=normal(T, B, H).cpu().pin_memory(), h0=normal(B, H, std=0.1), c0=normal(B, H, std=0.1))
        for name in ("x", "h0", "c0"):
            state[name].requires_grad_(True)
    else:
        f32 = torch.float32
        state.update(handle=_V1(T, B, I, H, params[0], params[1]), b_ih=params[2], b_hh=params[3],
                     x=normal(T, B, I, kind_of=f32), h0=normal(B, H, std=0.1, kind_of=f32),
                     c0=normal(B, H, std=0.1, kind_of=f32), y=torch.empty(T, B, H, device="cuda"),
                     hn=torch.empty(B, H, device="cuda"), cn=torch.empty(B, H, device="cuda"))
        torch.cuda.current_stream().synchronize()  # the C interface works on a stream of its own
    return state


def run(state):
    kind = state["kind"]
    if kind == "infer":
        return state["engine"].forward(state["x"], state["h0"], state["c0"])
    if kind == "v1":
        out = state["y"], state["hn"], state["cn"]
        state["handle"].forward(state["x"], state["b_ih"], state["b_hh"], state["h0"], state["c0"], *out)
        return out
    if kind == "eval":
        with torch.no_grad():
            y, (hn, cn) = state["model"](state["x"], (state["h0"], state["c0"]))
        return y, hn, cn
    inputs = [state["x"], state["h0"], state["c0"], *state["params"]]
    if kind == "train":
        y, (hn, cn) = state["model"](state["x"], (state["h0"], state["c0"]))
        grads = torch.autograd.grad(y, inputs, state["dy"])
        return (y.detach(), hn.detach(), cn.detach(), *grads)
    y, cache, (hn, cn) = state["model"](state["x"], state["h0"], state["c0"], recompute_interval=state["recompute"])
    grads = torch.autograd.grad(y, inputs, state["dy"])
    return (y.detach(), hn.detach(), cn.detach(), cache.h, cache.c, *grads)


def work(case):
    """Each input read once and each output written once; parameters and their gradients are fp32, a handle's packed
    weights have the arithmetic type.  Operations: the matrix products of both GEMMs of a cell, times three with backward."""
    kind = case["kind"]
    L, B, I, H, T = (case[k] for k in ("layers", "batch", "input_size", "hidden_size", "steps"))
    train = kind in ("train", "stream")
    size = 4 if kind == "v1" else DTYPES[case["dtype"]].itemsize
    weights = sum(4 * H * ((I if layer == 0 else H) + H) for layer in range(L))
    sequences = T * B * (I + H)
    states = L * B * H
    moved = sequences * size + 4 * states * size
    moved += weights * (4 if kind in ("train", "eval", "stream") else 2 if kind == "v1" else size) + L * 8 * H * 4
    flops = 2.0 * T * B * weights
    if train:
        moved += sequences * size + 2 * states * size + weights * 4 + L * 8 * H * 4
        flops *= 3
    if kind == "stream":
        moved += 2 * ((T + case["recompute"] - 1) // case["recompute"]) * B * H * 4
    return {"bytes": float(moved), "flops": float(flops)}


def tolerance(case):
    # fp32 sums; fp16 and bf16 operands (11 and 8 significant bits) with fp32 accumulation, rounded once per step
    return {"f32": {"rel": 1e-5}, "f16": {"rel": 2e-3}, "bf16": {"rel": 1e-2}}[case["dtype"]]
