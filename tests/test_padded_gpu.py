"""16-bit shapes that the tensor-core path runs zero-padded (engine_padded.cu), against the oracle: odd widths around the
padding's edges, each recurrent schedule behind it (clusters, grid-wide persistent, wide batch), the caches in logical
layout, step ranges, and tensors that start off a 16-byte boundary."""
import numpy as np
import pytest
import torch

from flashlstm_poc_b200.engine import TORCH_DTYPES, Engine
from flashlstm_poc_b200.workloads import Workload, make_inputs
from oracle import lstm_oracle as orc
from tests.gpu_helpers import assert_parity, run_engine, run_oracle
from tests.helpers import to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,L,T,B,I,H", [
    ("f16", 2, 6, 20, 650, 650), ("bf16", 1, 5, 3, 5, 5), ("f16", 3, 4, 7, 63, 65), ("bf16", 1, 7, 33, 12, 100),
    ("f16", 2, 5, 9, 3, 64),       # only the input is padded
    ("bf16", 2, 4, 40, 130, 1217),  # grid-wide persistent kernels
    ("f16", 1, 3, 150, 64, 1270),   # wide batch
])
def test_padded_shapes_match_the_oracle(dtype, L, T, B, I, H):
    w = Workload("t", dtype, L, I, H, B, T, seed=51, state_std=0.3)
    inp = make_inputs(w)
    gen = torch.Generator().manual_seed(5)
    dhn, dcn = torch.randn(L, B, H, generator=gen), torch.randn(L, B, H, generator=gen)
    td = TORCH_DTYPES[dtype]
    dhn, dcn = dhn.to(td).float(), dcn.to(td).float()
    got, eng = run_engine(w, inp, dhn=dhn, dcn=dcn, repeat=2)
    assert eng.backend == "tc"
    ref = run_oracle(inp, dhn=dhn, dcn=dcn)
    assert_parity(got, ref, dtype)
    for l in range(L):
        assert orc.max_abs_err(to_np(eng.gate_cache(l, T)), ref["gates"][l]) < 2e-2  # gates in (-1, 1), 16-bit h behind them
        assert np.isfinite(to_np(eng.cell_states(l, T))).all()
    eng.close()


# the padded form of every kernel that holds W_hh in tensor memory, and of those that run their short launches: dtype, T, B, H,
# kernel and batch tile forward and backward
PADDED_TMEM = [(dtype, *shape) for dtype in ("f16", "bf16") for shape in (
    (30, 20, 1000, "lstm_fwd_tm_kernel", 32, "lstm_bwd_tm_kernel", 32), (4, 60, 1000, "lstm_fwd_kernel", 32, "lstm_bwd_kernel", 32),
    (4, 20, 1080, "lstm_fwd_tm_kernel", 32, "lstm_bwd_tm_kernel", 32), (4, 70, 1080, "lstm_fwd_tm_kernel", 64, "lstm_bwd_tm_kernel", 64),
    (4, 3, 2430, "lstm_fwd_tm_kernel", 16, "lstm_bwd_kernel", 32), (4, 17, 2430, "lstm_fwd_tm_kernel", 32, "lstm_bwd_kernel", 32),
    (4, 33, 2430, "lstm_fwd_tm_kernel", 64, "step_kernel", 0),
    (4, 140, 1000, "lstm_fwd_wide_kernel", 64, "lstm_bwd_tm_kernel", 64),
    (4, 259, 1080, "lstm_fwd_wide_kernel", 128, "lstm_bwd_tm_kernel", 64))]


@pytest.mark.parametrize("dtype,T,B,H,forward,fwd_tile,backward,bwd_tile", PADDED_TMEM)
def test_padded_shapes_in_tensor_memory(dtype, T, B, H, forward, fwd_tile, backward, bwd_tile):
    eng = Engine(dtype, 1, B, 64, H, T, device=torch.device("cuda", 0))
    got = eng.recurrent_kernel(T), eng.recurrent_kernel(T, backward=True)
    eng.close()
    assert [(k["name"], k["batch_tile"]) for k in got] == [(forward, fwd_tile), (backward, bwd_tile)]
    test_padded_shapes_match_the_oracle(dtype, 1, T, B, 64, H)
    test_padded_gate_functions_keep_their_relative_accuracy_near_zero(dtype, B, 64, H, True, steps=T)
    if B > 4:
        test_an_infinite_input_stays_out_of_the_padding(dtype, T, B, 64, H, True)


def test_padded_ranges_and_unaligned_tensors():
    T, B, I, H = 7, 5, 33, 70
    w = Workload("t", "f16", 2, I, H, B, T, seed=52, state_std=0.3)
    inp = make_inputs(w)
    dev, td = torch.device("cuda", 0), torch.float16
    eng = Engine("f16", 2, B, I, H, T, device=dev)
    for l in range(2):
        eng.set_weights(l, inp.w_ih[l].to(dev), inp.w_hh[l].to(dev), inp.b_ih[l].to(dev), inp.b_hh[l].to(dev))

    def odd(t):  # the same values one element past an aligned start
        flat = torch.zeros(t.numel() + 1, dtype=t.dtype, device=dev)
        flat[1:] = t.to(dev).flatten()
        return flat[1:].view(t.shape)

    x, h0, c0, dy = (t.to(dev, td) for t in (inp.x, inp.h0, inp.c0, inp.dy))
    y, hn, cn = eng.forward(x, h0, c0)
    dx, dh0, dc0 = eng.backward(dy)
    cells = eng.cell_states(1, T).clone()
    want = [t.clone() for t in (y, hn, cn, dx, dh0, dc0, *eng.grads(0), *eng.grads(1))]
    x2, dy2, y2, dx2 = odd(x), odd(dy), odd(torch.zeros_like(y)), odd(torch.zeros_like(dx))
    hn2, cn2, dh2, dc2 = torch.zeros_like(hn), torch.zeros_like(cn), torch.zeros_like(dh0), torch.zeros_like(dc0)
    for t0, t1 in ((0, 2), (2, 3), (3, 7)):
        eng.forward_range_into(T, t0, t1, x2, h0, c0, y2, hn2, cn2)
    for t0, t1 in ((4, 7), (0, 4)):
        eng.backward_range_into(T, t0, t1, dy2, None, None, dx2, dh2, dc2)
    torch.cuda.synchronize()
    for a, b in zip(want, (y2, hn2, cn2, dx2, dh2, dc2, *eng.grads(0), *eng.grads(1))):
        assert torch.equal(a, b)
    assert torch.equal(cells, eng.cell_states(1, T))  # the logical copy follows the later calls
    eng.close()


@pytest.mark.parametrize("dtype,B,I,H,training", [
    ("f16", 9, 8, 70, True), ("bf16", 9, 8, 70, True),  # clusters
    ("bf16", 40, 16, 1217, True),                       # grid-wide persistent kernels
    ("f16", 150, 64, 1270, True),                       # wide batch
    ("bf16", 5, 8, 70, False),                          # one launch per step
])
def test_padded_gate_functions_keep_their_relative_accuracy_near_zero(dtype, B, I, H, training, steps=1):
    """Only the cell candidate has a pre-activation, exact in 16 bits and down to 2^-13 (f16) or 2^-20 (bf16), so that
    c_1 = tanh(a) / 2.  tanh is good to 2 units in the last place there and sigmoid(0) = 1/2 is exact: 2^-22 relative."""
    dev, td = torch.device("cuda", 0), TORCH_DTYPES[dtype]
    u = torch.arange(H)
    low = 13 if dtype == "f16" else 20
    a = (128 + (37 * u) % 128) / 128 * torch.pow(2.0, -(4 + u % (low - 3)).float()) * torch.where(u % 2 == 0, 1.0, -1.0)
    w_ih, w_hh, b = torch.zeros(4 * H, I), torch.zeros(4 * H, H), torch.zeros(4 * H)
    w_ih[2 * H:3 * H, 0] = a * 64
    x = torch.zeros(steps, B, I)
    x[0, :, 0] = 1 / 64
    eng = Engine(dtype, 1, B, I, H, steps, training=training, device=dev)
    eng.set_weights(0, w_ih.to(dev), w_hh.to(dev), b.to(dev), b.to(dev))
    eng.forward(x.to(dev, td))
    got = eng.cell_states(0, steps)[1].double().cpu()
    eng.close()
    want = (torch.tanh(a.double()) / 2).expand(B, H)
    assert float(((got - want) / want).abs().max()) < 2 ** -22


@pytest.mark.parametrize("dtype,T,B,I,H", [
    ("f16", 5, 9, 10, 70), ("bf16", 4, 5, 16, 100),  # clusters
    ("bf16", 4, 40, 16, 1217),                       # grid-wide persistent kernels
    ("f16", 3, 150, 64, 1270),                       # wide batch
])
@pytest.mark.parametrize("training", [True, False])
def test_an_infinite_input_stays_out_of_the_padding(dtype, T, B, I, H, training):
    """An infinite x or h0 saturates the real units' gates, which leaves every result finite; a padding unit must not make
    NaN of it (0 * inf) and hand that to the next step.  An infinite dy makes its own row's dG infinite, and nothing else."""
    if not training:
        T = min(T, 4)  # with B <= 32 one launch per step
    w = Workload("t", dtype, 1, I, H, B, T, seed=53, state_std=0.3, training=training)
    inp = make_inputs(w)
    inp.x[1, 2, 3], inp.x[0, 4, 1], inp.h0[0, 3, 2] = float("inf"), float("-inf"), float("inf")
    if not training:
        inp.dy = None
    got, eng = run_engine(w, inp)
    with np.errstate(over="ignore"):
        ref = run_oracle(inp)
    keys = ("y", "hn", "cn") + (("dx", "dh0", "dc0") if training else ())
    assert_parity(got, ref, dtype, keys=keys)
    if training:
        inp.dy[T - 1, 1, 0] = float("inf")
        dev, td = torch.device("cuda", 0), TORCH_DTYPES[dtype]
        x = inp.x.to(dev, td)
        eng.forward(x, inp.h0.to(dev, td), inp.c0.to(dev, td))
        dx, dh0, dc0 = (to_np(t) for t in eng.backward(inp.dy.to(dev, td)))
        rest = [b for b in range(B) if b != 1]
        clean = {"dx": dx[:, rest], "dh0": dh0[:, rest], "dc0": dc0[:, rest]}
        want = {"dx": got["dx"][:, rest], "dh0": got["dh0"][:, rest], "dc0": got["dc0"][:, rest]}
        for k in clean:
            assert np.array_equal(clean[k], want[k]), k
    eng.close()


@pytest.mark.parametrize("I,H", [(33, 70), (64, 70), (33, 64)])
def test_padded_calls_allocate_nothing_and_can_be_captured(I, H):
    """An engine's workspace is sized for max_seq_len when it is made: neither its first call nor the first one with tensors
    off a 16-byte boundary allocates, so either may be the one that a stream capture records."""
    T, B, dev, td = 6, 64, torch.device("cuda", 0), torch.float16
    w = Workload("t", "f16", 1, I, H, B, T, seed=54, state_std=0.3)
    inp = make_inputs(w)

    def odd(t):
        flat = torch.zeros(t.numel() + 1, dtype=t.dtype, device=dev)
        flat[1:] = t.to(dev).flatten()
        return flat[1:].view(t.shape)

    x, dy, h0, c0 = (t.to(dev, td) for t in (inp.x, inp.dy, inp.h0, inp.c0))
    inputs = {"even": (x, dy), "odd": (odd(x), odd(dy))}
    out = {k: [f(torch.zeros(s, dtype=td, device=dev)) for f, s in ((make, (T, B, H)), (make, (T, B, I)))]
           for k, make in (("even", lambda t: t), ("odd", odd))}
    states = [torch.zeros(1, B, H, dtype=t, device=dev) for t in (td, td, torch.float32, torch.float32)]
    params = [p[0].to(dev) for p in (inp.w_ih, inp.w_hh, inp.b_ih, inp.b_hh)]

    def made():
        eng = Engine("f16", 1, B, I, H, T, device=dev)
        eng.set_weights(0, *params)
        return eng

    def step(eng, kind):
        (xk, dyk), (y, dx) = inputs[kind], out[kind]
        eng.forward_into(T, xk, h0, c0, y, states[0], states[1])
        eng.backward_into(T, dyk, None, None, dx, states[2], states[3])

    eng = made()  # loads the kernels
    for kind in ("even", "odd"):
        step(eng, kind)
    torch.cuda.synchronize()
    want = [t.clone() for t in (*out["even"], *states, *eng.grads(0))]
    eng.close()
    eng = made()
    torch.cuda.synchronize()
    held, free = eng.workspace_bytes, torch.cuda.mem_get_info()[0]
    for kind in ("even", "odd"):
        step(eng, kind)
        torch.cuda.synchronize()
        assert eng.workspace_bytes == held
        assert torch.cuda.mem_get_info()[0] == free
    eng.close()
    eng = made()
    for t in out["odd"] + states:
        t.zero_()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step(eng, "odd")
    graph.replay()
    torch.cuda.synchronize()
    for a, b in zip(want, (*out["odd"], *states, *eng.grads(0))):
        assert torch.equal(a, b)
    del graph
    eng.close()


def test_what_fits_only_unpadded_runs_on_the_cuda_cores():
    """H = 65 pads to 128 and twice the memory.  Here the padded workspace takes 225 GB, the plain one 114 GB."""
    B, H, dev, td = 80000, 65, torch.device("cuda", 0), torch.float16
    torch.cuda.empty_cache()
    w = Workload("t", "f16", 1, 8, H, 9, 2, seed=55, state_std=0.3)
    inp = make_inputs(w)
    want, small = run_engine(w, inp)
    assert small.backend == "tc"
    small.close()
    eng = Engine("f16", 1, B, 8, H, 1000, device=dev)
    assert eng.backend == "simt"
    eng.set_weights(0, *(p[0].to(dev) for p in (inp.w_ih, inp.w_hh, inp.b_ih, inp.b_hh)))
    x, h0, c0 = (torch.zeros(n, B, k, dtype=td, device=dev) for n, k in ((2, 8), (1, H), (1, H)))
    x[:, :9], h0[:, :9], c0[:, :9] = (t.to(dev, td) for t in (inp.x, inp.h0, inp.c0))
    y, hn, cn = eng.forward(x, h0, c0)
    got = {"y": to_np(y[:, :9]), "hn": to_np(hn[:, :9]), "cn": to_np(cn[:, :9])}
    eng.close()
    assert_parity(got, want, "f16", keys=("y", "hn", "cn"))


@pytest.mark.parametrize("dtype,L,T,B,I,H", [("f16", 2, 6, 20, 40, 70), ("bf16", 2, 4, 40, 130, 1217)])
def test_padded_state_caches_match_the_oracle(dtype, L, T, B, I, H):
    """The logical copies of the cell and hidden states behind flstm_engine_cache_ptrs, slot by slot, of every layer."""
    import ctypes

    from flashlstm_poc_b200._lib import check
    from tests.helpers import params_from_inputs

    w = Workload("t", dtype, L, I, H, B, T, seed=56, state_std=0.3)
    inp = make_inputs(w)
    got, eng = run_engine(w, inp)
    fwd = orc.lstm_forward(inp.x.numpy(), params_from_inputs(inp), inp.h0.numpy(), inp.c0.numpy(), dtype=np.float32)
    for l in range(L):
        ptr = ctypes.c_void_p()
        check(eng.lib.flstm_engine_cache_ptrs(eng._h, l, None, None, ctypes.byref(ptr), None))
        hs = to_np(eng._wrap(ptr.value, (T + 1, B, H), TORCH_DTYPES[dtype]))
        cs = to_np(eng.cell_states(l, T))
        for t in range(T + 1):
            assert orc.rel_l2_err(hs[t], fwd.caches[l].h_s[t]) < 1e-2, (l, t)
            assert orc.rel_l2_err(cs[t], fwd.caches[l].c_s[t]) < 1e-2, (l, t)
        assert np.array_equal(hs[T], got["hn"][l])
    assert np.array_equal(hs[1:], got["y"])
    eng.close()
