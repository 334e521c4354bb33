"""The bounded-wait exit path of the persistent kernels, exercised without faulting, trapping or hanging anything.

The host asks the step barrier to wait for one arrival more than the CTAs of a batch group make
(flstm_engine_selftest_missing_arrivals) and shortens the limit of every device-side wait to a few
milliseconds (flstm_engine_set_wait_limit).  The wait of the second time step then runs out: the kernel raises
its error word, every role drains and the launch RETURNS; the host sees FLSTM_ERR_TIMEOUT, and the same engine
then computes a normal step whose results are bit-identical to the ones it produced before.

In the kernels without a step barrier the missing arrival is that of the launch's one barrier, ahead of the first result that crosses.
Their waits from step to step run out on words that one CTA leaves out (flstm_engine_selftest_lost_words)."""
import time

import numpy as np
import pytest
import torch

from flashlstm_poc_b200._lib import FlashLstmError
from flashlstm_poc_b200.engine import TORCH_DTYPES, Engine
from flashlstm_poc_b200.workloads import Workload, make_inputs

pytestmark = pytest.mark.gpu

LIMIT_US = 5000  # 5 ms


def _engine(w, inp, backend):
    dev = torch.device("cuda", 0)
    eng = Engine(w.dtype, w.layers, w.batch, w.input_size, w.hidden_size, w.seq_len, backend=backend, device=dev)
    for l in range(w.layers):
        eng.set_weights(l, inp.w_ih[l].to(dev), inp.w_hh[l].to(dev), inp.b_ih[l].to(dev), inp.b_hh[l].to(dev))
    return eng, dev


def _step(eng, inp, dev, td):
    y, hn, cn = eng.forward(inp.x.to(dev, td), inp.h0.to(dev, td), inp.c0.to(dev, td))
    dx, dh0, dc0 = eng.backward(inp.dy.to(dev, td))
    torch.cuda.synchronize()
    out = [y, hn, cn, dx, dh0, dc0] + [g for l in range(eng.layers) for g in eng.grads(l)]
    return [t.detach().float().cpu().numpy().copy() for t in out]


@pytest.mark.parametrize("dtype,backend,where", [
    ("f16", "tc", "forward"), ("f16", "tc", "backward"), ("bf16", "tc", "forward"),
    ("f32", "simt", "forward"), ("f32", "simt", "backward"),
    ("bf16", "tc", "forward-wide"),  # 96 sequences at H = 1024: the wide-batch forward kernel (all steps in one launch)
    # H = 2048: W_hh is streamed, and part of it is fetched into the ring ahead of the barrier that then fails
    ("bf16", "tc", "forward-streamed"), ("bf16", "tc", "backward-streamed"),
    # clusters of several CTAs in either direction (H = 64: BPTT on one CTA)
    ("f16", "tc", "forward-several"), ("bf16", "tc", "backward-several"),
])
def test_step_barrier_timeout_returns_and_engine_recovers(dtype, backend, where):
    where, _, variant = where.partition("-")
    shape = {"": (64, 64, 8), "wide": (128, 1024, 96), "streamed": (128, 2048, 8), "several": (64, 512, 8)}[variant]
    _time_out_and_recover(dtype, backend, where, shape, 4)


def _time_out_and_recover(dtype, backend, where, shape, steps, kernel=None, lost=None):
    w = Workload("timeout", dtype, 1, *shape, steps, seed=11, state_std=0.1)
    inp = make_inputs(w)
    td = TORCH_DTYPES[dtype]
    eng, dev = _engine(w, inp, backend)
    assert eng.backend == backend
    assert kernel in (None, eng.recurrent_kernel(steps, backward=where == "backward")["name"])
    before = _step(eng, inp, dev, td)
    assert all(np.isfinite(a).all() for a in before) and np.abs(before[0]).max() <= 1.0  # every row of y was written

    def ask(on):
        if lost is None:
            eng.selftest_missing_arrivals(int(on))
        else:
            eng.selftest_lost_words(*(lost if on else (0,)))

    eng.set_wait_limit(LIMIT_US)
    x, h0, c0, dy = (t.to(dev, td) for t in (inp.x, inp.h0, inp.c0, inp.dy))
    t_start = time.perf_counter()
    if where == "forward":
        ask(True)
        eng.forward(x, h0, c0)          # enqueued; the kernel gives up at the barrier of the second step
    else:
        eng.forward(x, h0, c0)
        ask(True)
        eng.backward(dy)
    with pytest.raises(FlashLstmError) as exc:
        eng.wait(20.0)                  # host watchdog: the launch has returned, the error word is set
    waited = time.perf_counter() - t_start
    assert exc.value.status == 3, exc.value  # FLSTM_ERR_TIMEOUT
    assert waited < 5.0, f"the kernel took {waited:.2f} s to give up with a {LIMIT_US} us limit"
    torch.cuda.synchronize()            # the context is intact

    ask(False)
    eng.set_wait_limit(0)
    after = _step(eng, inp, dev, td)
    eng.close()
    for a, b in zip(before, after):
        assert np.array_equal(a, b)
    return str(exc.value)


@pytest.mark.parametrize("dtype,backend,where", [
    ("f16", "tc", "forward"), ("f16", "tc", "backward"), ("bf16", "tc", "forward"), ("bf16", "tc", "backward"),
    ("f32", "simt", "forward"), ("f32", "simt", "backward"), ("f16", "simt", "forward"), ("bf16", "simt", "backward"),
])
def test_grid_wide_kernels_return_and_recover(dtype, backend, where, monkeypatch):
    """The grid-wide kernels with resident weights, whose CTAs clear the step counters on their way out (after an abort too):
    the shape above runs on clusters unless they are switched off."""
    monkeypatch.setenv("FLSTM_CLUSTER", "0")
    eng = Engine(dtype, 1, 8, 64, 64, 4, backend=backend, device=torch.device("cuda", 0))
    assert eng.recurrent_path()[0] == eng.recurrent_path(backward=True)[0] == "grid"
    eng.close()
    test_step_barrier_timeout_returns_and_engine_recovers(dtype, backend, where)


def test_which_kernels_the_cases_above_time_out():
    dev = torch.device("cuda", 0)
    for dtype, shape, forward, backward in (("f16", (64, 64, 8), "cluster", "cluster"), ("f32", (64, 64, 8), "cluster", "cluster"),
                                            ("f16", (64, 512, 8), "cluster", "cluster"), ("bf16", (128, 1024, 96), "grid", "steps"),
                                            ("bf16", (128, 2048, 8), "grid", "grid")):
        I, H, B = shape
        eng = Engine(dtype, 1, B, I, H, 4, device=dev)
        paths = eng.recurrent_path(), eng.recurrent_path(backward=True)
        eng.close()
        assert [p[0] for p in paths] == [forward, backward]
        if H == 512:
            assert all(p[1] == 16 for p in paths)


@pytest.mark.parametrize("dtype,where,shape,steps,kernel,switches", [
    # I, H, B: W_hh in tensor memory, one batch tile of 32 or 64 sequences, several in turn, part of W_hh streamed
    ("f16", "forward", (64, 1024, 40), 6, "lstm_fwd_tm_kernel", {}), ("bf16", "forward", (64, 1088, 70), 4, "lstm_fwd_tm_kernel", {}),
    ("f16", "forward", (64, 1024, 140), 4, "lstm_fwd_wide_kernel", {}), ("bf16", "forward", (64, 2048, 200), 4, "lstm_fwd_wide_kernel", {}),
    ("bf16", "forward", (64, 2432, 3), 4, "lstm_fwd_tm_kernel", {}),
    ("f16", "backward", (64, 1088, 8), 4, "lstm_bwd_tm_kernel", {}), ("bf16", "backward", (64, 1024, 140), 4, "lstm_bwd_tm_kernel", {}),
    # the grid-wide kernels that take their place elsewhere: output-tiled, streamed
    ("bf16", "forward", (64, 1024, 1600), 4, "wide_fwd_kernel", {}), ("bf16", "forward", (128, 1024, 96), 4, "wide_fwd_kernel", {"FLSTM_TMEM": "0"}),
    ("bf16", "forward", (128, 2048, 8), 4, "lstm_fwd_kernel", {"FLSTM_TMEM": "0"}),
    ("bf16", "backward", (128, 2048, 8), 4, "lstm_bwd_kernel", {"FLSTM_TMEM": "0"}),
])
def test_each_grid_wide_kernel_returns_and_recovers(dtype, where, shape, steps, kernel, switches, monkeypatch):
    for name, value in switches.items():
        monkeypatch.setenv(name, value)
    _time_out_and_recover(dtype, "tc", where, shape, steps, kernel)


@pytest.mark.parametrize("where,shape,lost", [
    # I, H, B; what a CTA sends or its count of resets (2, 4), step, sequence: the first batch group and others, first steps, last ones and
    # some behind the slots' first reuse
    ("forward", (64, 1024, 64), (2, 14, 40)), ("forward", (64, 576, 96), (2, 0, 95)), ("forward", (64, 1536, 32), (2, 24, 30)),
    ("forward", (64, 1024, 64), (4, 9, 3)), ("forward", (64, 2048, 31), (4, 0, 30)),
    ("backward", (64, 1024, 64), (2, 14, 40)), ("backward", (64, 1088, 8), (2, 0, 7)), ("backward", (64, 1536, 32), (2, 24, 31)),
    ("backward", (64, 576, 96), (4, 9, 70)),
])
def test_words_that_never_come_end_the_launch(where, shape, lost):
    """The gathers of all CTAs of a batch group (the other groups go on to their end), and the wait for the resets of a CTA's own slots."""
    steps = 26
    eng = Engine("f16", 1, shape[2], shape[0], shape[1], steps, device=torch.device("cuda", 0))
    assert eng.exchanges_directly(steps, backward=where == "backward")
    eng.close()
    _time_out_and_recover("f16", "tc", where, shape, steps, lost=lost)


@pytest.mark.parametrize("I,H,B,step,sequence", [(64, 1024, 64, 14, 40), (64, 1088, 8, 0, 7), (64, 1536, 32, 24, 31), (64, 576, 96, 9, 70)])
def test_a_piece_read_in_part_ends_the_launch(I, H, B, step, sequence):
    """The BPTT looks at one word of a 16-byte piece: one that came without another of its words would be taken for whole."""
    message = _time_out_and_recover("f16", "tc", "backward", (I, H, B), 26, lost=(1, step, sequence))
    assert "before all of it was written" in message
