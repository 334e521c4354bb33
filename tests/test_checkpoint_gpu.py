"""Activation checkpoints (recompute interval R): the forward keeps only the h/c state entering every R-th step,
the backward rebuilds the gate cache one segment at a time.  Outputs and state gradients must be bit-identical
to the full-cache engine (same kernels on the same values), weight gradients equal up to the fp32 order of the
segment-by-segment sum, everything within the parity bar against the CPU oracle, and the workspace smaller."""
import numpy as np
import pytest
import torch

from flashlstm_poc_b200.engine import TORCH_DTYPES, Engine
from flashlstm_poc_b200.workloads import Workload, make_inputs
from tests.gpu_helpers import assert_parity, run_oracle
from tests.helpers import to_np

pytestmark = pytest.mark.gpu


def _run(w, inp, interval, dhn, dcn, repeat=1):
    dev = torch.device("cuda", 0)
    td = TORCH_DTYPES[w.dtype]
    eng = Engine(w.dtype, w.layers, w.batch, w.input_size, w.hidden_size, w.seq_len, device=dev, backend="tc")
    for l in range(w.layers):
        eng.set_weights(l, inp.w_ih[l].to(dev), inp.w_hh[l].to(dev), inp.b_ih[l].to(dev), inp.b_hh[l].to(dev))
    if interval:
        eng.set_recompute_interval(interval)
    out = {}
    x, h0, c0, dy = inp.x.to(dev, td), inp.h0.to(dev, td), inp.c0.to(dev, td), inp.dy.to(dev, td)  # x must outlive backward
    for _ in range(repeat):
        y, hn, cn = eng.forward(x, h0, c0)
        dx, dh0, dc0 = eng.backward(dy, dhn.to(dev, td), dcn.to(dev, td))
        out = dict(y=to_np(y), hn=to_np(hn), cn=to_np(cn), dx=to_np(dx), dh0=to_np(dh0), dc0=to_np(dc0),
                   dw_ih=[to_np(eng.grads(l)[0]) for l in range(w.layers)],
                   dw_hh=[to_np(eng.grads(l)[1]) for l in range(w.layers)],
                   db=[to_np(eng.grads(l)[2]) for l in range(w.layers)])
    torch.cuda.synchronize()
    bytes_ = eng.workspace_bytes
    eng.close()
    return out, bytes_


def _compare(dtype, L, T, B, I, H, R):
    w = Workload("ck", dtype, L, I, H, B, T, seed=77, state_std=0.3)
    inp = make_inputs(w)
    torch.manual_seed(9)
    td = TORCH_DTYPES[dtype]
    dhn, dcn = torch.randn(L, B, H).to(td), torch.randn(L, B, H).to(td)
    full, full_bytes = _run(w, inp, 0, dhn, dcn)
    ck, ck_bytes = _run(w, inp, R, dhn, dcn, repeat=2)   # twice: the carries and accumulators start over
    for k in ("y", "hn", "cn", "dx", "dh0", "dc0"):
        assert np.array_equal(full[k], ck[k]), k
    for k in ("dw_ih", "dw_hh", "db"):
        for a, b in zip(full[k], ck[k]):
            assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(a) + 1e-7, k
    ref = run_oracle(inp, dhn.float(), dcn.float())
    assert_parity(ck, ref, dtype)
    if R < T:
        assert ck_bytes < full_bytes


@pytest.mark.parametrize("dtype,L,T,B,I,H,R,step_path", [
    ("f16", 2, 23, 16, 64, 64, 5, False),     # persistent kernels, ragged last segment, stacked layers
    ("bf16", 1, 12, 32, 128, 128, 1, False),  # R = 1: a checkpoint at every step
    ("f16", 1, 9, 8, 64, 128, 16, False),     # R >= T: a single segment
    ("bf16", 2, 9, 256, 128, 128, 4, True),   # per-step GEMM path (wide batch), dh carried as fp32 partial sums
    ("f16", 1, 7, 300, 64, 256, 3, True),     # per-step path, ragged batch tile, K split
])
def test_checkpoint_mode_matches_full_cache(dtype, L, T, B, I, H, R, step_path, monkeypatch):
    monkeypatch.setenv("FLSTM_STEP_MIN_BATCH", "1" if step_path else "0")
    _compare(dtype, L, T, B, I, H, R)


@pytest.mark.parametrize("dtype,L,T,B,I,H,R", [
    ("f16", 2, 23, 16, 64, 64, 5), ("bf16", 1, 12, 37, 128, 256, 1), ("f16", 1, 9, 20, 64, 512, 16), ("bf16", 2, 10, 300, 64, 256, 4),
])
def test_checkpoint_mode_on_clusters(dtype, L, T, B, I, H, R):
    """The same on the cluster-resident kernels: a segment's backward continues from the dG of the step after it."""
    eng = Engine(dtype, L, B, I, H, T, device=torch.device("cuda", 0))
    assert eng.recurrent_path()[0] == eng.recurrent_path(backward=True)[0] == "cluster"
    eng.close()
    _compare(dtype, L, T, B, I, H, R)


def test_checkpoint_mode_with_streamed_weights():
    """Segments that start at an odd step, at a width whose W_hh is streamed in alternating directions."""
    _compare("bf16", 1, 7, 3, 64, 2432, 3)


@pytest.mark.parametrize("dtype,L,T,B,I,H,R,forward,backward", [
    ("f16", 1, 30, 32, 64, 1024, 26, "lstm_fwd_tm_kernel", "lstm_bwd_tm_kernel"),  # a last segment of four steps runs without them
    ("bf16", 2, 9, 256, 64, 1024, 4, "lstm_fwd_wide_kernel", "lstm_bwd_tm_kernel"),  # two batch tiles in turn
    ("bf16", 1, 9, 5, 64, 2048, 5, "lstm_fwd_tm_kernel", "lstm_bwd_tm_kernel"),
    ("f16", 1, 7, 130, 64, 1088, 3, "lstm_fwd_wide_kernel", "lstm_bwd_tm_kernel"),
])
def test_checkpoint_mode_in_tensor_memory(dtype, L, T, B, I, H, R, forward, backward):
    eng = Engine(dtype, L, B, I, H, T, device=torch.device("cuda", 0))
    assert eng.recurrent_kernel(R)["name"] == forward and eng.recurrent_kernel(R, backward=True)["name"] == backward
    eng.close()
    _compare(dtype, L, T, B, I, H, R)


def test_checkpoint_mode_limits():
    from flashlstm_poc_b200._lib import FlashLstmError

    dev = torch.device("cuda", 0)
    eng = Engine("f32", 1, 4, 16, 16, 8, device=dev)   # fp32 runs on the SIMT backend
    with pytest.raises(FlashLstmError, match="tensor-core backend"):
        eng.set_recompute_interval(4)
    eng.close()
    w = Workload("ck", "f16", 1, 64, 64, 8, 8, seed=1)
    inp = make_inputs(w)
    eng = Engine("f16", 1, 8, 64, 64, 8, device=dev)
    eng.set_weights(0, inp.w_ih[0].to(dev), inp.w_hh[0].to(dev), inp.b_ih[0].to(dev), inp.b_hh[0].to(dev))
    eng.set_recompute_interval(4)
    x = inp.x.to(dev, torch.float16)
    y = torch.empty(8, 8, 64, dtype=torch.float16, device=dev)
    with pytest.raises(FlashLstmError, match="step ranges"):
        eng.forward_range_into(8, 0, 4, x, None, None, y, None, None)
    eng.set_recompute_interval(0)   # back to the full gate cache
    eng.forward_range_into(8, 0, 4, x, None, None, y, None, None)
    eng.forward_range_into(8, 4, 8, x, None, None, y, None, None)
    torch.cuda.synchronize()
    eng.close()


def test_a_padded_shape_says_why_it_has_no_checkpoints():
    from flashlstm_poc_b200._lib import FlashLstmError

    eng = Engine("f16", 1, 4, 33, 70, 8, device=torch.device("cuda", 0))
    assert eng.backend == "tc"
    with pytest.raises(FlashLstmError, match="hidden_size % 64 == 0 and input_size % 8 == 0"):
        eng.set_recompute_interval(4)
    eng.close()


@pytest.mark.parametrize("dtype,L,T,B,H,R", [("bf16", 3, 9, 140, 1024, 4), ("f16", 2, 8, 100, 1984, 3), ("bf16", 2, 7, 290, 1024, 3), ("f16", 2, 5, 259, 1024, 3)])
def test_kept_states_spare_the_recurrence_a_second_run(dtype, L, T, B, H, R):
    """Tiles of 64 and of 128 in turn: all layers but the last rebuild a segment from the h_t that the layer above was given."""
    eng = Engine(dtype, L, B, 64, H, R, device=torch.device("cuda", 0), backend="tc")
    assert eng.recurrent_kernel(R)["name"] == "lstm_fwd_wide_kernel"
    eng.close()
    _compare(dtype, L, T, B, 64, H, R)
