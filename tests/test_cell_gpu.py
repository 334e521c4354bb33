"""Inference over a few steps (tc_cell.cu, one launch per layer and step) against the oracle: one to four tiles of 8
sequences, input widths with a partial K chunk, both warp counts, absent states, padded widths, and the rule's edge."""
import pytest
import torch

from flashlstm_poc_b200.engine import TORCH_DTYPES, Engine
from flashlstm_poc_b200.workloads import Workload, make_inputs
from tests.gpu_helpers import assert_parity, run_engine, run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,L,T,B,I,H", [("f16", 2, 1, 1, 1024, 1024), ("bf16", 1, 2, 8, 40, 64), ("f16", 3, 4, 9, 8, 128),
                                             ("bf16", 2, 3, 16, 200, 192), ("f16", 1, 4, 17, 72, 320), ("bf16", 2, 1, 32, 96, 512),
                                             ("f16", 2, 2, 5, 33, 70), ("f16", 1, 5, 4, 64, 64), ("f16", 1, 2, 33, 64, 64)])
def test_few_step_inference(dtype, L, T, B, I, H):
    w = Workload("t", dtype, L, I, H, B, T, seed=91, state_std=0.3, training=False)
    inp = make_inputs(w)
    inp.dy = None
    got, eng = run_engine(w, inp, repeat=2)
    eng.close()
    assert_parity(got, run_oracle(inp), dtype)


def test_absent_states_and_fp32_cell_io():
    w = Workload("t", "f16", 2, 64, 128, 3, 2, seed=92, training=False)  # zero states
    inp = make_inputs(w)
    dev, td = torch.device("cuda", 0), TORCH_DTYPES["f16"]
    eng = Engine("f16", 2, 3, 64, 128, 2, training=False, device=dev)
    for l in range(2):
        eng.set_weights(l, inp.w_ih[l].to(dev), inp.w_hh[l].to(dev), inp.b_ih[l].to(dev), inp.b_hh[l].to(dev))
    x = inp.x.to(dev, td)
    zeros = torch.zeros(2, 3, 128, device=dev, dtype=td)
    want = eng.forward(x, zeros, zeros)
    got = eng.forward(x)
    assert all(torch.equal(a, b) for a, b in zip(want, got))
    eng.set_cell_io_f32()
    y, hn = torch.empty_like(want[0]), torch.empty_like(want[1])
    cn = torch.empty(2, 3, 128, device=dev)
    eng.forward_into(2, x, zeros, torch.zeros(2, 3, 128, device=dev), y, hn, cn)
    torch.cuda.synchronize()
    assert torch.equal(y, want[0]) and torch.equal(hn, want[1]) and torch.equal(cn.to(td), want[2])
    eng.close()


def test_states_updated_in_place():
    """h0 / c0 handed over as h_n / c_n as well: the same results as with buffers of their own."""
    w = Workload("t", "bf16", 2, 64, 512, 4, 1, seed=93, state_std=0.3, training=False)
    inp = make_inputs(w)
    dev, td = torch.device("cuda", 0), TORCH_DTYPES["bf16"]
    eng = Engine("bf16", 2, 4, 64, 512, 1, training=False, device=dev)
    for l in range(2):
        eng.set_weights(l, inp.w_ih[l].to(dev), inp.w_hh[l].to(dev), inp.b_ih[l].to(dev), inp.b_hh[l].to(dev))
    x, h, c = inp.x.to(dev, td), inp.h0.to(dev, td), inp.c0.to(dev, td)
    want = eng.forward(x, h, c)
    y = torch.empty_like(want[0])
    eng.forward_into(1, x, h, c, y, h, c)
    torch.cuda.synchronize()
    for a, b in zip(want, (y, h, c)):  # fp32 sums of 1088 terms in another order, rounded to bf16
        assert torch.allclose(a.float(), b.float(), rtol=2 ** -7, atol=2 ** -9)
    eng.close()


@pytest.mark.parametrize("L,T,B,I,H,cells", [
    (1, 1, 16, 64, 3136, True), (1, 1, 32, 64, 3072, True), (1, 1, 17, 64, 3136, False),
    (1, 2, 16, 64, 1344, True), (1, 2, 32, 64, 1280, True), (1, 2, 17, 64, 1344, False),
    (1, 3, 16, 64, 1216, True), (1, 3, 32, 64, 1152, True), (1, 3, 17, 64, 1216, False),
    (1, 4, 16, 64, 512, True), (2, 4, 8, 64, 512, False), (4, 4, 8, 64, 128, True), (2, 4, 16, 64, 576, True),
    (1, 4, 17, 64, 1152, True), (2, 4, 17, 64, 64, False), (1, 4, 17, 64, 1216, False), (1, 4, 8, 64, 1344, False),
    (1, 5, 1, 64, 64, False), (1, 2, 1, 2048, 2112, False),
    (1, 4, 16, 64, 1152, True), (1, 4, 16, 64, 1216, False), (1, 3, 16, 1536, 1536, True), (1, 3, 16, 2048, 2048, False),
])
def test_which_calls_run_step_by_step(L, T, B, I, H, cells):
    """The edges of the rule, by the launches of a call: one per layer and step, or the other path's (states in, a projection
    and a recurrence per layer, states out).  Both give the oracle's results."""
    w = Workload("t", "f16", L, I, H, B, T, seed=94, state_std=0.3, training=False)
    inp = make_inputs(w)
    inp.dy = None
    got, eng = run_engine(w, inp)
    dev, td = torch.device("cuda", 0), TORCH_DTYPES["f16"]
    before = eng.launch_count
    eng.forward(inp.x.to(dev, td), inp.h0.to(dev, td), inp.c0.to(dev, td))
    torch.cuda.synchronize()
    launches = eng.launch_count - before
    eng.close()
    assert launches == (L * T if cells else 2 * L + 2)
    assert_parity(got, run_oracle(inp), "f16")
