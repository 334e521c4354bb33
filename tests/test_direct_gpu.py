"""The tensor-memory kernels that exchange without a step barrier (tc_direct.cuh): words that announce themselves, slots that are
used again after eight steps.  What the oracle tests of test_tmem_gpu.py do not reach: results that are no numbers, a y that starts
at any element, many launches in a row, and sequences of every length around the slots."""
import pytest
import torch

from flashlstm_poc_b200.engine import TORCH_DTYPES, Engine
from flashlstm_poc_b200.workloads import Workload, make_inputs
from tests.gpu_helpers import assert_parity, run_engine, run_oracle

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


def engine(dtype, B, H, T, training=True):
    w = Workload("t", dtype, 1, 64, H, B, T, seed=91, state_std=0.3, training=training)
    inp = make_inputs(w)
    eng = Engine(dtype, 1, B, 64, H, T, training=training, device=DEV)
    eng.set_weights(0, inp.w_ih[0].to(DEV), inp.w_hh[0].to(DEV), inp.b_ih[0].to(DEV), inp.b_hh[0].to(DEV))
    return eng, [t if t is None else t.to(DEV, TORCH_DTYPES[dtype]) for t in (inp.x, inp.h0, inp.c0, inp.dy)]


# One batch group, an odd number of 64-wide chunks of K, partly filled tiles, the neighbouring form with a counter (tiles of 64, and a BPTT
# too wide); then two and three groups on one ring, the last of them partly filled.
SHAPES = [("f16", 32, 1024), ("bf16", 5, 1088), ("bf16", 70, 1088), ("f16", 64, 2048), ("bf16", 31, 2048),
          ("f16", 64, 1024), ("bf16", 41, 1024), ("bf16", 96, 576)]
# the widest: its training is not on the tensor cores
FORWARD_SHAPES = SHAPES + [("bf16", 31, 2304)]


@pytest.mark.parametrize("B,H,forward,backward,groups", [(32, 1024, True, True, 1), (5, 1088, True, True, 1), (70, 1088, False, False, None),
                                                         (64, 2048, False, False, None), (31, 2048, True, False, 1), (64, 1024, True, True, 2),
                                                         (41, 1024, True, True, 2), (96, 576, True, True, 3), (31, 2304, True, None, 1)])
def test_which_kernels_the_shapes_here_run(B, H, forward, backward, groups):
    eng = Engine("bf16", 1, B, 64, H, 26, training=backward is not None, device=DEV)
    assert eng.exchanges_directly(26) == forward
    if groups:
        assert eng.recurrent_kernel(26)["batch_groups"] == groups
    if backward is not None:
        assert eng.exchanges_directly(26, backward=True) == backward
        assert not eng.exchanges_directly(1) or H % 128  # short launches, where there is another kernel for them
    eng.close()


@pytest.mark.parametrize("dtype,B,H,training", [("f16", 64, 1024, True), ("bf16", 41, 1024, True), ("bf16", 96, 576, True), ("f16", 20, 1408, True),
                                                ("bf16", 31, 2304, False), ("f16", 7, 2368, False)])
def test_slots_used_three_times_match_the_oracle(dtype, B, H, training):
    w = Workload("t", dtype, 1, 40, H, B, 26, seed=93, state_std=0.3, training=training)
    inp = make_inputs(w)
    got, eng = run_engine(w, inp, repeat=2)
    assert eng.exchanges_directly(26) and (not training or eng.exchanges_directly(26, backward=True))
    eng.close()
    assert_parity(got, run_oracle(inp), dtype)


@pytest.mark.parametrize("dtype,B,H", FORWARD_SHAPES)
def test_sequences_that_are_no_numbers_stay_their_own(dtype, B, H):
    """From a step with an infinite and a NaN input on, one sequence's h is NaN, of either sign; it crosses like any other value and
    reaches no other sequence, whose results stay the same bit for bit."""
    T = 26
    eng, (x, h0, c0, _) = engine(dtype, B, H, T, training=False)
    want, _, _ = eng.forward(x, h0, c0)
    want = want.clone()
    for value in (float("nan"), -float("nan"), float("inf"), -float("inf")):
        bad = x.clone()
        bad[7, B // 2] = value
        bad[7, B // 2, ::2] = -value
        y, _, _ = eng.forward(bad, h0, c0)
        others = [b for b in range(B) if b != B // 2]
        assert torch.equal(y[:, others], want[:, others])
        assert torch.equal(y[:7, B // 2], want[:7, B // 2])
        assert torch.isnan(y[8:, B // 2]).all()
    y, _, _ = eng.forward(x, h0, c0)
    assert torch.equal(y, want)
    eng.close()


@pytest.mark.parametrize("dtype,B,H", FORWARD_SHAPES)
def test_y_may_start_at_any_element(dtype, B, H):
    T = 14
    eng, (x, h0, c0, _) = engine(dtype, B, H, T, training=False)
    want, hn, cn = eng.forward(x, h0, c0)
    room = torch.empty(T * B * H + 1, dtype=want.dtype, device=DEV)
    y = room[1:].view(T, B, H)
    eng.forward_into(T, x, h0, c0, y, hn, cn)
    torch.cuda.synchronize()
    assert torch.equal(y, want)
    eng.close()


@pytest.mark.parametrize("dtype,B,H", SHAPES)
def test_every_length_around_the_slots_and_many_launches(dtype, B, H):
    """A call of n steps gives the first n steps of a longer one, forward, and repeated calls the same bits."""
    T = 40
    eng, (x, h0, c0, dy) = engine(dtype, B, H, T)
    y, _, _ = eng.forward(x, h0, c0)
    want = y.clone()
    grads = [g.clone() for g in eng.backward(dy)]
    for n in [*range(1, 22), 39]:
        y, hn, _ = eng.forward(x[:n], h0, c0)
        assert torch.equal(y, want[:n]) and torch.equal(hn[0], want[n - 1])
    for _ in range(20):
        y, _, _ = eng.forward(x, h0, c0)
        assert torch.equal(y, want)
        for a, b in zip(grads, eng.backward(dy)):
            assert torch.equal(a, b)
    eng.close()


@pytest.mark.parametrize("dtype,B,H", SHAPES)
def test_gradients_that_are_no_numbers_stay_their_own(dtype, B, H):
    """A NaN and an infinity in one sequence's dY: its gradients of that step and before are NaN, no other sequence's change."""
    T = 26
    eng, (x, h0, c0, dy) = engine(dtype, B, H, T)
    eng.forward(x, h0, c0)
    want = [g.clone() for g in eng.backward(dy)]
    others = [b for b in range(B) if b != B // 2]
    for value in (float("nan"), -float("nan"), float("inf"), -float("inf")):
        bad = dy.clone()
        bad[18, B // 2, ::2] = value
        bad[18, B // 2, 1::2] = -value
        eng.forward(x, h0, c0)
        dx, dh0, dc0 = eng.backward(bad)
        assert torch.equal(dx[:, others], want[0][:, others]) and torch.equal(dx[19:], want[0][19:])
        assert torch.equal(dh0[:, others], want[1][:, others]) and torch.equal(dc0[:, others], want[2][:, others])
        assert torch.isnan(dx[:18, B // 2]).all() and torch.isnan(dh0[0, B // 2]).all()
    eng.close()


# batch, hidden size, whether the forward and the backward pass stay in clusters
CROSSING = [(56, 576, True, True), (57, 570, False, False), (64, 576, False, False), (112, 448, True, True), (112, 576, False, False),
            (113, 448, True, False), (48, 768, False, True), (40, 768, True, True), (96, 640, False, False)]


@pytest.mark.parametrize("B,H,cluster_fwd,cluster_bwd", CROSSING)
def test_both_sides_of_the_line_to_the_clusters_match_the_oracle(B, H, cluster_fwd, cluster_bwd):
    """A direction leaves the cluster-resident kernel where a step without a barrier over the grid is shorter; short sequences too."""
    dtype = "bf16" if H % 128 else "f16"
    for T in (3, 14):
        w = Workload("t", dtype, 1, 40, H, B, T, seed=92, state_std=0.3)
        inp = make_inputs(w)
        got, eng = run_engine(w, inp, repeat=2)
        names = [eng.recurrent_kernel(T, backward=back)["name"].startswith("cluster_") for back in (False, True)]
        eng.close()
        assert names == [cluster_fwd, cluster_bwd]
        assert_parity(got, run_oracle(inp), dtype)
