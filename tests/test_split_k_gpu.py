"""Weight gradients whose GEMM is split along K = T * B (few output tiles, long contraction) against the oracle: a last split
that is shorter than the others, row counts that no K block divides, output widths with and without a 16-byte row pitch,
and accumulation over checkpoint segments."""
import pytest
import torch

from flashlstm_poc_b200.engine import Engine
from flashlstm_poc_b200.workloads import Workload, make_inputs
from tests.gpu_helpers import assert_parity, run_engine, run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,T,B,I,H", [("f16", 64, 16, 64, 64), ("bf16", 103, 10, 8, 128), ("f16", 61, 37, 200, 192),
                                           ("bf16", 40, 130, 24, 320)])
def test_split_weight_gradients(dtype, T, B, I, H):
    w = Workload("t", dtype, 1, I, H, B, T, seed=61, state_std=0.2)
    inp = make_inputs(w)
    got, eng = run_engine(w, inp, repeat=2)
    eng.close()
    assert_parity(got, run_oracle(inp), dtype)


def test_split_weight_gradients_accumulate_over_segments():
    w = Workload("t", "f16", 1, 64, 128, 32, 96, seed=62)
    inp = make_inputs(w)
    dev = torch.device("cuda", 0)
    x, dy = inp.x.to(dev, torch.float16), inp.dy.to(dev, torch.float16)
    grads = []
    for interval in (0, 40):  # whole segments of 40 steps, the last one of 16
        eng = Engine("f16", 1, 32, 64, 128, 96, device=dev)
        eng.set_recompute_interval(interval)
        eng.set_weights(0, *(p[0].to(dev) for p in (inp.w_ih, inp.w_hh, inp.b_ih, inp.b_hh)))
        eng.forward(x)
        eng.backward(dy)
        torch.cuda.synchronize()
        grads.append([g.clone() for g in eng.grads(0)])
        eng.close()
    # the same fp32 sums of 3072 products in another order: sqrt(3072) * 2^-24 relative, with room for unlucky signs
    for a, b in zip(*grads):
        assert float((a - b).norm() / a.norm()) < 1e-5
