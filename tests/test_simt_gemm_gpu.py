"""The fp32 GEMMs of the CUDA-core path (projection, input gradient, split-K weight gradients, bias gradient) at sizes around
their tiles and K blocks, through one training step against the oracle."""
import numpy as np
import pytest
import torch

from flashlstm_poc_b200.workloads import Workload, make_inputs
from tests.gpu_helpers import assert_parity, run_engine, run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,B,I,H", [(3, 5, 7, 9), (2, 64, 130, 33), (40, 33, 65, 64), (64, 40, 17, 65), (130, 16, 256, 96),
                                     (12, 130, 128, 200), (90, 32, 500, 150)])
def test_f32_gemms_at_tile_edges(T, B, I, H):
    w = Workload("t", "f32", 1, I, H, B, T, seed=81, state_std=0.2)
    inp = make_inputs(w)
    got, eng = run_engine(w, inp, repeat=2)
    eng.close()
    # weight gradients sum up to 2880 terms of order 1 in fp32: 2880 * 2^-24 * |term| is about 2e-4
    assert_parity(got, run_oracle(inp), "f32", fp32_max_abs=4e-4)


def test_training_without_room_for_the_split_scratch():
    """The partial products of the split-K weight gradients take up to 64 MiB.  An engine that fits without them is made
    without them, and its GEMMs run unsplit."""
    w = Workload("t", "f32", 1, 1024, 1024, 2, 4, seed=82, state_std=0.2)
    inp = make_inputs(w)
    want, eng = run_engine(w, inp)  # also loads the kernels
    eng.close()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    filler = torch.empty(free - (122 << 20), dtype=torch.uint8, device="cuda")  # weights and gradients take 64 MiB
    try:
        got, eng = run_engine(w, inp)
        eng.close()
    finally:
        del filler
        torch.cuda.empty_cache()
    for k, a in want.items():
        for x, y in zip(a if isinstance(a, list) else [a], got[k] if isinstance(a, list) else [got[k]]):
            assert np.abs(x - y).max() <= 2e-5  # fp32 sums of 8 terms of order 1 (dW) in another order at most
