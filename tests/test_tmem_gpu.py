"""The recurrent kernels that hold W_hh in tensor memory (tc_lstm_fwd_tm.cu, tc_lstm_fwd_wide.cu, tc_lstm_bwd_tm.cu) against
the oracle, at the edges of their tiling: an odd and an even number of 64-wide K chunks per half, weights in tensor memory only,
beside shared memory and streamed, every batch-tile width, partly filled and empty tiles, one and two batch groups, one to six
batch tiles in turn, and step ranges that continue a launch.  KERNELS names the kernel that each shape runs."""
import pytest
import torch

from flashlstm_poc_b200.engine import TORCH_DTYPES, Engine
from flashlstm_poc_b200.workloads import Workload, make_inputs
from tests.gpu_helpers import assert_parity, run_engine, run_oracle

pytestmark = pytest.mark.gpu

# batch, hidden size, training, steps
SHAPES = [(1, 1088, True, 5), (70, 1088, True, 5), (33, 1152, True, 5), (100, 1152, True, 5), (40, 1216, True, 5), (32, 1280, True, 5),
          (32, 1024, True, 25), (40, 768, True, 25), (5, 2048, True, 5), (64, 2048, True, 33), (31, 2304, True, 5), (50, 2368, True, 5),
          # batch tiles in turn
          (140, 1024, True, 5), (256, 1024, True, 5), (259, 1024, False, 5), (300, 704, True, 5), (130, 1088, True, 5), (65, 1984, False, 5),
          (100, 2048, True, 5), (256, 2048, True, 5), (530, 320, True, 5), (290, 576, True, 5), (150, 2176, False, 5),
          # streamed
          (3, 2432, False, 5), (16, 2496, False, 5), (17, 3072, False, 5), (33, 4096, False, 5), (8, 4096, False, 5), (64, 2560, False, 5)]


@pytest.mark.parametrize("B,H,training,T", SHAPES)
def test_tensor_memory_kernels_match_the_oracle(B, H, training, T):
    dtype = "bf16" if (B + H // 64) % 2 else "f16"
    w = Workload("t", dtype, 1, 64, H, B, T, seed=51, state_std=0.3, training=training)
    inp = make_inputs(w)
    got, eng = run_engine(w, inp, repeat=2)
    eng.close()
    assert_parity(got, run_oracle(inp), dtype)


@pytest.mark.parametrize("B,H", [(7, 1088), (40, 2048), (140, 1024)])
def test_ranges_continue_one_another(B, H):
    """Forward and backward in step ranges equal one call."""
    w = Workload("t", "f16", 1, 64, H, B, 7, seed=52, state_std=0.3)
    inp = make_inputs(w)
    dev, td = torch.device("cuda", 0), TORCH_DTYPES["f16"]
    eng = Engine("f16", 1, B, 64, H, 7, device=dev)
    eng.set_weights(0, inp.w_ih[0].to(dev), inp.w_hh[0].to(dev), inp.b_ih[0].to(dev), inp.b_hh[0].to(dev))
    x, h0, c0, dy = (t.to(dev, td) for t in (inp.x, inp.h0, inp.c0, inp.dy))
    y, hn, cn = eng.forward(x, h0, c0)
    dx, dh0, dc0 = eng.backward(dy)
    want = [t.clone() for t in (y, hn, cn, dx, dh0, dc0)]
    got = [torch.empty_like(t) for t in want]
    for t0, t1 in ((0, 3), (3, 4), (4, 7)):
        eng.forward_range_into(7, t0, t1, x, h0, c0, *got[:3])
    for t0, t1 in ((5, 7), (1, 5), (0, 1)):
        eng.backward_range_into(7, t0, t1, dy, None, None, *got[3:])
    torch.cuda.synchronize()
    eng.close()
    for a, b in zip(want, got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("H,dtype", [(2432, "bf16"), (2496, "f16"), (4096, "f16")])
def test_ranges_of_a_streamed_forward_continue_one_another(H, dtype):
    """Part of W_hh is streamed in a direction that alternates from step to step: it goes by the step's number in the sequence,
    whatever step a launch starts at."""
    B, T = 3, 7
    w = Workload("t", dtype, 1, 64, H, B, T, seed=53, state_std=0.3, training=False)
    inp = make_inputs(w)
    dev, td = torch.device("cuda", 0), TORCH_DTYPES[dtype]
    eng = Engine(dtype, 1, B, 64, H, T, training=False, device=dev)
    eng.set_weights(0, inp.w_ih[0].to(dev), inp.w_hh[0].to(dev), inp.b_ih[0].to(dev), inp.b_hh[0].to(dev))
    x, h0, c0 = (t.to(dev, td) for t in (inp.x, inp.h0, inp.c0))
    want = [t.clone() for t in eng.forward(x, h0, c0)]
    got = [torch.empty_like(t) for t in want]
    for ranges in (((0, 3), (3, 4), (4, 7)), ((0, 1), (1, 6), (6, 7))):
        for t in got:
            t.zero_()
        for t0, t1 in ranges:
            eng.forward_range_into(T, t0, t1, x, h0, c0, *got)
        torch.cuda.synchronize()
        for a, b in zip(want, got):
            assert torch.equal(a, b)
    eng.close()


# batch, hidden size, training, steps, then (kernel, batch tile, tiles in turn) forward and backward.  ANY: the BPTT's batch groups
# depend on how many clusters of four CTAs the GPU holds at once (33 of 37 that its SMs would make on the one measured).
TM, WIDE, BACK = "lstm_fwd_tm_kernel", "lstm_fwd_wide_kernel", "lstm_bwd_tm_kernel"
ANY = (BACK, None, None)
KERNELS = [
    (1, 1088, True, 5, (TM, 32, 1), (BACK, 32, 1)), (70, 1088, True, 5, (TM, 64, 1), ANY),
    (33, 1152, True, 5, (TM, 32, 1), ANY), (100, 1152, True, 5, (TM, 64, 1), ANY),
    (40, 1216, True, 5, ("lstm_fwd_kernel", 64, 1), (BACK, 64, 1)), (32, 1280, True, 5, (TM, 32, 1), (BACK, 32, 1)),
    (32, 1024, True, 25, (TM, 32, 1), (BACK, 32, 1)), (40, 768, True, 25, ("cluster_fwd_kernel", 6, 1), ("cluster_bwd_kernel", 6, 1)),
    (5, 2048, True, 5, (TM, 32, 1), (BACK, 32, 1)), (64, 2048, True, 33, (TM, 64, 1), (BACK, 64, 1)),
    # (training at these widths needs more clusters than fit and runs on the CUDA cores)
    (31, 2304, True, 5, None, None), (50, 2368, True, 5, None, None),
    (31, 2304, False, 5, (TM, 32, 1), None), (50, 2368, False, 5, (TM, 64, 1), None),
    # batch tiles in turn
    (140, 1024, True, 5, (WIDE, 64, 2), (BACK, 64, 2)), (256, 1024, True, 5, (WIDE, 64, 2), (BACK, 64, 2)),
    (259, 1024, False, 5, (WIDE, 128, 2), None), (300, 704, True, 5, (WIDE, 64, 2), ANY),
    (130, 1088, True, 5, (WIDE, 64, 2), ANY), (65, 1984, False, 5, (WIDE, 64, 2), None),
    (100, 2048, True, 5, (WIDE, 64, 2), (BACK, 64, 2)), (256, 2048, True, 5, (WIDE, 128, 2), ("step_kernel", 0, 1)),
    (530, 320, True, 5, (WIDE, 64, 2), ANY), (290, 576, True, 5, (WIDE, 64, 2), ANY),
    (150, 2176, False, 5, (WIDE, 128, 2), None),
    # streamed
    (3, 2432, False, 5, (TM, 16, 1), None), (16, 2496, False, 5, (TM, 16, 1), None), (17, 3072, False, 5, (TM, 32, 1), None),
    (33, 4096, False, 5, (TM, 64, 1), None), (8, 4096, False, 5, (TM, 16, 1), None), (64, 2560, False, 5, (TM, 64, 1), None)]


def check_kernels(table):
    for B, H, training, T, forward, backward in table:
        eng = Engine("f16", 1, B, 64, H, T, training=training, device=torch.device("cuda", 0))
        for back, want in ((False, forward), (True, backward)):
            if want is not None:
                got = eng.recurrent_kernel(T, backward=back)
                have = got["name"], got["batch_tile"], got["tiles_in_turn"]
                assert have == want if want is not ANY else have[0] == BACK, (B, H, back, have)
                if got["name"] in (TM, WIDE, BACK):
                    assert bool(got["weights_streamed"]) == (H > 2368)
        eng.close()


def test_which_kernels_the_shapes_run():
    assert set(SHAPES) <= {s[:4] for s in KERNELS}
    check_kernels(KERNELS)


@pytest.mark.parametrize("dtype,B,H,short_fwd,long_fwd,short_bwd,long_bwd", [
    ("f16", 32, 1024, "lstm_fwd_kernel", "lstm_fwd_tm_kernel", "lstm_bwd_kernel", "lstm_bwd_tm_kernel"),
    ("bf16", 64, 1024, "lstm_fwd_kernel", "lstm_fwd_tm_kernel", "lstm_bwd_kernel", "lstm_bwd_tm_kernel"),
    ("bf16", 40, 768, "lstm_fwd_kernel", "lstm_fwd_tm_kernel", "lstm_bwd_kernel", "lstm_bwd_tm_kernel"),
    ("f16", 20, 1152, "lstm_fwd_kernel", "lstm_fwd_tm_kernel", "lstm_bwd_kernel", "lstm_bwd_tm_kernel"),
    ("f16", 32, 1280, "lstm_fwd_kernel", "lstm_fwd_tm_kernel", "lstm_bwd_kernel", "lstm_bwd_tm_kernel"),
    ("bf16", 40, 2048, "lstm_fwd_kernel", "lstm_fwd_tm_kernel", "lstm_bwd_kernel", "lstm_bwd_tm_kernel"),
    ("f16", 140, 1024, "lstm_fwd_kernel", "lstm_fwd_wide_kernel", "lstm_bwd_tm_kernel", "lstm_bwd_tm_kernel"),
    ("bf16", 256, 2048, "wide_fwd_kernel", "lstm_fwd_wide_kernel", "step_kernel", "step_kernel"),
])
def test_the_length_of_a_launch_chooses_its_kernel_and_not_its_bits(dtype, B, H, short_fwd, long_fwd, short_bwd, long_bwd, monkeypatch):
    """Short launches run other kernels than long ones, whatever length the engine was made for, and every way to cut a sequence
    gives the same bits."""
    monkeypatch.setenv("FLSTM_CLUSTER", "0")
    I, T = 64, 40
    w = Workload("t", dtype, 1, I, H, B, T, seed=54, state_std=0.3)
    inp = make_inputs(w)
    dev, td = torch.device("cuda", 0), TORCH_DTYPES[dtype]
    params = [p[0].to(dev) for p in (inp.w_ih, inp.w_hh, inp.b_ih, inp.b_hh)]
    x, h0, c0, dy = (t.to(dev, td) for t in (inp.x, inp.h0, inp.c0, inp.dy))

    def made_for(steps):
        eng = Engine(dtype, 1, B, I, H, steps, device=dev)
        eng.set_weights(0, *params)
        return eng

    def whole(eng):
        out = [t.clone() for t in eng.forward(x, h0, c0)]
        out += [t.clone() for t in eng.backward(dy)]
        return out + [t.clone() for t in eng.grads(0)]

    long = made_for(T)
    want = whole(long)
    short = made_for(2)
    short.forward(x[:2].contiguous(), h0, c0)
    for eng in (long, short):
        assert eng.recurrent_kernel(1)["name"] == short_fwd and eng.recurrent_kernel(T)["name"] == long_fwd
        assert eng.recurrent_kernel(1, backward=True)["name"] == short_bwd
        assert eng.recurrent_kernel(T, backward=True)["name"] == long_bwd
    for a, b in zip(want, whole(short)):  # the engine has grown
        assert torch.equal(a, b)
    short.close()
    got = [torch.zeros_like(t) for t in want[:6]]
    for t0, t1 in ((0, 1), (1, 4), (4, 36), (36, 40)):
        long.forward_range_into(T, t0, t1, x, h0, c0, *got[:3])
    for t0, t1 in ((39, 40), (30, 39), (5, 30), (0, 5)):
        long.backward_range_into(T, t0, t1, dy, None, None, *got[3:])
    torch.cuda.synchronize()
    for a, b in zip(want, got + list(long.grads(0))):
        assert torch.equal(a, b)
    long.close()


def test_step_trace_of_the_wide_forward():
    """The kernel with batch tiles in turn stamps the first tile of each step."""
    import numpy as np

    from flashlstm_poc_b200 import step_trace

    w = Workload("trace", "f16", 1, 64, 1024, 140, 24, seed=56)
    inp = make_inputs(w)
    dev, td = torch.device("cuda", 0), TORCH_DTYPES["f16"]
    eng = Engine("f16", 1, 140, 64, 1024, 24, device=dev)
    eng.set_weights(0, inp.w_ih[0].to(dev), inp.w_hh[0].to(dev), inp.b_ih[0].to(dev), inp.b_hh[0].to(dev))
    x, dy = inp.x.to(dev, td), inp.dy.to(dev, td)

    def run_step():
        eng.forward(x)
        eng.backward(dy)

    run_step()
    stamps = step_trace.collect(eng, run_step, steps=16)
    eng.close()
    forward = stamps[0]
    points = forward[:, [0, 2, 3, 4, 5, 7, 8]]
    assert (points[:, 0] > 0).all() and (np.diff(points, axis=1) > 0).all() and (forward[:, 0] < forward[:, 1]).all()
    assert (forward[1:, 0] > forward[:-1, 8]).all()  # a step's barrier waits for the release of the step before
    summary = step_trace.summarize(stamps, skip=2)
    assert summary["forward"]["period"] > 0 and summary["bptt"]["period"] > 0


IN_TURN = [(384, 1024, True, 4, (WIDE, 128, 2), (BACK, 64, 3)), (256, 1536, True, 3, (WIDE, 128, 2), (BACK, 64, 4)),
           (300, 1216, True, 3, (WIDE, 128, 3), (BACK, 64, 5)), (380, 1216, True, 3, (WIDE, 128, 3), (BACK, 64, 6)),
           (500, 1216, False, 3, (WIDE, 128, 4), None), (1400, 1024, False, 3, (WIDE, 128, 6), None),
           (310, 1024, True, 3, (WIDE, 128, 2), (BACK, 64, 3)), (31, 2304, False, 5, (TM, 32, 1), None),
           (50, 2368, False, 5, (TM, 64, 1), None)]


def test_which_kernels_the_shapes_below_run():
    check_kernels(IN_TURN)


@pytest.mark.parametrize("B,H,training,T,forward,backward", IN_TURN)
def test_three_to_six_tiles_in_turn_and_the_widest_layers(B, H, training, T, forward, backward):
    test_tensor_memory_kernels_match_the_oracle(B, H, training, T)


@pytest.mark.parametrize("B,H,T", [(40, 2048, 70), (384, 1024, 9), (300, 1216, 9)])
def test_long_ranges_continue_one_another(B, H, T):
    """The same with ranges that are long enough for these kernels, and several tiles in turn."""
    w = Workload("t", "bf16", 1, 64, H, B, T, seed=55, state_std=0.3)
    inp = make_inputs(w)
    dev, td = torch.device("cuda", 0), TORCH_DTYPES["bf16"]
    eng = Engine("bf16", 1, B, 64, H, T, device=dev)
    eng.set_weights(0, inp.w_ih[0].to(dev), inp.w_hh[0].to(dev), inp.b_ih[0].to(dev), inp.b_hh[0].to(dev))
    half = T // 2
    assert eng.recurrent_kernel(half)["name"] in (TM, WIDE) and eng.recurrent_kernel(half, backward=True)["name"] == BACK
    x, h0, c0, dy = (t.to(dev, td) for t in (inp.x, inp.h0, inp.c0, inp.dy))
    want = [t.clone() for t in (*eng.forward(x, h0, c0), *eng.backward(dy))]
    got = [torch.empty_like(t) for t in want]
    for t0, t1 in ((0, half), (half, T)):
        eng.forward_range_into(T, t0, t1, x, h0, c0, *got[:3])
    for t0, t1 in ((half, T), (0, half)):
        eng.backward_range_into(T, t0, t1, dy, None, None, *got[3:])
    torch.cuda.synchronize()
    eng.close()
    for a, b in zip(want, got):
        assert torch.equal(a, b)


# copies of four chunks with one, two and three left over; the widest that has three such copies, and one that takes copies of two
@pytest.mark.parametrize("B,H", [(530, 320), (140, 1152), (65, 1984), (100, 2176), (100, 2240),
                                 # three, four and five tiles of 64 rather than half as many of 128
                                 (550, 768), (450, 1024), (130, 1792), (190, 2048)])
def test_tiles_in_turn_with_every_remainder_of_a_copy(B, H):
    w = Workload("t", "bf16" if H % 128 else "f16", 1, 64, H, B, 4, seed=54, state_std=0.3, training=False)
    inp = make_inputs(w)
    got, eng = run_engine(w, inp, repeat=2)
    kernel = eng.recurrent_kernel(4)
    assert (kernel["name"], kernel["batch_tile"]) == (WIDE, 64)
    eng.close()
    assert_parity(got, run_oracle(inp), w.dtype)
