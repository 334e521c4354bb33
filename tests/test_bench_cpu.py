"""bench.py names the kernels that the engine runs (no GPU needed): labels, launches and stored traffic follow them."""
import pytest

from bench import recurrent_roofline
from flashlstm_poc_b200.workloads import WORKLOADS

PEAKS = {"hbm_gbs": 6500.0, "bf16_tflops": 1600.0, "source": "test"}


def kernel(name, launches_per_step=0):
    return {"name": name, "launches_per_step": launches_per_step}


@pytest.mark.parametrize("forward,backward,slower,label,launches,per_launch,traffic", [
    ("lstm_fwd_wide_kernel", kernel("step_kernel", 2), "bptt", "tc::step_bwd_pointwise_kernel + tc::step_kernel (launched per time step)",
     2048, 1, 57.7e6),
    ("lstm_fwd_wide_kernel", kernel("lstm_bwd_tm_kernel"), "bptt", "tc::lstm_bwd_tm_kernel", 2, 1024, None),
    ("lstm_fwd_wide_kernel", kernel("step_kernel", 2), "recurrent_fwd", "tc::lstm_fwd_wide_kernel", 2, 1024, None),
])
def test_roofline_entry_follows_the_kernels(forward, backward, slower, label, launches, per_launch, traffic):
    w = WORKLOADS["c3_bf16_l2_h2048"]
    phases = {"recurrent_fwd": 30.0, "bptt": 30.0, slower: 35.0}
    out = recurrent_roofline(w, 256, {"recurrent_fwd": kernel(forward), "bptt": backward}, w.seq_len, phases, PEAKS, True)
    assert (out["kernel"], out["launches_in_phase"], out["timesteps_per_launch"], out["traffic"]) == (label, launches, per_launch, traffic)
    assert "traffic_recurrent_fwd_kernel" not in out  # no stored figure of that kernel


def test_roofline_entry_with_checkpoints():
    w = WORKLOADS["c3_bf16_l2_h2048"]
    kernels = {"recurrent_fwd": kernel("lstm_fwd_wide_kernel"), "bptt": kernel("lstm_bwd_tm_kernel")}
    out = recurrent_roofline(w, 128, kernels, 100, {"recurrent_fwd": 30.0, "bptt": 35.0}, PEAKS, True)
    assert (out["launches_in_phase"], out["timesteps_per_launch"]) == (22, 100)
