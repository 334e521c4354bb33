"""The cluster-resident recurrent kernels (tc_cluster_fwd.cu, tc_cluster_bwd.cu) against the oracle, at the edges of
their tiling: every width and most cluster sizes they are built for, one, two and four tiles of 8 sequences per cluster
(BPTT: one and two), partly filled tiles and clusters, CTAs of a cluster that own no units, weights partly in shared memory, both ways of sending
h_t (from 4 sequences per cluster on whole rows), and step ranges that continue an earlier launch."""
import pytest
import torch

from flashlstm_poc_b200.engine import TORCH_DTYPES, Engine
from flashlstm_poc_b200.workloads import Workload, make_inputs
from tests.gpu_helpers import assert_parity, run_engine, run_oracle

pytestmark = pytest.mark.gpu

# CTAs per cluster, batch, hidden size
SHAPES = [(1, 3, 64), (1, 200, 64), (4, 5, 64), (2, 1, 128), (2, 150, 128), (1, 9, 128), (2, 33, 192), (4, 100, 192),
          (4, 300, 256), (8, 64, 256), (16, 33, 256), (8, 61, 320), (16, 5, 320), (8, 100, 384), (16, 20, 384),
          (16, 20, 448), (16, 37, 512), (16, 64, 512), (16, 20, 576), (16, 3, 640), (16, 30, 704), (16, 9, 768)]


@pytest.mark.parametrize("cluster,B,H", SHAPES)
def test_cluster_kernels_match_the_oracle(cluster, B, H, monkeypatch):
    monkeypatch.setenv("FLSTM_CLUSTER_SIZE", str(cluster))
    dtype = "bf16" if (B + H // 64) % 2 else "f16"
    w = Workload("t", dtype, 1, 64, H, B, 5, seed=41, state_std=0.3)
    inp = make_inputs(w)
    got, eng = run_engine(w, inp, repeat=2)
    eng.close()
    assert_parity(got, run_oracle(inp), dtype)


@pytest.mark.parametrize("B,H", [(7, 64), (37, 256), (20, 512)])
def test_ranges_and_an_unaligned_gradient(B, H):
    """Forward and backward in step ranges equal one call, also with y and dY that start off a 16-byte boundary."""
    w = Workload("t", "f16", 1, 64, H, B, 7, seed=42, state_std=0.3)
    inp = make_inputs(w)
    dev, td = torch.device("cuda", 0), TORCH_DTYPES["f16"]
    eng = Engine("f16", 1, B, 64, H, 7, device=dev)
    eng.set_weights(0, inp.w_ih[0].to(dev), inp.w_hh[0].to(dev), inp.b_ih[0].to(dev), inp.b_hh[0].to(dev))
    x, h0, c0, dy = (t.to(dev, td) for t in (inp.x, inp.h0, inp.c0, inp.dy))
    y, hn, cn = eng.forward(x, h0, c0)
    dx, dh0, dc0 = eng.backward(dy)
    want = [t.clone() for t in (y, hn, cn, dx, dh0, dc0)]

    def odd(t):  # the same values one element further on
        flat = torch.zeros(t.numel() + 1, dtype=t.dtype, device=dev)
        flat[1:] = t.flatten()
        return flat[1:].view(t.shape)

    y2, dy2 = odd(torch.zeros_like(y)), odd(dy)
    hn2, cn2, dx2 = torch.empty_like(hn), torch.empty_like(cn), torch.empty_like(dx)
    dh2, dc2 = torch.empty_like(dh0), torch.empty_like(dc0)
    for t0, t1 in ((0, 3), (3, 4), (4, 7)):
        eng.forward_range_into(7, t0, t1, x, h0, c0, y2, hn2, cn2)
    for t0, t1 in ((5, 7), (1, 5), (0, 1)):
        eng.backward_range_into(7, t0, t1, dy2, None, None, dx2, dh2, dc2)
    torch.cuda.synchronize()
    eng.close()
    for a, b in zip(want, (y2, hn2, cn2, dx2, dh2, dc2)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("cluster,B,H", SHAPES)
def test_the_shapes_above_run_on_clusters(cluster, B, H, monkeypatch):
    monkeypatch.setenv("FLSTM_CLUSTER_SIZE", str(cluster))
    eng = Engine("f16", 1, B, 64, H, 1, device=torch.device("cuda", 0))
    forward, backward = eng.recurrent_path(), eng.recurrent_path(backward=True)
    eng.close()
    assert forward[:2] == ("cluster", cluster)
    # the BPTT kernel has no form for 4 CTAs at H = 64
    assert backward[:2] == (("grid", 0) if (cluster, H) == (4, 64) else ("cluster", cluster))


@pytest.mark.parametrize("B,H,tiles,backward_tiles", [(2400, 64, 4, 0), (1250, 64, 2, 2), (600, 192, 2, 2), (600, 256, 4, 0), (300, 256, 2, 2),
                                                      (130, 320, 2, 2), (128, 512, 4, 0), (60, 512, 2, 2)])
def test_several_tiles_of_sequences_per_cluster(B, H, tiles, backward_tiles):
    """Batches at which the planner itself gives a cluster more than 8 or 16 sequences."""
    w = Workload("t", "bf16" if H % 128 else "f16", 1, 32, H, B, 3, seed=43, state_std=0.3)
    inp = make_inputs(w)
    got, eng = run_engine(w, inp, repeat=2)
    per_cluster = [eng.recurrent_path(b)[2] for b in (False, True)]
    eng.close()
    assert [(n + 7) // 8 if n <= 16 else 4 for n in per_cluster] == [tiles, backward_tiles]
    assert_parity(got, run_oracle(inp), w.dtype)
