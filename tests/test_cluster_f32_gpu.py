"""The cluster-resident fp32 recurrent kernels (simt_cluster.cu) against the oracle: widths that are no multiple of 4, 32 or
64, partly filled blocks of four sequences, CTAs without units, weights partly in shared memory, step ranges."""
import pytest
import torch

from flashlstm_poc_b200.engine import Engine
from flashlstm_poc_b200.workloads import Workload, make_inputs
from tests.gpu_helpers import assert_parity, run_engine, run_oracle

pytestmark = pytest.mark.gpu

# CTAs per cluster (0: the planner's choice), layers, batch, input size, hidden size
SHAPES = [(0, 1, 1, 3, 5), (1, 1, 2, 8, 30), (2, 1, 150, 16, 62), (4, 2, 9, 24, 71), (0, 1, 37, 40, 130), (8, 1, 32, 64, 256),
          (16, 1, 33, 64, 256), (0, 1, 100, 16, 200), (16, 1, 6, 32, 333), (16, 2, 20, 16, 509), (0, 1, 64, 8, 512)]


@pytest.mark.parametrize("cluster,L,B,I,H", SHAPES)
def test_f32_cluster_kernels_match_the_oracle(cluster, L, B, I, H, monkeypatch):
    if cluster:
        monkeypatch.setenv("FLSTM_CLUSTER_SIZE", str(cluster))
    w = Workload("t", "f32", L, I, H, B, 6, seed=71, state_std=0.3)
    inp = make_inputs(w)
    gen = torch.Generator().manual_seed(6)
    dhn, dcn = torch.randn(L, B, H, generator=gen), torch.randn(L, B, H, generator=gen)
    got, eng = run_engine(w, inp, dhn=dhn, dcn=dcn, repeat=2)
    eng.close()
    # fp32 sums of at most 4 * 509 terms of order 1/sqrt(H) and 600-term weight gradients: errors of order 1e-5
    assert_parity(got, run_oracle(inp, dhn=dhn, dcn=dcn), "f32", fp32_max_abs=1e-4)


@pytest.mark.parametrize("B,H", [(5, 36), (32, 256)])
def test_f32_ranges_equal_one_call(B, H):
    T = 9
    w = Workload("t", "f32", 1, 16, H, B, T, seed=72, state_std=0.3)
    inp = make_inputs(w)
    dev = torch.device("cuda", 0)
    eng = Engine("f32", 1, B, 16, H, T, device=dev)
    eng.set_weights(0, inp.w_ih[0].to(dev), inp.w_hh[0].to(dev), inp.b_ih[0].to(dev), inp.b_hh[0].to(dev))
    x, h0, c0, dy = (t.to(dev) for t in (inp.x, inp.h0, inp.c0, inp.dy))
    y, hn, cn = eng.forward(x, h0, c0)
    dx, dh0, dc0 = eng.backward(dy)
    want = [t.clone() for t in (y, hn, cn, dx, dh0, dc0, *eng.grads(0))]
    out = [torch.zeros_like(t) for t in (y, hn, cn, dx, dh0, dc0)]
    for t0, t1 in ((0, 1), (1, 6), (6, 9)):
        eng.forward_range_into(T, t0, t1, x, h0, c0, out[0], out[1], out[2])
    for t0, t1 in ((8, 9), (3, 8), (0, 3)):
        eng.backward_range_into(T, t0, t1, dy, None, None, out[3], out[4], out[5])
    torch.cuda.synchronize()
    for a, b in zip(want, (*out, *eng.grads(0))):
        assert torch.equal(a, b)
    eng.close()


@pytest.mark.parametrize("cluster,L,B,I,H", SHAPES)
def test_the_shapes_above_run_on_clusters(cluster, L, B, I, H, monkeypatch):
    if cluster:
        monkeypatch.setenv("FLSTM_CLUSTER_SIZE", str(cluster))
    eng = Engine("f32", L, B, I, H, 1, device=torch.device("cuda", 0))
    paths = [eng.recurrent_path(b) for b in (False, True)]
    eng.close()
    assert all(p[0] == "cluster" and p[1] == (cluster or p[1]) for p in paths)


@pytest.mark.parametrize("L,B,I,H,path", [(1, 8, 24, 520, "grid"), (2, 5, 16, 800, "grid"), (1, 40, 16, 700, "steps"), (1, 3, 16, 1100, "steps"),
                                          (1, 9, 8, 256, "grid-small"), (1, 300, 8, 200, "steps-small")])
def test_f32_beyond_the_clusters(L, B, I, H, path, monkeypatch):
    """The kernels of fp32 layers wider than 512: one grid-wide launch while its CTAs fit the machine at once, else a launch per
    step; small widths reach them with the clusters switched off."""
    path, _, small = path.partition("-")
    if small:
        monkeypatch.setenv("FLSTM_CLUSTER", "0")
    w = Workload("t", "f32", L, I, H, B, 5, seed=73, state_std=0.3)
    inp = make_inputs(w)
    gen = torch.Generator().manual_seed(7)
    dhn, dcn = torch.randn(L, B, H, generator=gen), torch.randn(L, B, H, generator=gen)
    got, eng = run_engine(w, inp, dhn=dhn, dcn=dcn, repeat=2)
    paths = [eng.recurrent_path(b)[0] for b in (False, True)]
    eng.close()
    assert paths == [path, path]
    # fp32 sums of up to 4400 terms of order 1/sqrt(H) and 1500-term weight gradients: errors of order 1e-5
    assert_parity(got, run_oracle(inp, dhn=dhn, dcn=dcn), "f32", fp32_max_abs=1e-4)
