"""The warm-start GEMM at the edges of its tiling (tile widths 16 to 128, ring
refills, K tails, rows of C that 16-byte stores cannot reach) and the
evaluation at row counts around its tiles and its workspace."""
import os
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "oracle"))


# tile width: 16 (few tiles), 32, 64, 128 (148 tiles and more); K beyond the
# ring's 8 (6 at width 128) chunks of 64, with and without a tail
@pytest.mark.parametrize("m,n,k", [(128, 48, 16), (256, 256, 528), (128, 16, 1040), (1280, 512, 64), (2560, 512, 128),
                                   (5120, 512, 464), (4736, 128, 512)])
@pytest.mark.parametrize("pad", [0, 1])
def test_gemm_tiles(m, n, k, pad):
    import torch
    from ekpnp.mlp import gemm_bf16
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda", generator=g).to(torch.bfloat16)
    b = torch.randn(n, k, device="cuda", generator=g).to(torch.bfloat16)
    c = torch.full((m, n + pad), float("nan"), device="cuda")
    gemm_bf16(a, b, c[:, :n])
    ref = a.double() @ b.double().T
    # FP32 accumulation of k products of magnitude ~1 (the bar of test_gemm_matches_torch)
    assert (c[:, :n].double() - ref).abs().max().item() <= 2e-6 * k
    if pad:
        assert bool(torch.isnan(c[:, n:]).all())


@pytest.mark.parametrize("rows", [1, 127, 128, 129, 1000, 8193])
def test_forward_rows(rows):
    import ekpnp.mlp as em
    import mlp_oracle as mo
    x = np.random.default_rng(rows).uniform(-1, 1, (rows, 4)).astype(np.float32)
    with em.Mlp(batch=128, seed=9) as net:
        small = net.forward(x[:1])
        y = net.forward(x)   # grows the workspace
        again = net.forward(x[:1])
        p = net.params
    ref, _ = mo.forward(p.astype(np.float64), x.astype(np.float64))
    # the bar of test_forward_and_gradients_match_oracle
    assert np.linalg.norm(y - ref) < 5e-3 * np.linalg.norm(ref)
    assert np.array_equal(small, again)


# the weight gradients run beside the deltas: whatever the overlap, gradients
# asked for again (outside a graph) and a training run started again (a graph)
# give the same bits, apart from the loss (summed by atomics)
@pytest.mark.parametrize("batch", [128, 256, 1024])
def test_gradient_streams_repeat(batch):
    import ekpnp.mlp as em
    import mlp_oracle as mo
    r = np.random.default_rng(batch)
    x = r.uniform(-1, 1, (batch, 4)).astype(np.float32)
    t = r.standard_normal((batch, 512)).astype(np.float32)
    runs = []
    for _ in range(2):
        with em.Mlp(batch=batch, seed=11) as net:
            p = net.params
            grads = [net.gradients(x, t)[0] for _ in range(4)]
            net.set_data(x, t)
            net.train(40, 1e-3)
            runs.append((grads, net.params))
    first = runs[0][0][0]
    for grads, _ in runs:
        assert all(np.array_equal(g, first) for g in grads)
    assert np.array_equal(runs[0][1], runs[1][1])
    _, ref = mo.loss_and_gradients(p.astype(np.float64), x.astype(np.float64), t.astype(np.float64))
    # the bar of test_forward_and_gradients_match_oracle
    for ws, _, bs in em.layer_slices():
        for part in (ws, bs):
            assert np.linalg.norm(first[part] - ref[part]) < 2e-2 * np.linalg.norm(ref[part])
