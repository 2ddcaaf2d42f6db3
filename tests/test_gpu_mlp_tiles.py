"""The network's GEMM at each tile width (mlp.cu gemm) with more slices than a
tile keeps in shared memory, and its gradients at ragged sizes: odd tiles of
the transposed outputs, of the column sums and of the loss's parts. The bounds
are test_gpu_mlp.py's: FP32 accumulation, and the oracle's BF16 roundings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(129, 33, 520), (1300, 500, 776), (2600, 700, 600), (2600, 700, 8)])
def test_gemm_at_each_tile_width(pkg, m, n, k):
    rng = np.random.default_rng(m + n + k)
    a = rng.standard_normal((m, k)).astype(np.float32)
    b = rng.standard_normal((n, k)).astype(np.float32)
    import torch
    ab = torch.from_numpy(a).to(torch.bfloat16).to(torch.float64)
    bb = torch.from_numpy(b).to(torch.bfloat16).to(torch.float64)
    scale = (ab.abs() @ bb.abs().T).numpy()
    assert np.all(np.abs(pkg.mlp.gemm_bf16(a, b) - (ab @ bb.T).numpy()) <= 1e-4 * scale + 1e-6)


@pytest.mark.parametrize("n_in,hidden,n_out", [(8, 24, 40), (72, 136, 1000)])
@pytest.mark.parametrize("rows", [8, 136, 264, 512])
def test_gradients_at_ragged_sizes(pkg, n_in, hidden, n_out, rows):
    import mlp_oracle as mo
    rng = np.random.default_rng(rows)
    x = rng.standard_normal((rows, n_in)).astype(np.float32)
    t = rng.standard_normal((rows, n_out)).astype(np.float32)
    params = mo.init_params(n_in, hidden, n_out, seed=2)
    with pkg.mlp.Mlp(n_in, hidden, n_out) as net:
        net.set_params(params)
        g, loss = net.gradients(x, t)
        # a step on the same rows in another order: the targets follow the inputs
        first = net.train(x, t, epochs=1, batch=rows, lr=1e-9)
    g_ref, loss_ref = mo.gradients(params, x, t, n_in, hidden, n_out)
    assert abs(loss - loss_ref) <= 1e-4 * loss_ref
    assert abs(first[0] - loss_ref) <= 1e-4 * loss_ref
    o = 0
    for s in (hidden * n_in, hidden, hidden * hidden, hidden, n_out * hidden, n_out):
        a, b = g[o:o + s].astype(np.float64), g_ref[o:o + s]
        o += s
        assert np.max(np.abs(a - b)) <= 1e-2 * np.max(np.abs(b))
