"""Batches of more rows, and networks of more inputs, than 65,535 tiles of 32."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in,rows", [(8, 65536 * 32 + 8), (65536 * 32 + 8, 8)])
def test_forward(pkg, n_in, rows):
    import mlp_oracle as mo
    rng = np.random.default_rng(3)
    x = rng.standard_normal((rows, n_in), dtype=np.float32)
    params = mo.init_params(n_in, 8, 8, seed=4)
    with pkg.mlp.Mlp(n_in, 8, 8, max_batch=rows) as net:
        net.set_params(params)
        y = net.forward(x)
    check = np.r_[0:16, rows - 16:rows] if rows > 32 else np.arange(rows)
    y_ref = mo.forward(params, x[check], n_in, 8, 8)[3]
    assert np.max(np.abs(y[check] - y_ref)) <= 1e-2 * np.max(np.abs(y_ref))
