"""The network's GEMMs share an SM's 512 TMEM columns with the launch after
them, which starts early (mlp.cu k_gemm_tn, pass.cuh)."""
import os
import re

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_the_next_launch_starts_after_the_columns_are_held():
    # a CTA of the next launch holds its columns until this grid is done, so no
    # CTA of this grid may still be waiting for columns then
    with open(os.path.join(ROOT, "sovereign-solver_b200", "csrc", "mlp.cu")) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    kernel = src[src.index("k_gemm_tn("):]
    order = [kernel.index(s) for s in ("tmem_alloc(", "__syncthreads()", "pass_begin()", "pass_wait()")]
    assert order == sorted(order)


@pytest.mark.gpu
def test_many_wide_tiles_of_one_slice(pkg):
    # 157 tiles of 128 columns with one slice each (32 KB of shared memory):
    # the form of which most CTAs would fit an SM
    import mlp_oracle as mo
    rows, d = 20000, 64
    rng = np.random.default_rng(5)
    x = rng.standard_normal((rows, d)).astype(np.float32)
    t = rng.standard_normal((rows, d)).astype(np.float32)
    params = mo.init_params(d, d, d, seed=6)
    with pkg.mlp.Mlp(d, d, d, max_batch=rows) as net:
        net.set_params(params)
        g, loss = net.gradients(x, t)
    g_ref, loss_ref = mo.gradients(params, x, t, d, d, d)
    assert abs(loss - loss_ref) <= 1e-4 * loss_ref
    o = 0
    for s in (d * d, d) * 3:
        a, b = g[o:o + s].astype(np.float64), g_ref[o:o + s]
        o += s
        assert np.max(np.abs(a - b)) <= 1e-2 * np.max(np.abs(b))
