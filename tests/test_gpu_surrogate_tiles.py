"""The surrogate's products at the edges of their tiles: one row and one more than
a row tile, a batch deeper than one staged round of the weight gradients, every
padded layer width, forward passes of one and several chunks.  The oracle and its
bound are those of test_gpu_surrogate.py (one BF16 ulp, norm-relative)."""
import numpy as np
import pytest

from test_gpu_surrogate import REL_TOL, _padded_x, _rel, mlp_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,batch,max_batch", [((3, 5, 7, 2), 1, 64), ((64, 256, 256, 64), 129, 200),
                                                   ((65, 130, 200, 100), 300, 300), ((256, 64, 192, 256), 513, 600),
                                                   ((16, 128, 64, 50), 33, 40)])
def test_tile_edges_match_oracle(sizes, batch, max_batch):
    from cerebellum_simulation_b200.surrogate import MLP
    rng = np.random.Generator(np.random.PCG64(batch))
    n_in, h1, h2, n_out = sizes
    net = MLP(*sizes, max_batch=max_batch, seed=5)
    p = net.get_params()
    W1, b1, W2, b2, W3, b3 = net.unpack(p)
    b1[:h1] = rng.normal(0, 0.1, h1); b2[:h2] = rng.normal(0, 0.1, h2); b3[:n_out] = rng.normal(0, 0.1, n_out)
    net.set_params(p)
    params = net.unpack(net.get_params())
    I, _, _, O = net.padded
    x = rng.normal(0, 1, (2 * max_batch + 3, n_in)).astype(np.float32)
    t = rng.normal(0, 1, (batch, n_out)).astype(np.float32)
    y_ref = mlp_oracle.forward(params, _padded_x(x, I))[3][:, :n_out]
    for rows in (1, batch, x.shape[0]):
        assert _rel(net.forward(x[:rows]), y_ref[:rows]) < REL_TOL, rows
    g, loss = net.gradients(x[:batch], t)
    t_pad = np.zeros((batch, O))
    t_pad[:, :n_out] = t
    g_ref, loss_ref = mlp_oracle.gradients(params, _padded_x(x[:batch], I), t_pad, n_out)
    assert abs(loss - loss_ref) / loss_ref < REL_TOL
    for name, a, b in zip(["W1", "b1", "W2", "b2", "W3", "b3"], net.unpack(g), g_ref):
        assert _rel(a, b) < REL_TOL, name
        a[tuple(slice(0, k) for k in {"W1": (h1, n_in), "b1": (h1,), "W2": (h2, h1), "b2": (h2,),
                                      "W3": (n_out, h2), "b3": (n_out,)}[name])] = 0
        assert not a.any(), name  # the padding's gradients
