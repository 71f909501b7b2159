"""Backward pass of the band network at the edges of its row splits and tiles
(one row, a tile of 64 and one more, a split of 256 rows and two, the most
splits, more rows than partial sums), and with features that start off a
16-byte boundary, against the float64 CPU reference.  The tolerance is that of
bf16 operands: 2e-2 of each parameter block's norm."""
import numpy as np
import pytest

import bandnet
import bandnet_ref as REF
import mvg

pytestmark = pytest.mark.gpu

SIZES = [256 * 528, 256, 256 * 256, 256, 256 * 256, 256, 2 * 256, 2]


@pytest.fixture(scope="module")
def net():
    import build as pkg_build
    pkg_build.build()
    c = mvg.Context(0)
    yield bandnet.BandNet(c, seed=4)
    c.close()


@pytest.mark.parametrize("n,offset", [(1, 0), (15, 0), (64, 0), (65, 1), (511, 0), (512, 8), (513, 4), (4100, 0),
                                      (9000, 0), (9000, 2)])
def test_gradients_at_tile_edges(net, n, offset):
    import torch
    rng = np.random.default_rng(n)
    x = np.zeros((n, bandnet.N_IN), np.float32)
    x[:, :512] = rng.poisson(1.0, (n, 512))
    x[:, 512:514] = rng.uniform(0.5, 2.0, (n, 2))
    buf = torch.zeros(offset + n * bandnet.N_IN, dtype=torch.bfloat16, device="cuda")
    X = buf[offset:]
    X.copy_(torch.from_numpy(x).cuda().reshape(-1))
    T = rng.normal(0, 1, (n, 2)).astype(np.float32)
    T_dev = torch.from_numpy(T).cuda()
    g, loss = net.grad_dev(X.data_ptr(), T_dev.data_ptr(), n)
    rloss, rg = REF.loss_and_grads(net.get_params(), X.float().cpu().numpy().astype(np.float64).reshape(n, -1),
                                   T.astype(np.float64))
    assert abs(loss - rloss) <= 2e-2 * abs(rloss) + 1e-6
    off = 0
    for s in SIZES:
        a, b = g[off:off + s], rg[off:off + s]
        assert np.linalg.norm(a - b) <= 2e-2 * np.linalg.norm(b) + 1e-7, (off, s)
        off += s
