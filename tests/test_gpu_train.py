"""The training kernels against the FP64 statement of the network, at batches that leave rows of a tile, chunks of the
weight gradients' runs and CTAs over: less than a tile, a tile, one row group more, a run more, and more tiles
than the GPU has SMs; and with the inputs off their 16-byte boundary."""
import numpy as np
import pytest

import ntg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("batch,offset", [(8, 0), (128, 0), (136, 1), (264, 0), (19584, 0)])
def test_gradients_match_oracle(batch, offset):
    import mlp_oracle
    rng = np.random.default_rng(batch)
    x = rng.random((batch, 48)).astype(np.float32)
    t = rng.random((batch, 8)).astype(np.float32)
    net = ntg.MLP(seed=batch)
    try:
        buf = torch.zeros(batch * 48 + 4, dtype=torch.float32, device="cuda")
        dx = buf[offset:offset + batch * 48].reshape(batch, 48)
        dx.copy_(torch.from_numpy(x))
        g, loss = net.gradients(dx, torch.from_numpy(t).cuda())
        g = g.cpu().numpy().astype(np.float64)
        ref, ref_loss = mlp_oracle.gradients(net.get_params(), x, t)
        assert abs(loss - ref_loss) <= 1e-3 * ref_loss
        offs = np.cumsum([0, 256 * 48, 256, 256 * 256, 256, 8 * 256, 8])
        for a, b in zip(offs[:-1], offs[1:]):  # the bound of the oracle test at other batches
            assert np.linalg.norm(g[a:b] - ref[a:b]) < 2e-2 * np.linalg.norm(ref[a:b]), (a, b)
    finally:
        net.close()


@pytest.mark.parametrize("batch", [1, 5, 129, 257])
def test_batches_are_multiples_of_eight(batch):
    """Other batches are refused, as they always were, and leave the network as it was."""
    net = ntg.MLP(seed=3)
    try:
        x, t = torch.rand((batch, 48), device="cuda"), torch.rand((batch, 8), device="cuda")
        before = net.get_params()
        for call in (net.gradients, net.train_step):
            with pytest.raises(ntg.NtgError) as e:
                call(x, t)
            assert e.value.code == ntg.NTG_ERROR_INVALID_INPUT
        assert np.array_equal(net.get_params(), before)
    finally:
        net.close()
