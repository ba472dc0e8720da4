"""The persistent convolution kernel over batch sizes: fewer bands than CTAs, as many, one more round for
some CTAs, and several rounds (16 bands of 4 rows per image, two CTAs on each of 148 SMs).  An image's
output does not depend on its batch, bit for bit, and the single image is checked against the float64
oracle (bf16 activations: 1e-2 relative L2, the bar of the network's other forward test)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [1, 2, 18, 19, 56])
def test_forward_batches(n):
    from oracle import cnn_oracle
    from summationbyparts_b200.learned import CorrectionNet
    g = torch.Generator(device="cuda").manual_seed(n)
    coarse = torch.rand((n, 4, 64, 64), dtype=torch.float64, device="cuda", generator=g) * 2.0 - 1.0
    net = CorrectionNet(max_batch=n, seed=3)
    rng = np.random.default_rng(7)
    p = net.params()
    net.set_params((p + 0.05 * rng.standard_normal(p.size) * (p != 0)).astype(np.float32))
    mean, scale = [0.1, -0.2, 0.0, 0.3], [0.7, 0.6, 0.8, 0.5]
    net.set_normalisation(mean, scale, [1.0, 2.0, 0.5, 1.5])
    y = net.output(coarse).cpu().numpy()
    single = CorrectionNet(max_batch=1, seed=3)
    single.set_params(net.params())
    single.set_normalisation(mean, scale, [1.0, 2.0, 0.5, 1.5])
    for k in {0, n // 2, n - 1}:
        assert single.output(coarse[k:k + 1].contiguous()).cpu().numpy()[0].tobytes() == y[k].tobytes(), k
    ref, _, _ = cnn_oracle.forward(net.params(), coarse[n - 1:].cpu().numpy(), mean, scale)
    out = y[n - 1].reshape(64, 64, 8)[..., :4]
    assert np.linalg.norm(out - ref[0, ..., :4]) <= 1e-2 * np.linalg.norm(ref[0, ..., :4])
    # the apply pass: coarse + y * out_scale from the same kernel's epilogue
    corrected = net.apply(coarse)
    want = coarse.cpu().numpy() + y[..., :4].reshape(n, 64, 64, 4).transpose(0, 3, 1, 2).astype(np.float64) * \
        np.array([1.0, 2.0, 0.5, 1.5])[:, None, None]
    assert np.array_equal(corrected.cpu().numpy(), want)
    net.close()
    single.close()
