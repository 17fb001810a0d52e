"""Weight gradients of large batches: more pixels than 256 chunks of 512 (longer chunks), a
last chunk that is not full, rows that are no multiple of the staging step.  The loss is a mean
over pixels, so the gradient of 64 images is the mean of their gradients; the factor 64 is a
power of two, which the BF16 gradients carry exactly, so only the order of the FP32 sums
differs (1e-5 of the gradient's norm)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w", [(48, 48), (37, 50), (9, 130)])
def test_batch_gradient_is_the_mean_of_image_gradients(rg, h, w):
    n = 64
    rng = np.random.default_rng(h * w)
    noisy = np.concatenate([rng.exponential(0.5, (n, h, w, 3)), np.ones((n, h, w, 1))], -1).astype(np.float32)
    normal, albedo = (rng.random((n, h, w, 3)).astype(np.float32) for _ in range(2))
    depth = rng.random((n, h, w)).astype(np.float32)
    ref = np.concatenate([rng.random((n, h, w, 3)), np.ones((n, h, w, 1))], -1).astype(np.float32)
    d = rg.Denoiser(seed=3)
    loss, grad = d.gradients(noisy, normal, albedo, depth, ref)
    one = [d.gradients(*(a[k:k + 1] for a in (noisy, normal, albedo, depth, ref))) for k in range(n)]
    mean = np.mean([g.astype(np.float64) for _, g in one], axis=0)
    assert abs(loss - np.mean([l for l, _ in one])) < 1e-5 * abs(loss)
    assert np.linalg.norm(grad - mean) < 1e-5 * np.linalg.norm(mean)
    d.close()
