"""The A-Trous kernels at the edges of their launch shapes: images narrower than a thread
block, heights that leave a thread's second row outside, steps larger than the image, one and
two pixels a thread (from 148 * 1024 pixels), all against the CPU oracle with the tolerance of
the parity test (1e-4 relative: float sums of 25 weights in another order of exponents); and
the no-allocation entry point captured into a CUDA graph."""
import numpy as np
import pytest

from test_zz_no_alloc import bind, make_inputs, run_noalloc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w,levels", [(1, 1, 1), (3, 31, 5), (33, 5, 7), (64, 97, 3), (296, 512, 5), (295, 512, 5),
                                        (607, 257, 6), (131, 1157, 9)])
def test_sizes_match_oracle(rg, orc, h, w, levels):
    inputs = make_inputs(h * 1000 + w, h, w)
    got = rg.denoise_atrous(*inputs, levels=levels)
    np.testing.assert_allclose(got, orc.denoise(*inputs, levels=levels), rtol=1e-4, atol=1e-6)


def test_zero_normal_exponent(rg, orc):
    """Exponent 0: every normal weight is 1, also of opposite normals."""
    color, normal, depth, albedo, alpha = make_inputs(5, 40, 70)
    normal[::3] = 1.0 - normal[::3]
    got = rg.denoise_atrous(color, normal, depth, albedo, alpha, levels=3, sigma_normal=0.0)
    ref = orc.denoise(color, normal, depth, albedo, alpha, levels=3, sigma_normal=0.0)
    np.testing.assert_allclose(got, ref, rtol=1e-4, atol=1e-6)


def test_captured_call_equals_direct_call(rg):
    torch = pytest.importorskip("torch")
    f = bind(rg.load_library())
    inputs = make_inputs(9, 90, 130)
    rc, want = run_noalloc(f, torch, inputs, torch.cuda.Stream().cuda_stream)
    assert rc == 0
    rgba = np.concatenate([inputs[0], np.ones(inputs[0].shape[:2] + (1,), np.float32)], axis=2)
    bufs = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (rgba,) + inputs[1:]]
    out = torch.zeros((90, 130, 4), device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        assert f(130, 90, *[b.data_ptr() for b in bufs], 5, 0.4, 128.0, 0.1, 1.0, out.data_ptr(),
                 torch.cuda.current_stream().cuda_stream) == 0
    for _ in range(2):
        out.fill_(7.0)
        g.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(out.cpu().numpy(), want)
