"""The A-Trous passes are launched as programmatic dependents, so the grids of several passes are
alive together and buffers are rewritten and read again two passes later.  Calls put on one stream
one after another, without a wait between them and with other inputs each, must give what each gives
alone, bit for bit: from images whose passes all fit on the chip at once to images of many waves."""
import numpy as np
import pytest

from test_zz_no_alloc import bind, make_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w,levels", [(9, 33, 16), (40, 54, 6), (333, 257, 5), (700, 900, 8)])
def test_calls_in_a_row_equal_calls_alone(rg, h, w, levels):
    torch = pytest.importorskip("torch")
    f = bind(rg.load_library())
    sets = [make_inputs(100 * k + h, h, w) for k in range(3)]
    stream = torch.cuda.Stream()
    want, calls = [], []
    for inputs in sets:
        rgba = np.concatenate([inputs[0], np.ones((h, w, 1), np.float32)], axis=2)
        bufs = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (rgba,) + inputs[1:]]
        out = torch.zeros((h, w, 4), device="cuda")
        torch.cuda.synchronize()
        call = [w, h, *[b.data_ptr() for b in bufs], levels, 0.4, 128.0, 0.1, 1.0]
        assert f(*call, out.data_ptr(), stream.cuda_stream) == 0
        torch.cuda.synchronize()
        want.append(out.clone())
        calls.append((call, bufs))
    outs = [torch.zeros((h, w, 4), device="cuda") for _ in range(30)]
    torch.cuda.synchronize()
    for k, out in enumerate(outs):
        assert f(*calls[k % 3][0], out.data_ptr(), stream.cuda_stream) == 0
    torch.cuda.synchronize()
    for k, out in enumerate(outs):
        assert torch.equal(out, want[k % 3]), k
