"""Register-tile dumps on both sides of the 3 MB from which an output that is not
16-byte aligned is formatted in device memory and copied."""
import ctypes

import numpy as np
import pytest

from test_gpu_parity import expected_words

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,f", [(176, 6), (176, 7), (256, 10)])   # 2.9, 3.3 and 10.1 MB
@pytest.mark.parametrize("skip", [0, 1, 2, 3])
def test_register_tile_dump(xg, oracle_mod, n, f, skip):
    import torch
    t = 32
    x = oracle_mod.gaussian_input(n, f, t, seed=n + f, sigma=30.0)
    want = expected_words(oracle_mod, oracle_mod.xengine_i64(x, n, f, t), n, f, "rt", "int32")
    want = want.view(np.uint32)
    buf = torch.full((want.size + 8,), -7, dtype=torch.int32, pin_memory=True)
    with xg.Correlator(n, f, t, ntimepipe=16, order="rt", flags=xg.XGPU_DONT_REGISTER_MATRIX) as c:
        c.set_input(x)
        c.ctx.matrix_h, c.ctx.matrix_len = buf.data_ptr(), buf.numel() // 2
        xg.check("output", xg.lib().xgpuSetHostOutputBuffer(ctypes.byref(c.ctx)))
        c.ctx.output_offset = skip
        c.run(xg.SYNCOP_DUMP)
    got = buf.numpy().view(np.uint32)
    assert np.array_equal(got[2 * skip: 2 * skip + want.size], want)
    rest = np.delete(got, np.s_[2 * skip: 2 * skip + want.size])
    assert (rest == np.uint32(2**32 - 7)).all()
