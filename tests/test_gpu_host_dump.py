"""Dumps stored straight into page-locked host memory, in every order, output
type and buffer type: sizes on both sides of the 512 KB where the wide-store
kernel takes over (with channels whose words do not fill its last block), and
outputs 16-byte and only 8-byte aligned.  A pageable output is formatted in
device memory and copied.  Words outside the dump stay as they were; the slots
of register-tile order that hold no baseline come out zero."""
import ctypes

import numpy as np
import pytest

from test_gpu_parity import expected_words

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine,compute", [("tensor", "int8"), ("plain", "fp32")])
@pytest.mark.parametrize("order", ["tri", "ri", "rt"])
@pytest.mark.parametrize("n,f", [(16, 1), (48, 13), (48, 14), (80, 7), (144, 3), (176, 2)])
@pytest.mark.parametrize("where", ["pinned", "pinned + 8 bytes", "pageable"])
def test_dump_into_host_memory(xg, oracle_mod, engine, compute, order, n, f, where):
    import torch
    t = 32
    x = oracle_mod.gaussian_input(n, f, t, seed=n + f, sigma=30.0)
    exact = oracle_mod.xengine_i64(x, n, f, t)
    for output in ("int32", "float32"):
        want = expected_words(oracle_mod, exact, n, f, order, output).view(np.uint32)
        buf = torch.full((want.size + 8,), -7, dtype=torch.int32, pin_memory=where != "pageable")
        skip = 1 if where == "pinned + 8 bytes" else 2        # Complex before the output
        with xg.Correlator(n, f, t, ntimepipe=16, engine=engine, compute=compute, output=output,
                           order=order, flags=xg.XGPU_DONT_REGISTER_MATRIX) as c:
            c.set_input(x)
            c.ctx.matrix_h, c.ctx.matrix_len = buf.data_ptr(), buf.numel() // 2
            xg.check("output", xg.lib().xgpuSetHostOutputBuffer(ctypes.byref(c.ctx)))
            c.ctx.output_offset = skip
            c.run(xg.SYNCOP_DUMP)
        got = buf.numpy().view(np.uint32)
        assert np.array_equal(got[2 * skip: 2 * skip + want.size], want)
        rest = np.delete(got, np.s_[2 * skip: 2 * skip + want.size])
        assert (rest == np.uint32(2**32 - 7)).all()
