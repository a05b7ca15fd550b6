"""Calls over device input recorded into a CUDA graph: on the context's own stream,
whose handle the program took, and on another stream of the thread while the context
calls go to its own.  The settings that a call chooses by asking whether the stream is
idle must neither end the capture nor change sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def buffers(oracle_mod, fmt, n, f, t):
    import torch
    xs, sums = [], []
    for q in range(3):
        if fmt == "packed4":
            x = oracle_mod.generate(t * f * n * 2, 1, 30 + q)
            sums.append(oracle_mod.xengine_i64(oracle_mod.unpack4(x), n, f, t))
        else:
            x = oracle_mod.gaussian_input(n, f, t, seed=30 + q, sigma=30.0)
            sums.append(oracle_mod.xengine_i64(x, n, f, t))
        xs.append(torch.from_numpy(np.ascontiguousarray(x).view(np.int8)).cuda())
    torch.cuda.synchronize()
    return xs, sums


# long packed calls ask whether the stream is idle (32,256 stages); so do chains of
# untuned calls of the second shape
@pytest.mark.parametrize("fmt,n,f,t", [("packed4", 400, 9, 16384), ("int8", 256, 10, 1024)])
def test_calls_on_a_captured_own_stream(xg, oracle_mod, fmt, n, f, t):
    import torch
    xs, sums = buffers(oracle_mod, fmt, n, f, t)
    with xg.Correlator(n, f, t, ntimepipe=16, input_format=fmt, flags=xg.XGPU_DONT_REGISTER) as c:
        stream = torch.cuda.ExternalStream(c.stream)
        for x in xs:      # maps and kernels in place
            c.run_device(x.data_ptr())
        torch.cuda.synchronize()
        c.clear()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            for x in xs:
                c.run_device(x.data_ptr())
        for _ in range(2):     # the first recorded call stores: each replay starts anew
            g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(c.dump_int64(), sum(sums))


@pytest.mark.parametrize("fmt,n,f,t", [("packed4", 400, 9, 16384), ("int8", 256, 10, 1024)])
def test_calls_while_another_stream_is_captured(xg, oracle_mod, fmt, n, f, t):
    import torch
    xs, sums = buffers(oracle_mod, fmt, n, f, t)
    y = torch.zeros(1024, device="cuda")
    with xg.Correlator(n, f, t, ntimepipe=16, input_format=fmt, flags=xg.XGPU_DONT_REGISTER) as c:
        for x in xs:
            c.run_device(x.data_ptr())
        torch.cuda.synchronize()
        c.clear()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            y += 1
            for x in xs:
                c.run_device(x.data_ptr())
            y += 1
        assert np.array_equal(c.dump_int64(), sum(sums))
        g.replay()
        torch.cuda.synchronize()
        assert float(y[0]) == 2.0
