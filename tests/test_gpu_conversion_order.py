"""Conversions beside engine launches where the order rests on the launch before
the last one: calls of several launches (more than 32768 samples), whose later
launches let the next conversion start at once, and calls over host and device
input in turn, which share the two conversion buffers.  Every call's input
differs; sums are bit-exact."""
import numpy as np
import pytest

from test_gpu_conversions import encode

pytestmark = pytest.mark.gpu


def inputs(oracle_mod, fmt, n, f, t, count, seed):
    import torch
    host, dev, sums = [], [], []
    for q in range(count):
        b, x = encode(oracle_mod, fmt, n, f, t, seed + q)
        host.append(np.ascontiguousarray(b).view(np.int8))
        dev.append(torch.from_numpy(host[-1]).cuda())
        sums.append(oracle_mod.xengine_i64(x, n, f, t))
    torch.cuda.synchronize()
    return host, dev, sums


@pytest.mark.parametrize("fmt", ["packed4", "dp4a_swizzled", "block32"])
@pytest.mark.parametrize("engine,grid", [("tensor", 0), ("tensor", 4), ("plain", 0)])
def test_calls_of_several_launches(xg, oracle_mod, fmt, engine, grid):
    n, f, t = 32, 2, 65536 + 256
    host, dev, sums = inputs(oracle_mod, fmt, n, f, t, 4, 300)
    with xg.Correlator(n, f, t, ntimepipe=16, engine=engine, input_format=fmt) as c:
        if engine == "tensor":
            c.tune(1, grid, 0)
        for _ in range(2):
            for d in dev:
                c.run_device(d.data_ptr())
        assert np.array_equal(c.dump_int64(), 2 * sum(sums))


@pytest.mark.parametrize("fmt", ["packed4", "dp4a_swizzled", "block32"])
@pytest.mark.parametrize("engine", ["tensor", "plain"])
@pytest.mark.parametrize("sync", ["SYNCOP_NONE", "SYNCOP_SYNC_TRANSFER"])
def test_host_and_device_calls_in_turn(xg, oracle_mod, fmt, engine, sync):
    n, f, t = 96, 3, 1024
    host, dev, sums = inputs(oracle_mod, fmt, n, f, t, 5, 400)
    with xg.Correlator(n, f, t, ntimepipe=16, engine=engine, input_format=fmt) as c:
        want = np.zeros_like(sums[0])
        for q in range(15):
            if q % 3 == 1:
                # the host buffer may be refilled once the transfer before is done
                c.set_input(host[q % 5])
                c.run(getattr(xg, sync))
                if sync == "SYNCOP_NONE":
                    c.run_device(dev[(q + 1) % 5].data_ptr(), xg.SYNCOP_SYNC_TRANSFER)
                    want += sums[(q + 1) % 5]
            else:
                c.run_device(dev[q % 5].data_ptr())
            want += sums[q % 5]
        assert np.array_equal(c.dump_int64(), want)


@pytest.mark.parametrize("compute", ["int8", "fp32"])
@pytest.mark.parametrize("fmt", ["packed4", "dp4a_swizzled", "block32"])
def test_plain_grids_that_fill_the_gpu(xg, oracle_mod, fmt, compute):
    """648 blocks: their launches come at the conversion's start."""
    n, f, t = 256, 9, 128
    host, dev, sums = inputs(oracle_mod, fmt, n, f, t, 4, 500)
    out = "int32" if compute == "int8" else "float32"
    with xg.Correlator(n, f, t, ntimepipe=16, engine="plain", compute=compute, output=out,
                       input_format=fmt) as c:
        for q in range(8):
            c.run_device(dev[q % 4].data_ptr())
        assert np.array_equal(c.dump(), (2 * sum(sums)).astype(out))


@pytest.mark.parametrize("band,off", [(0, 0), (18, 1)])
def test_long_calls_on_a_callers_stream(xg, band, off):
    """134 MB of int8 samples a call, converted with nothing beside: launched plainly.
    Every format gives the sums of the same samples as int8."""
    import torch
    n, f, t = 512, 16, 4096
    gen = torch.Generator(device="cuda").manual_seed(7)
    xs = [torch.randint(-8, 8, (t, (band or f) * n * 2, 2), generator=gen, device="cuda",
                        dtype=torch.int8) for _ in range(2)]
    encoded = {
        "int8": lambda x: x,
        "packed4": lambda x: (x[..., 0] << 4) | (x[..., 1] & 15),
        "dp4a_swizzled": lambda x: x.view(t // 4, 4, -1).transpose(1, 2),
        "block32": lambda x: x.view(-1, 32, 2).transpose(1, 2),
    }
    want, stream = None, torch.cuda.Stream()
    for fmt, encode_as in encoded.items():
        bufs = [encode_as(x).contiguous() for x in xs]
        torch.cuda.synchronize()
        with xg.Correlator(n, f, t, input_format=fmt, channel_offset=off, input_nfrequency=band,
                           flags=xg.XGPU_DONT_REGISTER) as c:
            c.tune(1, 0, 0)
            c.set_stream(stream.cuda_stream)
            for q in (0, 1, 0):
                c.run_device(bufs[q].data_ptr())
            got = c.dump_int64()
        want = got if want is None else want
        assert np.array_equal(got, want), fmt
