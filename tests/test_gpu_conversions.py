"""Input conversions that run beside the previous call's engine launch: chains of
device-input calls in each converted format, on each engine, over whole inputs
and channel ranges read in place, on the context's own stream and on a caller's,
with waits, dumps and clears between the calls.  Every call's input differs and
both conversion buffers are in use, so an order violated shows in the sums
(bit-exact against the oracle; the FP32 engine against its float sums).  Long packed calls on CTA pairs switch from the
kernel's own expansion to a conversion ahead of it in mid-chain."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def encode(oracle_mod, fmt, n, f, t, seed):
    """(device bytes, plain samples) of one call over the whole band."""
    if fmt == "packed4":
        p = oracle_mod.generate(t * f * n * 2, 1, seed)
        return p, oracle_mod.unpack4(p)
    x = oracle_mod.gaussian_input(n, f, t, seed=seed, sigma=30.0)
    return (oracle_mod.swizzle(x, n, f, t) if fmt == "dp4a_swizzled" else oracle_mod.block32(x)), x


@pytest.mark.parametrize("fmt", ["packed4", "dp4a_swizzled", "block32"])
@pytest.mark.parametrize("engine,compute", [("tensor", "int8"), ("plain", "int8"),
                                            ("plain", "fp32")])
@pytest.mark.parametrize("n,f,t,band,off,own", [(48, 5, 208, 0, 0, True), (80, 3, 336, 8, 2, True),
                                                (256, 4, 1024, 0, 0, True),
                                                (64, 6, 512, 7, 1, False)])
def test_chains_of_converted_calls(xg, oracle_mod, fmt, engine, compute, n, f, t, band, off, own):
    import torch
    fin = band or f
    bufs, sums, samples = [], [], []
    for q in range(5):
        b, x = encode(oracle_mod, fmt, n, fin, t, 900 + q)
        bufs.append(torch.from_numpy(np.ascontiguousarray(b).view(np.int8)).cuda())
        mine = np.ascontiguousarray(x.reshape(t, fin, 4 * n)[:, off:off + f]).reshape(-1)
        sums.append(oracle_mod.xengine_i64(mine, n, f, t))
        samples.append(mine)

    def expected(calls):
        if compute == "fp32":   # the float engine's sums over the calls in order
            return oracle_mod.xengine_f32(np.concatenate([samples[q] for q in calls]), n, f,
                                          t * len(calls))
        return sum(sums[q] for q in calls).astype(np.int32)

    torch.cuda.synchronize()
    out = "int32" if compute == "int8" else "float32"
    stream = torch.cuda.Stream()
    with xg.Correlator(n, f, t, ntimepipe=16, engine=engine, compute=compute, output=out,
                       input_format=fmt, channel_offset=off, input_nfrequency=band) as c:
        if not own:
            c.set_stream(stream.cuda_stream)
        for q in range(9):
            sync = {3: xg.SYNCOP_SYNC_COMPUTE, 8: xg.SYNCOP_DUMP}.get(q, xg.SYNCOP_NONE)
            c.run_device(bufs[q % 5].data_ptr(), sync)
        assert np.array_equal(c.output_view()[: c.info.matLength * 2],
                              expected([q % 5 for q in range(9)]))
        c.run_device(bufs[0].data_ptr())
        c.clear()
        for q in range(3):
            c.run_device(bufs[q].data_ptr())
        assert np.array_equal(c.dump(), expected([0, 1, 2]))


def test_long_packed_calls_convert_ahead(xg):
    """36,864 and 110,592 pipeline stages a call: the third call on, and every
    call, convert ahead of the CTA-pair kernel.  The same samples as int8 give
    the same sums."""
    import torch
    for n, f, t in [(512, 16, 8192), (512, 48, 8192)]:
        gen = torch.Generator(device="cuda").manual_seed(f)
        plain, packed = [], []
        for _ in range(2):
            x = torch.randint(-8, 8, (t * f * n * 2, 2), generator=gen, device="cuda",
                              dtype=torch.int8)
            plain.append(x)
            packed.append(((x[:, 0] << 4) | (x[:, 1] & 15)).contiguous())
        torch.cuda.synchronize()
        got = []
        for fmt, bufs in (("int8", plain), ("packed4", packed)):
            with xg.Correlator(n, f, t, input_format=fmt, flags=xg.XGPU_DONT_REGISTER) as c:
                for q in range(5):
                    c.run_device(bufs[q % 2].data_ptr())
                got.append(c.dump_int64())
        assert np.array_equal(got[0], got[1])
