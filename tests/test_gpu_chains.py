"""Untuned contexts choose the tensor-core kernel per call: chains of calls over
device input run CTA pairs on part of the SMs from the second call on.  Chains
of every length up to eight, over shapes below and above the work where the rule
takes over, others whose tiles or whose size it leaves to the default, with items that use the word buffer or not, word buffers small
enough to be left zero by a fold and larger ones, packed input that the chain's
calls expand in the kernel and the first call converts, and integrations that
are dumped, continued, or cleared with words pending: bit-exact sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(32, 3, 256), (128, 10, 1024), (176, 13, 1552), (256, 24, 256), (400, 5, 384),
          (80, 37, 400), (400, 30, 512)]


@pytest.mark.parametrize("fmt", ["int8", "packed4"])
@pytest.mark.parametrize("n,f,t", SHAPES)
def test_chains_of_untuned_calls(xg, oracle_mod, n, f, t, fmt):
    import torch
    ring, sums, bufs = 3, [], []
    for q in range(ring):
        if fmt == "packed4":
            x = oracle_mod.generate(t * f * n * 2, 1, 50 + q)
            sums.append(oracle_mod.xengine_i64(oracle_mod.unpack4(x), n, f, t))
        else:
            x = oracle_mod.gaussian_input(n, f, t, seed=50 + q, sigma=40.0)
            sums.append(oracle_mod.xengine_i64(x, n, f, t))
        bufs.append(torch.from_numpy(x.view(np.int8)).cuda())
    torch.cuda.synchronize()

    with xg.Correlator(n, f, t, ntimepipe=16, input_format=fmt) as c:
        def words():
            return c.output_view()[: c.info.matLength * 2]

        for k in (1, 2, 3, 8):
            # a chain whose last call dumps
            c.clear()
            want = np.zeros_like(sums[0])
            for q in range(k):
                c.run_device(bufs[q % ring].data_ptr(),
                             xg.SYNCOP_DUMP if q == k - 1 else xg.SYNCOP_NONE)
                want += sums[q % ring]
            order = c.info.matrix_order
            assert order == xg.TRIANGULAR_ORDER
            assert np.array_equal(words(), want.astype(np.int32))
            # the integration goes on, first to a wait, then to an exact dump
            for q in range(k):
                c.run_device(bufs[(q + 1) % ring].data_ptr(),
                             xg.SYNCOP_SYNC_COMPUTE if q == k - 1 else xg.SYNCOP_NONE)
                want += sums[(q + 1) % ring]
            assert np.array_equal(c.dump_int64(), want)
            # a chain that is discarded, words pending
            for q in range(k):
                c.run_device(bufs[q % ring].data_ptr())
        c.clear()
        for q in range(3):
            c.run_device(bufs[q].data_ptr())
        assert np.array_equal(c.dump(), sum(sums).astype(np.int32))
