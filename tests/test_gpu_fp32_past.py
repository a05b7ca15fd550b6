"""An FP32 integration whose sums have passed 2^24 in the middle of the array runs one
CTA a block from then on where four would be slower (120 and 200 blocks; 60 keep
theirs), until the integration is cleared: the float engine's bits throughout, also when
calls are queued ahead of what they find, and clears come between queued calls."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,f,t", [(64, 20, 512), (128, 10, 512), (64, 10, 512)])
@pytest.mark.parametrize("wait", [False, True])
def test_loud_integrations_and_clears(xg, oracle_mod, n, f, t, wait):
    import torch
    rng = np.random.default_rng(n + f)
    shape = t * f * n * 4
    loud = [rng.choice(np.array([-128, 127], np.int8), shape) for _ in range(2)]
    quiet = [rng.integers(-8, 9, shape).astype(np.int8) for _ in range(2)]
    dev = {id(x): torch.from_numpy(x).cuda() for x in loud + quiet}
    torch.cuda.synchronize()
    sync = xg.SYNCOP_SYNC_COMPUTE if wait else xg.SYNCOP_NONE
    with xg.Correlator(n, f, t, ntimepipe=16, engine="plain", compute="fp32",
                       output="float32") as c:
        for xs in ([loud[0], loud[1], loud[0], quiet[0], loud[1]], [quiet[1], quiet[0]],
                   [quiet[0], loud[0], loud[0], quiet[1]]):
            for _ in range(2):    # once discarded with its calls queued
                c.clear()
                for x in xs:
                    c.run_device(dev[id(x)].data_ptr(), sync)
            want = oracle_mod.xengine_f32(np.concatenate(xs), n, f, t * len(xs))
            assert np.array_equal(c.dump().view(np.uint32), want.view(np.uint32))
