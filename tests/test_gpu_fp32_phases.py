"""The FP32 engine's two phases (integer arithmetic while every float sum is
exact, float arithmetic from there on) give the bits of xGPU's float engine:
integrations that stay exact, that leave the exact phase in the first chunk, in
a later one, at the check that covers four chunks or one, calls that start
from sums already past 2^24, and launches of every number of time pieces (one
to eight: 256 stations x 6 channels and more than 32768 samples run whole).  The oracle's float engine restates
omp_xengine.c:24-28 term for term, so the tolerance is zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def samples(kind, n, f, t, rng):
    shape = (t, f, n, 2, 2)
    if kind == "full":      # every sample -128 - 128i: autocorrelations grow by 2^15 a sample
        return np.full(shape, -128, np.int8)
    if kind == "mixed":     # a few loud stations: only some blocks leave the exact phase
        x = np.clip(np.round(rng.normal(0, 12, shape)), -127, 127).astype(np.int8)
        x[:, :, ::7] = rng.choice(np.array([-128, 127], np.int8), (t, f, len(range(0, n, 7)), 2, 2))
        return x
    if kind == "late":      # loud from the middle of a chunk on
        x = rng.integers(-8, 9, shape).astype(np.int8)
        x[t // 2 + 13:] = rng.choice(np.array([-128, 127], np.int8), x[t // 2 + 13:].shape)
        return x
    return np.clip(np.round(rng.normal(0, 40, shape)), -127, 127).astype(np.int8)


@pytest.mark.parametrize("kind", ["gauss", "full", "mixed", "late"])
@pytest.mark.parametrize("n,f,t,calls", [(16, 1, 64, 1), (48, 2, 448, 1), (32, 1, 512, 2),
                                         (64, 2, 1040, 3), (80, 1, 2064, 2), (32, 10, 6400, 1),
                                         (256, 6, 192, 3), (128, 13, 528, 2), (16, 1, 33024, 1)])
def test_phases_equal_the_float_engine(xg, oracle_mod, kind, n, f, t, calls):
    rng = np.random.default_rng(n * 7919 + t)
    xs = [samples(kind, n, f, t, rng).reshape(-1) for _ in range(calls)]
    want = oracle_mod.xengine_f32(np.concatenate(xs), n, f, t * calls)
    with xg.Correlator(n, f, t, ntimepipe=16, engine="plain", compute="fp32",
                       output="float32") as c:
        for q, x in enumerate(xs):
            c.set_input(x)
            c.run(xg.SYNCOP_SYNC_COMPUTE)
        got = c.dump()
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
