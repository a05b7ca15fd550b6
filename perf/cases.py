"""Performance cases of the X-engine: what a user's program has it correlate,
through the package's public entry points, from the smallest calls to the
largest blocks.

A case is one of three uses (``api``):

* ``device``: a context whose input is already in device memory (a receiver
  that writes HBM): clear, ``calls`` calls over a ring of input buffers, the
  last one dumping to a pinned output buffer;
* ``host``: the drop-in use of xGPU's own driver: input in pinned host memory,
  ``SYNCOP_SYNC_TRANSFER`` on all calls but the last, ``SYNCOP_DUMP`` on it;
* ``batch``: a planned batch of uneven subarrays replayed as a CUDA graph.

Inputs are clipped, rounded Gaussian int8 samples (sigma 16, the benchmark's),
or uniform 4+4-bit samples in [-7, 7] for packed input.
"""
import ctypes
import math
import random

import torch

import xgpu_b200 as xg

SIGMA = 16.0
RING_BYTES = 160 << 20   # inputs rotate over more than the L2 cache where a case has enough calls
MAX_RING = 16


def _case(name, api="device", n=0, f=0, t=0, calls=1, engine="tensor", compute="int8",
          output="int32", order="tri", fmt="int8", band=0, offset=0, ksplit=0, grid=0, pair=0):
    c = {"api": api, "n": n, "f": f, "t": t, "calls": calls, "engine": engine, "compute": compute,
         "output": output, "order": order, "fmt": fmt, "band": band, "offset": offset,
         "ksplit": ksplit, "grid": grid, "pair": pair}
    if name:
        c["name"] = name
    return c


def _batch_case(name, jobs, nmax, fmax, tmax, shapes, autotune):
    c = {"api": "batch", "jobs": jobs, "nmax": nmax, "fmax": fmax, "tmax": tmax, "shapes": shapes,
         "autotune": autotune}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # The smallest useful call: one short block of a small array, dumped at once; all latency.
        _case("small_dump", n=32, f=4, t=256),
        # An xGPU program relinked: the build's default shape, output type and order, host
        # buffers, one dump per call.
        _case("dropin_default", api="host", n=256, f=10, t=1024, output="float32", order="rt"),
        # The default shape as a stream over device buffers, with a setting an earlier autotuning
        # chose (CTA pairs on a quarter of the SMs), one dump per 32 blocks.
        _case("stream_tuned", n=256, f=10, t=1024, calls=32, ksplit=1, grid=36, pair=1),
        # A mid-size array with more channels, untuned, dumped as separate real and imaginary
        # planes of floats.
        _case("stream_real_imag", n=128, f=64, t=2048, calls=8, output="float32", order="ri"),
        # One GPU's channels of a shared band, with a station count and a block length that leave
        # partial tiles and stages.
        _case("odd_range", n=176, f=13, t=1552, calls=4, band=40, offset=9),
        # A large array integrating long blocks (the benchmark's large configuration, a quarter of
        # its channels): tensor-bound.
        _case("large_block", n=512, f=64, t=8192, calls=16),
        # The same array fed with packed 4+4-bit samples.
        _case("large_packed", n=512, f=64, t=8192, calls=8, fmt="packed4"),
        # Uneven subarrays in one launch (the benchmark's mix, a quarter of its jobs).
        _batch_case("batch_uneven", 24, 1024, 64, 8192, 3, True),
        # A handful of tiny subarrays: launch and scheduling latency.
        _batch_case("batch_small", 8, 64, 4, 512, 5, False),
        # xGPU's dp4a build: the CUDA-core integer engine at the default shape.
        _case("plain_dp4a", n=256, f=10, t=1024, calls=4, engine="plain"),
        # xGPU's FP32 build: float sums at the benchmark's small shape, in the default order.
        _case("plain_fp32", n=64, f=10, t=1024, calls=4, engine="plain", compute="fp32",
              output="float32", order="rt"),
        # A pipeline that already swizzles its samples for xGPU's dp4a kernel.
        _case("swizzled_stream", n=256, f=10, t=1024, calls=8, order="rt", fmt="dp4a_swizzled"),
    ]


def _log_int(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi, max(lo, int(round(v / step)) * step))


def _ops(n, f, t):
    return xg.ops_per_integration(n, f, t)


def draw(rng):
    kind = rng.choice(["device", "device", "device", "host", "format", "dp4a", "fp32", "batch"])
    if kind == "batch":
        jobs = _log_int(rng, 2, 24)
        return _batch_case(None, jobs, _log_int(rng, 64, 1024, 16), _log_int(rng, 2, 64),
                           _log_int(rng, 256, 8192, 256), rng.randrange(1 << 20),
                           rng.random() < 0.5)
    n = _log_int(rng, 16, 768, 16)
    f = _log_int(rng, 1, 128)
    t = _log_int(rng, 128, 8192, 16)
    calls = _log_int(rng, 1, 32)
    # bounds on one pass: tensor, dp4a and float arithmetic, and the host link
    most = {"device": 2e13, "host": 5e12, "format": 5e12, "dp4a": 1e12, "fp32": 2e11}[kind]
    link = (1 << 28) if kind == "host" else (1 << 33)

    def too_much():
        return calls * _ops(n, f, t) > most or calls * 4 * n * f * t > link or n * n * f > 2 ** 24

    while too_much():
        if calls > 2:
            calls = max(1, calls // 2)
        elif f > 4:
            f = f // 2
        elif t > 512:
            t = max(256, t // 2 // 16 * 16)
        elif n > 128:
            n = n // 2 // 16 * 16
        else:
            calls = 1
            f = max(1, f // 2)
    c = _case(None, n=n, f=f, t=t, calls=calls,
              api="host" if kind == "host" else "device",
              output=rng.choice(["int32", "float32"]),
              order=rng.choice(["tri", "tri", "ri", "rt"]))
    if kind == "device" and rng.random() < 0.3:
        c["band"] = f + rng.randrange(1, 2 * f + 2)
        c["offset"] = rng.randrange(0, c["band"] - f + 1)
    if kind == "device" and rng.random() < 0.25:
        c["ksplit"], c["grid"], c["pair"] = 1, 36, 1
    if kind == "format":
        c["fmt"] = rng.choice(["packed4", "dp4a_swizzled", "block32"])
    if kind in ("dp4a", "fp32"):
        c["engine"] = "plain"
    if kind == "fp32":
        c["compute"], c["output"] = "fp32", "float32"
    return c


# ---- inputs -----------------------------------------------------------------

def _gaussian(nbytes, gen, sigma=SIGMA):
    out = torch.empty(nbytes, dtype=torch.int8, device="cuda")
    chunk = 1 << 26
    for a in range(0, nbytes, chunk):
        m = min(chunk, nbytes - a)
        r = torch.randn(m, generator=gen, device="cuda").mul_(sigma).round_().clamp_(-127, 127)
        out[a:a + m] = r.to(torch.int8)
    return out


def _generator(seed, q):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + q) % (1 << 62))
    return g


def _samples(case, seed, q):
    """Input buffer q as plain int8 [t][band][n][pol][re, im], flat."""
    nbytes = 4 * case["n"] * (case["band"] or case["f"]) * case["t"]
    gen = _generator(seed, q)
    if case["fmt"] == "packed4":
        return torch.randint(-7, 8, (nbytes,), generator=gen, device="cuda", dtype=torch.int8)
    return _gaussian(nbytes, gen)


def _encode(case, x):
    """The same samples in the case's input format."""
    fmt, t = case["fmt"], case["t"]
    if fmt == "packed4":
        v = x.view(-1, 2)
        return ((v[:, 0] << 4) | (v[:, 1] & 15)).contiguous()
    if fmt == "dp4a_swizzled":   # [t/4][f][s][p][c][t%4]
        return x.view(t // 4, 4, -1).transpose(1, 2).contiguous().view(-1)
    if fmt == "block32":         # per 16 stations: 32 real bytes, then 32 imaginary bytes
        return x.view(-1, 32, 2).transpose(1, 2).contiguous().view(-1)
    return x


def _ring(case):
    nbytes = 4 * case["n"] * (case["band"] or case["f"]) * case["t"]
    return max(1, min(case["calls"], MAX_RING, max(2, -(-RING_BYTES // nbytes))))


def _batch_shapes(case):
    """(stations, channels, samples, sigma) of each subarray: stations log-uniform."""
    rng = random.Random(case["shapes"])
    lo = min(32, case["nmax"])
    return [(_log_int(rng, lo, case["nmax"], 16), rng.randint(1, case["fmax"]),
             256 * rng.randint(1, max(1, case["tmax"] // 256)), rng.uniform(4.0, 32.0))
            for _ in range(case["jobs"])]


# ---- the program's state ----------------------------------------------------

class _Correlation:
    def __init__(self, case, seed):
        n, f, t = case["n"], case["f"], case["t"]
        host = case["api"] == "host"
        self.c = xg.Correlator(
            n, f, t, ntimepipe=128 if t % 128 == 0 else 16, compute=case["compute"],
            output=case["output"], order=case["order"], engine=case["engine"],
            input_format=case["fmt"], device=torch.cuda.current_device(),
            flags=xg.XGPU_DONT_REGISTER_MATRIX if host else xg.XGPU_DONT_REGISTER,
            channel_offset=case["offset"], input_nfrequency=case["band"])
        # dumps go to a page-locked buffer of the program's own
        words = int(self.c.info.matLength) * 2
        self.out = torch.zeros(words, dtype=torch.int32 if case["output"] == "int32"
                               else torch.float32, pin_memory=True)
        self.c.ctx.matrix_h, self.c.ctx.matrix_len = self.out.data_ptr(), words // 2
        xg.check("xgpuSetHostOutputBuffer",
                 xg.lib().xgpuSetHostOutputBuffer(ctypes.byref(self.c.ctx)))
        if not host:
            self.inputs = [_encode(case, _samples(case, seed, q)) for q in range(_ring(case))]
            ptrs = [x.data_ptr() for x in self.inputs]
            self.feeds = [ptrs[k % len(ptrs)] for k in range(case["calls"])]
        else:
            self.c.set_input(_encode(case, _samples(case, seed, 0)).cpu().numpy())
            self.feeds = None
        if case["ksplit"]:
            self.c.tune(case["ksplit"], case["grid"], case["pair"])
        self.calls = case["calls"]
        torch.cuda.synchronize()

    def run(self):
        c, last = self.c, self.calls - 1
        c.clear()
        if self.feeds is None:
            for _ in range(last):
                c.run(xg.SYNCOP_SYNC_TRANSFER)
            c.run(xg.SYNCOP_DUMP)
        else:
            for ptr in self.feeds[:last]:
                c.run_device(ptr)
            c.run_device(self.feeds[last], xg.SYNCOP_DUMP)
        return self.out

    def __del__(self):
        if hasattr(self, "c"):
            self.c.close()


class _BatchOfSubarrays:
    def __init__(self, case, seed):
        self.inputs, self.states, jobs = [], [], []
        for q, (n, f, t, sigma) in enumerate(_batch_shapes(case)):
            x = _gaussian(4 * n * f * t, _generator(seed, q), sigma)
            s = torch.zeros(xg.state_elems(n, f), dtype=torch.int64, device="cuda")
            self.inputs.append(x)
            self.states.append(s)
            jobs.append({"input": x.data_ptr(), "state": s.data_ptr(), "nstation": n,
                         "nfrequency": f, "ntime": t})
        torch.cuda.synchronize()
        self.b = xg.Batch(jobs, device=torch.cuda.current_device(),
                          stream=torch.cuda.current_stream().cuda_stream,
                          autotune=case["autotune"], graph=True, pair=not case["autotune"])

    def run(self):
        self.b.run()
        return self.states

    def __del__(self):
        if hasattr(self, "b"):
            torch.cuda.synchronize()
            self.b.close()


def prepare(case, seed):
    return _BatchOfSubarrays(case, seed) if case["api"] == "batch" else _Correlation(case, seed)


def run(state):
    return state.run()


def _mat_length(case):
    n, f = case["n"], case["f"]
    if case["order"] == "rt":
        return f * (n // 2 + 1) * (n // 4) * 16
    return f * (n * (n + 1) // 2) * 4


def work(case):
    if case["api"] == "batch":
        shapes = _batch_shapes(case)
        return {"bytes": sum(4 * n * f * t + 8 * xg.state_elems(n, f) for n, f, t, _ in shapes),
                "flops": sum(_ops(n, f, t) for n, f, t, _ in shapes)}
    n, f, t, calls = case["n"], case["f"], case["t"], case["calls"]
    per = 2 if case["fmt"] == "packed4" else 4
    return {"bytes": calls * per * n * f * t + 8 * _mat_length(case),
            "flops": calls * _ops(n, f, t)}


# ---- the same sums in 64 bits -----------------------------------------------

def _visibilities(x, n, f0, f, fin, t):
    """float64 [f][baseline][p1][p2][re, im] of int8 samples [t][fin][n][pol][c]."""
    v = x.view(t, fin, 4 * n)
    i, j = torch.tril_indices(n, n, device="cuda")
    out = torch.empty((f, i.numel(), 2, 2, 2), dtype=torch.float64, device="cuda")
    for q in range(f):
        a = v[:, f0 + q, :].to(torch.float64)
        g = (a.T @ a).view(n, 2, 2, n, 2, 2)            # [s][p][c][s'][p'][c']
        re = g[:, :, 0, :, :, 0] + g[:, :, 1, :, :, 1]   # [s][p][s'][p']
        im = g[:, :, 1, :, :, 0] - g[:, :, 0, :, :, 1]
        out[q, ..., 0] = re[i, :, j, :]
        out[q, ..., 1] = im[i, :, j, :]
    return out


def _ordered(case, vis):
    """Triangular sums -> the case's matrix order, flat words."""
    n, f, order = case["n"], case["f"], case["order"]
    if order == "tri":
        return vis.reshape(-1)
    if order == "ri":
        return torch.cat([vis[..., 0].reshape(-1), vis[..., 1].reshape(-1)])
    i, j = torch.tril_indices(n, n, device="cuda")
    tile = (n // 2 + 1) * (n // 4)
    a, b = i // 2, j // 2
    slot = (2 * (j % 2) + i % 2) * tile + a * (a + 1) // 2 + b
    out = torch.zeros((2, f, 4 * tile, 4), dtype=torch.float64, device="cuda")
    out[0, :, slot] = vis[..., 0].reshape(f, -1, 4)
    out[1, :, slot] = vis[..., 1].reshape(f, -1, 4)
    return out.reshape(-1)


def exact(case, seed):
    if case["api"] == "batch":
        outs = []
        for q, (n, f, t, sigma) in enumerate(_batch_shapes(case)):
            x = _gaussian(4 * n * f * t, _generator(seed, q), sigma)
            outs.append(_visibilities(x, n, 0, f, f, t).reshape(-1).to(torch.int64))
        return outs
    n, f, t, calls = case["n"], case["f"], case["t"], case["calls"]
    ring = 1 if case["api"] == "host" else _ring(case)
    vis = None
    for q in range(ring):
        times = (calls - q + ring - 1) // ring   # calls that read buffer q
        v = _visibilities(_samples(case, seed, q), n, case["offset"], f, case["band"] or f, t)
        vis = v.mul_(times) if vis is None else vis.add_(v, alpha=times)
    words = _ordered(case, vis)
    if case["output"] == "int32":
        words = words.to(torch.int64).to(torch.int32)   # an int32 dump wraps
    return words.cpu().numpy()
