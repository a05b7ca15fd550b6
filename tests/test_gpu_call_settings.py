"""The kernel and grid of a call over device input, read from the launches that
a profiler records (in a process of its own).  An untuned context runs CTA pairs
on part of the SMs only for calls that the calls before them can overlap: not
for a call whose predecessors have finished, however the program waited for
them, and not once the program holds the stream and may queue its own work
between the calls."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import ctypes, json, os, tempfile, time
import torch
from torch.profiler import profile, ProfilerActivity
import xgpu_b200 as xg

def recorded(f, times=0, kinds=("kernel",)):
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        f()
        torch.cuda.synchronize()
    path = os.path.join(tempfile.mkdtemp(), "trace.json")
    p.export_chrome_trace(path)
    with open(path) as fh:
        ev = [e for e in json.load(fh)["traceEvents"] if e.get("cat") in kinds]
    ev.sort(key=lambda e: e["ts"])
    return [[e["name"].split("(")[0].split("::")[-1], e["args"].get("grid", [0])[0]] + times * [e["ts"], e["ts"] + e["dur"]]
            for e in ev]

def context(n, f, t, fmt="int8", **kind):
    c = xg.Correlator(n, f, t, input_format=fmt, **kind, flags=xg.XGPU_DONT_REGISTER)
    x = torch.randint(-8, 8, (4 * n * f * t,), device="cuda", dtype=torch.int8)
    torch.cuda.synchronize()
    return c, x

def calls(c, x, k, sync=xg.SYNCOP_NONE, wait=None):
    for _ in range(k):
        c.run_device(x.data_ptr(), sync)
        if wait:
            wait()

def chain(c, x, sync=xg.SYNCOP_NONE):
    # of three, the one least interrupted on the host: a call that the host queues
    # late finds the ones before it finished
    runs = []
    for _ in range(3):
        c.clear()
        runs.append(recorded(lambda: calls(c, x, 6, sync)))
    return min(runs, key=lambda r: sum(grid for name, grid in r))

out = {}
c, x = context(256, 10, 8192)      # a call takes about 0.1 ms
recorded(lambda: calls(c, x, 1))
c.clear()
out["lone"] = recorded(lambda: calls(c, x, 1))
out["chain"] = chain(c, x)
out["transfer"] = chain(c, x, xg.SYNCOP_SYNC_TRANSFER)
c.clear()
out["waited"] = recorded(lambda: calls(c, x, 6, wait=torch.cuda.synchronize))
c.clear()
out["slow"] = recorded(lambda: calls(c, x, 6, wait=lambda: time.sleep(0.005)))
c.clear()
c.stream
out["stream held"] = recorded(lambda: calls(c, x, 6))
c.close()
c, x = context(512, 48, 8192, "packed4")    # 110,592 pipeline stages, 0.9 ms a call
for how, sync, wait in (("api", xg.SYNCOP_SYNC_COMPUTE, None),
                        ("device", xg.SYNCOP_NONE, torch.cuda.synchronize)):
    calls(c, x, 1, sync, wait)
    out["packed " + how] = recorded(lambda: calls(c, x, 3, sync, wait))
calls(c, x, 3)
torch.cuda.synchronize()
out["packed chain"] = recorded(lambda: calls(c, x, 4))
c.close()
c, x = context(384, 64, 8192, "packed4")    # 86,016 stages of six tile rows
out["packed chain, six rows"] = recorded(lambda: calls(c, x, 4))
c.close()
c, x = context(64, 20, 1024, engine="plain", compute="fp32", output="float32")
x.random_(-128, 128)     # two calls take the diagonal blocks' sums past 2^24
torch.cuda.synchronize()
out["loud"] = recorded(lambda: (calls(c, x, 6, xg.SYNCOP_SYNC_COMPUTE), c.clear(),
                                calls(c, x, 1, xg.SYNCOP_SYNC_COMPUTE)))
c.close()
for skip in (0, 1):      # Complex before the output: 16-byte aligned, and not
    c, x = context(176, 13, 32, order="rt", ntimepipe=16)
    buf = torch.zeros(int(c.info.matLength) * 2 + 2, dtype=torch.int32, pin_memory=True)
    c.ctx.matrix_h, c.ctx.matrix_len = buf.data_ptr(), buf.numel() // 2
    xg.check("output", xg.lib().xgpuSetHostOutputBuffer(ctypes.byref(c.ctx)))
    c.ctx.output_offset = skip
    out["dump %d" % skip] = recorded(lambda: c.run_device(x.data_ptr(), xg.SYNCOP_DUMP),
                                     kinds=("kernel", "gpu_memcpy"))
    c.close()
for name, kind in (("dp4a", {}), ("fp32", {"compute": "fp32", "output": "float32"})):
    c, x = context(64, 10, 1024, "dp4a_swizzled", engine="plain", **kind)
    calls(c, x, 4)
    torch.cuda.synchronize()
    out["converted " + name] = recorded(lambda: calls(c, x, 8), times=1)
    c.close()
for name, sync in (("first", xg.SYNCOP_NONE), ("first transfer", xg.SYNCOP_SYNC_TRANSFER),
                   ("first waited", xg.SYNCOP_SYNC_COMPUTE)):
    c, x = context(400, 5, 384)    # short items: a call that may be one of many uses the words
    out[name] = recorded(lambda: (calls(c, x, 1, sync), c.flush()))
    c.close()
print(json.dumps(out))
"""


@pytest.fixture(scope="module")
def launches(xg):
    root = os.path.dirname(os.path.dirname(os.path.abspath(xg.__file__)))
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=root, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return json.loads(r.stdout.splitlines()[-1])


def test_chain_runs_pairs_on_part_of_the_sms(launches):
    assert len(launches["chain"]) == 6
    assert launches["chain"][0] == launches["lone"][0]
    assert all("tc2" in name and grid < 148 for name, grid in launches["chain"][1:])


@pytest.mark.parametrize("how", ["waited", "slow"])
def test_call_after_finished_calls_has_the_gpu(launches, how):
    assert launches[how] == 6 * launches["lone"]


def test_held_stream_keeps_the_default(launches):
    assert launches["stream held"] == 6 * launches["lone"]


def test_transfer_sync_waits_for_no_engine(launches):
    """SYNCOP_SYNC_TRANSFER returns with the engine at work (device input has no
    transfer), so its calls are a chain's like any others."""
    assert launches["transfer"] == launches["chain"]
    assert launches["first transfer"] == launches["first"]
    assert launches["first waited"] != launches["first"]


@pytest.mark.parametrize("how", ["api", "device"])
def test_lone_packed_calls_expand_in_the_kernel(launches, how):
    """A conversion ahead of the kernel passes beside the call before; calls that come
    one by one have none.  (Under the power cap they take 7% longer with it.)"""
    assert [name for name, grid in launches["packed " + how]] == 3 * ["xengine_tc2_kernel<true, false>"]


def test_chained_packed_calls_convert_ahead(launches):
    names = [name for name, grid in launches["packed chain"]]
    assert names[-6:] == 3 * ["unpack4_kernel<false>", "xengine_tc2_kernel<false, false>"]


def test_chained_packed_calls_of_few_tile_rows_expand_in_the_kernel(launches):
    names = [name for name, grid in launches["packed chain, six rows"]]
    assert names == 4 * ["xengine_tc2_kernel<true, false>"]


@pytest.mark.parametrize("engine", ["dp4a", "fp32"])
def test_small_plain_grids_come_after_their_conversion(launches, engine):
    """Let in beside the conversion, their CTAs would crowd on the SMs that it leaves
    room on."""
    rows = launches["converted " + engine]
    assert len(rows) == 16
    for conversion, launch in zip(rows[::2], rows[1::2]):
        assert "unswizzle" in conversion[0] and engine in launch[0]
        # times in us: a few for the launch itself, where the conversion that waits for
        # the launch before takes 15 to 30
        assert launch[2] > conversion[3] - 4


def test_narrow_stores_of_large_dumps_are_copied(launches):
    """A register-tile dump of 6.5 MB that is 16-byte aligned goes to the host in wide
    stores; one that is not is formatted on the device and copied."""
    wide, narrow = ([name for name, grid in launches["dump %d" % skip]] for skip in (0, 1))
    assert "format_host_kernel" in wide[-1]
    assert "format_kernel" in narrow[-2] and "DtoH" in narrow[-1]


def test_saturated_float_sums_run_one_cta_a_block(launches):
    names = [name for name, grid in launches["loud"]]
    four, one = "xengine_fp32_kernel<4>", "xengine_fp32_kernel<1>"
    assert names[0] == four and names[3:] == [one, one, one, four]
