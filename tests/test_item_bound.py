"""The tensor-core kernels combine a work item's products in 32 bits, which hold
kSegment (32768) samples: what launches or plans them refuses longer items, on
either kernel, whatever its caller split.  The launchers are linked from the
library's objects and run with no device in sight, so that what they accept ends
at the missing device."""
import os
import subprocess

PROGRAM = r"""
#include "internal.h"
using namespace xgpu;

int main() {
  XGPUConfig c;
  xgpuDefaultConfig(&c);
  c.nstation = 16; c.nfrequency = 1; c.ntime = 1 << 17; c.ntimepipe = 16;
  const Sizes s = make_sizes(c);
  CUtensorMap map;
  const int samples[] = {32768, 32768 + 16, 65536, 65536 + 16, 3 * 32768};
  for (int wide = 0; wide < 2; ++wide)
    for (int t : samples)
      for (int k = 1; k <= 3; ++k) {
        TcTuning tune;
        tune.ksplit = k;
        tune.wide = wide;
        const cudaError_t e = launch_tc_tuned(map, s, 0, t, nullptr, 0, nullptr, 0, tune, 0);
        Job job;
        const int r = tc_fill_job(&job, nullptr, s, 0, t, nullptr, 0, k, 0, wide);
        printf("%d %d %d %d %d\n", wide, t, k, e == cudaErrorInvalidValue, r == kItemTooLong);
      }
}
"""


def test_items_longer_than_the_drain_holds(tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    lib = os.path.join(root, "xgpu_b200")
    subprocess.run(["make", "-s", "-j", "8", "-C", lib], check=True)
    src, exe = tmp_path / "bound.cu", tmp_path / "bound"
    src.write_text(PROGRAM)
    objects = [os.path.join(lib, "_build", o) for o in sorted(os.listdir(os.path.join(lib, "_build")))
               if o.endswith(".o")]
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-ccbin", "g++",
                    "-I", os.path.join(lib, "csrc"), "-o", str(exe), str(src), *objects,
                    "-Xcompiler", "-fopenmp", "-lgomp"], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True,
                         env={**os.environ, "CUDA_VISIBLE_DEVICES": ""}).stdout
    rows = [tuple(map(int, line.split())) for line in out.splitlines()]
    assert len(rows) == 2 * 5 * 3
    for wide, t, k, launch_refused, fill_refused in rows:
        stages = -(-t // 128)
        too_long = -(-stages // k) * 128 > 32768
        assert (launch_refused, fill_refused) == (too_long, too_long), (wide, t, k)
