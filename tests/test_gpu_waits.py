"""The bounded waits every staged kernel is built from (csrc/tma.cuh), in a small kernel of their own: a wait that runs out
ends, says so, and - the warp forms - says the same to every lane. Skipped where nvcc is missing."""
import ctypes
import os
import shutil
import subprocess

import pytest
import torch

from conftest import ROOT
from helpers import ptr, sync

pytestmark = pytest.mark.gpu

# One block of two warps and one barrier of one arrival. Lane l of the first warp starts its wait l x `stagger` ns late, with a
# limit of `limit` ns; the second warp's first lane arrives `arrive` ns after the start, or (0) not at all. Nothing waits
# without a bound: the delays end by the clock, the waits by their limit.
PROGRAM = r"""
#include "tma.cuh"
using namespace osmos;
__device__ void delay(uint64_t from, uint64_t ns) {
  for (int i = 0; i < (1 << 20) && tma::global_ns() - from < ns; i++) __nanosleep(200);
}
__global__ void waits(int* out, int is_long, uint64_t stagger, uint64_t limit, uint64_t arrive) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    tma::bar_init(&bar, 1);
    tma::bar_init_fence();
  }
  __syncthreads();
  const uint64_t t0 = tma::global_ns();
  if (threadIdx.x < kWarp) {
    if (stagger) delay(t0, threadIdx.x * stagger);
    const bool ok = is_long ? tma::bar_wait_long(&bar, 0, limit) : tma::bar_wait_warp(&bar, 0, limit);
    out[threadIdx.x] = ok ? 1 : 0;
  } else if (threadIdx.x == kWarp && arrive) {
    if (arrive > 1) delay(t0, arrive);
    tma::bar_arrive(&bar);
  }
}
extern "C" int run_waits(int* out, int is_long, uint64_t stagger, uint64_t limit, uint64_t arrive) {
  waits<<<1, 2 * kWarp>>>(out, is_long, stagger, limit, arrive);
  return (int) cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def waits(tmp_path_factory):
    nvcc = shutil.which("nvcc")
    if not nvcc:
        pytest.skip("nvcc not available")
    from libosmos_b200 import build
    d = tmp_path_factory.mktemp("waits")
    src, so = d / "waits.cu", d / "waits.so"
    src.write_text(PROGRAM)
    cmd = [nvcc, *build.NVCC_FLAGS, "-I" + os.path.join(ROOT, "libosmos_b200", "csrc"), "-shared", "-o", str(so), str(src)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    f = ctypes.CDLL(str(so)).run_waits
    f.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_uint64, ctypes.c_uint64, ctypes.c_uint64]
    return f


@pytest.mark.parametrize("form,stagger,limit,arrive,landed", [
    ("warp", 0, 50_000_000, 1, 1),                # the arrival comes at once: every lane sees it
    ("long", 0, 50_000_000, 1, 1),
    ("warp", 20_000, 50_000_000, 300_000, 1),     # ... in the middle of the lanes' starts
    ("long", 20_000, 50_000_000, 300_000, 1),
    ("warp", 0, 2_000_000, 0, 0),                 # it never comes: every lane gives up
    ("long", 40_000, 2_000_000, 0, 0),
    ("warp", 40_000, 2_000_000, 2_600_000, 0),    # it comes when the first lanes have given up and the last have not: all have
    ("long", 40_000, 2_000_000, 2_600_000, 1),    # (the long form's lanes look together: its limit starts with the last one)
])
def test_warp_wait_has_one_outcome(dev, waits, form, stagger, limit, arrive, landed):
    out = torch.full((32,), -1, dtype=torch.int32, device=dev)
    assert waits(ptr(out), int(form == "long"), stagger, limit, arrive) == 0
    sync()
    assert out.tolist() == [landed] * 32
