"""A process that asked for blocking synchronisation (cudaDeviceScheduleBlockingSync)
sleeps while a correction's ticks run, instead of spinning on their counters."""

import subprocess
import sys
import os

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import ctypes, resource, sys
sched = int(sys.argv[1])
cu = ctypes.CDLL("libcuda.so.1")
assert cu.cuInit(0) == 0
assert cu.cuDevicePrimaryCtxSetFlags_v2(0, sched) == 0
import numpy as np, torch
from extrem_z_b200 import api, synth
fld = synth.make_field(160, 160, 160, n_gauss=64, seed=3, rel=1e-3)
f, start = torch.from_numpy(fld.f).cuda(), torch.from_numpy(fld.decp).cuda()
ctx = api.context(0)
for rep in range(3):
    g = start.clone()
    torch.cuda.synchronize()
    before = resource.getrusage(resource.RUSAGE_THREAD).ru_nvcsw
    report, _ = ctx.correct_device(f, g, fld.eb)
    slept = resource.getrusage(resource.RUSAGE_THREAD).ru_nvcsw - before
print(slept, report.manifold_rounds - report.manifold_reused)
"""


def run(sched):
    out = subprocess.run([sys.executable, "-c", PROGRAM, str(sched)], cwd=ROOT, check=True,
                         capture_output=True, text=True, timeout=300).stdout
    return [int(x) for x in out.split()[-2:]]


def test_blocking_sync_sleeps():
    """Every computed manifold round of this field takes some hundred microseconds
    and ends in a wait for its counters: at least as many sleeps."""
    slept, rounds = run(4)  # CU_CTX_SCHED_BLOCKING_SYNC
    assert rounds >= 3
    assert slept >= rounds
