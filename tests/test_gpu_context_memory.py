"""Contexts of lattices past the FP32 gain kernel's 1024 orbits do not build its
tables on the host: their entries grow with the seventh power of the lattice's
size (32^3, R = 5.5: gigabytes)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import resource, sys
sys.path.insert(0, {root!r})
import torch
torch.zeros(1).cuda()
import gpu_determ_gb300 as gd
gd.Context(gd.GridSpec(8, R=4.8)).close()
before = resource.getrusage(resource.RUSAGE_SELF).ru_maxrss
ctx = gd.Context(gd.GridSpec(32, R=5.5))
print("MB", (resource.getrusage(resource.RUSAGE_SELF).ru_maxrss - before) // 1024)
"""


def test_large_lattice_needs_little_host_memory(cuda, gdlib):
    r = subprocess.run([sys.executable, "-c", CODE.format(root=ROOT)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr
    mb = int(r.stdout.split("MB")[1])
    # the weight rows and the pair sums' items are some hundred MB, products and
    # targets of every pair sum another 3 GB
    assert mb < 1500, mb
