"""Host memory of a call does not grow with its number of chunks."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import resource, torch
from pyscfad_b200 import triples
g = torch.Generator(device="cuda").manual_seed(0)
def inputs(o, v):
    r = lambda *s: 0.01 * torch.randn(*s, generator=g, device="cuda", dtype=torch.float64)
    e = torch.cat([torch.full((o,), -1.0), torch.full((v,), 1.0)]).to("cuda", torch.float64)
    return [e, r(o, v), r(o, o, v, v), r(o, v, o, o), r(o, v, o, v), r(o, v, v * (v + 1) // 2), r(v, o)]
for n in (20, 120):
    x = inputs(2, n)
    triples.energy(*x, precision="fp64", block_size=1)
    print(resource.getrusage(resource.RUSAGE_SELF).ru_maxrss)
"""


# nvir 120 in blocks of one: 295 240 chunks (1540 at nvir 20, which brings in the context and
# the kernels).  A list of their descriptors (over 300 bytes each) is 88 MB and more; a few MB is
# what the driver's queues and the allocator may take.
@pytest.mark.gpu
def test_chunks_are_not_listed_on_the_host():
    out = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=120, check=True)
    small, large = (int(line) for line in out.stdout.split())   # KB
    assert large - small < 40 << 10
