"""Kernel variants at the sizes where their tile rules change: remainders, one
past a tile, the smallest and largest of each range, against the CPU oracle."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from pyscfad_b200 import triples
from pyscfad_b200.synthetic import make_inputs
from tests import golden_util as G

pytestmark = pytest.mark.gpu


def _relerr(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-7))


# M and N of the FP64 contractions are nocc * (virtual block), nvir and nocc:
# N tiles of 16, 32, 48 and 64 (nocc 2-16, 17, 33, 49), 128-wide tiles with a
# remainder (nvir 65, 130), K in one slice and in many
@pytest.mark.parametrize("o,v", [(2, 130), (3, 65), (16, 7), (17, 5), (33, 3), (49, 2), (65, 2)])
def test_fp64_contraction_tiles(o, v):
    inp = make_inputs(o, v, 40, seed=o, fvo_sigma=1e-3)
    e_ref, g_ref = O.oracle_energy_vjp(inp)
    e, g = triples.energy_vjp(*(getattr(inp, k) for k in G.KEYS), precision="fp64", device="cuda")
    torch.cuda.synchronize()
    # FP64 sums of at most o*o*16 + v products in another order: a few 1e-16 times sqrt(K), and the parity bounds
    assert abs(float(e) - e_ref) <= 1e-12 * abs(e_ref)
    for k in G.KEYS:
        assert _relerr(g[k].cpu().numpy(), g_ref[k]) < 1e-10, k
