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


# What only makes a call faster: more than one chunk slot (an extra scratch), and
# the V-term tables (a scratch without room for them: the entries are gathered).
# Short sub-ranges (nvir 27: blocks 16, 8, 2, 1) start inside an 8-wide table block
@pytest.mark.parametrize("o,v,tv", [(3, 27, 16), (2, 40, 8), (5, 9, 2)])
@pytest.mark.parametrize("precision", ["mixed", "mixed_bf16", "fp64"])
def test_scratch_sizes_give_the_same(o, v, tv, precision):
    import ctypes

    from pyscfad_b200 import _lib

    inp = make_inputs(o, v, 40, seed=v, fvo_sigma=1e-3)
    ins = [torch.as_tensor(np.ascontiguousarray(getattr(inp, k)), device="cuda") for k in G.KEYS]
    lib, opt, prec = _lib.load(), _lib.options(tv), _lib.PRECISION[precision]
    full = lib.triples_workspace_size_ex(prec, o, v, 0, 1, ctypes.byref(opt))

    def run(nbytes):
        ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        e = torch.zeros((), dtype=torch.float64, device="cuda")
        g = {k: torch.empty_like(a) for k, a in zip(G.KEYS, ins)}
        rc = lib.triples_energy_vjp_ex(torch.cuda.current_stream().cuda_stream, prec, o, v, 0,
                                       *[a.data_ptr() for a in ins], 1.0, 1, ctypes.byref(opt), ws.data_ptr(), nbytes,
                                       e.data_ptr(), *[g[k].data_ptr() for k in G.KEYS])
        if rc == 0:
            rc = lib.triples_check_device_status(torch.cuda.current_stream().cuda_stream, ws.data_ptr())
        return rc, float(e), g

    rc, e0, g0 = run(full)
    assert rc == 0
    extra = lib.triples_workspace_extra(prec, o, v, 0, 1, ctypes.byref(opt))
    assert extra > 0
    sizes = [full + extra, full + extra // 2]
    if precision != "fp64":
        sizes.append(full - 256)
    else:
        assert run(full - 256)[0] != 0
    # the same FP32 values either way; only FP64 sums may be ordered differently
    for nbytes in sizes:
        rc, e1, g1 = run(nbytes)
        assert rc == 0
        assert abs(e1 - e0) <= 1e-13 * abs(e0)
        for k in G.KEYS:
            assert _relerr(g1[k].cpu().numpy(), g0[k].cpu().numpy()) < 1e-12, k
    assert run(4096)[0] != 0


# W-contraction tiles of 2 to 16 r values (nocc 1-17, with and without a second
# tile), adjoint tiles of 16 to 128 columns (nvir 7-130), K tails of every length
@pytest.mark.parametrize("o,v", [(1, 17), (2, 130), (3, 65), (8, 18), (9, 33), (13, 7), (17, 20), (33, 5)])
@pytest.mark.parametrize("tile_n", [0, 128, 256])
def test_mixed_contraction_tiles(o, v, tile_n):
    inp = make_inputs(o, v, 40, seed=o, fvo_sigma=1e-3)
    ins = [getattr(inp, k) for k in G.KEYS]
    e0, g0 = triples.energy_vjp(*ins, precision="fp64", device="cuda")
    e, g = triples.energy_vjp(*ins, precision="mixed", device="cuda", tile_n=tile_n)
    scale = 1e-14 if o == 1 else 0.0   # one occupied orbital has no triples: both are rounding noise
    assert abs(float(e) - float(e0)) <= 1e-6 * abs(float(e0)) + scale
    if o > 1:
        for k in G.KEYS:
            assert _relerr(g[k].cpu().numpy(), g0[k].cpu().numpy()) < 1e-5, k


# The adjoint tiles of x blocks of 16 and 8 virtuals (two and one 8 x 8 tiles
# wide: K blocks of 64 and of half as many stored values) and of the shorter
# remainder blocks kept in rows, for occupied counts off the 4 per K block and
# the 8 and 16 per M tile.  The mixed mode's parity bounds.
@pytest.mark.parametrize("o,v,tv", [(2, 24, 16), (5, 40, 16), (9, 28, 8), (17, 40, 16), (18, 27, 8)])
@pytest.mark.parametrize("precision", ["mixed", "mixed_bf16"])
def test_adjoint_tiles(o, v, tv, precision):
    inp = make_inputs(o, v, 40, seed=v, fvo_sigma=1e-3)
    ins = [getattr(inp, k) for k in G.KEYS]
    e0, g0 = triples.energy_vjp(*ins, precision="fp64", device="cuda")
    e, g = triples.energy_vjp(*ins, precision=precision, device="cuda", block_size=tv)
    e_tol, g_tol = (1e-6, 1e-5) if precision == "mixed" else (1e-4, 1e-3)
    assert abs(float(e) - float(e0)) <= e_tol * abs(float(e0))
    for k in G.KEYS:
        assert _relerr(g[k].cpu().numpy(), g0[k].cpu().numpy()) < g_tol, k


# The 64 x 64 tiles in which a packed ovvv is split and its gradient folded, and in
# which t2 is transposed and its gradient folded (nocc 66: a second tile): one short
# of a tile, exact, one past, several.  The packed and the full ovvv hold the same
# values, so the results differ by the order of FP64 sums.
@pytest.mark.parametrize("o,v", [(2, 63), (2, 64), (3, 65), (2, 130), (66, 2)])
@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed_bf16"])
def test_packed_layout_tiles(o, v, precision):
    inp = make_inputs(o, v, 40, seed=v, fvo_sigma=1e-3)
    ins = {k: getattr(inp, k) for k in G.KEYS}
    e0, g0 = triples.energy_vjp(**ins, precision=precision, device="cuda")
    e, g = triples.energy_vjp(**dict(ins, ovvv=inp.ovvv_tril()), precision=precision, device="cuda")
    assert abs(float(e) - float(e0)) <= 1e-12 * abs(float(e0))
    full = g0["ovvv"].cpu().numpy()
    il, jl = np.tril_indices(v)
    fold = full[:, :, il, jl] + np.where(il != jl, full[:, :, jl, il], 0.0)
    assert _relerr(g["ovvv"].cpu().numpy(), fold) < 1e-11
    for k in G.KEYS:
        if k != "ovvv":
            assert _relerr(g[k].cpu().numpy(), g0[k].cpu().numpy()) < 1e-11, k


# The LNO projection's kernels for up to 16, 32 and 64 occupied orbitals, at and past
# the 8-row tiles: Gram tiles shared by eight warps (nocc 8), by two (9-16), one or
# more per warp (17-64); the energy of an energy-only call comes from them as well.
@pytest.mark.parametrize("o,v", [(8, 5), (9, 4), (12, 17), (16, 3), (17, 3), (24, 3), (32, 2), (33, 2), (40, 2), (64, 2)])
def test_lno_projection_tiles(o, v):
    inp = make_inputs(o, v, 40, seed=o, fvo_sigma=1e-3)
    mat = np.random.default_rng(o).normal(size=(o, o))
    e_ref, g_ref = O.np_lno_energy_vjp(inp, mat)
    ins = [getattr(inp, k) for k in G.KEYS]
    e, g = triples.lno_energy_vjp(mat, *ins, precision="fp64", device="cuda")
    e1 = triples.lno_energy(mat, *ins, precision="fp64", device="cuda")
    # FP64 sums of up to nocc^3 nvir^3 terms of both signs in another order, and the parity bounds
    assert abs(float(e) - e_ref) <= 1e-11 * abs(e_ref)
    assert abs(float(e1) - float(e)) <= 1e-12 * abs(e_ref)
    for k in ("mat",) + G.KEYS:
        assert _relerr(g[k].cpu().numpy(), g_ref[k]) < 1e-10, k
