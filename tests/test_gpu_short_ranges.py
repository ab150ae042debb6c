"""Chunks with a short virtual sub-range (remainder blocks, blocks of 4 and
less): their kernels take a thread per element, so items share warps and CTAs
and an LNO box has as many slots as the blocks have virtual triples."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from pyscfad_b200 import triples
from pyscfad_b200.synthetic import make_inputs
from tests import golden_util as G


def _relerr(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-7))


@pytest.mark.parametrize("o,v", [(64, 1), (64, 2), (64, 3), (49, 5), (30, 7), (20, 12)])
def test_lno_scratch_follows_the_blocks(o, v):
    """Four FP64 box arrays over (i, j, k, virtual triple of the largest chunk) and what a canonical call needs;
    512 slots whatever the blocks were 4.4 GB at nocc 64 nvir 2."""
    largest = 1 << (v.bit_length() - 1)                   # nvir below 16: the largest block is its leading bit
    slots = max(2, largest ** 3)
    for precision in ("fp64", "mixed"):
        box = 4 * 8 * o ** 3 * slots
        canonical = triples.workspace_size(o, v, True, True, precision)
        assert triples.lno_workspace_size(o, v, True, True, precision) <= canonical + box + (1 << 20)


# Element kernels of every item size and warp layout: 1 to 256 elements (blocks 1, 2, 4, 8, 16 in
# every combination of nvir 31 = 16 + 8 + 4 + 2 + 1), equal occupied and equal virtual ranges,
# against the oracle; FP64 sums in another order.
@pytest.mark.gpu
@pytest.mark.parametrize("o,v,tv", [(2, 31, 0), (5, 23, 0), (4, 21, 4), (3, 9, 1), (6, 6, 2), (9, 19, 0)])
def test_lno_short_ranges_match_the_oracle(o, v, tv):
    inp = make_inputs(o, v, 40, seed=v, fvo_sigma=1e-3)
    mat = np.random.default_rng(o).normal(size=(o, o))
    e_ref, g_ref = O.np_lno_energy_vjp(inp, mat)
    ins = [getattr(inp, k) for k in G.KEYS]
    e, g = triples.lno_energy_vjp(mat, *ins, precision="fp64", device="cuda", block_size=tv)
    e1 = triples.lno_energy(mat, *ins, precision="fp64", device="cuda", block_size=tv)
    assert abs(float(e) - e_ref) <= 1e-11 * abs(e_ref)
    assert abs(float(e1) - float(e)) <= 1e-12 * abs(e_ref)
    for k in ("mat",) + G.KEYS:
        assert _relerr(g[k].cpu().numpy(), g_ref[k]) < 1e-10, k
    # the mixed modes' parity bounds
    for precision, e_tol, g_tol in (("mixed", 1e-6, 1e-5), ("mixed_bf16", 1e-4, 1e-3)):
        e, g = triples.lno_energy_vjp(mat, *ins, precision=precision, device="cuda", block_size=tv)
        assert abs(float(e) - e_ref) <= e_tol * abs(e_ref)
        for k in ("mat",) + G.KEYS:
            assert _relerr(g[k].cpu().numpy(), g_ref[k]) < g_tol, (precision, k)


# The projection's forms for up to 16, 32 and 64 occupied orbitals over boxes of several sub-range
# triples, many tiles a CTA, full and short: the identity projector is the canonical energy
# (another path and another order of FP64 sums).
@pytest.mark.gpu
@pytest.mark.parametrize("o,v", [(14, 33), (17, 17), (20, 33), (33, 17), (33, 20), (40, 16)])
@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed_bf16"])
def test_lno_projection_over_several_ranges(o, v, precision):
    inp = make_inputs(o, v, 40, seed=o, fvo_sigma=1e-3)
    ins = [getattr(inp, k) for k in G.KEYS]
    e0, g0 = triples.energy_vjp(*ins, precision="fp64", device="cuda")
    e, g = triples.lno_energy_vjp(np.eye(o), *ins, precision=precision, device="cuda")
    e_tol, g_tol = {"fp64": (1e-12, 1e-10), "mixed": (1e-6, 1e-5), "mixed_bf16": (1e-4, 1e-3)}[precision]
    assert abs(float(e) - float(e0)) <= e_tol * abs(float(e0))
    for k in G.KEYS:
        assert _relerr(g[k].cpu().numpy(), g0[k].cpu().numpy()) < g_tol, k
    torch.cuda.synchronize()


# FP64 items of 1 to 256 elements in both kernels that take them (nocc 5 and 6 lie on either
# side of the rule), chunks of both kinds in one group, several warps to an item (energy partials
# of nvir 36: 8 warps), nocc above 128; against the oracle or, where that is slow, against the same
# problem cut into 16-wide blocks.  FP64 sums in another order.
@pytest.mark.gpu
@pytest.mark.parametrize("o,v,tv", [(5, 31, 0), (6, 31, 0), (7, 20, 4), (6, 9, 1), (8, 13, 2), (6, 36, 0), (9, 23, 0)])
def test_fp64_short_ranges_match_the_oracle(o, v, tv):
    inp = make_inputs(o, v, 40, seed=v, fvo_sigma=1e-3)
    e_ref, g_ref = O.oracle_energy_vjp(inp)
    ins = [getattr(inp, k) for k in G.KEYS]
    e, g = triples.energy_vjp(*ins, precision="fp64", device="cuda", block_size=tv)
    e1 = triples.energy(*ins, precision="fp64", device="cuda", block_size=tv)
    assert abs(float(e) - e_ref) <= 1e-12 * abs(e_ref)
    assert abs(float(e1) - e_ref) <= 1e-12 * abs(e_ref)
    for k in G.KEYS:
        assert _relerr(g[k].cpu().numpy(), g_ref[k]) < 1e-10, k


@pytest.mark.gpu
@pytest.mark.parametrize("o,v,tv", [(20, 33, 2), (33, 19, 4), (130, 3, 0), (40, 17, 8)])
def test_fp64_short_ranges_against_other_blocks(o, v, tv):
    inp = make_inputs(o, v, 40, seed=v, fvo_sigma=1e-3)
    ins = [getattr(inp, k) for k in G.KEYS]
    e0, g0 = triples.energy_vjp(*ins, precision="fp64", device="cuda", block_size=1 if o > 128 else 16)
    e, g = triples.energy_vjp(*ins, precision="fp64", device="cuda", block_size=tv)
    e1 = triples.energy(*ins, precision="fp64", device="cuda", block_size=tv)
    assert abs(float(e) - float(e0)) <= 1e-12 * abs(float(e0))
    assert abs(float(e1) - float(e0)) <= 1e-12 * abs(float(e0))
    for k in G.KEYS:
        assert _relerr(g[k].cpu().numpy(), g0[k].cpu().numpy()) < 1e-10, k


# The mixed modes' items of up to 32 elements (nocc 14 on: the rule's number of items), in calls that also
# hold larger ones (nvir 17, 19, 23), with the parity bounds of these modes against FP64.
@pytest.mark.gpu
@pytest.mark.parametrize("o,v,tv", [(13, 7, 0), (14, 7, 0), (14, 1, 0), (15, 19, 0), (16, 23, 0), (14, 9, 2), (20, 6, 1)])
@pytest.mark.parametrize("precision", ["mixed", "mixed_bf16"])
def test_mixed_short_ranges(o, v, tv, precision):
    inp = make_inputs(o, v, 40, seed=v, fvo_sigma=1e-3)
    ins = [getattr(inp, k) for k in G.KEYS]
    e0, g0 = triples.energy_vjp(*ins, precision="fp64", device="cuda", block_size=tv)
    e, g = triples.energy_vjp(*ins, precision=precision, device="cuda", block_size=tv)
    e1 = triples.energy(*ins, precision=precision, device="cuda", block_size=tv)
    e_tol, g_tol = (1e-6, 1e-5) if precision == "mixed" else (1e-4, 1e-3)
    scale = 1e-14 if v == 1 else 0.0   # one virtual orbital has no triples: both are rounding noise
    assert abs(float(e) - float(e0)) <= e_tol * abs(float(e0)) + scale
    assert abs(float(e1) - float(e0)) <= e_tol * abs(float(e0)) + scale
    if v > 1:
        for k in G.KEYS:
            assert _relerr(g[k].cpu().numpy(), g0[k].cpu().numpy()) < g_tol, k


# An item of up to 32 elements (64 without the adjoint) gives the same FP32 values in its element kernel as
# in the persistent epilogue, which the batch engine uses for every chunk (nvir below 13: no item of three
# distinct full ranges, whose FP32 sums a batch orders in its own way; two ranges of 8 at nvir 9 and
# 12); only FP64 sums are ordered differently.
@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["mixed", "mixed_bf16"])
def test_mixed_short_ranges_have_the_values_of_the_persistent_epilogue(precision):
    from pyscfad_b200.batched import BatchedTriples

    problems = []
    for o, v in ((14, 2), (14, 3), (15, 5), (16, 7), (17, 6), (20, 1), (14, 9), (15, 12)):
        inp = make_inputs(o, v, 40, seed=o + v, fvo_sigma=1e-3)
        problems.append({k: getattr(inp, k) for k in G.KEYS})
    batch = BatchedTriples(problems, precision=precision, engine="batch", tune=False)
    batch.run()
    for prob, (e0, g0) in zip(problems, batch.results()):
        e, g = triples.energy_vjp(*(prob[k] for k in G.KEYS), precision=precision, device="cuda")
        if prob["t1"].shape[1] == 1:
            continue   # one virtual orbital has no triples: both are rounding noise
        e1 = triples.energy(*(prob[k] for k in G.KEYS), precision=precision, device="cuda")
        assert abs(float(e) - e0) <= 1e-12 * abs(e0)
        assert abs(float(e1) - e0) <= 1e-12 * abs(e0)
        for k in G.KEYS:
            assert _relerr(g[k].cpu().numpy(), g0[k].cpu().numpy()) < 1e-11, k


# Host threads with different nocc share the projection kernel of their range; each call must find the shared
# memory that it asks for, whatever another thread is launching.
@pytest.mark.gpu
def test_lno_calls_of_host_threads_do_not_disturb_each_other():
    from concurrent.futures import ThreadPoolExecutor

    sizes = (9, 10, 12, 14, 16, 9, 13, 16)
    problems = []
    for t, o in enumerate(sizes):
        inp = make_inputs(o, 3, 20, seed=t, fvo_sigma=1e-3)
        ins = [torch.as_tensor(np.ascontiguousarray(getattr(inp, k)), device="cuda") for k in G.KEYS]
        problems.append((torch.eye(o, dtype=torch.float64, device="cuda"), ins, torch.cuda.Stream()))
    e_ref = [float(triples.lno_energy(m, *ins)) for m, ins, _ in problems]
    torch.cuda.synchronize()

    def work(t):
        m, ins, st = problems[t]
        with torch.cuda.stream(st):
            return [float(triples.lno_energy(m, *ins)) for _ in range(300)]

    with ThreadPoolExecutor(len(sizes)) as pool:
        results = list(pool.map(work, range(len(sizes))))
    for t in range(len(sizes)):
        assert max(abs(e - e_ref[t]) for e in results[t]) <= 1e-12 * abs(e_ref[t])
