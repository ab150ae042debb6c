"""Device memory that suffices for a call's needs but not for its optional
scratch (chunk groups, V-term tables): the call runs all the same."""
import numpy as np
import pytest
import torch

from pyscfad_b200 import _lib, triples
from pyscfad_b200.synthetic import make_inputs
from tests import golden_util as G


class _Stream:
    cuda_stream = 0


@pytest.fixture
def room(monkeypatch):
    """Host buffers in place of device scratch, of at most room[0] bytes at once."""
    limit, log = [1 << 60], []

    def alloc(nbytes, device, stream):
        log.append(nbytes)
        if nbytes + sum(b.numel() for b in triples._workspaces.values()) > limit[0]:
            raise torch.cuda.OutOfMemoryError("no room")
        return torch.empty(nbytes, dtype=torch.uint8)

    triples.release_workspace()
    monkeypatch.setattr(triples, "_alloc", alloc)
    yield limit, log
    triples.release_workspace()


def test_scratch_falls_back_to_what_the_call_needs(room):
    limit, log = room
    cpu = torch.device("cpu")
    assert triples._workspace(1000, cpu, _Stream, 500, 900).numel() == 1500
    assert triples._workspace(1000, cpu, _Stream, 500, 900).numel() == 1500    # kept
    triples.release_workspace()
    limit[0] = 1200
    assert triples._workspace(1000, cpu, _Stream, 500, 900).numel() == 1000
    triples.release_workspace()
    limit[0] = 950
    assert triples._workspace(1000, cpu, _Stream, 500, 900).numel() == 900
    del log[:]
    assert triples._workspace(1000, cpu, _Stream, 500, 900).numel() == 900     # no further attempt at more
    assert log == []
    triples.release_workspace()
    limit[0] = 800
    with pytest.raises(torch.cuda.OutOfMemoryError):
        triples._workspace(1000, cpu, _Stream, 500, 900)
    assert triples._workspaces == {}


def test_outputs_get_the_room_of_the_optional_scratch(room):
    """An allocation beside the scratch that fails: the scratch is given back and the call tried once more."""
    cpu, tries = torch.device("cpu", 0), []

    def call(device, t1):
        ws = triples._workspace(1000, cpu, _Stream, 500, 900)
        tries.append(ws.numel())
        if ws.numel() > 900:
            raise torch.cuda.OutOfMemoryError("no room for the outputs")
        return "done"

    assert triples._with_room(call, cpu, None) == "done" and tries == [1500, 1000, 900]
    # nothing optional left to give back: the error reaches the caller

    def never(device, t1):
        raise torch.cuda.OutOfMemoryError("no room")

    with pytest.raises(torch.cuda.OutOfMemoryError):
        triples._with_room(never, cpu, None)


def test_scratch_of_captured_calls_stays(room):
    """A recorded graph holds its scratch's address: it is not given back for another stream's sake."""
    cpu = torch.device("cpu", 0)

    class Other:
        cuda_stream = 1

    kept = triples._workspace(1000, cpu, _Stream, 500, 900)
    triples._captured.add(triples._key(cpu, _Stream))
    triples._workspace(1000, cpu, Other, 500, 900)
    assert triples._give_back(cpu)
    assert list(triples._workspaces.values()) == [kept] and triples._workspaces[triples._key(cpu, _Stream)] is kept
    assert not triples._give_back(cpu)


@pytest.mark.parametrize("o,v", [(5, 19), (20, 180), (40, 360), (50, 450)])
def test_least_scratch_is_without_the_tables(o, v):
    lib = _lib.load()
    for grad in (0, 1):
        least, size = (lib.triples_workspace_least(1, o, v, 1, grad, None), lib.triples_workspace_size(1, o, v, 1, grad))
        nb = (v + 7) // 8
        tables = o * o * nb * nb * 64 * 8 + o * nb * 8 * 8
        assert size - 512 <= least + tables <= size + 512
        assert lib.triples_workspace_least(0, o, v, 1, grad, None) == lib.triples_workspace_size(0, o, v, 1, grad)
    arr = (_lib.Problem * 2)()
    for q in arr:
        q.nocc, q.nvir, q.ovvv_packed = o, v, 1
    for prec in (0, 1):
        n = lib.triples_batch_workspace_size(prec, 2, arr) - lib.triples_batch_workspace_least(prec, 2, arr)
        assert n == 2 * (lib.triples_workspace_size(prec, o, v, 1, 1) - lib.triples_workspace_least(prec, o, v, 1, 1, None))


@pytest.mark.gpu
def test_captured_call_is_noted_and_replays():
    inp = make_inputs(4, 20, 30, seed=3, fvo_sigma=1e-3)
    ins = [torch.as_tensor(np.ascontiguousarray(getattr(inp, k)), device="cuda") for k in G.KEYS]
    e0, g0 = triples.energy_vjp(*ins, precision="mixed")
    triples.release_workspace()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        e, g = triples.energy_vjp(*ins, precision="mixed", check=False)
    assert len(triples._captured) == 1 and triples._captured <= set(triples._workspaces)
    assert not triples._give_back(torch.device("cuda"))
    graph.replay()
    torch.cuda.synchronize()
    assert abs(float(e) - float(e0)) <= 1e-12 * abs(float(e0))
    for k in G.KEYS:
        ref = g0[k].cpu().numpy()
        assert float(np.abs(g[k].cpu().numpy() - ref).max()) <= 1e-11 * max(float(np.abs(ref).max()), 1e-7), k
    triples.release_workspace()


@pytest.mark.gpu
@pytest.mark.parametrize("entry", ["ovvv", "df"])
def test_call_fits_where_the_optional_scratch_does_not(entry):
    """Torch's allocator limited to the inputs, the outputs and the needed scratch (as a full device
    would be), on a first call and on one that finds larger scratch cached."""
    o, v, naux = 14, 150, 40
    inp = make_inputs(o, v, naux, seed=1, fvo_sigma=1e-3)
    if entry == "ovvv":
        ins = {k: torch.as_tensor(np.ascontiguousarray(getattr(inp, k)), device="cuda") for k in G.KEYS}
        ins["ovvv"] = torch.as_tensor(inp.ovvv_tril(), device="cuda")
        call, own = triples.energy_vjp, 0
    else:
        ins = {k: torch.as_tensor(np.ascontiguousarray(getattr(inp, k)), device="cuda") for k in G.KEYS if k != "ovvv"}
        ins["Lov"] = torch.randn(naux, o * v, dtype=torch.float64, device="cuda") * 0.01
        ins["Lvv"] = torch.randn(naux, v * (v + 1) // 2, dtype=torch.float64, device="cuda") * 0.01
        call, own = triples.energy_vjp_df, 2 * 8 * o * v * v * (v + 1) // 2
    lib = _lib.load()
    least = lib.triples_workspace_least(1, o, v, 1, 1, None) + own
    assert lib.triples_workspace_extra(1, o, v, 1, 1, None) > 300 << 20
    e0, g0 = call(**ins, precision="mixed", device="cuda")
    g0 = {k: t.cpu() for k, t in g0.items()}
    outputs = sum(t.numel() * 8 for t in ins.values())
    triples.release_workspace()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    limit = torch.cuda.memory_reserved() + outputs + least + (100 << 20)   # (rounding of the allocator's blocks)
    try:
        for cached in (False, True):
            triples.release_workspace()
            torch.cuda.empty_cache()
            if cached:   # scratch of an earlier call, as large as the limit lets it be
                st = torch.cuda.current_stream()
                triples._workspaces[("cuda", None, int(st.cuda_stream))] = torch.empty(
                    least + (80 << 20) + outputs // 2, dtype=torch.uint8, device="cuda")
            torch.cuda.set_per_process_memory_fraction(limit / total)
            e, g = call(**ins, precision="mixed", device="cuda")
            assert abs(float(e) - float(e0)) <= 1e-12 * abs(float(e0))
            for k in g0:
                ref = g0[k].numpy()
                assert float(np.abs(g[k].cpu().numpy() - ref).max()) <= 1e-10 * max(float(np.abs(ref).max()), 1e-7), k
            del e, g
            torch.cuda.set_per_process_memory_fraction(1.0)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
        triples.release_workspace()
