"""Scratch that a problem's call gets in a lane and in the tuner."""
import torch

from pyscfad_b200 import _lib, batched


class _Recorder:
    """The library with the workspace bytes of every E + VJP call noted instead of the call made."""

    def __init__(self):
        self.real, self.bytes = _lib.load(), []

    def __getattr__(self, name):
        return getattr(self.real, name)

    def triples_energy_vjp_ex(self, *args):
        self.bytes.append(args[16])
        return 0


class _Stream:
    cuda_stream = 0


def _problem(o, v):
    ins = [torch.zeros(1, dtype=torch.float64) for _ in batched.KEYS]
    return batched._Problem(o, v, True, ins, dict(zip(batched.KEYS, ins)), torch.zeros(()))


def test_a_call_gets_the_same_scratch_whatever_else_shares_it():
    """The scratch decides how many chunks run in one launch: a candidate must be timed with the scratch
    that its lane will give it, not with that of the largest problem or candidate."""
    lib = _Recorder()
    for prec in (0, 1, 2):
        for o, v in ((5, 40), (8, 61), (12, 30)):
            prob = _problem(o, v)
            for tv in batched.TV_CANDIDATES:
                need, own = batched._scratch(lib, prec, prob, tv)
                assert lib.real.triples_workspace_size_ex(prec, o, v, 1, 1, _lib.options(tv)) == need <= own
                del lib.bytes[:]
                for size in (own, 2 * own, own + (3 << 30)):
                    batched._call(lib, prec, prob, torch.empty(size, dtype=torch.uint8, device="meta"), _Stream, tv)
                assert lib.bytes == [own] * 3
                batched._call(lib, prec, prob, torch.empty(need, dtype=torch.uint8, device="meta"), _Stream, tv)
                assert lib.bytes[-1] == need
