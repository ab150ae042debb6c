"""A workspace off the 16-byte boundary is refused before any launch (the kernels' vectors and bulk
copies would fault on it)."""
import ctypes

import pytest
import torch

from pyscfad_b200 import _lib


# (without a device only: were a call not refused, it would go on to the made-up addresses)
@pytest.mark.skipif(torch.cuda.is_available(), reason="made-up device addresses")
@pytest.mark.parametrize("offset", [8, 4, 1])
@pytest.mark.parametrize("prec", [0, 1, 2])
def test_misaligned_workspace_is_refused(prec, offset):
    lib = _lib.load()
    p, big = ctypes.c_void_p(4096), 1 << 40
    ws = ctypes.c_void_p((1 << 20) + offset)
    assert lib.triples_energy(None, prec, 5, 19, 1, *[p] * 7, ws, big, p) == 1
    assert lib.triples_energy_vjp(None, prec, 5, 19, 1, *[p] * 7, 1.0, ws, big, p, *[p] * 7) == 1
    assert lib.triples_lno_energy(None, prec, 5, 19, 1, *[p] * 8, ws, big, p) == 1
    assert lib.triples_lno_energy_vjp(None, prec, 5, 19, 1, *[p] * 8, 1.0, ws, big, p, *[p] * 8) == 1
    assert lib.triples_energy_df(None, prec, 5, 19, 60, *[p] * 8, ws, big, p) == 1
    assert lib.triples_energy_vjp_df(None, prec, 5, 19, 60, *[p] * 8, 1.0, ws, big, p, *[p] * 8) == 1
    arr = (_lib.Problem * 1)()
    arr[0].nocc, arr[0].nvir, arr[0].ovvv_packed = 5, 19, 1
    for name, _ in _lib.Problem._fields_:
        if getattr(arr[0], name) is None:
            setattr(arr[0], name, 4096)
    handle = ctypes.c_void_p()
    assert lib.triples_batch_create(prec, 1, arr, 1.0, ws, big, ctypes.byref(handle)) == 1 and not handle.value
