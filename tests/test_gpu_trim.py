"""The device scratch that a measurement leaves in its context: kept for the next
call, given back by trim and when the context ends."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_trim():
    import torch
    from lsquantumed_gb300.build import build
    build()
    import lsquantumed_gb300 as ed
    env = ed.Environment(nspins=24)
    b = ed.Basis(env, 0)
    psi = torch.zeros(b.size, dtype=torch.complex128, device='cuda')
    psi[:7] = 1.0
    op = ed.SiSj(env, b)
    first = op.AllPairs(psi)
    torch.cuda.synchronize()
    kept = torch.cuda.mem_get_info()[0]
    env.trim()
    assert torch.cuda.mem_get_info()[0] - kept >= 8 * b.size  # the copy of the real parts, at least
    env.trim()  # nothing left to give back
    assert np.array_equal(op.AllPairs(psi), first)
