"""Kernels at the sizes where their tiling can go wrong (remainders, one-chunk grids, smallest and largest of a range),
against the CPU oracle."""
import pytest
import torch

from oracle import nsa_oracle as O
from tests.test_gpu_tensorcore import DEV, _grad_close, _inputs, _no_timeouts, _random_indices
from tests.util import max_abs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dk,dv,H,G,T,n", [(64, 64, 8, 2, 64, 1), (64, 64, 8, 1, 192, 3), (128, 128, 16, 1, 320, 17),
                                           (64, 64, 4, 1, 2112, 32), (192, 128, 16, 1, 448, 16)])
def test_selection_over_ragged_chunks_and_short_ranges(dk, dv, H, G, T, n):
    """Query counts that leave a partial 128-query chunk of the inverse index, slot counts that are no power of two, index
    ranges of a few entries per CTA; ids repeat and rows have holes."""
    from nsa import ops
    q, k, v, do = _inputs(2, H, G, T, dk, dv, seed=T + n)
    gen = torch.Generator().manual_seed(n)
    idx = _random_indices(2, G, T, max(n, 4), 64, gen)[..., :n].contiguous()
    idx[:, :, ::3, -1] = idx[:, :, ::3, 0]             # a repeated id counts once
    scale = dk ** -0.5
    d = lambda t: t.to(DEV)
    o, L, M = ops.slc_fwd(d(q), d(k), d(v), d(idx), 64, scale)
    dq, dkey, dval = ops.slc_bwd(d(q), d(k), d(v), d(idx), o, d(do), L, M, 64, scale)
    torch.cuda.synchronize()
    _no_timeouts()
    qf, kf, vf = (t.float().requires_grad_(True) for t in (q, k, v))
    ref = O.selection_attention(qf, kf, vf, idx, 64, scale)
    gq, gk, gv = torch.autograd.grad(ref, (qf, kf, vf), do.float())
    assert max_abs(o.float(), ref) < 2e-2
    _grad_close(dq, gq, "dq")
    _grad_close(dkey, gk.transpose(-1, -2), "dk")
    _grad_close(dval, gv, "dv")
