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


@pytest.mark.parametrize("T", [20, 33, 100, 129, 200, 637, 1030])
@pytest.mark.parametrize("dk,dv,H,G", [(64, 64, 4, 2), (192, 128, 16, 1)])
def test_bf16_layer_at_any_length(dk, dv, H, G, T):
    """Sequences that are no multiple of a tile, of 64 or of 8, shorter than a key tile, and with fewer compressed blocks
    than a tile holds run on the tensor-core kernels: ids, outputs and all gradients against the oracle."""
    import nsa
    from nsa import _lib
    from nsa.kernels import nsa_layer
    from tests.util import check_layer_against_oracle
    c = dict(B=2, H=H, G=G, T=T, dk=dk, dv=dv, d_model=64, l=32, d=16, l_prime=64, n=16, w=150)
    inp = O.make_inputs(2, H, G, T, dk, dv, 64, 32, seed=T, block_offset_std=0.5, dtype=torch.bfloat16)
    check_layer_against_oracle(f"bf16 layer dk={dk} T={T}", nsa, c, inp, torch.bfloat16)
    _no_timeouts()
    if T >= 32:
        cfg = nsa.NSAConfig(d_model=64, head_dim_qk=dk, head_dim_v=dv, n_heads=H, n_kv_groups=G, w=150)
        q, k, v = (inp[x].to(DEV, torch.bfloat16).requires_grad_(True) for x in ("q", "k", "v"))
        phi = tuple(getattr(inp["phi"], n_).to(DEV) for n_ in ("pos_embed", "w1", "b1", "w2", "b2"))
        logits = torch.zeros(2, T, 3 * H, device=DEV)
        ran = _lib.profile_kernels(lambda: torch.autograd.grad(nsa_layer(q, k, v, logits, phi, cfg).sum(), (q, k, v)))
        assert {"fa_fwd_win", "fa_fwd_cmp_exact", "slc_bwd_fused", "fa_bwd_dkv_cmp", "fa_bwd_dqds_win"} <= set(ran), ran


@pytest.mark.parametrize("Tk,lo", [(384, 128), (200, 72)])
def test_keys_and_values_read_as_slices_of_a_longer_buffer(Tk, lo):
    """Keys with padded rows and time slices of a longer key/value buffer are read where they lie."""
    from nsa import ops
    B, H, G, dk, dv = 2, 4, 2, 64, 64
    q, _, _, _ = _inputs(B, H, G, Tk, dk, dv, seed=3)
    _, k, v, _ = _inputs(B, H, G, 1024, dk, dv, seed=4)
    ks, vs = k[..., lo:lo + Tk], v[:, :, lo:lo + Tk]
    o, L, M = ops.sliding_fwd(q.to(DEV), k.to(DEV)[..., lo:lo + Tk], v.to(DEV)[:, :, lo:lo + Tk], 100, 0.125)
    torch.cuda.synchronize()
    _no_timeouts()
    ref = O.sliding_window_attention(q.float(), ks.float().contiguous(), vs.float().contiguous(), 100, 0.125)
    assert max_abs(o.float(), ref) < 2e-2
