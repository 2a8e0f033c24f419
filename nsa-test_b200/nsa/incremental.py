"""Incremental (prefill-in-chunks / decode) forward of the NSA layer against a key/value cache.

The reference has no incremental path (its module accepts and ignores ``attention_mask``,
nsa/kernels.py:2213, and always recomputes the whole sequence); this is the same layer arithmetic
(nsa/kernels.py:2298-2463) evaluated for the newest query rows only, so that the rows it returns equal the
corresponding rows of the full-sequence forward.  Forward only, no autograd.

``NSACache`` keeps, per layer, the three key/value streams of the module (selection, sliding window and the
source of the compression), zero-padded to a fixed capacity, and the compressed keys/values, which grow by
one block every ``d`` tokens once ``l`` tokens are there.  ``nsa_layer_incremental`` runs the scoring/top-n,
the three branches and the gate mix for the new rows with a query position offset, for bf16 calls in one library
call:

* up to 64 (sequence, group, token) rows on the decode kernels (``nsa_decode_fwd``; ``module_forward_incremental``
  hands it the hidden states of up to eight tokens, whose projections and cache update then run in the same call);
* more rows on the layer's own tile kernels, which read the caches where they lie (``nsa_incremental_fwd``).

Everything else (other types, head dims or block sizes) is composed here from the branch entry points, on new rows
padded to a 128-row tile and key slices copied out of the cache.  Both one-call forms choose the blocks that this
composition chooses for the same rows, bit for bit: the choice is made from the same products and sums in the same order.
"""
from __future__ import annotations

import math
from typing import Optional

import torch

from . import _lib, ops
from .kernels import (NSAConfig, PAD_BLOCK_END, _PhiCompress, _next_pow2, _project_heads, _selection_fallback,
                      gate_logits_from_hidden)

__all__ = ["NSACache", "nsa_layer_incremental", "module_forward_incremental"]

_TILE = 128
_FEW_ROWS = 64       # (sequence, group, row) count up to which scoring takes the unpadded rows
_PLAIN = (torch.Tensor, torch.nn.Parameter)


def _round_up(x: int, m: int) -> int:
    return (x + m - 1) // m * m


class NSACache:
    """Key/value cache of one NSA layer for ``batch`` sequences of up to ``capacity`` tokens.

    Layouts are the kernels' own: keys ``[B,G,dk,capacity]``, values ``[B,G,capacity,dv]`` (zeros beyond
    ``length``), compressed keys fp32 ``[B,G,dk,nbp]`` (+ a copy in the compute dtype for the compressed
    attention) and compressed values ``[B,G,nbp,dv]`` with ``n_blocks`` valid blocks.
    """

    def __init__(self, config: NSAConfig, batch: int, capacity: int, device, dtype=torch.bfloat16,
                 shared_kv: bool = False):
        c = config
        self.config, self.dtype, self.shared_kv = c, dtype, shared_kv
        self.capacity = _round_up(capacity, _TILE)
        G, dk, dv = c.n_kv_groups, c.head_dim_qk, c.head_dim_v

        def kv():
            return (torch.zeros(batch, G, dk, self.capacity, device=device, dtype=dtype),
                    torch.zeros(batch, G, self.capacity, dv, device=device, dtype=dtype))

        self.k_slc, self.v_slc = kv()
        (self.k_win, self.v_win) = (self.k_slc, self.v_slc) if shared_kv else kv()
        (self.k_src, self.v_src) = (self.k_slc, self.v_slc) if shared_kv else kv()
        nb_cap = max((self.capacity - c.l) // c.d + 1, 1)
        self.nbp = max(_next_pow2(nb_cap), _TILE)
        self.k_cmp = torch.zeros(batch, G, dk, self.nbp, device=device, dtype=torch.float32)
        self.k_cmp_lp = torch.zeros(batch, G, dk, self.nbp, device=device, dtype=dtype)
        self.v_cmp = torch.zeros(batch, G, self.nbp, dv, device=device, dtype=dtype)
        self.block_ends = torch.full((self.nbp,), PAD_BLOCK_END, device=device, dtype=torch.int32)
        self.length = 0
        self.n_blocks = 0

    @torch.no_grad()
    def append(self, phi_params, k_slc, v_slc, kv_compress=None, kv_sliding=None) -> int:
        """Add ``Tn`` tokens: k_* ``[B,G,dk,Tn]``, v_* ``[B,G,Tn,dv]`` (one pair feeds all branches unless the
        cache was built with separate streams).  Compresses the blocks the new tokens complete.  Returns the
        position of the first new token."""
        c = self.config
        Tn = k_slc.shape[-1]
        p0, p1 = self.length, self.length + Tn
        if p1 > self.capacity:
            raise ValueError(f"NSACache: {p1} tokens exceed the capacity {self.capacity}")
        if not self.shared_kv and (kv_compress is None or kv_sliding is None):
            raise ValueError("NSACache: built with separate streams, kv_compress and kv_sliding are required")
        nb_new = (p1 - c.l) // c.d + 1 if p1 >= c.l else 0
        tensors = (k_slc, v_slc) if self.shared_kv else (k_slc, v_slc, *kv_compress, *kv_sliding)
        if not self._append_in_place(phi_params, tensors, p0, Tn, max(nb_new, self.n_blocks)):
            self._append_by_copies(phi_params, k_slc, v_slc, kv_compress, kv_sliding, p0, p1, nb_new)
        self.length, self.n_blocks = p1, max(nb_new, self.n_blocks)
        return p0

    def _append_in_place(self, phi_params, tensors, p0: int, Tn: int, nb: int) -> bool:
        """The append as one library call; False where a tensor is not of the cache's type, shape and CUDA device."""
        c, dev = self.config, self.k_slc.device
        if dev.type != "cuda":
            return False
        B = self.k_slc.shape[0]
        for i, t in enumerate(tensors):
            want = (B, c.n_kv_groups, c.head_dim_qk, Tn) if i % 2 == 0 else (B, c.n_kv_groups, Tn, c.head_dim_v)
            if type(t) not in _PLAIN or t.shape != want or t.dtype != self.dtype or t.device != dev:
                return False
        pe, w1, b1, w2, b2 = phi_params
        U, dk, pdt = w1.shape[0], c.head_dim_qk, w1.dtype
        for t, n in ((pe, c.l * c.l), (w1, U * (dk + c.l)), (b1, U), (w2, dk * U), (b2, dk)):
            if t is not None and (type(t) not in _PLAIN or t.dtype != pdt or t.numel() != n or t.device != dev or not t.is_contiguous()):
                return False
        if Tn == 0 or self.dtype not in (torch.float32, torch.bfloat16) or pdt not in (torch.float32, torch.bfloat16):
            return False
        if B * c.n_kv_groups * len(tensors) > 65535:
            return False
        d = _cache_desc(self, B, Tn, p0, nb)
        if d is None:
            return False
        d.nb_new, d.U = nb - self.n_blocks, U
        ops.cache_append(d, tensors, phi_params)
        return True

    def _append_by_copies(self, phi_params, k_slc, v_slc, kv_compress, kv_sliding, p0: int, p1: int, nb_new: int) -> None:
        c = self.config
        self.k_slc[..., p0:p1] = k_slc
        self.v_slc[:, :, p0:p1] = v_slc
        if not self.shared_kv:
            self.k_src[..., p0:p1], self.v_src[:, :, p0:p1] = kv_compress[0], kv_compress[1]
            self.k_win[..., p0:p1], self.v_win[:, :, p0:p1] = kv_sliding[0], kv_sliding[1]
        if nb_new > self.n_blocks:
            b0, cnt = self.n_blocks, nb_new - self.n_blocks
            lo, hi = b0 * c.d, (nb_new - 1) * c.d + c.l
            keys = self.k_src[..., lo:hi].transpose(-1, -2).contiguous()
            vals = self.v_src[:, :, lo:hi].contiguous()
            kc, vc = _PhiCompress.apply(keys, vals, *phi_params, c.l, c.d)
            self.k_cmp[..., b0:nb_new] = kc[..., :cnt]
            self.k_cmp_lp[..., b0:nb_new] = kc[..., :cnt].to(self.dtype)
            self.v_cmp[:, :, b0:nb_new] = vc[:, :, :cnt].to(self.dtype)
            self.block_ends[b0:nb_new] = (torch.arange(b0, nb_new, device=self.block_ends.device, dtype=torch.int32)
                                          * c.d + (c.l - 1))


def _cache_desc(cache: NSACache, B: int, Tn: int, pos: int, nb: int, scale: float = 0.0):
    """Descriptor of ``Tn`` tokens at ``pos`` of ``cache`` with ``nb`` valid compressed blocks for the library's entry points, or
    None when the cache's tensors are not laid out as those read and write them."""
    c = cache.config
    H, G, dk, dv, cap, nbp = c.n_heads, c.n_kv_groups, c.head_dim_qk, c.head_dim_v, cache.capacity, cache.nbp
    dev, dt = cache.k_slc.device, cache.dtype
    for t, n, want in ((cache.k_slc, dk * cap, dt), (cache.v_slc, dv * cap, dt), (cache.k_win, dk * cap, dt), (cache.v_win, dv * cap, dt),
                       (cache.k_src, dk * cap, dt), (cache.v_src, dv * cap, dt), (cache.k_cmp, dk * nbp, torch.float32),
                       (cache.k_cmp_lp, dk * nbp, dt), (cache.v_cmp, dv * nbp, dt)):
        if t.numel() != B * G * n or t.dtype != want or t.device != dev or not t.is_contiguous() or t.data_ptr() % 16:
            return None
    if cache.block_ends.numel() != nbp or cache.block_ends.dtype != torch.int32 or cache.block_ends.device != dev:
        return None
    return _lib.DecodeDesc(B=B, Tn=Tn, H=H, G=G, dk=dk, dv=dv, l=c.l, d=c.d, l_prime=c.l_prime, n=c.n,
                           n_fixed=c.n_fixed if c.include_fixed_in_selection else 0, window=c.w,
                           gate_mode=_lib.GATE_SOFTMAX if c.gate_mode == "softmax" else _lib.GATE_SIGMOID, pos=pos, nb=nb, cap=cap,
                           nbp=nbp, scale=scale, k_slc=cache.k_slc.data_ptr(), v_slc=cache.v_slc.data_ptr(),
                           k_src=cache.k_src.data_ptr(), v_src=cache.v_src.data_ptr(), k_win=cache.k_win.data_ptr(),
                           v_win=cache.v_win.data_ptr(), k_cmp=cache.k_cmp.data_ptr(), k_cmp_lp=cache.k_cmp_lp.data_ptr(),
                           v_cmp=cache.v_cmp.data_ptr(), block_ends=cache.block_ends.data_ptr())


def _layer_rows(q: torch.Tensor, gate_logits: torch.Tensor, cache: NSACache, scale: float, return_info: bool):
    """``nsa_layer_incremental`` in one library call: the decode kernels for a handful of rows, the tile kernels with a query
    offset for more; None where neither applies."""
    B, H, Tn, dk = q.shape
    dv, dev = cache.config.head_dim_v, q.device
    if (q.dtype != torch.bfloat16 or cache.dtype != torch.bfloat16 or dev != cache.k_slc.device or H != cache.config.n_heads
            or dk != cache.config.head_dim_qk or gate_logits.shape != (B, Tn, 3 * H) or gate_logits.device != dev):
        return None
    d = _cache_desc(cache, B, Tn, cache.length - Tn, cache.n_blocks, scale)
    if d is None:
        return None
    few = bool(_lib.lib.nsa_decode_supported(d))
    if not few and not _lib.lib.nsa_incremental_supported(d):
        return None
    if q.data_ptr() % 16 or (q.stride(3) != 1 or any(q.stride(i) % 8 for i in range(3)) if few else not q.is_contiguous()):
        q = q.clone(memory_format=torch.contiguous_format)
    lg = gate_logits.float().contiguous()
    out = torch.empty(B, Tn, H, dv, device=dev, dtype=q.dtype)
    d.q, d.gate_logits, d.out = q.data_ptr(), lg.data_ptr(), out.data_ptr()
    d.sq = q.stride()[:3] if few else (H * Tn * dk, Tn * dk, dk)
    info = None
    if return_info:
        o = lambda: torch.empty(B, H, Tn, dv, device=dev, dtype=q.dtype)
        info = dict(indices=torch.empty(B, cache.config.n_kv_groups, Tn, cache.config.n, device=dev, dtype=torch.int32),
                    gates=torch.empty(B, H, Tn, 3, device=dev, dtype=torch.float32), o_cmp=o(), o_slc=o(), o_win=o())
        for name, t in info.items():
            setattr(d, name, t.data_ptr())
    (ops.decode_fwd if few else ops.incremental_fwd)(d, dev)
    out = out.transpose(1, 2)
    return (out, info) if return_info else out


def _decode_module(module, x: torch.Tensor, cache: NSACache):
    """``module_forward_incremental`` up to the output projection for at most eight tokens in one library call: mixed output
    [B,Tn,H*dv], or None where its kernels do not apply (other types or sizes, too short a cache, autocast, tensor
    subclasses).  The same products, roundings and cache contents as the general path."""
    c = module.config
    if x.dim() != 3 or type(x) not in _PLAIN or x.dtype != torch.bfloat16 or cache.shared_kv or cache.config != c:
        return None
    B, Tn, dm = x.shape
    p1 = cache.length + Tn
    dev = x.device
    if (B * Tn > 8 or Tn == 0 or p1 > cache.capacity or p1 < c.l or dm != c.d_model or dev != cache.k_slc.device
            or cache.dtype != torch.bfloat16 or torch.is_autocast_enabled("cuda") or x.stride(2) != 1 or x.stride(0) % 8
            or x.stride(1) % 8 or x.data_ptr() % 16):
        return None
    nb = (p1 - c.l) // c.d + 1
    G, dk, dv, H = c.n_kv_groups, c.head_dim_qk, c.head_dim_v, c.n_heads
    d = _cache_desc(cache, B, Tn, cache.length, nb, module.scale)
    if d is None:
        return None
    lins = (module.k_select, module.v_select, module.v_compress, module.k_sliding, module.v_sliding)
    g0, g2 = module.gate_mlp[0], module.gate_mlp[2]
    pe, pw1, pb1, pw2, pb2 = module._phi_params()
    D2, U = g0.weight.shape[0], pw1.shape[0]
    rows = (G * dk, G * dv, G * dv, G * dk, G * dv)
    params = [(lin.weight, r * dm) for lin, r in zip(lins, rows)] + [(lin.bias, r) for lin, r in zip(lins, rows)]
    params += [(g0.weight, D2 * dm), (g0.bias, D2), (g2.weight, 3 * H * D2), (g2.bias, 3 * H), (pe, c.l * c.l), (pw1, U * (dk + c.l)),
               (pb1, U), (pw2, dk * U), (pb2, dk)]
    ptrs = []
    for t, n in params:
        if t is None:
            ptrs.append(None)
            continue
        if type(t) not in _PLAIN or t.dtype != torch.bfloat16 or t.numel() != n or t.device != dev or not t.is_contiguous():
            return None
        ptrs.append(t.data_ptr())
    (d.gate_w1, d.gate_b1, d.gate_w2, d.gate_b2, d.pos_embed, d.phi_w1, d.phi_b1, d.phi_w2, d.phi_b2) = ptrs[10:]
    if any(p_ is None or p_ % 16 for p_ in ptrs[:5] + [d.gate_w1, d.gate_w2]) or not (d.pos_embed and d.phi_w1 and d.phi_w2):
        return None
    d.project, d.nb_new, d.d_model, d.d_gate, d.U = 1, nb - cache.n_blocks, dm, D2, U
    if not _lib.lib.nsa_decode_supported(d):
        return None
    # What the block choice depends on comes out of the library's products, as on the general path: rounded otherwise, near-ties
    # would fall the other way.  (One product for q of all sequences: for up to eight tokens it has the bits of one batched over the
    # heads per sequence, at every one of 1176 shapes tried, and reads the weights once; eight of those took 115 us a token.)
    q = torch.nn.functional.linear(x, module.q_proj.weight).view(B, Tn, H, dk)
    if module.q_proj.bias is not None:
        q = q + module.q_proj.bias.view(H, dk)
    k_new = _project_heads(x, module.k_compress, G, dk, transposed=True)
    if any(type(t) not in _PLAIN or t.dtype != torch.bfloat16 or t.device != dev for t in (q, k_new)):
        return None
    out = torch.empty(B, Tn, H * dv, device=dev, dtype=x.dtype)
    d.q, d.sq, d.k_new, d.sk = q.data_ptr(), (q.stride(0), q.stride(2), q.stride(1)), k_new.data_ptr(), k_new.stride()
    d.x, d.sx, d.out = x.data_ptr(), x.stride()[:2], out.data_ptr()
    d.w, d.bias = tuple(ptrs[:5]), tuple(ptrs[5:10])
    ops.decode_fwd(d, dev)
    cache.length, cache.n_blocks = p1, nb
    return out


def _pad_rows(x: torch.Tensor, dim: int, rows: int) -> torch.Tensor:
    have = x.shape[dim]
    if have == rows:
        return x.contiguous()
    shape = list(x.shape)
    shape[dim] = rows - have
    return torch.cat([x, x.new_zeros(shape)], dim=dim)


@torch.no_grad()
def nsa_layer_incremental(q_new: torch.Tensor, gate_logits_new: torch.Tensor, cache: NSACache,
                          scale: Optional[float] = None, return_info: bool = False):
    """Output rows ``[B,H,Tn,dv]`` of the NSA layer for the ``Tn`` newest tokens of ``cache`` (the keys/values
    of these tokens must have been appended already).  q_new ``[B,H,Tn,dk]``, gate_logits_new ``[B,Tn,3H]``.

    Row r is the query at position ``cache.length - Tn + r`` and sees exactly what the full-sequence forward
    shows it: the compressed blocks that end at or before it, its top-n selected blocks (causally clipped)
    and the last ``w`` keys.
    """
    c = cache.config
    B, H, Tn, dk = q_new.shape
    pos = cache.length - Tn
    if pos < 0:
        raise ValueError("nsa_layer_incremental: more query rows than cached tokens")
    if cache.n_blocks == 0:
        # The full-sequence layer lets rows without a visible compressed block attend block 0; before that
        # block exists there is nothing to reproduce, so the first chunk has to bring at least l tokens.
        raise ValueError(f"nsa_layer_incremental: the cache needs at least l={c.l} tokens")
    scale = 1.0 / math.sqrt(dk) if scale is None else scale
    if Tn > 0:
        res = _layer_rows(q_new, gate_logits_new, cache, scale, return_info)
        if res is not None:
            return res
    rows = _round_up(Tn, _TILE)
    q = _pad_rows(q_new, 2, rows)
    n_fixed = c.n_fixed if c.include_fixed_in_selection else 0
    nb = cache.n_blocks

    G = c.n_kv_groups
    blocks = (c.l, c.d, nb)
    if Tn < rows and B * G * Tn <= _FEW_ROWS:
        # A handful of rows (decode): the tile kernel would run one CTA per (sequence, group) over all compressed
        # blocks; unpadded rows take the generic scoring path, whose q.k products spread over the whole GPU.
        real = ops.score_topn(q_new.contiguous(), cache.k_cmp, cache.block_ends, c.l, c.d, c.l_prime, c.n, n_fixed, scale,
                              nb, pos)
        indices = torch.cat([real, real.new_full((B, G, rows - Tn, c.n), -1)], dim=2)
        o_cmp, _, _ = ops.cmp_attn_fwd(q, cache.k_cmp_lp, cache.v_cmp, cache.block_ends, scale, blocks, pos)
    elif ops.cmp_exact_supported(q, cache.k_cmp_lp, cache.v_cmp):
        # as the full-sequence layer does it: the compressed attention runs on the fp32 keys (as bf16 hi + lo halves)
        # and hands its log-sum-exp to the scoring kernel, so the two agree on every row, near-ties included
        hi, lo = ops.split_keys(cache.k_cmp)
        o_cmp, _, _, lse2 = ops.cmp_attn_fwd(q, hi, cache.v_cmp, cache.block_ends, scale, blocks, pos, k_lo=lo)
        indices = ops.score_topn(q, cache.k_cmp, cache.block_ends, c.l, c.d, c.l_prime, c.n, n_fixed, scale, nb, pos,
                                 cmp_lse2=lse2)
    else:
        indices = ops.score_topn(q, cache.k_cmp, cache.block_ends, c.l, c.d, c.l_prime, c.n, n_fixed, scale, nb, pos)
        o_cmp, _, _ = ops.cmp_attn_fwd(q, cache.k_cmp_lp, cache.v_cmp, cache.block_ends, scale, blocks, pos)
    idx = _selection_fallback(indices, c.l_prime, pos).to(torch.int32).contiguous()
    o_slc, _, _ = ops.slc_fwd(q, cache.k_slc, cache.v_slc, idx, c.l_prime, scale, pos)

    # Sliding window: the window reaches w - 1 positions back, so the dense kernel runs on the key slice that
    # starts at a tile boundary at or before pos - (w - 1); the query rows sit at their offset inside it.
    lo = max(0, (pos - (c.w - 1)) // _TILE * _TILE)
    span = _round_up(pos - lo + Tn, _TILE)
    qw = q_new.new_zeros(B, H, span, dk)
    qw[:, :, pos - lo:pos - lo + Tn] = q_new
    ks = cache.k_win[..., lo:lo + span].contiguous()
    vs = cache.v_win[:, :, lo:lo + span].contiguous()
    o_win, _, _ = ops.sliding_fwd(qw, ks, vs, c.w, scale)
    o_win = _pad_rows(o_win[:, :, pos - lo:pos - lo + Tn], 2, rows)

    out, gates = ops.gate_mix_fwd(_pad_rows(gate_logits_new, 1, rows), o_cmp, o_slc, o_win, c.gate_mode)
    out = out[:, :, :Tn]
    if return_info:
        return out, dict(indices=indices[:, :, :Tn], gates=gates[:, :, :Tn], o_cmp=o_cmp[:, :, :Tn],
                         o_slc=o_slc[:, :, :Tn], o_win=o_win[:, :, :Tn])
    return out


@torch.no_grad()
def module_forward_incremental(module, hidden_new: torch.Tensor, cache: NSACache) -> torch.Tensor:
    """``NSAAttention`` applied to the ``Tn`` newest tokens ``hidden_new [B,Tn,d_model]``: projects them, appends
    their keys/values to ``cache`` (built with ``shared_kv=False``) and returns ``[B,Tn,d_model]``, equal to the
    last ``Tn`` rows of ``module(hidden_all)[0]`` in eval mode."""
    c = module.config
    B, Tn, _ = hidden_new.shape
    H, G, dk, dv = c.n_heads, c.n_kv_groups, c.head_dim_qk, c.head_dim_v
    few = _decode_module(module, hidden_new, cache)
    if few is not None:
        return module.o_proj(few)
    q = _project_heads(hidden_new, module.q_proj, H, dk)

    def kv(kp, vp):
        return _project_heads(hidden_new, kp, G, dk, transposed=True), _project_heads(hidden_new, vp, G, dv)

    k_sel, v_sel = kv(module.k_select, module.v_select)
    cache.append(module._phi_params(), k_sel, v_sel, kv_compress=kv(module.k_compress, module.v_compress),
                 kv_sliding=kv(module.k_sliding, module.v_sliding))
    out = nsa_layer_incremental(q, gate_logits_from_hidden(hidden_new, module.gate_mlp), cache, module.scale)
    return module.o_proj(out.transpose(1, 2).reshape(B, Tn, H * dv))
