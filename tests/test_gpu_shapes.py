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


@pytest.mark.parametrize("T", [20, 100, 129, 200, 637, 1030, 2061])
@pytest.mark.parametrize("dk,dv,H,G", [(64, 64, 4, 2), (192, 128, 16, 1)])
def test_bf16_layer_at_any_length(dk, dv, H, G, T):
    """Sequences that are no multiple of a tile, of 64 or of 8, shorter than a key tile, and with fewer compressed blocks
    than a tile holds: ids, outputs and all gradients against the oracle.  From 2048 tokens on the tensor-core kernels run,
    whose probabilities are bf16; shorter ones keep fp32 probabilities."""
    import nsa
    from nsa import _lib
    from nsa.kernels import nsa_layer
    from tests.util import check_layer_against_oracle
    B = 1 if T > 2000 else 2
    c = dict(B=B, H=H, G=G, T=T, dk=dk, dv=dv, d_model=64, l=32, d=16, l_prime=64, n=16, w=150)
    inp = O.make_inputs(B, H, G, T, dk, dv, 64, 32, seed=T, block_offset_std=0.5, dtype=torch.bfloat16)
    check_layer_against_oracle(f"bf16 layer dk={dk} T={T}", nsa, c, inp, torch.bfloat16)
    _no_timeouts()
    if T >= 32:
        cfg = nsa.NSAConfig(d_model=64, head_dim_qk=dk, head_dim_v=dv, n_heads=H, n_kv_groups=G, w=150)
        q, k, v = (inp[x].to(DEV, torch.bfloat16).requires_grad_(True) for x in ("q", "k", "v"))
        phi = tuple(getattr(inp["phi"], n_).to(DEV) for n_ in ("pos_embed", "w1", "b1", "w2", "b2"))
        logits = torch.zeros(B, T, 3 * H, device=DEV)
        ran = set(_lib.profile_kernels(lambda: torch.autograd.grad(nsa_layer(q, k, v, logits, phi, cfg).sum(), (q, k, v))))
        tc = {"fa_fwd_win", "fa_fwd_cmp_exact", "slc_bwd_fused", "fa_bwd_dkv_cmp", "fa_bwd_dqds_win"}
        assert tc <= ran if T >= 2048 else not tc & ran and {"attn_fwd_mma", "attn_bwd_mma"} <= ran, ran


@pytest.mark.parametrize("Tk,lo", [(384, 128), (200, 72)])
def test_keys_and_values_read_as_slices_of_a_longer_buffer(Tk, lo):
    """Keys with padded rows and time slices of a longer key/value buffer are read where they lie."""
    from nsa import ops
    B, H, G, dk, dv = 2, 4, 2, 64, 64
    q, _, _, _ = _inputs(B, H, G, Tk, dk, dv, seed=3)
    _, k, v, _ = _inputs(B, H, G, 1024, dk, dv, seed=4)
    ks, vs = k[..., lo:lo + Tk], v[:, :, lo:lo + Tk]
    o, L, M = ops.sliding_fwd(q.to(DEV), k.to(DEV)[..., lo:lo + Tk], v.to(DEV)[:, :, lo:lo + Tk], 100, 0.125, any_length=True)
    torch.cuda.synchronize()
    _no_timeouts()
    ref = O.sliding_window_attention(q.float(), ks.float().contiguous(), vs.float().contiguous(), 100, 0.125)
    assert max_abs(o.float(), ref) < 2e-2


@pytest.mark.parametrize("dk,dv,G,B", [(192, 128, 4, 1), (192, 128, 4, 8), (128, 128, 2, 2), (64, 64, 2, 1)])
def test_appended_blocks_are_those_of_the_copies(dk, dv, G, B, monkeypatch):
    """One block at a time and many: the compressed keys rank blocks, so they are the same bit for bit on either route."""
    import nsa
    from nsa import incremental as I
    cfg = nsa.NSAConfig(d_model=64, head_dim_qk=dk, head_dim_v=dv, n_heads=G * 4, n_kv_groups=G)
    gen = torch.Generator(device=DEV).manual_seed(B)
    rn = lambda *s_: torch.randn(*s_, generator=gen, device=DEV).bfloat16()
    phi = (rn(32, 32), rn(2 * dk, dk + 32), rn(2 * dk), rn(dk, 2 * dk), rn(dk))
    a, b = (I.NSACache(cfg, B, 1200, DEV, shared_kv=True) for _ in range(2))
    for Tn in (32, 16, 1, 15, 17, 31, 48, 1, 700, 16):
        k, v = rn(B, G, dk, Tn), rn(B, G, Tn, dv)
        a.append(phi, k, v)
        with monkeypatch.context() as mp:
            mp.setattr(I.NSACache, "_append_in_place", lambda *x: False)
            b.append(phi, k, v)
    assert a.n_blocks == b.n_blocks == (877 - 32) // 16 + 1
    for name in ("k_cmp", "k_cmp_lp", "v_cmp"):
        assert torch.equal(getattr(a, name), getattr(b, name)), name


def _rows_close(got, want, tol, what):
    """Relative 2-norm of the difference, row by row."""
    got, want = got.double().cpu(), want.double().cpu()
    err = (got - want).norm(dim=-1) / want.norm(dim=-1).clamp_min(1e-6)
    assert err.max().item() < tol, (what, err.max().item())


def _exact_rows(q, k, v, see):
    """Attention of q [B,H,Tn,dk] over k [B,G,dk,N], v [B,G,N,dv] under see [B,G,Tn,N], in 64 bits on the CPU."""
    hpg = q.shape[1] // k.shape[1]
    q, k, v = (t.double().cpu() for t in (q, k, v))
    s = q @ k.repeat_interleave(hpg, 1) * q.shape[-1] ** -0.5
    s = s.masked_fill(~see.cpu().repeat_interleave(hpg, 1), float("-inf"))
    return torch.softmax(s, -1) @ v.repeat_interleave(hpg, 1)


def _peaked_module(cfg, seed):
    """Projections that keep unit variance, queries of four times that (logits of standard deviation 4: a row attends a few
    keys), compression weights that leave compressed keys of order one."""
    import nsa
    m = nsa.NSAAttention(cfg).to(DEV).bfloat16().eval()
    gen = torch.Generator(device=DEV).manual_seed(seed)
    with torch.no_grad():
        for name, p in m.named_parameters():
            std = 0.1 if p.dim() == 1 else {"q_proj.weight": 4.0, "compress_mlp.2.weight": 8.0}.get(name, 1.0) * p.shape[1] ** -0.5
            p.copy_(torch.randn(p.shape, generator=gen, device=DEV) * std)
    return m


@pytest.mark.parametrize("heads,B,cached,news,w,gate,bias,l", [
    ((8, 2, 64, 64), 3, 61, (1, 2, 1, 1, 2), 100, "softmax", True, 32),      # a chunk edge, completed blocks, several tokens
    ((16, 1, 192, 128), 1, 31, (1, 1, 8), 512, "sigmoid", False, 32),        # the first block completes with the first token
    ((32, 2, 128, 128), 8, 1999, (1, 1), 130, "sigmoid", True, 32),
    ((8, 4, 64, 64), 2, 6000, (1, 4, 3), 64, "sigmoid", False, 32),          # two heads per group; more candidates than one pass
    ((8, 2, 64, 64), 1, 700, (4, 1), 200, "sigmoid", False, 64),             # a block overlaps three others on either side
])
def test_decode_kernels_match_the_tile_kernels(monkeypatch, heads, B, cached, news, w, gate, bias, l):
    """A handful of tokens through the decode kernels against the same call through the tile kernels: the chosen blocks and what
    they are chosen from are the same bit for bit, outputs and values agree as bf16 rounds them (a row of dv outputs of the tile
    kernels is off by 2^-9 for P, for the branch outputs and for the mix, the compressed branch by 2^-9 of logits of size 4 for its
    bf16 keys: 1.5e-2 of a row's norm).  The branch outputs against 64 bits on the cache's own contents: P has 16 bits here, so the
    rounding of the outputs is left, 2^-9 of each value."""
    import nsa
    from nsa import incremental as I
    H, G, dk, dv = heads
    cfg = nsa.NSAConfig(d_model=128, head_dim_qk=dk, head_dim_v=dv, n_heads=H, n_kv_groups=G, w=w, gate_mode=gate, use_bias=bias, l=l)
    m = _peaked_module(cfg, 3)
    gen = torch.Generator(device=DEV).manual_seed(cached)
    x = torch.randn(B, cached + sum(news), 128, generator=gen, device=DEV)
    x += torch.randn(B, -(-x.shape[1] // 64), 128, generator=gen, device=DEV).mul_(0.5).repeat_interleave(64, dim=1)[:, :x.shape[1]]
    x = x.bfloat16()
    new, old = I.NSACache(cfg, B, cached + 16, DEV), I.NSACache(cfg, B, cached + 16, DEV)
    for c in (new, old):
        if cached >= l:
            I.module_forward_incremental(m, x[:, :cached], c)
        else:
            c.append(m._phi_params(), *_kv(m, x[:, :cached], "select"), kv_compress=_kv(m, x[:, :cached], "compress"),
                     kv_sliding=_kv(m, x[:, :cached], "sliding"))
    p, ids = cached, []
    real, score = I.ops.decode_fwd, I.ops.score_topn

    def with_ids(d, dev):
        if d.indices:
            return real(d, dev)
        ids.append(torch.empty(d.B, d.G, d.Tn, d.n, device=dev, dtype=torch.int32))
        d.indices = ids[-1].data_ptr()
        real(d, dev)

    monkeypatch.setattr(I.ops, "decode_fwd", with_ids)
    for Tn in news:
        y = I.module_forward_incremental(m, x[:, p:p + Tn], new)
        assert len(ids) == (1 if B * Tn <= 8 or B * Tn * G <= 64 else 0), "the decode kernels did not run"
        with monkeypatch.context() as mp:
            mp.setattr(I, "_decode_module", lambda *a: None)
            mp.setattr(I, "_layer_rows", lambda *a: None)
            mp.setattr(I.ops, "score_topn", lambda *a, **k: (ids.append(score(*a, **k)), ids[-1])[1])
            z = I.module_forward_incremental(m, x[:, p:p + Tn], old)
        torch.cuda.synchronize()
        _no_timeouts()
        p += Tn
        if len(ids) == 2:
            assert torch.equal(*ids), (Tn, (ids[0] != ids[1]).any(-1).sum())
        ids.clear()
        _rows_close(y, z, 1.5e-2, Tn)
        assert (new.length, new.n_blocks) == (old.length, old.n_blocks) == (p, (p - l) // 16 + 1)
    for name in ("k_src", "k_cmp", "k_cmp_lp", "block_ends"):
        assert torch.equal(getattr(new, name), getattr(old, name)), name
    for name in ("k_slc", "v_slc", "v_src", "k_win", "v_win", "v_cmp"):
        a, b = getattr(new, name).float(), getattr(old, name).float()
        # bf16 products of another summation order may round to the neighbour (2^-8 relative)
        assert ((a - b).abs() <= 2 ** -7 * b.abs() + 1e-6).all() and (a != b).float().mean().item() < 1e-2, name
    # the layer call with its diagnostics
    q, lg = torch.randn(B, H, 1, dk, device=DEV).mul_(4).bfloat16(), torch.randn(B, 1, 3 * H, device=DEV)
    out, info = I.nsa_layer_incremental(q, lg, new, return_info=True)
    with monkeypatch.context() as mp:
        mp.setattr(I, "_layer_rows", lambda *a: None)
        _, want = I.nsa_layer_incremental(q, lg, new, return_info=True)
    torch.cuda.synchronize()
    assert torch.equal(info["indices"], want["indices"]) and max_abs(info["gates"], want["gates"]) < 1e-6
    t, pos = p - 1, torch.arange(p)
    every = lambda see: see.expand(B, G, 1, -1)
    chosen = (info["indices"].cpu().unsqueeze(-2) == (pos // 64).view(1, 1, 1, p, 1)).any(-1)
    ref = dict(o_cmp=_exact_rows(q, new.k_cmp[..., :new.n_blocks], new.v_cmp[:, :, :new.n_blocks], every(torch.ones(new.n_blocks, dtype=torch.bool))),
               o_win=_exact_rows(q, new.k_win[..., :p], new.v_win[:, :, :p], every(pos > t - w)),
               o_slc=_exact_rows(q, new.k_slc[..., :p], new.v_slc[:, :, :p], chosen))
    for name, r in ref.items():
        _rows_close(info[name], r, 2 ** -8, name)
    mix = sum(g.double().cpu().unsqueeze(-1) * ref[n_] for n_, g in zip(("o_cmp", "o_slc", "o_win"), info["gates"].unbind(-1)))
    _rows_close(out, mix, 2 ** -8, "out")


@pytest.mark.parametrize("dm,H,dk", [(2560, 64, 192), (2048, 32, 128), (512, 8, 64), (8192, 8, 64), (64, 48, 128)])
def test_queries_of_a_few_tokens_from_one_product(dm, H, dk):
    """The decode path forms q of all sequences with one product, the general path with one batched over the heads per sequence:
    the block choice wants the same bits of both."""
    from nsa.kernels import _project_heads
    lin = torch.nn.Linear(dm, H * dk, bias=False, device=DEV, dtype=torch.bfloat16)
    gen = torch.Generator(device=DEV).manual_seed(dm)
    with torch.no_grad():
        for B, Tn in ((1, 1), (1, 3), (1, 8), (2, 1), (5, 1), (8, 1), (3, 2), (2, 4)):
            x = torch.randn(B, Tn + 2, dm, generator=gen, device=DEV).bfloat16()[:, 1:1 + Tn]
            one = torch.nn.functional.linear(x, lin.weight).view(B, Tn, H, dk).transpose(1, 2)
            assert torch.equal(one, _project_heads(x, lin, H, dk)), (B, Tn)


@pytest.mark.parametrize("B,G,hpg,dk,dv,cached", [(8, 4, 16, 192, 128, 32000), (1, 4, 16, 192, 128, 2100), (2, 2, 16, 128, 128, 60000), (4, 2, 4, 64, 64, 9001)])
def test_decoded_rows_choose_the_tile_paths_blocks(monkeypatch, B, G, hpg, dk, dv, cached):
    """Long caches, where the n-th and the next block of some rows agree to 1e-7: ids bit for bit, over queries enough to meet such
    rows (one decoded row in 200 did when the sums ran in an order of their own)."""
    import nsa
    from nsa import incremental as I
    H = G * hpg
    cfg = nsa.NSAConfig(d_model=64, head_dim_qk=dk, head_dim_v=dv, n_heads=H, n_kv_groups=G)
    gen = torch.Generator(device=DEV).manual_seed(cached)
    rn = lambda *s, std=1.0: torch.randn(*s, generator=gen, device=DEV) * std
    phi = tuple(t.bfloat16() for t in (rn(32, 32, std=0.02), rn(2 * dk, dk + 32, std=0.02), rn(2 * dk, std=0.0), rn(dk, 2 * dk, std=0.02), rn(dk, std=0.0)))
    cache = I.NSACache(cfg, B, cached, DEV, shared_kv=True)
    k = rn(B, G, dk, cached) + rn(B, G, dk, -(-cached // 64), std=0.5).repeat_interleave(64, -1)[..., :cached]
    cache.append(phi, k.bfloat16(), rn(B, G, cached, dv).bfloat16())
    for _ in range(12):
        q, lg = rn(B, H, 1, dk).bfloat16(), rn(B, 1, 3 * H)
        _, a = I.nsa_layer_incremental(q, lg, cache, return_info=True)
        with monkeypatch.context() as mp:
            mp.setattr(I, "_layer_rows", lambda *a_: None)
            _, b = I.nsa_layer_incremental(q, lg, cache, return_info=True)
        assert torch.equal(a["indices"], b["indices"])
    _no_timeouts()


def _kv(m, x, name):
    from nsa.kernels import _project_heads
    c = m.config
    with torch.no_grad():
        return (_project_heads(x, getattr(m, "k_" + name), c.n_kv_groups, c.head_dim_qk, transposed=True),
                _project_heads(x, getattr(m, "v_" + name), c.n_kv_groups, c.head_dim_v))


@pytest.mark.parametrize("dtype,pdtype,shared", [(torch.bfloat16, torch.bfloat16, False), (torch.bfloat16, torch.float32, True),
                                                 (torch.float32, torch.float32, False)])
def test_append_kernel_matches_the_copies(dtype, pdtype, shared, monkeypatch):
    """Appends of every alignment, from tensors of either order in memory, against the copies through tensor operations."""
    import nsa
    from nsa import incremental as I
    H, G, dk, dv, B = 4, 2, 48, 40, 2
    cfg = nsa.NSAConfig(d_model=64, head_dim_qk=dk, head_dim_v=dv, n_heads=H, n_kv_groups=G)
    gen = torch.Generator().manual_seed(5)
    rn = lambda *s: torch.randn(*s, generator=gen).to(DEV)
    phi = (rn(32, 32), rn(2 * dk, dk + 32) * 0.1, rn(2 * dk), rn(dk, 2 * dk) * 0.1, rn(dk))
    phi = tuple(p.to(pdtype) for p in phi)
    a, b = (I.NSACache(cfg, B, 700, DEV, dtype=dtype, shared_kv=shared) for _ in range(2))
    for i, Tn in enumerate((20, 11, 1, 33, 300, 1, 64)):
        def kv():
            k, v = rn(B, G, dk, Tn).to(dtype), rn(B, G, Tn, dv).to(dtype)
            if i % 2:
                k, v = k.transpose(2, 3).contiguous().transpose(2, 3), v.permute(0, 2, 1, 3).contiguous().permute(0, 2, 1, 3)
            return k, v
        args = kv()
        more = {} if shared else dict(kv_compress=kv(), kv_sliding=kv())
        calls = []
        real = I.ops.cache_append
        with monkeypatch.context() as mp:
            mp.setattr(I.ops, "cache_append", lambda *x: (calls.append(1), real(*x)))
            a.append(phi, *args, **more)
        assert calls
        with monkeypatch.context() as mp:
            mp.setattr(I.NSACache, "_append_in_place", lambda *x: False)
            b.append(phi, *args, **more)
    torch.cuda.synchronize()
    assert (a.length, a.n_blocks) == (b.length, b.n_blocks) == (430, 25)
    for name in ("k_slc", "v_slc", "k_src", "v_src", "k_win", "v_win", "block_ends"):
        assert torch.equal(getattr(a, name), getattr(b, name)), name
    for name in ("k_cmp", "k_cmp_lp", "v_cmp"):          # the same products through other GEMM shapes: fp32 sums of 96 terms
        x, y = getattr(a, name), getattr(b, name)
        tol = 1e-5 if x.dtype == torch.float32 else 2 ** -8
        assert max_abs(x.float(), y.float()) <= tol * max(1.0, y.float().abs().max().item()), name


@pytest.mark.parametrize("dk,dv,H,G,T,w,lp,n", [(40, 24, 6, 2, 65, 1, 48, 3), (64, 64, 3, 3, 129, 33, 16, 5), (100, 256, 34, 1, 40, 500, 64, 4),
                                               (8, 8, 40, 2, 70, 64, 32, 30)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_generic_kernels_off_every_tile(dk, dv, H, G, T, w, lp, n, dtype):
    """Head dims off the 32-channel columns, groups of 1, 3, 20 and 34 heads (a 32-row tile holds part of one, or several queries),
    blocks that are no multiple of a 32-key tile, windows of one key and past the sequence; gradients included."""
    from nsa import ops
    q, k, v, do = (t.to(dtype) for t in _inputs(2, H, G, T, dk, dv, seed=T + dk))
    gen = torch.Generator().manual_seed(n)
    nblk = -(-T // lp)
    idx = torch.randint(-1, nblk, (2, G, T, n), generator=gen, dtype=torch.int32)
    idx[..., 0] = (torch.arange(T) // lp).int()
    scale = dk ** -0.5
    d = lambda t: t.to(DEV)
    ends = torch.full((T,), 999999, dtype=torch.int32)
    ends[:T // 2] = torch.randperm(T, generator=gen)[:T // 2].int()          # in no order
    for name, fwd, bwd, ref in (
            ("win", lambda *a: ops.sliding_fwd(*a, w, scale, generic=True), lambda *a: ops.sliding_bwd(*a, w, scale, generic=True),
             lambda a, b, c: O.sliding_window_attention(a, b, c, w, scale)),
            ("cmp", lambda *a: ops.cmp_attn_fwd(*a, d(ends), scale, generic=True),
             lambda a, b, c, *r: ops.cmp_attn_bwd(a, b, c, d(ends), *r, scale, generic=True),
             lambda a, b, c: _masked(a, b, c, ends[None, :] <= torch.arange(T)[:, None], scale)),
            ("slc", lambda *a: ops.slc_fwd(*a, d(idx), lp, scale, generic=True),
             lambda a, b, c, *r: ops.slc_bwd(a, b, c, d(idx), *r, lp, scale, generic=True),
             lambda a, b, c: O.selection_attention(a, b, c, idx, lp, scale))):
        o, L, M = fwd(d(q), d(k), d(v))
        dq, dkey, dval = bwd(d(q), d(k), d(v), o, d(do), L, M)
        torch.cuda.synchronize()
        qf, kf, vf = (t.float().requires_grad_(True) for t in (q, k, v))
        want = ref(qf, kf, vf)
        gq, gk, gv = torch.autograd.grad(want, (qf, kf, vf), do.float())
        if dtype == torch.float32:
            # fp32 sums of at most 40 * T terms in another order: 1e-5 of the largest entry is 80 roundings in a row
            for a, b in ((o, want), (dq, gq), (dkey, gk.transpose(-1, -2)), (dval, gv)):
                assert max_abs(a, b) < 1e-5 * max(1.0, b.abs().max().item()), name
        else:
            assert max_abs(o.float(), want) < 2e-2, name
            for a, b, what in ((dq, gq, "dq"), (dkey, gk.transpose(-1, -2), "dk"), (dval, gv, "dv")):
                _grad_close(a, b, f"{name} {what}")


def _masked(q, k, v, mask, scale):
    """Attention under a [T, keys] mask; rows that see nothing give zeros."""
    hpg = q.shape[1] // k.shape[1]
    s = (q * scale) @ k.repeat_interleave(hpg, 1)
    some = mask.any(-1)[:, None]
    p = torch.softmax(torch.where(some, s.masked_fill(~mask, float("-inf")), torch.zeros_like(s)), -1)
    return torch.where(mask, p, torch.zeros_like(p)) @ v.repeat_interleave(hpg, 1)


def test_generic_kernels_ignore_what_a_row_does_not_see():
    """Keys, values and upstream gradients of later positions that are not finite leave earlier rows and keys alone."""
    from nsa import ops
    B, H, G, T, D = 1, 4, 2, 96, 32
    q, k, v, do = (t.float().to(DEV) for t in _inputs(B, H, G, T, D, D, seed=11))
    idx = (torch.arange(T) // 16).int().view(1, 1, T, 1).expand(B, G, T, 1).contiguous().to(DEV)
    be = torch.arange(T, dtype=torch.int32, device=DEV)
    bad = T - 5
    for fwd, bwd in ((lambda *a: ops.sliding_fwd(*a, 40, 0.2, generic=True), lambda *a: ops.sliding_bwd(*a, 40, 0.2, generic=True)),
                     (lambda *a: ops.cmp_attn_fwd(*a, be, 0.2, generic=True), lambda a, b, c, *r: ops.cmp_attn_bwd(a, b, c, be, *r, 0.2, generic=True)),
                     (lambda *a: ops.slc_fwd(*a, idx, 16, 0.2, generic=True), lambda a, b, c, *r: ops.slc_bwd(a, b, c, idx, *r, 16, 0.2, generic=True))):
        kk, vv, dd = k.clone(), v.clone(), do.clone()
        kk[..., bad:], vv[:, :, bad:] = float("nan"), float("inf")
        dd[:, :, :8] = float("nan")                                  # keys from 8 on are seen by no such row
        o, L, M = fwd(q, k, v)
        dq, dkey, dval = bwd(q, k, v, o, do, L, M)
        _, dkey2, dval2 = bwd(q, k, v, o, dd, L, M)
        o2, L2, M2 = fwd(q, kk, vv)
        dq2, _, _ = bwd(q, kk, vv, o2, do, L2, M2)
        torch.cuda.synchronize()
        for a, b in ((o[:, :, :bad], o2[:, :, :bad]), (dq[:, :, :bad], dq2[:, :, :bad]), (dkey[:, :, 8:], dkey2[:, :, 8:]),
                     (dval[:, :, 8:], dval2[:, :, 8:])):
            assert torch.isfinite(b).all() and max_abs(a, b) < 1e-5


@pytest.mark.parametrize("dk,dv,H,G,T,w", [(64, 64, 8, 2, 128, 150), (192, 128, 16, 1, 640, 512), (128, 128, 4, 2, 896, 30), (192, 128, 6, 1, 256, 600)])
def test_window_backward_with_heads_split_over_a_cluster(dk, dv, H, G, T, w):
    """Few key tiles: clusters of 2, 4 and 8 CTAs share a tile's heads (and none where the heads are odd in number).  The row sums
    dO.O are computed here; the outputs are added into."""
    from nsa import ops
    q, k, v, do = _inputs(2, H, G, T, dk, dv, seed=T)
    qd, kd, vd, dd = (t.to(DEV) for t in (q, k, v, do))
    scale = dk ** -0.5
    o, L, M = ops.sliding_fwd(qd, kd, vd, w, scale)
    qf, kf, vf = (t.float().requires_grad_(True) for t in (q, k, v))
    want = torch.autograd.grad(O.sliding_window_attention(qf, kf, vf, w, scale), (qf, kf, vf), do.float())
    dq, dkey, dval = ops.sliding_bwd(qd, kd, vd, o, dd, L, M, w, scale)
    torch.cuda.synchronize()
    _no_timeouts()
    _grad_close(dq, want[0], "dq")
    _grad_close(dkey, want[1].transpose(-1, -2), "dk")
    _grad_close(dval, want[2], "dv")


@pytest.mark.parametrize("dk,dv,H,G,T,pos", [(64, 64, 4, 2, 4500, 0), (64, 64, 16, 8, 7201, 0), (192, 128, 32, 8, 7200, 0), (128, 128, 16, 8, 7130, 600)])
def test_block_scores_from_the_forward_match_the_scoring_kernel(dk, dv, H, G, T, pos):
    """Keys that grow along the sequence move the softmax reference from key tile to key tile; sums cross tile edges.  Ids of the
    layer (and of a chunk against a cache), whose scores come out of the compressed forward, against the scoring kernel on the
    same compressed keys: the same blocks but for near-ties at the cut."""
    import nsa
    from nsa import incremental as I, ops
    from nsa.kernels import nsa_layer
    cfg = nsa.NSAConfig(d_model=64, head_dim_qk=dk, head_dim_v=dv, n_heads=H, n_kv_groups=G, w=128)
    Tk = pos + T
    inp = O.make_inputs(1, H, G, Tk, dk, dv, 64, 32, seed=T, block_offset_std=0.5, dtype=torch.bfloat16)
    grow = torch.linspace(0.2, 6.0, Tk).view(1, 1, 1, Tk)
    q, k, v = inp["q"].to(DEV, torch.bfloat16), (inp["k"] * grow).to(DEV, torch.bfloat16), inp["v"].to(DEV, torch.bfloat16)
    phi = tuple(getattr(inp["phi"], n_).to(DEV) * (20.0 if n_ in ("w1", "w2") else 1.0) for n_ in ("pos_embed", "w1", "b1", "w2", "b2"))
    logits = torch.zeros(1, Tk, 3 * H, device=DEV)
    qn = q[:, :, pos:].contiguous()
    if pos == 0:
        _, info = nsa_layer(q, k, v, logits, phi, cfg, return_info=True)
        k_cmp, nb = info["k_cmp"], (Tk - 32) // 16 + 1
    else:
        cache = I.NSACache(cfg, 1, Tk, DEV, shared_kv=True)
        cache.append(phi, k, v)
        _, info = I.nsa_layer_incremental(qn, logits[:, pos:], cache, return_info=True)
        k_cmp, nb = cache.k_cmp, cache.n_blocks
    be = torch.full((k_cmp.shape[-1],), 999999, device=DEV, dtype=torch.int32)
    be[:nb] = torch.arange(nb, device=DEV, dtype=torch.int32) * 16 + 31
    want = ops.score_topn(qn, k_cmp, be, 32, 16, 64, 16, 3, dk ** -0.5, nb, pos, any_length=True)
    torch.cuda.synchronize()
    _no_timeouts()
    other = (info["indices"].unsqueeze(-1) != want.unsqueeze(-2)).all(-1).sum(-1)
    assert int(other.max()) <= 1 and (other > 0).float().mean().item() < 0.02, (int(other.max()), (other > 0).float().mean().item())
    # on one log-sum-exp the two choose the same blocks: rows whose cut rounding could move go to the scoring kernel itself.  So do
    # rows of equal scores (constant keys): every row of that call.
    for keys in (k_cmp.float(), torch.ones_like(k_cmp, dtype=torch.float32)):
        hi, lo = ops.split_keys(keys)
        val = torch.randn(1, G, keys.shape[-1], dv, device=DEV, dtype=torch.bfloat16)
        _, _, _, lse2, got = ops.cmp_attn_topn_fwd(qn, hi, lo, keys, val, be, 32, 16, 64, 16, 3, nb, dk ** -0.5, pos, any_length=True)
        want = ops.score_topn(qn, keys, be, 32, 16, 64, 16, 3, dk ** -0.5, nb, pos, any_length=True, cmp_lse2=lse2)
        torch.cuda.synchronize()
        _no_timeouts()
        assert torch.equal(got.sort(-1).values, want.sort(-1).values)


@pytest.mark.parametrize("rows,dv", [((1, 2, 33), 128), ((2, 3, 21), 64), ((1, 1, 1), 128), ((2, 20, 7), 128), ((1, 32, 5), 256)])
def test_row_kernels_at_any_row_count(rows, dv):
    """Rows that do not fill a warp's share: gate/mix backward with its row sums, against the formulas."""
    from nsa import ops
    B, H, T = rows
    gen = torch.Generator().manual_seed(T)
    oc, os_, ow, do = (torch.randn(B, H, T, dv, generator=gen).bfloat16() for _ in range(4))
    lg = torch.randn(B, T, 3 * H, generator=gen)
    out, gates = ops.gate_mix_fwd(lg.to(DEV), oc.to(DEV), os_.to(DEV), ow.to(DEV), "sigmoid")
    dc, ds, dw, dlog, delta = ops.gate_mix_bwd(gates, oc.to(DEV), os_.to(DEV), ow.to(DEV), do.to(DEV), "sigmoid", want_delta=True)
    torch.cuda.synchronize()
    g = torch.sigmoid(lg.view(B, T, H, 3).permute(0, 2, 1, 3))
    for i, (o, d) in enumerate(((oc, dc), (os_, ds), (ow, dw))):
        dot = (do.float() * o.float()).sum(-1)
        assert max_abs(d.float(), (g[..., i:i + 1] * do.float()).bfloat16().float()) <= 2 ** -8 * 4      # one rounding apart
        assert max_abs(delta[i], g[..., i] * dot) < 1e-4 * max(1.0, dot.abs().max().item())            # fp32 sums of dv terms
        assert max_abs(dlog.view(B, T, H, 3)[..., i], (dot * g[..., i] * (1 - g[..., i])).transpose(1, 2)) < 1e-4 * max(1.0, dot.abs().max().item())


@pytest.mark.parametrize("dk,dv,H,G,T,w,n", [(64, 64, 3, 1, 72, 1, 3), (192, 128, 16, 1, 200, 100, 4), (128, 128, 80, 1, 40, 512, 1),
                                             (64, 64, 4, 4, 1000, 333, 16)])
def test_mma_kernels_keep_32_bit_probabilities(dk, dv, H, G, T, w, n):
    """Ragged bf16 calls (groups of 1, 3, 16 and 80 heads, windows of one key and past the sequence, ends in no order) against the
    oracle on the same inputs; their error against it is that of the fp32-probability FMA kernels: what rounding the results to bf16
    leaves, with a tenth of room for sums in another order.  (A window of one key has a zero gradient, a difference of two equal
    sums of dv products in 32 bits: 1e-6 of what the products alone would give.)"""
    from nsa import _lib, ops
    q, k, v, do = _inputs(2, H, G, T, dk, dv, seed=T + dk)
    gen = torch.Generator().manual_seed(n)
    idx = torch.randint(-1, -(-T // 64), (2, G, T, n), generator=gen, dtype=torch.int32)
    idx[..., 0] = (torch.arange(T) // 64).int()
    ends = torch.full((T,), 999999, dtype=torch.int32)
    ends[:T // 2] = torch.randperm(T, generator=gen)[:T // 2].int()
    scale = dk ** -0.5
    d = lambda t: t.to(DEV)
    for name, fwd, bwd, ref in (
            ("win", lambda *a, **k_: ops.sliding_fwd(*a, w, scale, **k_), lambda *a, **k_: ops.sliding_bwd(*a, w, scale, **k_),
             lambda a, b, c: O.sliding_window_attention(a, b, c, w, scale)),
            ("cmp", lambda *a, **k_: ops.cmp_attn_fwd(*a, d(ends), scale, **k_),
             lambda a, b, c, *r, **k_: ops.cmp_attn_bwd(a, b, c, d(ends), *r, scale, **k_),
             lambda a, b, c: _masked(a, b, c, ends[None, :] <= torch.arange(T)[:, None], scale)),
            ("slc", lambda *a, **k_: ops.slc_fwd(*a, d(idx), 64, scale, **k_),
             lambda a, b, c, *r, **k_: ops.slc_bwd(a, b, c, d(idx), *r, 64, scale, **k_),
             lambda a, b, c: O.selection_attention(a, b, c, idx, 64, scale))):
        got = []
        for generic in (False, True):
            def run():
                o, L, M = fwd(d(q), d(k), d(v), generic=generic)
                got.append((o, *bwd(d(q), d(k), d(v), o, d(do), L, M, generic=generic), L, M))
            ran = set(_lib.profile_kernels(run))
            assert ("attn_fwd_mma" in ran and "attn_bwd_mma" in ran) != generic, ran
        qf, kf, vf = (t.double().requires_grad_(True) for t in (q, k, v))
        want = ref(qf, kf, vf)
        gq, gk, gv = torch.autograd.grad(want, (qf, kf, vf), do.double())
        for what, a, b, r in zip(("o", "dq", "dk", "dv"), *got, (want, gq, gk.transpose(-1, -2), gv)):
            ea, eb = (a.double().cpu() - r).norm().item(), (b.double().cpu() - r).norm().item()
            floor = do.double().norm() * v.double().norm(dim=-1).max() * max(k.double().norm(dim=-2).max(), q.double().norm(dim=-1).max()) * scale
            assert ea <= 1.1 * eb + 1e-6 * floor.item(), (name, what, ea, eb)
        for a, b in zip(got[0][4:], got[1][4:]):
            assert torch.equal(torch.isfinite(a), torch.isfinite(b)) and max_abs(a.nan_to_num(0, 0, 0), b.nan_to_num(0, 0, 0)) < 1e-4, name
    # values that are not finite behind what a row sees
    kk, vv = d(k).clone(), d(v).clone()
    kk[..., T - 5:], vv[:, :, T - 5:] = float("nan"), float("inf")
    dd = d(do).clone()
    dd[:, :, :8] = float("nan")
    o, L, M = ops.sliding_fwd(d(q), d(k), d(v), w, scale)
    dq, dkey, dval = ops.sliding_bwd(d(q), d(k), d(v), o, d(do), L, M, w, scale)
    _, dkey2, dval2 = ops.sliding_bwd(d(q), d(k), d(v), o, dd, L, M, w, scale)
    o2, L2, M2 = ops.sliding_fwd(d(q), kk, vv, w, scale)
    dq2, _, _ = ops.sliding_bwd(d(q), kk, vv, o2, d(do), L2, M2, w, scale)
    torch.cuda.synchronize()
    for a, b in ((o[:, :, :T - 5], o2[:, :, :T - 5]), (dq[:, :, :T - 5], dq2[:, :, :T - 5]), (dkey[:, :, 8:], dkey2[:, :, 8:]), (dval[:, :, 8:], dval2[:, :, 8:])):
        assert torch.isfinite(b).all() and max_abs(a.float(), b.float()) <= 2 ** -7 * max(1.0, a.float().abs().max().item())


@pytest.mark.parametrize("c_layer", [True, False])
@pytest.mark.parametrize("token_major", [True, False])
def test_layer_without_an_upstream_gradient(monkeypatch, c_layer, token_major):
    """A later node that hands back no gradient for the layer's output: zero gradients, as for a gradient of zeros."""
    import nsa
    from nsa import kernels as K
    from tests.test_host import DropGradient
    monkeypatch.setattr(K, "_USE_C_LAYER", c_layer)
    inp = O.make_inputs(1, 4, 2, 128, 64, 64, 64, 32, seed=1, dtype=torch.bfloat16)
    cfg = nsa.NSAConfig(d_model=64, head_dim_qk=64, head_dim_v=64, n_heads=4, n_kv_groups=2, w=64)
    q, k, v = (inp[x].to(DEV, torch.bfloat16).requires_grad_(True) for x in ("q", "k", "v"))
    phi = tuple(getattr(inp["phi"], n_).to(DEV).requires_grad_(True) for n_ in ("pos_embed", "w1", "b1", "w2", "b2"))
    logits = torch.zeros(1, 128, 12, device=DEV, requires_grad=True)
    out = K.nsa_layer(q, k, v, logits, phi, cfg, token_major_out=token_major)
    ins = (q, k, v, logits, *phi)
    for g, t in zip(torch.autograd.grad(DropGradient.apply(out).sum(), ins), ins):
        assert g.shape == t.shape and not g.any()


@pytest.mark.parametrize("pos", [0, 300])
def test_block_choice_in_the_smaller_scratch(monkeypatch, pos):
    """Where memory does not hold the scratch of the faster block choice, the layer and a chunk against a cache run in the smaller
    one, and choose the same blocks (the compressed branch's sums run alike: outputs bit for bit)."""
    import nsa
    from nsa import incremental as I, ops
    from nsa.kernels import nsa_layer
    H, G, T = 16, 8, 7201
    cfg = nsa.NSAConfig(d_model=64, head_dim_qk=64, head_dim_v=64, n_heads=H, n_kv_groups=G, w=128, n=4)      # (few slots: the choice's scratch is the largest)
    inp = O.make_inputs(1, H, G, pos + T, 64, 64, 64, 32, seed=T, block_offset_std=0.5, dtype=torch.bfloat16)
    q, k, v = (inp[x].to(DEV, torch.bfloat16) for x in ("q", "k", "v"))
    phi = tuple(getattr(inp["phi"], n_).to(DEV) for n_ in ("pos_embed", "w1", "b1", "w2", "b2"))
    logits = torch.zeros(1, pos + T, 3 * H, device=DEV)
    if pos:
        cache = I.NSACache(cfg, 1, pos + T, DEV, shared_kv=True)
        cache.append(phi, k, v)
        run = lambda: I.nsa_layer_incremental(q[:, :, pos:].contiguous(), logits[:, pos:], cache, return_info=True)
    else:
        run = lambda: nsa_layer(q, k, v, logits, phi, cfg, return_info=True)
    with torch.no_grad():
        a, info_a = run()
        real, sizes = ops._scratch, []

        def no_room(dev, nbytes, least):
            sizes.append((nbytes, least()))
            return real(dev, least(), None)
        monkeypatch.setattr(ops, "_scratch", no_room)
        b, info_b = run()
    torch.cuda.synchronize()
    _no_timeouts()
    assert sizes and all(more > less for more, less in sizes)
    assert torch.equal(info_a["o_cmp"], info_b["o_cmp"]) and torch.equal(info_a["indices"].sort(-1).values, info_b["indices"].sort(-1).values)
    assert max_abs(a.float(), b.float()) < 2e-2


def test_scratch_falls_back_where_memory_runs_out():
    from nsa import ops
    ws, n_ = ops._scratch(torch.device(DEV), 1 << 46, lambda: 1000)
    assert n_ == ws.numel() == 1000


@pytest.mark.parametrize("dk,dv,H,G,T", [(64, 64, 4, 2, 100), (192, 128, 16, 1, 637)])
def test_compressed_gradients_of_ragged_calls_add_up_to_zero(dk, dv, H, G, T):
    """A constant added to every compressed key leaves the softmax alone, so dK_cmp adds up to zero over the blocks but for the
    rounding of its entries, the output's in dO.O and dO's.  Given the gate backward's row sums, which are of the gradient before its rounding,
    a call must not be further off than one that forms them itself (as the FMA kernels do)."""
    from nsa import ops
    q, k, v, dout = (t.to(DEV) for t in _inputs(1, H, G, T, dk, dv, seed=T))
    nb = (T - 32) // 16 + 1
    kc, vc = k[..., :nb].contiguous(), v[:, :, :nb].contiguous()
    pad = (0, -nb % 8)
    kc, vc = torch.nn.functional.pad(kc, pad), torch.nn.functional.pad(vc, (0, 0, *pad))
    ends = torch.full((kc.shape[-1],), 999999, device=DEV, dtype=torch.int32)
    ends[:nb] = torch.arange(nb, device=DEV, dtype=torch.int32) * 16 + 31
    o, L, M = ops.cmp_attn_fwd(q, kc, vc, ends, dk ** -0.5)
    gates = torch.rand(1, H, T, 3, device=DEV)
    d_cmp, _, _, _, delta = ops.gate_mix_bwd(gates, o, o, o, dout, "sigmoid", want_delta=True)
    off = []
    for kw in (dict(row_delta=delta[0]), dict(generic=True)):
        _, dkc, _ = ops.cmp_attn_bwd(q, kc, vc, ends, o, d_cmp, L, M, dk ** -0.5, **kw)
        off.append(dkc.float().sum(2).norm().item())
    assert off[0] <= 1.15 * off[1], off


@pytest.mark.parametrize("branch", ["win", "slc"])
def test_ragged_backward_without_room_for_its_row_sums(monkeypatch, branch):
    """The row sums dO.O are formed in the products' kernels where the scratch has no room for them: the same gradients but for sums
    of dv products in another order (1e-6 of dS) and the rounding to bf16 that this may turn."""
    from nsa import ops
    B, H, G, T, dk, dv = 2, 8, 2, 203, 64, 64
    q, k, v, do = (t.to(DEV) for t in _inputs(B, H, G, T, dk, dv, seed=7))
    idx = (torch.arange(T) // 64).int().view(1, 1, T, 1).expand(B, G, T, 2).contiguous().to(DEV)
    idx[..., 1] = 0
    if branch == "win":
        fwd, bwd, size = (lambda: ops.sliding_fwd(q, k, v, 90, 0.125)), (lambda o, L, M: ops.sliding_bwd(q, k, v, o, do, L, M, 90, 0.125)), "nsa_attn_bwd_workspace_bytes"
        less = lambda real, a: 256
    else:
        fwd, bwd, size = (lambda: ops.slc_fwd(q, k, v, idx, 64, 0.125)), (lambda o, L, M: ops.slc_bwd(q, k, v, idx, o, do, L, M, 64, 0.125)), "nsa_slc_bwd_workspace_bytes"
        less = lambda real, a: real(*a) - 2 * (-(-B * H * T * 4 // 256) * 256)
    o, L, M = fwd()
    want = bwd(o, L, M)
    real = getattr(ops.lib, size)
    monkeypatch.setattr(ops.lib, size, lambda *a: less(real, a))
    for a, b in zip(bwd(o, L, M), want):
        assert ((a.float() - b.float()).abs() <= 2 ** -7 * b.float().abs() + 1e-5 * b.float().abs().max()).all()
        assert (a != b).float().mean().item() < 0.02
