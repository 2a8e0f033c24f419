"""CPU-side checks: the C-ABI library loads and exports what the header declares, the configuration
validates like the reference's, the launcher shims carry the reference's parameter order."""
import os
import re

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_library_exports_every_declared_symbol():
    import nsa._lib as L
    header = open(os.path.join(ROOT, "include", "nsa_b200.h")).read()
    declared = set(re.findall(r"NSA_API\s+[\w\s\*]+?\b(nsa_\w+)\s*\(", header))
    assert len(declared) >= 17
    for name in declared:
        assert hasattr(L.lib, name), f"{name} declared in the header but not exported"
    assert declared == set(L.PROTOTYPES), "ctypes prototypes out of sync with the header"
    assert b"sm_100a" in L.lib.nsa_version()


def test_argument_errors_without_a_gpu():
    """Bad arguments are rejected before any CUDA call, with a message."""
    import nsa._lib as L
    rc = L.lib.nsa_sliding_fwd(None, None, None, None, None, None, None, 1, 3, 2, 8, 8, 8, 4, 1.0, 0, 0, None)
    assert rc == -1 and b"H/G" in L.lib.nsa_last_error()
    rc = L.lib.nsa_sliding_fwd(None, None, None, None, None, None, None, 1, 4, 2, 8, 8, 8, 4, 1.0, 0, 0, None)
    assert rc == -1 and b"null" in L.lib.nsa_last_error()
    rc = L.lib.nsa_topn_from_scores(None, None, 1, 4, 2, 8, 8, 2, 100, 0, None)
    assert rc == -1
    assert L.lib.nsa_slc_bwd_workspace_bytes(1, 64, 4, 65536, 65536, 192, 128, 16, 64, 1, 0) > 4 * 65536 * 16 * 4
    # the stride-generic family only needs the inverse index
    assert L.lib.nsa_slc_bwd_workspace_bytes(1, 64, 4, 65536, 65536, 192, 128, 16, 64, 1, L.FLAG_GENERIC) < (1 << 28)


def test_config_defaults_and_validation():
    """Defaults of the paper configuration (nsa/kernels.py:516-591) and the rejected settings."""
    from nsa import NSAConfig
    c = NSAConfig()
    assert (c.d_model, c.head_dim_qk, c.head_dim_v, c.l, c.d, c.l_prime, c.n, c.w) == (2560, 192, 128, 32, 16, 64, 16, 512)
    assert (c.n_heads, c.n_kv_groups, c.n_fixed, c.n_dynamic, c.gate_mode) == (64, 4, 3, 13, "sigmoid")
    assert c.heads_per_group == 16 and c.head_dim_qk_padded == 256 and c.head_dim_v_padded == 128
    c = NSAConfig(include_fixed_in_selection=False)
    assert c.n_fixed == 0 and c.n_dynamic == 16
    for bad in (dict(l=0), dict(l_prime=0), dict(d=0), dict(n=0), dict(w=0), dict(gate_mode="tanh"),
                dict(n_heads=6, n_kv_groups=4), dict(l=24, d=16)):
        with pytest.raises((AssertionError, ValueError)):
            NSAConfig(**bad)


def test_package_surface():
    import nsa
    import nsa.kernels as K
    assert nsa.__version__ == "1.0.0"
    assert set(nsa.__all__) == {"NSAConfig", "NSAAttention", "_nsa_sliding_window_fwd_kernel",
                                "_nsa_sliding_window_bwd_kernel", "_nsa_compression_fwd_kernel",
                                "_nsa_compression_bwd_kernel", "_nsa_sparse_selection_fwd_kernel",
                                "_nsa_sparse_selection_bwd_kernel"}
    for n in ("CompressionAttention", "SelectionAttention", "SlidingWindowAttention",
              "derive_selection_from_compression_per_timestep", "select_top_k_blocks_per_query_with_gqa"):
        assert hasattr(K, n)
    # positional parameter counts of the six reference kernels (nsa/kernels.py:595, 837, 1152, 1304, 1534, 1691)
    counts = {"_nsa_sparse_selection_fwd_kernel": 34, "_nsa_sparse_selection_bwd_kernel": 50,
              "_nsa_sliding_window_fwd_kernel": 29, "_nsa_sliding_window_bwd_kernel": 45,
              "_nsa_compression_fwd_kernel": 30, "_nsa_compression_bwd_kernel": 46}
    for n, cnt in counts.items():
        assert len(getattr(nsa, n).positional) == cnt, n
    assert nsa._nsa_sliding_window_fwd_kernel.positional[:9] == ["Q", "K", "V", "Out", "sm_scale", "L", "M", "stride_qz", "stride_qh"]
    assert nsa._nsa_sliding_window_fwd_kernel.positional[11:15] == ["stride_kz", "stride_kg", "stride_kn", "stride_kk"]


def test_module_parameter_names_match_reference_state_dict():
    from nsa import NSAAttention, NSAConfig
    m = NSAAttention(NSAConfig(d_model=64, head_dim_qk=16, head_dim_v=16, n_heads=4, n_kv_groups=2, l=8, d=4, l_prime=8, n=4, w=8))
    names = set(m.state_dict())
    expect = {f"{p}.weight" for p in ("q_proj", "k_compress", "v_compress", "k_select", "v_select", "k_sliding", "v_sliding",
                                      "pos_embed", "compress_mlp.0", "compress_mlp.2", "gate_mlp.0", "gate_mlp.2", "o_proj")}
    expect |= {f"{p}.bias" for p in ("compress_mlp.0", "compress_mlp.2", "gate_mlp.0", "gate_mlp.2")}
    assert names == expect
    with pytest.raises(RuntimeError):      # no CPU path
        m(torch.zeros(1, 16, 64))


def test_reference_helpers():
    from nsa.reference import compare_outputs, create_block_ends
    assert create_block_ends(64, 8, 8, device="cpu").tolist() == list(range(7, 64, 8))
    assert create_block_ends(20, 8, 4, device="cpu").tolist() == [7, 11, 15, 19]
    ok, _ = compare_outputs(torch.ones(3), torch.ones(3))
    assert ok


def test_library_keeps_no_call_pairing_state():
    """Query offset, row sums and dQ addends travel in the argument lists: no setter is exported."""
    import nsa._lib as L
    for gone in ("nsa_set_query_offset", "nsa_set_row_delta", "nsa_set_dq_addends", "nsa_set_kernel_family"):
        assert not hasattr(L.lib, gone), gone


def test_launcher_checks_every_tensor_before_launching():
    """The launcher shims refuse, before any launch, strides that would make a kernel write past a tensor, negative
    strides, and serve over-reaching read-only tensors from a padded copy."""
    from nsa.kernels import _Launcher
    t = torch.zeros(2, 3, 8, 4)
    assert _Launcher._extent("t", t.stride(), t.shape) == t.numel()
    assert _Launcher._fits("t", t, t.stride(), t.shape) is t
    with pytest.raises(ValueError, match="storage holds"):
        _Launcher._fits("dK", t, (192, 64, 8, 1), (2, 3, 8, 8))         # strides of a tensor twice as wide
    with pytest.raises(ValueError, match="negative"):
        _Launcher._fits("Out", t, (96, 32, -4, 1), t.shape)
    wide = _Launcher._safe("K", t, (192, 64, 8, 1), (2, 3, 8, 8))       # read-only: padded copy, original values first
    assert wide.numel() >= _Launcher._extent("K", (192, 64, 8, 1), (2, 3, 8, 8)) and wide is not t
    assert _Launcher._fits("K^T", t, (96, 32, 1, 4), (2, 3, 4, 8)) is t   # a transposed view stays inside the storage
    assert _Launcher._safe("K", t, t.stride(), t.shape) is t
    view = t[:, :, 2:]                                                   # storage offset counts against the room left
    with pytest.raises(ValueError):
        _Launcher._fits("dQ", view, t.stride(), t.shape)


def test_projections_match_the_per_linear_products(monkeypatch):
    """The one autograd node of the seven projections against one product per linear: values and gradients in 64 bits."""
    import torch
    from nsa import kernels as K, ops
    monkeypatch.setattr(ops, "token_major", lambda x: x.transpose(1, 2).contiguous())
    torch.manual_seed(0)
    x = torch.randn(2, 5, 8, dtype=torch.double, requires_grad=True)
    layouts = ((4, 3, False), (2, 3, True), (2, 2, False))
    lins = [torch.nn.Linear(8, h * d, bias=False, dtype=torch.double) for h, d, _ in layouts]
    ws = [lin.weight for lin in lins]
    a = K._Projections.apply(x, layouts, *ws)
    b = [K._project_heads(x, lin, *lay) for lin, lay in zip(lins, layouts)]
    gs = [torch.randn_like(t) for t in b]
    for p, q in zip((*a, *torch.autograd.grad(a, [x, *ws], gs)), (*b, *torch.autograd.grad(b, [x, *ws], gs))):
        assert p.shape == q.shape and (p - q).abs().max().item() < 1e-12
    assert all(t.is_contiguous() for t in a)


class DropGradient(torch.autograd.Function):
    """A node that hands back no gradient for its input."""

    @staticmethod
    def forward(ctx, x):
        return x.clone()

    @staticmethod
    def backward(ctx, _g):
        return None


def test_gate_mix_without_an_upstream_gradient(monkeypatch):
    """An undefined gradient of the mixed output counts as zeros."""
    from nsa import kernels as K, ops
    monkeypatch.setattr(ops, "gate_mix_fwd", lambda lg, a, b, c, mode: (a + b + c, lg))
    monkeypatch.setattr(ops, "gate_mix_bwd", lambda g, a, b, c, d, mode: (d.contiguous(), d * 2, d * 3, g * d.sum()))
    lg, a, b, c = (torch.randn(1, 2, 6, requires_grad=True), *(torch.randn(1, 2, 2, 4, requires_grad=True) for _ in range(3)))
    out, _ = K._GateMix.apply(lg, a, b, c, "sigmoid")
    grads = torch.autograd.grad((DropGradient.apply(out)).sum(), (lg, a, b, c))
    assert all(g.shape == t.shape and not g.any() for g, t in zip(grads, (lg, a, b, c)))


def test_projection_weight_gradients_round_once(monkeypatch):
    """bf16 weights shared by several sequences: the gradient is one 32-bit sum over all of them, as through the linears' own
    products, so its error against 64 bits is one rounding, 2^-9 relative at most (and 2^-9 / sqrt(3) in the 2-norm)."""
    from nsa import kernels as K, ops
    monkeypatch.setattr(ops, "token_major", lambda x: x.transpose(1, 2).contiguous())
    torch.manual_seed(1)
    B, T, layouts = 4, 64, ((4, 8, False), (2, 8, True), (2, 4, False))
    x = torch.randn(B, T, 32).bfloat16().requires_grad_(True)
    ws = [torch.randn(h * d, 32).bfloat16().requires_grad_(True) for h, d, _ in layouts]
    outs = K._Projections.apply(x, layouts, *ws)
    gs = [torch.randn_like(t) for t in outs]
    for (h, d, transposed), g, dw in zip(layouts, gs, torch.autograd.grad(outs, ws, gs)):
        rows = g.transpose(2, 3) if transposed else g                  # [B,h,T,d]
        want = torch.einsum("bhtd,btm->hdm", rows.double(), x.double()).reshape(h * d, 32)
        assert ((dw.double() - want).norm() / want.norm()).item() < 2 ** -9


@pytest.mark.parametrize("BG,dk,dv", [(4, 192, 128), (8, 192, 128), (2, 128, 128), (4, 128, 128), (16, 64, 64)])
def test_compression_backward_scratch_covers_its_column_sums(BG, dk, dv):
    """The layer forms the products of ragged sequences over rows padded to 8, which may hold one block per plane more than the
    sequence; the bytes reserved for those rows have to hold the column sums' partial rows over the blocks that there are."""
    from nsa._lib import BF16, lib
    al = lambda n: -(-n // 256) * 256
    U, l, d = 2 * dk, 32, 16

    def chunks(rows, W):                  # rows of W values in chunks of 32 to 1024, as many as four thread blocks per SM need
        per_row = -(-W // 32)
        want = -(-4 * 148 // per_row)
        return -(-rows // min(1024, max(32, -(-rows // want))))

    for T in [*range(2049, 9000, 7), *range(13080, 13088), *range(9001, 65536, 53)]:
        rows = -(-T // 8) * 8
        nb, nb_rows = (T - l) // d + 1, (rows - l) // d + 1
        nbp = 1 << (nb - 1).bit_length()
        nseg = -(-rows // 16)
        assert nseg == -(-T // 16)        # the pooling kernel walks the segments of T, the scratch holds those of the padded rows
        parts = -(-nseg // max(4, -(-nseg * BG // 296)))
        others = [BG * nb_rows * dk * 4, BG * nb_rows * U * 4, BG * nbp * dv * 4, BG * rows * U * 2, parts * BG * l * U * 4, l * U * 4, U * dk * 2]
        reserved = lib.nsa_cmp_phi_workspace_bytes(1, BG, rows, dk, dv, l, d, U, nbp, BF16, 1) - 256 - sum(map(al, others))
        assert reserved >= chunks(BG * nb, dk) * dk * 4, (T, reserved)


def test_shared_memory_attributes_do_not_depend_on_the_call():
    """A kernel's dynamic shared memory attribute is shared by all host threads: set to one call's size, another thread's larger
    launch would be refused.  Every place sets a constant (k..., SM::..., or a size made of template arguments alone)."""
    import glob
    import os
    import re
    import nsa
    src = os.path.join(os.path.dirname(nsa.__file__), "..", "csrc", "*.cu")
    sizes = [(os.path.basename(f), m) for f in glob.glob(src)
             for m in re.findall(r"cudaFuncAttributeMaxDynamicSharedMemorySize,\s*([^;]*?)\)\s*(?:;|!=|==)", open(f).read())]
    assert len(sizes) > 10
    by_template = {("attn_generic.cu", "(int)sm"), ("attn_generic.cu", "(int)sm_dkv"), ("attn_mma.cu", "sm")}
    for f, size in sizes:
        assert re.fullmatch(r"(\(int\))?(k[A-Z]\w*|\w+(<[^>]*>)?::k\w+)", size) or (f, size) in by_template, (f, size)


def test_append_to_a_cache_in_host_memory():
    """Tokens before the first compressed block are only copied, wherever the cache lies."""
    from nsa import NSAConfig
    from nsa.incremental import NSACache
    cache = NSACache(NSAConfig(d_model=64, head_dim_qk=16, head_dim_v=8, n_heads=4, n_kv_groups=2), 1, 64, "cpu", shared_kv=True)
    phi = tuple(torch.zeros(*n_) for n_ in ((32, 32), (32, 48), (32,), (16, 32), (16,)))
    k, v = torch.randn(1, 2, 16, 20).bfloat16(), torch.randn(1, 2, 20, 8).bfloat16()
    assert cache.append(phi, k, v) == 0 and (cache.length, cache.n_blocks) == (20, 0)
    assert torch.equal(cache.k_slc[..., :20], k) and torch.equal(cache.v_slc[:, :, :20], v)
