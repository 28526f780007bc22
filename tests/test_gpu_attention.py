"""Parity of the tcgen05 attention kernel with the CPU oracle (the reference's PyTorch
attention), through triton_attn_func / the C ABI. Tolerance from the project baseline:
2e-2 max abs error in bf16."""
import ctypes
import math
import threading

import pytest
import torch

import trinix_b200 as T
from oracle import reference_port as R
from tests.util import Golden

pytestmark = pytest.mark.gpu
G = Golden()
TOL = 2e-2


def _qkv(B, Sq, Sk, Hq, Hk, D, seed=0, dtype=torch.bfloat16):
    g = torch.Generator().manual_seed(seed)
    q = torch.randn(B, Sq, Hq, D, generator=g).to(dtype)
    k = torch.randn(B, Sk, Hk, D, generator=g).to(dtype)
    v = torch.randn(B, Sk, Hk, D, generator=g).to(dtype)
    return q, k, v


def _check(cuda, q, k, v, causal=False, window=None, slopes=None, scale=None, tol=TOL):
    out = T.triton_attn_func(q.to(cuda), k.to(cuda), v.to(cuda), softmax_scale=scale,
                             causal=causal, window_size=window,
                             alibi_slopes=None if slopes is None else slopes.to(cuda))
    assert T.attention_status(cuda) == 0, "a bounded wait inside the kernel gave up"
    assert out.shape == q.shape and out.dtype == q.dtype
    # the oracle in the kernel's input dtype (what the reference computes) and in fp32 (truth)
    ref = R.attention_variant_ref(q, k, v, scale, causal, window, slopes).float()
    ref32 = R.attention_variant_ref(q.float(), k.float(), v.float(), scale, causal, window,
                                    None if slopes is None else slopes.float())
    o = out.float().cpu()
    assert not torch.isnan(o).any()
    err, err32 = float((o - ref).abs().max()), float((o - ref32).abs().max())
    # The 16-bit oracle rounds scores and probabilities to the input dtype (base.py:373,394),
    # so it sits up to `oracle_noise` away from the exact result itself; the kernel must be
    # within tol of the exact result and within tol + that noise of the 16-bit oracle.
    oracle_noise = float((ref - ref32).abs().max())
    assert err32 <= tol and err <= tol + oracle_noise, (err, err32, oracle_noise)
    return out


@pytest.mark.parametrize("D", [128, 64])
@pytest.mark.parametrize("S", [128, 256, 384, 1000])
def test_noncausal_mha(cuda, S, D):
    q, k, v = _qkv(1, S, S, 2, 2, D, seed=S + D)
    _check(cuda, q, k, v)


@pytest.mark.parametrize("D", [128, 64])
@pytest.mark.parametrize("S", [64, 129, 512, 777, 1536])
def test_causal_gqa(cuda, S, D):
    q, k, v = _qkv(2, S, S, 8, 2, D, seed=S)
    _check(cuda, q, k, v, causal=True)


def test_causal_mqa_with_expanded_kv_heads(cuda):
    """MQA as the reference's module presents it: one kv head expanded to all query heads
    (head stride 0), multi_query_attention.py:173-174."""
    q, k, v = _qkv(2, 300, 300, 4, 1, 128, seed=7)
    ref = R.attention_variant_ref(q, k, v, None, True).float()
    kd, vd = k.to("cuda").expand(-1, -1, 4, -1), v.to("cuda").expand(-1, -1, 4, -1)
    assert kd.stride(2) == 0
    out = T.triton_attn_func(q.to("cuda"), kd, vd, causal=True)
    assert T.attention_status() == 0
    assert float((out.float().cpu() - ref).abs().max()) <= TOL
    out1 = T.triton_attn_func(q.to("cuda"), k.to("cuda"), v.to("cuda"), causal=True)
    assert torch.equal(out, out1)  # native Hkv=1 and the expanded view are the same launch


def test_tiled_noncontiguous_kv_like_the_reference_module(cuda):
    """K/V tiled to all heads and handed over as transposed (B,S,H,D) views, the layout
    grouped_query_attention.py:189-194 produces."""
    q, k, v = _qkv(2, 260, 260, 8, 2, 128, seed=11)
    kt = R.tile_kv_heads_ref(k, 4).to("cuda").transpose(1, 2).contiguous().transpose(1, 2)
    vt = R.tile_kv_heads_ref(v, 4).to("cuda").transpose(1, 2).contiguous().transpose(1, 2)
    assert not kt.is_contiguous()
    out = T.triton_attn_func(q.to("cuda"), kt, vt, causal=True)
    native = T.triton_attn_func(q.to("cuda"), k.to("cuda"), v.to("cuda"), causal=True)
    assert T.attention_status() == 0
    assert torch.equal(out, native)


@pytest.mark.parametrize("S", [200, 1024])
def test_causal_alibi(cuda, S):
    H = 8
    q, k, v = _qkv(1, S, S, H, 2, 128, seed=S)
    slopes = R.alibi_slopes_ref(H)
    _check(cuda, q, k, v, causal=True, slopes=slopes)
    _check(cuda, q, k, v, causal=False, slopes=slopes)  # |i-j| on both sides


@pytest.mark.parametrize("Sq,Sk,causal,window", [
    (1300, 1300, True, None),          # many KV tiles, both Q tiles of a CTA, ragged tail
    (900, 900, False, (300, 0)),       # a window that ends at the query, no causal flag
    (1100, 1100, True, (200, 0)),      # causal and a left window: two boundary tiles per row block
    (130, 130, True, None),            # second Q tile nearly empty
    (256, 640, True, None),            # more keys than queries (top-left aligned mask)
])
def test_alibi_with_keys_visited_backwards(cuda, Sq, Sk, causal, window):
    """ALiBi under a causal mask, or a window that ends at the query, walks a row block's KV tiles
    from the last to the first; slopes from steep (an O rescale per tile in ascending order) to
    flat, grouped kv heads, head dims 128 and 64."""
    for D, H, Hk in ((128, 8, 2), (64, 4, 4)):
        q, k, v = _qkv(2, Sq, Sk, H, Hk, D, seed=Sq + D)
        slopes = torch.tensor([2.0 ** (-8.0 * (i + 1) / H) for i in range(H)])
        slopes[0] = 1.5  # steeper than any standard ALiBi head
        _check(cuda, q, k, v, causal=causal, window=window, slopes=slopes)


@pytest.mark.parametrize("S,window", [(700, (100, 0)), (1300, (256, 0)), (600, (64, 64)),
                                      (512, (0, 0)), (900, (1024, 0)), (520, (130, 7))])
def test_sliding_window(cuda, S, window):
    q, k, v = _qkv(1, S, S, 4, 2, 128, seed=S)
    _check(cuda, q, k, v, window=window)
    _check(cuda, q, k, v, causal=True, window=(window[0], max(window)))


def test_window_zero_zero_returns_v(cuda):
    q, k, v = _qkv(1, 300, 300, 2, 2, 64, seed=1)
    out = T.triton_attn_func(q.to(cuda), k.to(cuda), v.to(cuda), window_size=(0, 0))
    assert torch.equal(out.cpu(), v)  # softmax over a single key is exactly 1


def test_cross_lengths_scale_and_fp16(cuda):
    q, k, v = _qkv(2, 200, 333, 4, 4, 128, seed=3)
    _check(cuda, q, k, v, scale=0.05)
    q, k, v = _qkv(1, 130, 70, 2, 1, 64, seed=4, dtype=torch.float16)
    _check(cuda, q, k, v, tol=5e-3)
    q, k, v = _qkv(1, 260, 130, 2, 1, 128, seed=5)
    _check(cuda, q, k, v, causal=True)  # rows beyond the key count see every key


def test_large_logits_trigger_rescale(cuda):
    """Row maxima that keep growing along the keys force the O-rescale path."""
    g = torch.Generator().manual_seed(0)
    S, D = 1024, 128
    q = torch.randn(1, S, 1, D, generator=g)
    k = torch.randn(1, S, 1, D, generator=g) * torch.linspace(0.2, 3.0, S).view(1, S, 1, 1)
    v = torch.randn(1, S, 1, D, generator=g)
    _check(cuda, q.bfloat16(), k.bfloat16(), v.bfloat16(), scale=0.5, tol=3e-2)


def test_lse_output(cuda):
    q, k, v = _qkv(1, 300, 300, 2, 2, 128, seed=2)
    out, lse = T.attention(q.to(cuda), k.to(cuda), v.to(cuda), causal=True, return_lse=True)
    s = torch.einsum("bqhd,bkhd->bhqk", q.float(), k.float()) * 128 ** -0.5
    s = s.masked_fill(torch.triu(torch.ones(300, 300), 1).bool(), float("-inf"))
    torch.testing.assert_close(lse.cpu(), torch.logsumexp(s, -1), rtol=1e-3, atol=1e-3)


def test_golden_attention_vectors_from_the_reference(cuda):
    """The attention outputs the unmodified reference produced (its PyTorch backend, fp32 and
    bf16, head dim 32, GQA 4:2, causal / not / causal + ALiBi): the kernel meets them directly.
    Head dim 32 runs as 64 with zero columns appended."""
    q, k, v = (G(n).bfloat16().to(cuda) for n in ("attn_q", "attn_k", "attn_v"))
    for causal in (False, True):
        out = T.triton_attn_func(q, k, v, causal=causal)
        assert out.shape == q.shape
        want_bf16 = G(f"attn_out_bf16_causal{int(causal)}").float()
        want_f32 = G(f"attn_out_causal{int(causal)}")     # from the fp32 inputs
        assert float((out.float().cpu() - want_bf16).abs().max()) <= TOL
        assert float((out.float().cpu() - want_f32).abs().max()) <= 2 * TOL  # + input rounding
    out = T.triton_attn_func(q, k, v, causal=True, alibi_slopes=R.alibi_slopes_ref(4).to(cuda))
    assert float((out.float().cpu() - G("attn_out_alibi")).abs().max()) <= 2 * TOL
    assert T.attention_status(cuda) == 0
    # head dims between the two built ones, and the one beyond them
    g = torch.Generator().manual_seed(3)
    q96 = torch.randn(1, 200, 4, 96, generator=g).bfloat16()
    k96 = torch.randn(1, 200, 2, 96, generator=g).bfloat16()
    v96 = torch.randn(1, 200, 2, 96, generator=g).bfloat16()
    out96, lse96 = T.attention(q96.to(cuda), k96.to(cuda), v96.to(cuda), causal=True, return_lse=True)
    ref96 = R.attention_variant_ref(q96.float(), k96.float(), v96.float(), None, True)
    assert out96.shape == q96.shape and lse96.shape == (1, 4, 200)
    assert float((out96.float().cpu() - ref96).abs().max()) <= TOL
    q256 = torch.zeros(1, 128, 2, 256, dtype=torch.bfloat16, device=cuda)
    with pytest.raises(T._lib.TrinixB200Error) as e:     # a clear error, no fallback
        T.triton_attn_func(q256, q256, q256)
    assert e.value.code == -6


def test_full_size_properties(cuda):
    """Benchmark geometry (S=4096, 32 query / 8 kv heads, D=128), one batch element:
    causal output row 0 equals v[0]; batch sharding is bit-identical; window (S, 0) == causal."""
    g = torch.Generator(device=cuda).manual_seed(0)
    B, S, H, Hk, D = 2, 4096, 32, 8, 128
    q = torch.randn(B, S, H, D, generator=g, device=cuda).bfloat16()
    k = torch.randn(B, S, Hk, D, generator=g, device=cuda).bfloat16()
    v = torch.randn(B, S, Hk, D, generator=g, device=cuda).bfloat16()
    out = T.triton_attn_func(q, k, v, causal=True)
    assert T.attention_status(cuda) == 0
    assert torch.equal(out[:, 0], v[:, 0].repeat_interleave(4, dim=1))
    parts = torch.cat([T.triton_attn_func(q[b:b + 1], k[b:b + 1], v[b:b + 1], causal=True)
                       for b in range(B)])
    assert torch.equal(out, parts)
    w = T.triton_attn_func(q, k, v, window_size=(S, 0))
    assert torch.equal(out, w)
    # against torch's own fused attention on the GPU (a library used as checker only)
    ref = torch.nn.functional.scaled_dot_product_attention(
        q.transpose(1, 2), k.transpose(1, 2).repeat_interleave(4, 1),
        v.transpose(1, 2).repeat_interleave(4, 1), is_causal=True).transpose(1, 2)
    assert float((out.float() - ref.float()).abs().max()) <= TOL


def _mask_ref(q, k, v, mask4, causal, scale=None):
    """The reference's PyTorch attention (base.py:347-400) with K/V tiled to all query heads
    and the mask expanded to (B, H, Sq, Sk), in the input dtype and in fp32."""
    g = q.shape[2] // k.shape[2]
    kt, vt = k.repeat_interleave(g, dim=2), v.repeat_interleave(g, dim=2)
    B, Sq, H, _ = q.shape
    m = mask4.expand(B, H, Sq, k.shape[1]).float()
    ref = R.attention_ref(q, kt, vt, scale, causal, m.to(q.dtype)).float()
    ref32 = R.attention_ref(q.float(), kt.float(), vt.float(), scale, causal, m)
    return ref, ref32


@pytest.mark.parametrize("mask_kind", ["2d_f32", "3d_bool", "4d_b1", "4d_bh_bf16"])
@pytest.mark.parametrize("Sq,Sk,D", [(300, 300, 128), (257, 640, 64)])
def test_dense_additive_mask(cuda, mask_kind, Sq, Sk, D):
    """attn_mask in every shape _prepare_mask accepts (attention_kernel.py:479-495), float and
    bool, broadcast by stride: parity with the reference's PyTorch path on the expanded mask."""
    B, Hq, Hk = 2, 4, 2
    q, k, v = _qkv(B, Sq, Sk, Hq, Hk, D, seed=Sq + Sk)
    g = torch.Generator().manual_seed(7)
    if mask_kind == "2d_f32":
        mask = torch.randn(Sq, Sk, generator=g)
        mask[:, Sk // 3: Sk // 2] = float("-inf")          # a hidden band
        mask4 = mask[None, None]
    elif mask_kind == "3d_bool":
        hidden = torch.rand(B, Sq, Sk, generator=g) < 0.3
        hidden[..., 0] = False                              # no fully hidden row
        mask = hidden
        mask4 = torch.zeros(B, 1, Sq, Sk).masked_fill_(hidden[:, None], float("-inf"))
    elif mask_kind == "4d_b1":
        mask = torch.randn(B, 1, Sq, Sk, generator=g) * 2
        mask4 = mask
    else:
        mask = (torch.randn(B, Hq, Sq, Sk, generator=g) * 2).bfloat16()
        mask4 = mask.float()
    out = T.triton_attn_func(q.to(cuda), k.to(cuda), v.to(cuda), attn_mask=mask.to(cuda))
    assert T.attention_status(cuda) == 0
    ref, ref32 = _mask_ref(q, k, v, mask4, False)
    o = out.float().cpu()
    assert not torch.isnan(o).any()
    err, err32 = float((o - ref).abs().max()), float((o - ref32).abs().max())
    noise = float((ref - ref32).abs().max())
    assert err32 <= TOL and err <= TOL + noise, (err, err32, noise)


def test_dense_mask_combines_with_causal_and_alibi(cuda):
    B, S, Hq, Hk, D = 1, 400, 4, 1, 128
    q, k, v = _qkv(B, S, S, Hq, Hk, D, seed=11)
    g = torch.Generator().manual_seed(3)
    mask = torch.randn(S, S, generator=g)
    slopes = torch.tensor([0.5, 0.25, 0.125, 0.0625])
    out = T.triton_attn_func(q.to(cuda), k.to(cuda), v.to(cuda), attn_mask=mask.to(cuda),
                             causal=True, alibi_slopes=slopes.to(cuda))
    assert T.attention_status(cuda) == 0
    i = torch.arange(S)
    alibi = -slopes[:, None, None] * (i[:, None] - i[None, :]).abs().float()   # (H, S, S)
    ref, ref32 = _mask_ref(q, k, v, (mask[None] + alibi)[None], True)
    o = out.float().cpu()
    err, err32 = float((o - ref).abs().max()), float((o - ref32).abs().max())
    noise = float((ref - ref32).abs().max())
    assert err32 <= TOL and err <= TOL + noise, (err, err32, noise)


@pytest.mark.parametrize("p_drop", [0.1, 0.5])
@pytest.mark.parametrize("Sq,Sk,D,causal,with_mask", [(300, 300, 128, True, False),
                                                      (257, 640, 64, False, True)])
def test_dropout_matches_the_rebuilt_keep_mask(cuda, p_drop, Sq, Sk, D, causal, with_mask):
    """dropout_p > 0: the kernel's Philox stream is rebuilt on the CPU element for element, so the
    comparison with the reference's PyTorch arithmetic (softmax, then dropout, then times V,
    base.py:394-397) is exact up to the usual tolerance, not statistical."""
    B, Hq, Hk = 2, 4, 2
    q, k, v = _qkv(B, Sq, Sk, Hq, Hk, D, seed=Sq + Sk + int(100 * p_drop))
    mask = None
    if with_mask:
        mask = torch.randn(B, 1, Sq, Sk, generator=torch.Generator().manual_seed(5))
    seed, offset = 0x1234_5678_9ABC_DEF0 >> 2, 3
    out, lse = T.attention(q.to(cuda), k.to(cuda), v.to(cuda), causal=causal,
                           attn_mask=None if mask is None else mask.to(cuda), dropout_p=p_drop,
                           seed=seed, offset=offset, return_lse=True)
    assert T.attention_status(cuda) == 0
    keep = R.dropout_keep_mask_ref(seed, offset, B, Hq, Sq, Sk, p_drop)
    g = Hq // Hk
    kt, vt = k.repeat_interleave(g, dim=2), v.repeat_interleave(g, dim=2)
    m4 = None if mask is None else mask.expand(B, Hq, Sq, Sk).contiguous()
    ref32 = R.attention_dropout_ref(q.float(), kt.float(), vt.float(), None, causal, m4, keep, p_drop)
    ref = R.attention_dropout_ref(q, kt, vt, None, causal,
                                  None if m4 is None else m4.to(q.dtype), keep, p_drop).float()
    o = out.float().cpu()
    err32, err = float((o - ref32).abs().max()), float((o - ref).abs().max())
    noise = float((ref - ref32).abs().max())
    tol = TOL / (1.0 - p_drop)  # kept probabilities are scaled up by 1 / (1 - p)
    assert err32 <= tol and err <= tol + noise, (err32, err, noise)
    # the LSE is that of the undropped scores (another instantiation of the kernel computes it
    # here, with its own rounding of the score arithmetic: close, not bit-equal)
    _, lse0 = T.attention(q.to(cuda), k.to(cuda), v.to(cuda), causal=causal,
                          attn_mask=None if mask is None else mask.to(cuda), return_lse=True)
    torch.testing.assert_close(lse, lse0, rtol=1e-5, atol=1e-5)
    # same seed and offset: the same result bit for bit; another offset: another mask
    again = T.attention(q.to(cuda), k.to(cuda), v.to(cuda), causal=causal,
                        attn_mask=None if mask is None else mask.to(cuda), dropout_p=p_drop,
                        seed=seed, offset=offset)
    other = T.attention(q.to(cuda), k.to(cuda), v.to(cuda), causal=causal,
                        attn_mask=None if mask is None else mask.to(cuda), dropout_p=p_drop,
                        seed=seed, offset=offset + 1)
    assert torch.equal(again, out) and not torch.equal(other, out)


def test_dropout_keep_rate_and_module_path(cuda):
    """Statistics of the stream (v = 1 makes the output the kept mass of each row), and the
    module surface: training mode drops, eval mode does not, the seed follows torch.manual_seed."""
    B, S, H, D = 1, 2048, 2, 64
    q = torch.zeros(B, S, H, D, dtype=torch.bfloat16, device=cuda)       # uniform probabilities
    v = torch.ones(B, S, H, D, dtype=torch.bfloat16, device=cuda)
    for p_drop in (0.1, 0.5):
        out = T.attention(q, q, v, dropout_p=p_drop, seed=99)
        thr = R.dropout_threshold(p_drop)
        # every row: sum_j keep_j / (S * (1 - p_eff)), mean 1, std sqrt(p / ((1 - p) S))
        m = out.float()[..., 0]
        assert abs(float(m.mean()) - 1.0) < 5e-3
        p_eff = thr / 256.0
        assert abs(float(m.std()) - (p_eff / ((1 - p_eff) * S)) ** 0.5) < 5e-3
    attn = T.FastGroupedQueryAttention(512, 8, 2, dropout=0.3, bias=False, kernel_type="triton",
                                       causal=True).to(cuda).bfloat16()
    x = torch.randn(2, 256, 512, device=cuda, dtype=torch.bfloat16)
    with torch.no_grad():
        attn.eval()
        e1, e2 = attn(x)[0], attn(x)[0]
        attn.train()
        torch.manual_seed(5)
        t1 = attn(x)[0]
        t2 = attn(x)[0]
        torch.manual_seed(5)
        t3 = attn(x)[0]
    assert torch.equal(e1, e2) and not torch.equal(t1, e1)
    assert not torch.equal(t1, t2) and torch.equal(t1, t3)
    assert T.attention_status(cuda) == 0
    with pytest.raises(ValueError):
        T.attention(q, q, v, dropout_p=1.0)


def test_dense_mask_rejects_bad_shapes(cuda):
    q, k, v = (t.to(cuda) for t in _qkv(2, 128, 128, 2, 2, 64))
    with pytest.raises(ValueError):
        T.triton_attn_func(q, k, v, attn_mask=torch.zeros(128, 64, device=cuda))
    with pytest.raises(ValueError):
        T.triton_attn_func(q, k, v, attn_mask=torch.zeros(3, 128, 128, device=cuda))
    with pytest.raises(ValueError):
        T.triton_attn_func(q, k, v, attn_mask=torch.zeros(1, 1, 1, 128, 128, device=cuda))


def test_launch_after_recorded_failure_raises_then_recovers(cuda):
    """A non-zero status word (a bounded wait gave up in some earlier launch) makes every later
    launch skip its work on the device. The host learns of it without a synchronisation: a launch
    that skips its work (or gives up) writes the word into the pinned host memory attached to the
    workspace and the next call checks that first, raising status -8 instead of handing back
    unwritten output. The word is set from the host here; no wait on the device is ever made to
    run out."""
    from trinix_b200 import ops
    q, k, v = (t.to(cuda) for t in _qkv(1, 512, 512, 4, 2, 128, seed=21))
    good = T.attention(q, k, v, causal=True)
    assert T.attention_status(cuda) == 0
    ops._workspace(cuda)[:4].view(torch.int32).fill_(4)     # as if a softmax wait had run out
    T.attention(q, k, v, causal=True)                        # skipped on the device; word written
    torch.cuda.synchronize(cuda)
    with pytest.raises(T._lib.TrinixB200Error) as e:         # first call that can know: raises
        T.attention(q, k, v, causal=True)
    assert e.value.code == -8 and "0x4" in str(e.value)
    again = T.attention(q, k, v, causal=True)                # both copies were cleared
    assert T.attention_status(cuda) == 0
    assert torch.equal(again, good)
    # the C-level form of the same check
    import ctypes
    lib = T._lib.load()
    host = torch.zeros(1, dtype=torch.int32).pin_memory()
    ws = ops._workspace(cuda)
    P = ctypes.c_void_p
    st = P(torch.cuda.current_stream(cuda).cuda_stream)
    ws[:4].view(torch.int32).fill_(2)
    assert lib.trx_attn_status(P(ws.data_ptr()), P(host.data_ptr()), st) == 0
    torch.cuda.synchronize(cuda)
    assert int(host[0]) == 2
    assert lib.trx_attn_status(P(ws.data_ptr()), P(host.data_ptr()), st) == -8
    assert lib.trx_attn_status(None, P(host.data_ptr()), st) == -1
    assert T.attention_status(cuda) == 2 and T.attention_status(cuda) == 0


def test_views_the_tensor_maps_cannot_take_are_materialised(cuda):
    """Legal strided views whose base is not 16-byte aligned or whose strides are not multiples
    of 8 elements (a slice along D at an offset of 4, a head stride of 132) run all the same."""
    g = torch.Generator().manual_seed(5)
    big = torch.randn(2, 200, 4, 136, generator=g).bfloat16().to(cuda)
    q, k, v = big[..., 4:132], big[..., 4:132].clone(), big[..., 8:136]
    assert q.data_ptr() % 16 != 0 and q.stride(-1) == 1
    out = T.triton_attn_func(q, k, v, causal=True)
    ref = T.triton_attn_func(q.contiguous(), k, v.contiguous(), causal=True)
    assert T.attention_status(cuda) == 0 and torch.equal(out, ref)
    odd = torch.randn(1, 150, 2, 132, generator=g).bfloat16().to(cuda)[..., :128]
    assert odd.stride(2) % 8 != 0
    out = T.triton_attn_func(odd, odd, odd)
    assert torch.equal(out, T.triton_attn_func(*(odd.contiguous(),) * 3))


@pytest.mark.parametrize("shape,strides", [
    ((2, 5, 1, 64), (320, 64, 1, 1)),            # one head, few rows
    ((2, 300, 1, 64), (19200, 64, 1, 1)),        # one head, many rows
    ((1, 1, 8, 128), (3077, 3077, 128, 1)),      # one row of one sequence
    ((1, 200, 8, 128), (204803, 1024, 128, 1)),  # one sequence
    ((3, 1, 8, 128), (1024, 7, 128, 1)),         # one row each
])
def test_size_one_dims_of_any_stride(cuda, shape, strides):
    """The stride of a size-1 dim addresses nothing, whatever its value."""
    g = torch.Generator().manual_seed(shape[1])
    q = torch.randn(204803, generator=g).bfloat16().to(cuda).as_strided(shape, strides)
    out = T.triton_attn_func(q, q, q, causal=True)
    assert out.stride() == torch.empty(shape).stride()
    assert torch.equal(out, T.triton_attn_func(*(q.clone(memory_format=torch.contiguous_format),) * 3,
                                               causal=True))
    assert T.attention_status(cuda) == 0


def test_flash_stand_in_keeps_the_conventions_of_the_symbol_it_replaces(cuda):
    """flash_attn_func (the symbol bound at trinix/layers/attention/base.py:10-16): causal with
    Sq < Sk is aligned bottom-right (decode against a KV cache sees every cached key), unknown
    keywords raise instead of being dropped."""
    Sq, Sk = 70, 300
    q, k, v = _qkv(2, Sq, Sk, 4, 2, 128, seed=9)
    out = T.flash_attn_func(q.to(cuda), k.to(cuda), v.to(cuda), causal=True)
    assert T.attention_status(cuda) == 0
    i, j = torch.arange(Sq)[:, None], torch.arange(Sk)[None, :]
    mask = torch.zeros(Sq, Sk).masked_fill_(j > i + (Sk - Sq), float("-inf"))
    kt, vt = k.repeat_interleave(2, 2), v.repeat_interleave(2, 2)
    ref32 = R.attention_ref(q.float(), kt.float(), vt.float(), None, False, mask)
    assert float((out.float().cpu() - ref32).abs().max()) <= TOL
    # one query row against the cache: sees all keys
    out1 = T.flash_attn_func(q[:, :1].to(cuda), k.to(cuda), v.to(cuda), causal=True)
    full = T.triton_attn_func(q[:, :1].to(cuda), k.to(cuda), v.to(cuda), causal=False)
    assert torch.equal(out1, full)
    # equal lengths: identical to triton_attn_func
    q2, k2, v2 = (t.to(cuda) for t in _qkv(1, 200, 200, 4, 4, 64, seed=2))
    assert torch.equal(T.flash_attn_func(q2, k2, v2, causal=True),
                       T.triton_attn_func(q2, k2, v2, causal=True))
    assert torch.equal(T.flash_attn_func(q2, k2, v2, window_size=(50, 0)),
                       T.triton_attn_func(q2, k2, v2, window_size=(50, 0)))
    with pytest.raises(TypeError):
        T.flash_attn_func(q2, k2, v2, softcap=30.0)
    with pytest.raises(NotImplementedError):
        T.flash_attn_func(q.to(cuda), k.to(cuda), v.to(cuda), causal=True, window_size=(10, 0))


@pytest.mark.parametrize("Sq,Sk", [(1, 1000), (1, 128), (7, 2049), (130, 64)])
def test_decode_shapes_kv_longer_or_shorter_than_q(cuda, Sq, Sk):
    """KV-cache decode shapes (grouped_query_attention.py:179-187 concatenates past keys, so
    Sk > Sq, down to a single query row), GQA heads, no mask."""
    q, k, v = _qkv(2, Sq, Sk, 8, 2, 128, seed=Sq * 7 + Sk)
    _check(cuda, q, k, v)


@pytest.mark.parametrize("Sq,Sk,Hq,Hk,D,causal,window,alibi", [
    (1, 1, 8, 2, 128, False, None, False),        # one key: three warps of the CTA have none
    (1, 15, 4, 4, 64, False, None, True),         # less than one 16-key tile, one row per tile
    (1, 17, 32, 1, 128, False, None, False),      # MQA: 32 packed rows, two row tiles
    (3, 63, 8, 2, 64, True, None, True),          # rows that see one to three keys
    (5, 65, 12, 4, 128, False, None, False),      # 15 of 16 packed rows live
    (16, 4093, 8, 2, 128, False, (1 << 29, 4077), False),  # causal, aligned at the end of the cache
    (16, 300, 8, 1, 64, False, (1 << 29, 284), False),     # 128 packed rows: four double row tiles
    (2, 2100, 8, 8, 128, False, (100, 2098), False),       # a left edge inside the keys
    (9, 700, 6, 2, 128, False, (3, 2), True),     # a window of a few keys: most splits are empty
    (16, 5, 4, 2, 64, False, (2, 1), False),      # rows beyond the keys: nothing visible, output 0
    (17, 300, 8, 2, 128, False, None, False),     # one row more than the decode kernel takes
])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_few_query_rows(cuda, Sq, Sk, Hq, Hk, D, causal, window, alibi, dtype):
    """Few query rows against many keys: packed row tiles, key splits and their merge, at the edges
    of the 16-key tiles, the 16-row tiles and the splits. Bound: probabilities are rounded to
    2^-9 (bf16) of themselves and so is the result, each at most 2^-9 * max|v| ~ 9e-3."""
    q, k, v = _qkv(3, Sq, Sk, Hq, Hk, D, seed=Sq * 31 + Sk, dtype=dtype)
    slopes = R.alibi_slopes_ref(Hq) if alibi else None
    from trinix_b200 import ops
    out, lse = ops.attention(q.to(cuda), k.to(cuda), v.to(cuda), causal=causal, window=window,
                             alibi_slopes=None if slopes is None else slopes.to(cuda),
                             return_lse=True)
    assert T.attention_status(cuda) == 0
    qf, kf, vf = q.float(), k.float(), v.float()
    ref = R.attention_variant_ref(qf, kf, vf, None, causal, window, slopes)
    s = torch.einsum("bihd,bjhd->bhij", qf, R.tile_kv_heads_ref(kf, Hq // Hk)) * D ** -0.5
    i, j = torch.arange(Sq)[:, None], torch.arange(Sk)[None]
    if slopes is not None:
        s = s - slopes.view(1, -1, 1, 1) * (i - j).abs()
    if causal:
        s = s.masked_fill(j > i, float("-inf"))
    if window is not None:
        s = s.masked_fill((j - i < -window[0]) | (j - i > window[1]), float("-inf"))
    ref_lse = torch.logsumexp(s, -1)
    seen = ~torch.isinf(ref_lse)
    assert torch.equal(torch.isinf(lse.cpu()), ~seen)
    # fp32 scores of 128 terms of magnitude ~1 and fp32 sums: 1e-5 each
    assert float((lse.cpu()[seen] - ref_lse[seen]).abs().max()) <= 5e-5
    rows = seen.transpose(1, 2)
    assert float((out.float().cpu()[rows] - ref[rows]).abs().max()) <= TOL
    assert not out.float().cpu()[~rows].any()


@pytest.mark.parametrize("B,Sq,Sk,Hq,Hk,D", [
    (1, 16, 96, 32, 8, 128), (1, 16, 97, 32, 8, 128),      # the lines of the dispatch by keys
    (1, 16, 128, 32, 8, 128), (1, 16, 129, 32, 8, 128),
    (10, 16, 128, 32, 8, 128),     # more than one wave of the tcgen05 kernel
    (24, 16, 256, 32, 8, 128),     # one CTA per row tile, two waves
    (48, 1, 2093, 32, 8, 128),     # two, more than one wave
    (8, 16, 1024, 32, 8, 128),     # two, one wave
    (20, 1, 300, 8, 8, 64), (2, 2, 900, 32, 8, 128),       # one, four
    (2, 1, 4093, 8, 8, 64), (3, 16, 5000, 8, 2, 128),      # eight
    (1, 1, 9001, 8, 2, 64), (2, 3, 33000, 32, 1, 128),     # sixteen
])
def test_few_query_rows_with_every_number_of_splits(cuda, B, Sq, Sk, Hq, Hk, D):
    """Shapes for which the keys of a row tile go to 1, 2, 4, 8 and 16 CTAs, whatever the numbers the
    cost arrives at. Reference in fp32 on the device; bounds as in test_few_query_rows."""
    from trinix_b200 import ops
    q, k, v = (t.to(cuda) for t in _qkv(B, Sq, Sk, Hq, Hk, D, seed=Sk))
    out, lse = ops.attention(q, k, v, return_lse=True)
    assert T.attention_status(cuda) == 0
    qg = q.float().view(B, Sq, Hk, Hq // Hk, D)
    s = torch.einsum("bihgd,bjhd->bhgij", qg, k.float()) * D ** -0.5
    ref = torch.einsum("bhgij,bjhd->bihgd", torch.softmax(s, -1), v.float()).reshape(B, Sq, Hq, D)
    assert float((out.float() - ref).abs().max()) <= TOL
    ref_lse = torch.logsumexp(s, -1).reshape(B, Hq, Sq)
    # sums of up to 33000 fp32 terms in another order: below 33000 * 2^-24 of the sum
    assert float((lse - ref_lse).abs().max()) <= 5e-5 + Sk * 2.0 ** -24


@pytest.mark.parametrize("causal,window,alibi,scale", [
    (False, None, False, None), (True, None, False, None), (False, (5, 9), False, None),
    (False, (200, 0), True, None), (True, None, True, None), (False, None, True, None),
    (False, None, False, -0.1), (True, None, True, -0.1), (False, None, False, 0.0),
])
@pytest.mark.parametrize("B,Sq,Sk,Hq,Hk,D,dtype", [
    (2, 128, 128, 8, 2, 128, torch.bfloat16), (3, 300, 127, 4, 4, 64, torch.float16),
    (1, 33, 1, 6, 3, 128, torch.float16), (1, 16, 97, 32, 8, 128, torch.bfloat16),
    (2, 257, 65, 4, 4, 128, torch.bfloat16),
])
def test_single_key_tile(cuda, B, Sq, Sk, Hq, Hk, D, dtype, causal, window, alibi, scale):
    """Calls of one KV tile have a kernel of their own up to a wave of CTAs: every form that they take,
    contiguous, in other layouts and as part of a batch of more than a wave (bit for bit the same).
    Reference in 64 bits, bounds as in test_alibi_on_both_sides."""
    from trinix_b200 import ops
    q, k, v = (t.to(cuda) for t in _qkv(B, Sq, Sk, Hq, Hk, D, seed=Sq + Sk, dtype=dtype))
    slopes = R.alibi_slopes_ref(Hq).to(cuda) if alibi else None
    kw = dict(causal=causal, window=window, alibi_slopes=slopes, scale=scale, return_lse=True)
    out, lse = ops.attention(q, k, v, **kw)
    swap = lambda t: t.transpose(1, 2).contiguous().transpose(1, 2)  # noqa: E731
    cache = torch.full((B, 200, Hk, D), float("nan"), device=cuda, dtype=dtype)
    cache[:, 40:40 + Sk] = v  # the values around the slice are never used
    again = ops.attention(swap(q), swap(k), cache[:, 40:40 + Sk], **kw)
    assert T.attention_status(cuda) == 0
    assert torch.equal(again[0], out) and torch.equal(again[1], lse)
    if Sq > 16:  # the number of key splits of fewer rows goes by the batch
        n = torch.cuda.get_device_properties(cuda).multi_processor_count
        more = ops.attention(q.repeat(n, 1, 1, 1), k.repeat(n, 1, 1, 1), v.repeat(n, 1, 1, 1), **kw)
        assert torch.equal(more[0][:B], out) and torch.equal(more[1][-B:], lse)
    g = Hq // Hk
    s = torch.einsum("bihd,bjhd->bhij", q.double(), k.double().repeat_interleave(g, 2))
    s = s * (D ** -0.5 if scale is None else scale)
    i, j = torch.arange(Sq, device=cuda)[:, None], torch.arange(Sk, device=cuda)[None]
    if alibi:
        s = s - slopes.double().view(1, -1, 1, 1) * (i - j).abs()
    if causal:
        s = s.masked_fill(j > i, float("-inf"))
    if window is not None:
        s = s.masked_fill((j - i < -window[0]) | (j - i > window[1]), float("-inf"))
    ref_lse = torch.logsumexp(s, -1)
    seen = ~torch.isinf(ref_lse)
    assert torch.equal(torch.isinf(lse), ~seen)
    assert bool(((lse.double() - ref_lse).abs()[seen]
                 <= (1e-5 + 2.0 ** -22 * (ref_lse.abs() + 10))[seen]).all())
    p, vt = torch.softmax(s, -1).nan_to_num_(0.0), v.double().repeat_interleave(g, 2)
    ref = torch.einsum("bhij,bjhd->bihd", p, vt)
    u = 2.0 ** -8 if dtype is torch.bfloat16 else 2.0 ** -11
    bound = u * (ref.abs() + torch.einsum("bhij,bjhd->bihd", p, vt.abs())) + 1e-4
    assert bool(((out.double() - ref).abs() <= bound).all())
    assert not out[~seen.transpose(1, 2)].any()


@pytest.mark.parametrize("B,S,Hq,Hk", [
    (4, 2500, 32, 8),    # 41 MB of keys and values, 10 of a batch: all heads of a batch at a time
    (1, 6151, 32, 32),   # 101 MB of a batch: one head after the other, row pairs, heaviest first
])
def test_causal_orders_of_large_calls(cuda, B, S, Hq, Hk):
    """Causal calls whose keys and values do not fit L2 walk their work items in other orders. Rows at
    the edges of the tiles and some in between, against fp32 on the device."""
    from trinix_b200 import ops
    D = 128
    q, k, v = (t.to(cuda) for t in _qkv(B, S, S, Hq, Hk, D, seed=S))
    out, lse = ops.attention(q, k, v, causal=True, return_lse=True)
    assert T.attention_status(cuda) == 0
    rows = torch.tensor(sorted({r for e in range(0, S + 1, 128) for r in (e - 1, e, e + 77)
                                if 0 <= r < S} | {S - 1}), device=cuda)
    hidden = torch.arange(S, device=cuda)[None] > rows[:, None]
    for b in range(B):
        for h in range(Hq):
            kf, vf = k[b, :, h * Hk // Hq].float(), v[b, :, h * Hk // Hq].float()
            s = (q[b, rows, h].float() @ kf.t() * D ** -0.5).masked_fill(hidden, float("-inf"))
            p = torch.softmax(s, -1)
            ref, size = p @ vf, p @ vf.abs()
            assert bool(((out[b, rows, h].float() - ref).abs()
                         <= 2.0 ** -8 * (ref.abs() + size) + 1e-4).all()), (b, h)
            assert float((lse[b, h, rows] - torch.logsumexp(s, -1)).abs().max()) <= 1e-4, (b, h)


@pytest.mark.parametrize("B,Sq,Sk,H,D,window,dtype", [
    (1, 256, 256, 3, 128, None, torch.bfloat16),     # tiles before, across and after the queries
    (1, 300, 1000, 3, 64, None, torch.float16),      # most keys after every query
    (1, 1000, 130, 3, 128, None, torch.float16),     # most before; a tile of two keys
    (60, 513, 511, 4, 128, (300, 140), torch.bfloat16),    # cut at both ends, several items per CTA
    (60, 640, 640, 4, 64, (1, 400), torch.bfloat16),
])
def test_alibi_on_both_sides(cuda, B, Sq, Sk, H, D, window, dtype):
    """Tiles on one side of their queries take another path than those in between, and slopes from
    none to one that leaves a row little more than its own key. Reference in 64 bits: the scores carry
    an fp32 rounding of their size, results and probabilities u of themselves."""
    from trinix_b200 import ops
    q, k, v = (t.to(cuda) for t in _qkv(B, Sq, Sk, H, H, D, seed=Sq + Sk, dtype=dtype))
    slopes = torch.tensor([0.0, 0.01, 0.3, 4.0], device=cuda)[-H:].contiguous()
    out, lse = ops.attention(q, k, v, window=window, alibi_slopes=slopes, return_lse=True)
    assert T.attention_status(cuda) == 0
    i, j = torch.arange(Sq, device=cuda)[:, None], torch.arange(Sk, device=cuda)[None]
    u = 2.0 ** -8 if dtype is torch.bfloat16 else 2.0 ** -11
    for b in {0, B - 1}:
        s = torch.einsum("ihd,jhd->hij", q[b].double(), k[b].double()) * D ** -0.5
        s = s - slopes.double().view(-1, 1, 1) * (i - j).abs()
        if window is not None:
            s = s.masked_fill((j - i < -window[0]) | (j - i > window[1]), float("-inf"))
        ref_lse = torch.logsumexp(s, -1)
        seen = ~torch.isinf(ref_lse)
        assert torch.equal(torch.isinf(lse[b]), ~seen)
        # a score has up to 4 roundings of half an ulp of its terms; 1e-5 for dot products and sums
        size = ref_lse.abs() + 10
        assert bool(((lse[b].double() - ref_lse).abs()[seen] <= (1e-5 + 2.0 ** -22 * size)[seen]).all())
        p = torch.softmax(s, -1).nan_to_num_(0.0)
        ref = torch.einsum("hij,jhd->ihd", p, v[b].double())
        bound = u * (ref.abs() + torch.einsum("hij,jhd->ihd", p, v[b].double().abs())) + 1e-4
        assert bool(((out[b].double() - ref).abs() <= bound).all())


@pytest.mark.parametrize("extra", [0, 1])  # one work item per SM, and one more
@pytest.mark.parametrize("causal,alibi", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("Sq,Sk,D", [(17, 1, 128), (130, 128, 64), (256, 129, 128), (200, 700, 128)])
def test_one_item_per_sm(cuda, Sq, Sk, D, causal, alibi, extra):
    """Launches of one work item per SM have kernels of their own; one item more takes the others.
    Reference in fp32 on the device, bounds as in test_more_work_items_than_ctas."""
    from trinix_b200 import ops
    H = torch.cuda.get_device_properties(cuda).multi_processor_count + extra
    q, k, v = (t.to(cuda) for t in _qkv(1, Sq, Sk, H, H, D, seed=Sq + Sk))
    slopes = torch.linspace(0.01, 0.5, H, device=cuda) if alibi else None
    out, lse = ops.attention(q, k, v, causal=causal, alibi_slopes=slopes, return_lse=True)
    assert T.attention_status(cuda) == 0
    s = torch.einsum("bihd,bjhd->bhij", q.float(), k.float()) * D ** -0.5
    i, j = torch.arange(Sq, device=cuda)[:, None], torch.arange(Sk, device=cuda)[None]
    if alibi:
        s = s - slopes.view(1, -1, 1, 1) * (i - j).abs()
    if causal:
        s = s.masked_fill(j > i, float("-inf"))
    largest = max(1.0, float(s[~torch.isinf(s)].abs().max()))
    assert float((lse - torch.logsumexp(s, -1)).abs().max()) <= 1e-5 * (5 + largest)
    p = torch.softmax(s, -1)
    ref = torch.einsum("bhij,bjhd->bihd", p, v.float())
    bound = 2.0 ** -8 * (ref.abs() + torch.einsum("bhij,bjhd->bihd", p, v.float().abs())) + 1e-4
    assert bool(((out.float() - ref).abs() <= bound).all())


@pytest.mark.parametrize("Sq", [128, 256])  # an empty second Q tile, and two
def test_one_item_of_half_a_million_key_tiles(cuda, Sq):
    """2^26 keys in one work item: 2^19 visits of a microsecond or more, which is longer than the 400 ms
    after which a wait gives up. Keys of zeros and values of ones, so every sum is exact in fp32: the
    row sum 2^26 in shares of 2^24, O in steps of 16."""
    from trinix_b200 import ops
    Sk, D = 1 << 26, 64
    if torch.cuda.mem_get_info()[0] < 20 << 30:
        pytest.skip("needs 20 GB")
    q = torch.ones(1, Sq, 1, D, device=cuda, dtype=torch.bfloat16)
    k = torch.zeros(1, Sk, 1, D, device=cuda, dtype=torch.bfloat16)
    v = torch.ones(1, Sk, 1, D, device=cuda, dtype=torch.bfloat16)
    out, lse = ops.attention(q, k, v, return_lse=True)
    assert T.attention_status(cuda) == 0
    assert bool((out == 1).all())
    assert float((lse - 26 * math.log(2.0)).abs().max()) <= 4e-6  # 18.0 to an fp32 ulp or two
    del k, v
    torch.cuda.empty_cache()


@pytest.mark.parametrize("Sq", [17, 300])
@pytest.mark.parametrize("Sk", [128, 1024])
def test_row_sums_lose_no_more_than_chains_of_sixteen(cuda, Sq, Sk):
    """One key of weight 1 in the first eight columns, 2^-25 for every other: in fp32 those that are
    added behind the 1 in its chain are lost, and nothing else is. A row of a tile is summed in eight
    chains of 16, so 15 are; with a chain of 32 it would be 31."""
    from trinix_b200 import ops
    B, D = 8, 128
    q = torch.zeros(B, Sq, 2, D)
    q[..., 0] = 1.0
    k = torch.zeros(B, Sk, 2, D)
    k[..., 0] = -25.0
    for b in range(B):
        k[b, b, :, 0] = 0.0
    v = torch.zeros(B, Sk, 2, D)
    q, k, v = (t.bfloat16().to(cuda) for t in (q, k, v))
    # the score in the log2 domain is q.k to 1e-7, the weights 2^-25 (1 +- 3e-6)
    _, lse = ops.attention(q, k, v, scale=math.log(2.0), return_lse=True)
    exact = math.log1p((Sk - 1) * 2.0 ** -25)
    # one more of them for the last roundings, and the weights' own error
    assert float((lse.double() - exact).abs().max()) <= 16 * 2.0 ** -25 + Sk * 2.0 ** -25 * 3e-6


@pytest.mark.parametrize("B,Sq,Sk,Hq,Hk,D,causal,window,alibi,scale", [
    (40, 130, 130, 8, 8, 128, False, None, False, None),   # two rows in the second Q tile
    (40, 100, 300, 8, 8, 64, True, None, False, None),     # none
    (13, 700, 700, 24, 8, 128, True, None, False, None),   # row pairs, one to six KV tiles each
    (6, 1500, 1500, 16, 4, 128, True, None, False, None),  # pairs of heads
    (20, 1000, 1000, 8, 8, 64, False, (200, 0), False, None),   # tiles that start one later
    (20, 600, 600, 8, 8, 128, False, (30, 150), False, None),   # hidden at both ends
    (30, 700, 130, 8, 8, 64, False, (10, 3), False, None),      # items and rows without any key
    (30, 300, 0, 8, 8, 128, False, None, False, None),          # no key at all
    (20, 513, 513, 8, 2, 128, False, None, True, None),    # ALiBi on both sides of the query
    (20, 513, 513, 8, 8, 64, True, None, True, None),      # before it: last tile first, row pairs
    (20, 400, 400, 8, 2, 128, False, None, False, -0.1),   # a scale that is not positive
    (20, 700, 700, 8, 2, 128, False, None, False, 1.5),    # large scores: O is rescaled
])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_more_work_items_than_ctas(cuda, B, Sq, Sk, Hq, Hk, D, causal, window, alibi, scale, dtype):
    """Every CTA works on several items, of different lengths and with Q tiles that differ in their
    keys. Reference in fp32 on the device; the log sums' bound is relative to the scores."""
    from trinix_b200 import ops
    q, k, v = (t.to(cuda) for t in _qkv(B, Sq, Sk, Hq, Hk, D, seed=Sq + Sk, dtype=dtype))
    slopes = R.alibi_slopes_ref(Hq).to(cuda) if alibi else None
    out, lse = ops.attention(q, k, v, causal=causal, scale=scale, window=window,
                             alibi_slopes=slopes, return_lse=True)
    assert T.attention_status(cuda) == 0
    g = Hq // Hk
    s = torch.einsum("bihd,bjhd->bhij", q.float(), k.float().repeat_interleave(g, 2))
    s = s * (D ** -0.5 if scale is None else scale)
    i, j = torch.arange(Sq, device=cuda)[:, None], torch.arange(Sk, device=cuda)[None]
    if slopes is not None:
        s = s - slopes.view(1, -1, 1, 1) * (i - j).abs()
    if causal:
        s = s.masked_fill(j > i, float("-inf"))
    if window is not None:
        s = s.masked_fill((j - i < -window[0]) | (j - i > window[1]), float("-inf"))
    ref_lse = torch.logsumexp(s, -1)
    seen = ~torch.isinf(ref_lse)
    assert torch.equal(torch.isinf(lse), ~seen)
    if seen.any():
        largest = max(1.0, float(s[~torch.isinf(s)].abs().max()))
        assert float((lse[seen] - ref_lse[seen]).abs().max()) <= 1e-5 * (5 + largest)
        p, vt = torch.softmax(s, -1).nan_to_num_(0.0), v.float().repeat_interleave(g, 2)
        ref = torch.einsum("bhij,bjhd->bihd", p, vt)
        # probabilities and the result are each rounded to u of themselves
        u = 2.0 ** -8 if dtype is torch.bfloat16 else 2.0 ** -11
        bound = u * (ref.abs() + torch.einsum("bhij,bjhd->bihd", p, vt.abs())) + 1e-4
        assert bool(((out.float() - ref).abs() <= bound).all())
    assert not out[~seen.transpose(1, 2)].any()


@pytest.mark.parametrize("Sq", [1, 4])
def test_few_query_rows_in_every_layout(cuda, Sq):
    """The same call with contiguous tensors, transposed (B, H, S, D) storage, a slice of a longer
    cache, expanded kv heads (of both tensors and of K alone) and an expanded batch."""
    q, k, v = _qkv(2, Sq, 333, 8, 2, 128, seed=Sq)
    q, k, v = q.to(cuda), k.to(cuda), v.to(cuda)
    base = T.triton_attn_func(q, k, v)
    swap = lambda t: t.transpose(1, 2).contiguous().transpose(1, 2)  # noqa: E731
    assert torch.equal(T.triton_attn_func(swap(q), swap(k), swap(v)), base)
    cache = torch.full((2, 512, 2, 128), float("nan"), device=cuda, dtype=k.dtype)
    cache[:, 40:373] = k  # the keys around the slice are never used
    assert torch.equal(T.triton_attn_func(q, cache[:, 40:373], v), base)
    k1, v1 = k[:, :, :1], v[:, :, :1]
    mqa = T.triton_attn_func(q, k1, v1)
    assert torch.equal(T.triton_attn_func(q, k1.expand(-1, -1, 8, -1), v1.expand(-1, -1, 8, -1)), mqa)
    half = T.triton_attn_func(q, k1.expand(-1, -1, 2, -1), v)  # K shared by all heads, V by four
    ref = R.attention_variant_ref(q.float().cpu(), k1.expand(-1, -1, 2, -1).float().cpu(),
                                  v.float().cpu())
    assert float((half.float().cpu() - ref).abs().max()) <= TOL
    kb, vb = k[:1].expand(2, -1, -1, -1), v[:1].expand(2, -1, -1, -1)
    assert torch.equal(T.triton_attn_func(q, kb, vb),
                       T.triton_attn_func(q, kb.contiguous(), vb.contiguous()))
    assert T.attention_status(cuda) == 0


@pytest.mark.parametrize("Sk", [1, 31, 33, 127, 258, 264, 509])
@pytest.mark.parametrize("D,dtype", [(128, torch.bfloat16), (64, torch.float16)])
@pytest.mark.parametrize("wide", [True, False])
def test_dense_mask_at_every_alignment(cuda, Sk, D, dtype, wide):
    """The mask in fp32 and in the activation dtype, with rows that allow copies of 16, 4 and 2
    bytes (row lengths that are multiples of 8, even, odd; a view one element into its storage),
    keys hidden by -inf and by the type's lowest value, ragged last tiles. Bound as for the other
    masks: probabilities and result are each rounded once, 2^-9 * max|v| in bf16."""
    B, Sq, H = 2, 150, 4
    q, k, v = _qkv(B, Sq, Sk, H, 2, D, seed=Sk, dtype=dtype)
    mdt = torch.float32 if wide else dtype
    g = torch.Generator().manual_seed(Sk + D)
    mask = torch.randn(B, 1, Sq, Sk, generator=g)
    mask[torch.rand(B, 1, Sq, Sk, generator=g) < 0.2] = float("-inf")
    mask[:, :, :, 0] = 0.0  # every row sees a key
    if Sk > 8:
        mask[1, :, :, 5] = torch.finfo(mdt).min
    mask = mask.to(mdt)
    store = torch.zeros(mask.numel() + 1, dtype=mdt, device=cuda)
    for shift in (0, 1):
        m = store[shift:shift + mask.numel()].view(mask.shape).copy_(mask.to(cuda))
        out = T.triton_attn_func(q.to(cuda), k.to(cuda), v.to(cuda), attn_mask=m)
        assert T.attention_status(cuda) == 0
        _, ref32 = _mask_ref(q, k, v, mask.float(), False)
        assert float((out.float().cpu() - ref32).abs().max()) <= TOL


def test_recorded_failure_with_few_query_rows(cuda):
    """The decode kernel too skips its work on a recorded failure and writes the host mirror; with
    no failure the mirror stays untouched. The word is set from the host."""
    from trinix_b200 import ops
    q, k, v = (t.to(cuda) for t in _qkv(1, 2, 700, 8, 2, 128, seed=3))
    good = T.attention(q, k, v)
    torch.cuda.synchronize(cuda)
    assert int(ops._status_host[cuda.index or 0][0]) == 0
    ops._workspace(cuda)[:4].view(torch.int32).fill_(4)
    T.attention(q, k, v)
    torch.cuda.synchronize(cuda)
    assert int(ops._status_host[cuda.index or 0][0]) == 4
    with pytest.raises(T._lib.TrinixB200Error):
        T.attention(q, k, v)
    assert torch.equal(T.attention(q, k, v), good)
    assert T.attention_status(cuda) == 0


@pytest.mark.parametrize("B,Sq,Sk", [(16, 1, 4093), (40, 2, 3000), (1, 4, 20000), (64, 1, 300)])
def test_few_query_rows_while_a_failure_is_being_recorded(cuda, B, Sq, Sk):
    """The status word may turn non-zero while a launch runs (a launch on another stream gives up).
    Warps, CTAs and the CTAs of a cluster then read different values: every output row is either
    the whole result or untouched, never a sum of some of the parts. The word is written by a copy
    from the host beside the launch, at several distances; no wait is made to run out."""
    q, k, v = (t.to(cuda) for t in _qkv(B, Sq, Sk, 32, 8, 128, seed=B))
    good = T.attention(q, k, v)
    lib = T._lib.load()
    P, st3 = ctypes.c_void_p, T._lib.I64x3
    ws = torch.zeros(256, dtype=torch.uint8, device=cuda)
    word = torch.full((1,), 4, dtype=torch.int32).pin_memory()
    side, main = torch.cuda.Stream(cuda), torch.cuda.current_stream(cuda)
    mixed = 0
    for trial in range(60):
        ws.zero_()
        out = torch.full_like(q, 7.0)
        lse = torch.full((B, 32, Sq), 7.0, device=cuda)
        side.wait_stream(main)
        with torch.cuda.stream(side):
            torch.cuda._sleep(1500 * trial)  # 0 to 50 us
            ws[:4].view(torch.int32).copy_(word, non_blocking=True)
        assert lib.trx_attn_fwd(
            P(q.data_ptr()), P(k.data_ptr()), P(v.data_ptr()), P(out.data_ptr()), P(lse.data_ptr()),
            None, B, Sq, Sk, 32, 8, 128, st3(*q.stride()[:3]), st3(*k.stride()[:3]),
            st3(*v.stride()[:3]), st3(*out.stride()[:3]), 128 ** -0.5, 0, -1, -1, 2,
            P(ws.data_ptr()), 256, P(main.cuda_stream)) == 0
        torch.cuda.synchronize(cuda)
        same = (out == good).all(-1)
        untouched = (out == 7.0).all(-1)
        assert bool((same | untouched).all())
        assert torch.equal((lse == 7.0).transpose(1, 2), untouched)
        mixed += bool(same.any()) and bool(untouched.any())
    # nothing left over: the launch after it works
    assert torch.equal(T.attention(q, k, v), good) and T.attention_status(cuda) == 0
    print(f"{mixed} of 60 launches caught half way")


def test_recorded_failure_is_raised_once_with_calls_in_flight(cuda):
    """Launches that were queued before the host saw the failure skip their work and report it too,
    possibly after it was raised: that report belongs to the same failure."""
    from trinix_b200 import ops
    q, k, v = (t.to(cuda) for t in _qkv(1, 300, 300, 4, 2, 128, seed=13))
    good = T.attention(q, k, v)
    torch.cuda.synchronize(cuda)
    torch.cuda._sleep(60_000_000)  # some 30 ms, in which all of this is queued
    ops._workspace(cuda)[:4].view(torch.int32).fill_(4)
    T.attention(q, k, v)
    seen = torch.cuda.Event()
    seen.record()
    torch.cuda._sleep(60_000_000)
    T.attention(q, k, v)           # reports once more, long after the first one
    seen.synchronize()
    with pytest.raises(T._lib.TrinixB200Error):
        T.attention(q, k, v)
    for _ in range(3):
        assert torch.equal(T.attention(q, k, v), good)
        torch.cuda.synchronize(cuda)
    assert T.attention_status(cuda) == 0


@pytest.fixture
def no_workspace_yet(cuda, monkeypatch):
    """The state before a device's first attention call."""
    from trinix_b200 import ops
    T.attention(*(t.to(cuda) for t in _qkv(1, 16, 16, 2, 2, 64)))  # the library is loaded
    torch.cuda.synchronize(cuda)
    for name in ("_workspaces", "_status_host", "_status_word"):
        monkeypatch.setattr(ops, name, {})
    return ops


def test_first_calls_from_several_threads_share_one_workspace(cuda, no_workspace_yet):
    """One workspace and one host word per device, whoever comes first: a word that only a dropped
    workspace still points at would be written after it was given back."""
    ops, n = no_workspace_yet, 8
    start, got = threading.Barrier(n), [None] * n

    def first(i):
        start.wait()
        ws = ops._workspace(cuda)
        got[i] = (ws.data_ptr(), ops._status_host[0].data_ptr(), ctypes.addressof(ops._status_word[0]))

    threads = [threading.Thread(target=first, args=(i,)) for i in range(n)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(set(got)) == 1 and got[0][1] == got[0][2]
    attached = int(ops._workspace(cuda)[8:16].view(torch.int64).item())
    assert attached == got[0][1]  # unified addressing: the device's address of the word is the host's


def test_new_workspace_is_ready_for_every_stream(cuda, no_workspace_yet):
    side = torch.cuda.Stream(cuda)
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)
        ws = no_workspace_yet._workspace(cuda)
    assert side.query()  # nothing of its set-up is still to run when another stream uses it
    assert int(ws[:4].view(torch.int32).item()) == 0


def test_first_call_under_capture(cuda, no_workspace_yet):
    """The set-up is then part of the graph."""
    q, k, v = (t.to(cuda) for t in _qkv(1, 200, 200, 4, 2, 128, seed=17))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = T.attention(q, k, v, causal=True)
    graph.replay()
    torch.cuda.synchronize(cuda)
    assert torch.equal(out, T.attention(q, k, v, causal=True))
    assert T.attention_status(cuda) == 0
