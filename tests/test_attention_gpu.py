"""The hand-written tcgen05 flash-attention forward and backward (head_dim 128) against an fp32 softmax(QK^T)V
reference and its autograd gradients, through F.scaled_dot_product_attention (the default route on the device)."""
import math

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def ref_attention(q, k, v, causal):
    B, H, Sq, D = q.shape
    Hkv, Sk = k.shape[1], k.shape[2]
    kf = k.float().repeat_interleave(H // Hkv, dim=1)
    vf = v.float().repeat_interleave(H // Hkv, dim=1)
    s = q.float() @ kf.transpose(-1, -2) / math.sqrt(D)
    if causal:
        mask = torch.ones(Sq, Sk, dtype=torch.bool).tril()
        s = s.masked_fill(~mask, float("-inf"))
    return torch.softmax(s, -1) @ vf, torch.logsumexp(s, -1)


@pytest.fixture
def native_sdp(bw):
    prev = bw._C._sdp_impl()
    bw._C._set_sdp_impl(2)
    yield
    bw._C._set_sdp_impl(prev)


@pytest.mark.parametrize("B,H,Hkv,Sq,Sk,causal", [(1, 2, 2, 128, 128, False), (2, 4, 4, 256, 256, True),
                                                   (1, 4, 2, 384, 384, True), (1, 2, 1, 200, 200, True),
                                                   (2, 2, 2, 128, 320, False), (1, 8, 8, 1024, 1024, True)])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_native_forward(bw, dev, native_sdp, B, H, Hkv, Sq, Sk, causal, dt):
    torch.manual_seed(0)
    # [B, S, H, D] memory viewed as [B, H, S, D]: what a transformer block passes
    q = torch.randn(B, Sq, H, 128).to(dt).transpose(1, 2)
    k = torch.randn(B, Sk, Hkv, 128).to(dt).transpose(1, 2)
    v = torch.randn(B, Sk, Hkv, 128).to(dt).transpose(1, 2)
    ref, ref_lse = ref_attention(q, k, v, causal)
    before = bw._C._native_sdp_forward_calls()
    out = F.scaled_dot_product_attention(q.to(dev), k.to(dev), v.to(dev), is_causal=causal, enable_gqa=(H != Hkv))
    assert bw._C._native_sdp_forward_calls() == before + 1, "the hand-written forward did not run"
    tol = 2e-2 if dt == torch.bfloat16 else 4e-3
    err = (out.float().cpu() - ref).abs().max()
    assert err < tol, float(err)
    bw.synchronize()
    assert bw._C._gemm_status(False) == 0


def test_native_is_the_default_route(bw):
    assert bw._C._sdp_impl() == 2


@pytest.mark.parametrize("B,H,Hkv,Sq,Sk,causal", [(2, 4, 4, 256, 256, True), (1, 2, 2, 128, 128, False),
                                                   (1, 4, 2, 384, 384, True), (1, 2, 1, 200, 200, True),
                                                   (2, 2, 2, 128, 320, False), (1, 4, 4, 1024, 1024, True),
                                                   (1, 2, 2, 330, 200, False)])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_native_backward(bw, dev, native_sdp, B, H, Hkv, Sq, Sk, causal, dt):
    torch.manual_seed(1)
    q = torch.randn(B, Sq, H, 128).to(dt).transpose(1, 2)
    k = torch.randn(B, Sk, Hkv, 128).to(dt).transpose(1, 2)
    v = torch.randn(B, Sk, Hkv, 128).to(dt).transpose(1, 2)
    g = torch.randn(B, Sq, H, 128).to(dt).transpose(1, 2)
    qr, kr, vr = (t.float().requires_grad_() for t in (q, k, v))
    ref, _ = ref_attention(qr, kr, vr, causal)
    ref.backward(g.float())
    qd, kd, vd = (t.to(dev).requires_grad_() for t in (q, k, v))
    before = bw._C._native_sdp_backward_calls()
    out = F.scaled_dot_product_attention(qd, kd, vd, is_causal=causal, enable_gqa=(H != Hkv))
    out.backward(g.to(dev))
    assert bw._C._native_sdp_backward_calls() == before + 1, "the hand-written backward did not run"
    tol = 3e-2 if dt == torch.bfloat16 else 8e-3
    for name, a, b in (("dq", qd.grad, qr.grad), ("dk", kd.grad, kr.grad), ("dv", vd.grad, vr.grad)):
        assert a.shape == b.shape
        rel = (a.float().cpu() - b).abs().max() / b.abs().max()
        assert rel < tol, (name, float(rel))
    bw.synchronize()
    assert bw._C._gemm_status(False) == 0


def test_library_routes_still_work(bw, dev):
    """impl 0 / 1 (library flash / cuDNN kernels over the same memory) stay selectable."""
    torch.manual_seed(2)
    q, k, v = (torch.randn(1, 128, 2, 64).to(torch.bfloat16).transpose(1, 2) for _ in range(3))
    ref, _ = ref_attention(q, k, v, True)
    prev = bw._C._sdp_impl()
    try:
        for impl in (0, 1, 2):     # head_dim 64 is not covered by the hand-written kernels: impl 2 falls to flash
            bw._C._set_sdp_impl(impl)
            out = F.scaled_dot_product_attention(q.to(dev), k.to(dev), v.to(dev), is_causal=True)
            assert (out.float().cpu() - ref).abs().max() < 2e-2, impl
    finally:
        bw._C._set_sdp_impl(prev)


@pytest.mark.parametrize("H,Hkv,pos", [(4, 4, 0), (8, 2, 37), (4, 4, 255), (4, 1, 100), (4, 4, 31), (4, 2, 63), (4, 4, 64)])
def test_decode_attention(bw, dev, H, Hkv, pos):
    torch.manual_seed(0)
    B, L = 3, 256
    q = torch.randn(B, H, 128).to(torch.bfloat16)
    kc, vc = (torch.randn(B, Hkv, L, 128).to(torch.bfloat16) for _ in range(2))
    ref, _ = ref_attention(q.unsqueeze(2), kc[:, :, :pos + 1], vc[:, :, :pos + 1], False)
    p = torch.tensor([pos], dtype=torch.long, device=dev)
    out = torch.ops.blackwell.decode_attention(q.to(dev), kc.to(dev), vc.to(dev), p)
    assert (out.float().cpu() - ref.squeeze(2)).abs().max() < 2e-2


def test_bf16_graph_decode_runs_fused_kernel(bw, dev):
    from torch_musa_b200.models import Llama, LlamaConfig
    from torch_musa_b200.models.decode import LlamaDecoder

    cfg = LlamaConfig(vocab_size=512, dim=256, n_layers=2, n_heads=2, ffn_dim=512, max_seq_len=64)   # head_dim 128
    torch.manual_seed(0)
    model = Llama(cfg).to(dev).to(torch.bfloat16).eval()
    prompt = torch.randint(0, 512, (4, 9), device=dev)
    a = LlamaDecoder(model, 4, 64, device=dev)
    assert a._fused_decode
    a.prefill(prompt)
    eager = a.decode(6).cpu()
    b = LlamaDecoder(model, 4, 64, device=dev)
    b.prefill(prompt)
    b.capture()
    assert torch.equal(b.decode(6).cpu(), eager)


@pytest.mark.parametrize("lens,H,Hkv,causal", [([128, 256], 2, 2, False), ([77, 300, 1, 129], 4, 2, True),
                                               ([513], 2, 1, True), ([64, 64, 64, 200], 4, 4, False)])
def test_packed_variable_length_attention(bw, dev, lens, H, Hkv, causal):
    """Sequences of different lengths packed without padding: one launch each for forward and backward, lengths read
    on the device; compared per sequence with the fp32 reference and its autograd gradients."""
    from torch_musa_b200.ops import flash_attn_varlen_func

    torch.manual_seed(0)
    total = sum(lens)
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32)
    q0 = torch.randn(total, H, 128).to(torch.bfloat16)
    k0 = torch.randn(total, Hkv, 128).to(torch.bfloat16)
    v0 = torch.randn(total, Hkv, 128).to(torch.bfloat16)
    g0 = torch.randn(total, H, 128).to(torch.bfloat16)
    # fp32 oracle, sequence by sequence
    qr, kr, vr = (t.float().requires_grad_() for t in (q0, k0, v0))
    outs = []
    for i in range(len(lens)):
        s, e = int(cu[i]), int(cu[i + 1])
        o, _ = ref_attention(qr[s:e].transpose(0, 1).unsqueeze(0), kr[s:e].transpose(0, 1).unsqueeze(0),
                             vr[s:e].transpose(0, 1).unsqueeze(0), causal)
        outs.append(o.squeeze(0).transpose(0, 1))
    ref = torch.cat(outs, 0)
    ref.backward(g0.float())
    qd, kd, vd = (t.to(dev).requires_grad_() for t in (q0, k0, v0))
    f0, b0 = bw._C._native_sdp_forward_calls(), bw._C._native_sdp_backward_calls()
    out = flash_attn_varlen_func(qd, kd, vd, cu.to(dev), cu.to(dev), max(lens), max(lens), causal=causal)
    out.backward(g0.to(dev))
    assert bw._C._native_sdp_forward_calls() == f0 + 1 and bw._C._native_sdp_backward_calls() == b0 + 1
    assert bw._C._gemm_status() == 0
    assert (out.float().cpu() - ref).abs().max() < 2e-2
    for got, want in ((qd.grad, qr.grad), (kd.grad, kr.grad), (vd.grad, vr.grad)):
        assert (got.float().cpu() - want).abs().max() < 6e-2 * max(1.0, float(want.abs().max()))
    # the host-side composition of the same contract agrees with the oracle too
    cpu = flash_attn_varlen_func(q0.float(), k0.float(), v0.float(), cu, cu, max(lens), max(lens), causal=causal)
    assert (cpu - ref.detach()).abs().max() < 1e-3


@pytest.mark.parametrize("fused_qkv", [True, False])
def test_decode_rope_and_cache_update_in_one_launch(bw, dev, fused_qkv):
    """q rotated into a fresh buffer, k rotated into the key cache at the device-side position, v copied into the
    value cache; packed qkv views (strided) and separate tensors; against the fp32 rotate-half formula."""
    from torch_musa_b200.ops import precompute_rope_cache

    torch.manual_seed(0)
    B, H, Hkv, L, pos = 3, 4, 2, 32, 17
    cos, sin = precompute_rope_cache(L, 128)
    if fused_qkv:
        qkv = torch.randn(B, 1, H + 2 * Hkv, 128).to(torch.bfloat16)
        q, k, v = qkv.split([H, Hkv, Hkv], dim=2)
        qd, kd, vd = qkv.to(dev).split([H, Hkv, Hkv], dim=2)
    else:
        q, k, v = (torch.randn(B, 1, n, 128).to(torch.bfloat16) for n in (H, Hkv, Hkv))
        qd, kd, vd = q.to(dev), k.to(dev), v.to(dev)
    kc = torch.full((B, Hkv, L, 128), 9.0, dtype=torch.bfloat16, device=dev)
    vc = torch.full((B, Hkv, L, 128), 9.0, dtype=torch.bfloat16, device=dev)
    p = torch.tensor([pos], dtype=torch.long, device=dev)
    bw.reset_kernel_launch_count()
    qr = torch.ops.blackwell.decode_rope_cache(qd, kd, vd, cos.to(dev), sin.to(dev), p, kc, vc)
    assert bw.kernel_launch_count() == 1

    def rot(x):                                   # [B, 1, n, 128] -> rotate-half at position pos, fp32
        x = x.float()
        a, b = x[..., :64], x[..., 64:]
        c, s = cos[pos], sin[pos]
        return torch.cat([a * c - b * s, b * c + a * s], -1)

    assert (qr.float().cpu() - rot(q).squeeze(1)).abs().max() < 3e-2
    assert (kc[:, :, pos].float().cpu() - rot(k).squeeze(1)).abs().max() < 3e-2
    assert torch.equal(vc[:, :, pos].cpu(), v.squeeze(1))
    untouched = torch.ones(L, dtype=torch.bool)
    untouched[pos] = False
    assert bool((kc[:, :, untouched.to(dev)] == 9.0).all()) and bool((vc[:, :, untouched.to(dev)] == 9.0).all())


@pytest.mark.parametrize("S", [1, 127, 129, 385, 640])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_forward_maximum_rises_with_every_block(bw, dev, native_sdp, S, causal, dt):
    """The scores grow along the keys, so the softmax's reference maximum is raised and the output rescaled in every
    block of 128 keys, also in one that the first half of a block has already been computed for."""
    torch.manual_seed(5)
    q = torch.randn(1, S, 2, 128).abs().to(dt).transpose(1, 2)
    ramp = (torch.arange(S) / 32.0).view(1, S, 1, 1) * 0.4
    k = (torch.randn(1, S, 2, 128) * 0.1 + ramp).to(dt).transpose(1, 2)
    v = torch.randn(1, S, 2, 128).to(dt).transpose(1, 2)
    ref, _ = ref_attention(q, k, v, causal)
    before = bw._C._native_sdp_forward_calls()
    out = F.scaled_dot_product_attention(q.to(dev), k.to(dev), v.to(dev), is_causal=causal)
    assert bw._C._native_sdp_forward_calls() == before + 1
    # P is rounded to 16 bits before it multiplies V (|v| < 5): 5 * 2^-9 (bf16) or 5 * 2^-12 (fp16), plus the output's rounding
    tol = 2e-2 if dt == torch.bfloat16 else 4e-3
    assert (out.float().cpu() - ref).abs().max() < tol
    bw.synchronize()
    assert bw._C._gemm_status(False) == 0


@pytest.mark.parametrize("Sq,Sk,H,Hkv", [(1, 1, 1, 1), (129, 129, 4, 1), (257, 385, 2, 2), (64, 257, 4, 2), (513, 127, 2, 1)])
@pytest.mark.parametrize("causal", [False, True])
def test_backward_edges(bw, dev, native_sdp, Sq, Sk, H, Hkv, causal):
    """Remainders of the query and key blocks, one and several pairs per block of keys, grouped heads; causal with fewer
    and with more keys than queries (keys without any query get zero gradients)."""
    torch.manual_seed(6)
    q, g = (torch.randn(2, Sq, H, 128).bfloat16().transpose(1, 2) for _ in range(2))
    k, v = (torch.randn(2, Sk, Hkv, 128).bfloat16().transpose(1, 2) for _ in range(2))
    qr, kr, vr = (t.float().requires_grad_() for t in (q, k, v))
    ref, _ = ref_attention(qr, kr, vr, causal)
    ref.backward(g.float())
    qd, kd, vd = (t.to(dev).requires_grad_() for t in (q, k, v))
    before = bw._C._native_sdp_backward_calls()
    out = F.scaled_dot_product_attention(qd, kd, vd, is_causal=causal, enable_gqa=(H != Hkv))
    out.backward(g.to(dev))
    assert bw._C._native_sdp_backward_calls() == before + 1
    for name, a, b in (("dq", qd.grad, qr.grad), ("dk", kd.grad, kr.grad), ("dv", vd.grad, vr.grad)):
        a = a.float().cpu()
        if Sq == 1 and Sk == 1 and name != "dv":     # the softmax is constant: rounding noise of the two sums that cancel
            assert a.abs().max() < 3e-2, name
            continue
        # P and dS are rounded to bf16 (2^-9) before they are multiplied, the result is rounded again: 3e-2 of the largest entry
        # as above
        err = (a - b).abs().max()
        assert err < 3e-2 * b.abs().max(), (name, float(err))
        # and for every block of 128 rows by itself, in the 2-norm: those two roundings, the output's in delta, and the
        # cancellation in dP - delta come to a few times 2^-9; rows that no query sees are exact zeros
        for i, (ab, bb) in enumerate(zip(a.split(128, 2), b.split(128, 2))):
            assert (ab - bb).norm() <= 8 * 2.0 ** -9 * bb.norm(), (name, i, float((ab - bb).norm() / bb.norm()))
    bw.synchronize()
    assert bw._C._gemm_status(False) == 0
