"""tcgen05 causal attention (forward + backward) against fp32 SDPA on the same inputs."""

import math
import os

import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from bitscom_b200.ops import _native, attention as A


def _ref(qkv, B, S, nh, hd):
    H = nh * hd
    q, k, v = (qkv[:, i * H:(i + 1) * H].view(B, S, nh, hd).transpose(1, 2) for i in range(3))
    o = torch.nn.functional.scaled_dot_product_attention(q, k, v, is_causal=True)
    return o.transpose(1, 2).reshape(B * S, H)


@pytest.mark.parametrize("hd", [128, 64])
@pytest.mark.parametrize("B,S,nh", [(1, 128, 1), (2, 256, 2), (1, 512, 4), (1, 2048, 2)])
def test_attention_forward_backward(B, S, nh, hd):
    assert A.available() and A.supported(S, hd)
    H = nh * hd
    g = torch.Generator(device="cuda").manual_seed(S + nh)
    qkv = (torch.randn(B * S, 3 * H, device="cuda", generator=g) * 0.7).to(torch.bfloat16)
    d_out = (torch.randn(B * S, H, device="cuda", generator=g) * 0.5).to(torch.bfloat16)

    x = qkv.clone().requires_grad_()
    out = A.attention(x, B, S, nh, hd)
    out.backward(d_out)
    torch.cuda.synchronize()
    A.check_status()

    xr = qkv.float().requires_grad_()
    ref = _ref(xr, B, S, nh, hd)
    ref.backward(d_out.float())

    err = (out.float() - ref).abs().max().item()
    assert err < 2e-2, f"forward max err {err}"
    for name, lo in (("dq", 0), ("dk", H), ("dv", 2 * H)):
        got, want = x.grad[:, lo:lo + H].float(), xr.grad[:, lo:lo + H]
        e = (got - want).abs().max().item()
        tol = 3e-2 * max(1.0, want.abs().max().item())
        assert e < tol, f"{name} max err {e} (tol {tol})"


@pytest.mark.parametrize("variant", ["pipelined", "simple"])
@pytest.mark.parametrize("hd", [128, 64])
@pytest.mark.parametrize("B,S,nh", [(1, 128, 1), (2, 384, 2), (1, 2048, 2)])
def test_forward_variants_match_reference(B, S, nh, hd, variant):
    """Both forward kernels against fp32 SDPA: the software-pipelined one (issuer warp, scores
    double-buffered in TMEM, output accumulated in TMEM with rescaling on demand; the default)
    and the simple one whose MMA and softmax take turns.  The log-sum-exp each writes is
    checked through the backward pass of the same call."""
    H = nh * hd
    g = torch.Generator(device="cuda").manual_seed(S + nh + hd)
    qkv = (torch.randn(B * S, 3 * H, device="cuda", generator=g) * 0.7).to(torch.bfloat16)
    d_out = (torch.randn(B * S, H, device="cuda", generator=g) * 0.5).to(torch.bfloat16)
    before = A.set_forward_variant(variant)
    try:
        x = qkv.clone().requires_grad_()
        out = A.attention(x, B, S, nh, hd)
        out.backward(d_out)
        torch.cuda.synchronize()
        A.check_status()
    finally:
        A.set_forward_variant(before)
    xr = qkv.float().requires_grad_()
    ref = _ref(xr, B, S, nh, hd)
    ref.backward(d_out.float())
    err = (out.float() - ref).abs().max().item()
    assert err < 2e-2, f"forward max err {err}"
    e = (x.grad.float() - xr.grad).abs().max().item()
    assert e < 3e-2 * max(1.0, xr.grad.abs().max().item()), f"grad max err {e}"


@pytest.mark.parametrize("dq", ["tma", "atomic"])
@pytest.mark.parametrize("hd", [128, 64])
@pytest.mark.parametrize("B,S,nh", [(1, 128, 1), (2, 384, 2), (1, 1024, 3)])
def test_backward_dq_variants_match_reference(B, S, nh, hd, dq):
    """dQ accumulated by TMA reductions from a swizzled staging tile, and by float4 atomics,
    against fp32 autograd; two calls in a row (the accumulator must be left zeroed)."""
    H = nh * hd
    g = torch.Generator(device="cuda").manual_seed(7 * S + nh + hd)
    qkv = (torch.randn(B * S, 3 * H, device="cuda", generator=g) * 0.7).to(torch.bfloat16)
    d_out = (torch.randn(B * S, H, device="cuda", generator=g) * 0.5).to(torch.bfloat16)
    xr = qkv.float().requires_grad_()
    _ref(xr, B, S, nh, hd).backward(d_out.float())
    before = A.set_backward_dq_variant(dq)
    try:
        for _ in range(2):
            x = qkv.clone().requires_grad_()
            A.attention(x, B, S, nh, hd).backward(d_out)
            torch.cuda.synchronize()
            A.check_status()
            for name, lo in (("dq", 0), ("dk", H), ("dv", 2 * H)):
                got, want = x.grad[:, lo:lo + H].float(), xr.grad[:, lo:lo + H]
                e = (got - want).abs().max().item()
                tol = 3e-2 * max(1.0, want.abs().max().item())
                assert e < tol, f"{name} max err {e} (tol {tol})"
    finally:
        A.set_backward_dq_variant(before)


@pytest.mark.parametrize("hd", [128, 64])
@pytest.mark.parametrize("B,S,nh,growth", [(19, 128, 8, 0.0), (10, 384, 6, 0.0), (2, 1024, 10, 4.0)])
def test_persistent_kernels_match_reference(B, S, nh, growth, hd):
    """More tiles than SMs: the two-tile forward kernel and the persistent backward kernel, whose
    CTAs take several items each; single-block items, an odd number of query blocks (last pair
    without its second tile), and keys that grow along the sequence, so that the row maxima rise
    in every block.  bf16 P and output: 2^-8 relative of the largest value, with a factor 4."""
    H = nh * hd
    g = torch.Generator(device="cuda").manual_seed(B + S + hd)
    qkv = torch.randn(B * S, 3 * H, device="cuda", generator=g) * 0.7
    qkv[:, H:2 * H] *= (1 + growth * torch.arange(S, device="cuda") / S).repeat(B)[:, None]
    qkv = qkv.to(torch.bfloat16)
    d_out = (torch.randn(B * S, H, device="cuda", generator=g) * 0.5).to(torch.bfloat16)
    assert B * nh * (S // 128) > 148
    x = qkv.clone().requires_grad_()
    out = A.attention(x, B, S, nh, hd)
    out.backward(d_out)
    torch.cuda.synchronize()
    A.check_status()
    xr = qkv.float().requires_grad_()
    ref = _ref(xr, B, S, nh, hd)
    ref.backward(d_out.float())
    assert (out.float() - ref).abs().max().item() < 2 ** -6 * ref.abs().max().item()
    for name, lo in (("dq", 0), ("dk", H), ("dv", 2 * H)):
        got, want = x.grad[:, lo:lo + H].float(), xr.grad[:, lo:lo + H]
        e = (got - want).abs().max().item()
        assert e < 2 ** -6 * want.abs().max().item(), f"{name} max err {e}"


@pytest.mark.parametrize("hd", [128, 64])
@pytest.mark.parametrize("exponent", [-129, -140])
def test_backward_of_small_probabilities(hd, exponent):
    """One query that gives a key the probability 2^exponent, below fp32's normal range, and an
    output gradient that makes it count: P must reach dS as it is (dQ, dK), and P^T dO as far as bf16
    has it (dv of 2^-129: subnormal spacing 2^-133).  ex2 of an argument rounded to 2^-17 and one
    rounding to bf16; 2^-140 has 9 bits in fp32."""
    S, scale = 128, hd ** -0.5
    qkv = torch.zeros(S, 3 * hd, device="cuda")
    qkv[S - 1, 0] = 1.0
    qkv[0, hd] = (exponent + 7) * math.log(2) / scale   # 127 other keys share the rest
    qkv[0, 2 * hd + 1] = 2.0
    x = qkv.to(torch.bfloat16).requires_grad_()
    d_out = torch.zeros(S, hd, device="cuda", dtype=torch.bfloat16)
    d_out[S - 1] = 2.0 ** 115
    A.attention(x, 1, S, 1, hd).backward(d_out)
    xr = x.detach().double().requires_grad_()
    q, k, v = xr[:, :hd], xr[:, hd:2 * hd], xr[:, 2 * hd:]
    causal = torch.ones(S, S, dtype=torch.bool, device="cuda").tril()
    p = torch.softmax((q @ k.t() * scale).masked_fill(~causal, float("-inf")), -1)
    (p @ v).backward(d_out.double())
    assert 2.0 ** (exponent - 1) < p[S - 1, 0].item() < 2.0 ** (exponent + 1)
    got, want = x.grad.double(), xr.grad
    for row, col in ((S - 1, 0), (0, hd)):  # dq of the query, dk of the key
        assert abs(got[row, col] - want[row, col]) <= 2.0 ** -6 * abs(want[row, col])
    if exponent > -133:
        assert abs(got[0, 2 * hd] - want[0, 2 * hd]) <= 2.0 ** -4 * abs(want[0, 2 * hd])


def test_attention_second_call_reuses_zeroed_scratch():
    B, S, nh, hd = 1, 256, 2, 128
    H = nh * hd
    qkv = (torch.randn(B * S, 3 * H, device="cuda") * 0.5).to(torch.bfloat16)
    d_out = (torch.randn(B * S, H, device="cuda") * 0.5).to(torch.bfloat16)
    grads = []
    for _ in range(2):
        x = qkv.clone().requires_grad_()
        A.attention(x, B, S, nh, hd).backward(d_out)
        grads.append(x.grad.clone())
    assert torch.equal(grads[0], grads[1])


@pytest.mark.parametrize("variant", ["atomic", "tma", "pipelined"])
@pytest.mark.parametrize("B,S,nh,hd", [(1, 128, 1, 128), (3, 256, 5, 64), (1, 384, 3, 128)])
def test_backward_scratch_may_hold_anything(variant, B, S, nh, hd):
    """The dQ accumulator and the row sums are given to the C entry full of other values."""
    lib, stream, H, scale = A._get(), _native.stream_ptr(), nh * hd, hd ** -0.5
    qkv = (torch.randn(B * S, 3 * H, device="cuda") * 0.5).to(torch.bfloat16)
    d_out = (torch.randn(B * S, H, device="cuda") * 0.5).to(torch.bfloat16)
    out, lse = torch.empty_like(d_out), torch.empty(B, nh, S, device="cuda")
    check = _native.check
    check(lib.bcom_attention_fwd(qkv.data_ptr(), out.data_ptr(), lse.data_ptr(), B, S, nh, hd, scale,
                                 stream), "fwd")
    got = []
    before = A.set_backward_dq_variant(variant)
    try:
        for fill in (0.0, 3.0, float("nan")):
            acc = torch.full((B * S, H), fill, device="cuda")
            delta = torch.full((B, nh, S), fill, device="cuda")
            got.append(torch.empty_like(qkv))
            check(lib.bcom_attention_bwd(
                qkv.data_ptr(), out.data_ptr(), d_out.data_ptr(), lse.data_ptr(), got[-1].data_ptr(),
                acc.data_ptr(), delta.data_ptr(), B, S, nh, hd, scale, stream), "bwd")
    finally:
        A.set_backward_dq_variant(before)
    torch.cuda.synchronize()
    A.check_status()
    for other in got[1:]:  # dq is a sum in any order: up to 3 terms here
        assert torch.equal(other[:, H:], got[0][:, H:])
        assert torch.allclose(other[:, :H].float(), got[0][:, :H].float(), rtol=2 ** -7, atol=1e-5)


def test_backward_passes_on_two_streams_at_once():
    """Passes of one shape on two streams, queued behind a wait so that they run together.  Two key
    blocks per sequence: a sum of two dQ terms does not depend on their order."""
    B, S, nh, hd = 24, 256, 8, 128
    H, work = nh * hd, []
    for seed in range(2):
        g = torch.Generator(device="cuda").manual_seed(seed)
        qkv = (torch.randn(B * S, 3 * H, device="cuda", generator=g) * 0.5).to(torch.bfloat16)
        d_out = (torch.randn(B * S, H, device="cuda", generator=g) * 0.5).to(torch.bfloat16)
        qkv.requires_grad_()
        out = A.attention(qkv, B, S, nh, hd)
        want = torch.autograd.grad(out, qkv, d_out, retain_graph=True)[0]
        work.append((qkv, d_out, out, want, torch.cuda.Stream()))
    torch.cuda.synchronize()
    grads = [[], []]
    for qkv, d_out, _, _, stream in work:
        with torch.cuda.stream(stream):
            torch.cuda._sleep(20_000_000)
    for _ in range(8):
        for i, (qkv, d_out, _, _, stream) in enumerate(work):
            with torch.cuda.stream(stream):
                out = A.attention(qkv, B, S, nh, hd)
                grads[i].append(torch.autograd.grad(out, qkv, d_out)[0])
    torch.cuda.synchronize()
    A.check_status()
    for got, (_, _, _, want, _) in zip(grads, work):
        assert all(torch.equal(g, want) for g in got)


@pytest.mark.performance
def test_attention_throughput_report():
    B, S, nh, hd = 2, 2048, 32, 128
    H = nh * hd
    qkv = (torch.randn(B * S, 3 * H, device="cuda") * 0.5).to(torch.bfloat16).requires_grad_()
    d_out = (torch.randn(B * S, H, device="cuda") * 0.5).to(torch.bfloat16)
    flops_fwd = 4 * B * nh * S * S * hd / 2
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(3)]
    for _ in range(2):
        A.attention(qkv, B, S, nh, hd).backward(d_out)
    ev[0].record()
    out = A.attention(qkv, B, S, nh, hd)
    ev[1].record()
    out.backward(d_out)
    ev[2].record()
    torch.cuda.synchronize()
    A.check_status()
    f, b = ev[0].elapsed_time(ev[1]), ev[1].elapsed_time(ev[2])
    print(f"attention fwd {f:.3f} ms = {flops_fwd / f / 1e9:.0f} TFLOP/s; "
          f"bwd {b:.3f} ms = {2.5 * flops_fwd / b / 1e9:.0f} TFLOP/s")
