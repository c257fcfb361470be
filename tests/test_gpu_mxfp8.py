"""MXFP8: quantiser bit-exact against the PyTorch restatement, block-scaled GEMM against the fp32
product of the dequantised operands, linear layer against bf16."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K", [(128, 128), (300, 256), (4096, 1280), (77, 3584)])
def test_quantize_bit_exact(M, K):
    from kohakuwullm_b200.ops import mxfp8 as mx

    torch.manual_seed(0)
    x = (torch.randn(M, K, device="cuda") * torch.logspace(-3, 2, K, device="cuda")).to(torch.bfloat16)
    x[0, :32] = 0  # an all-zero block
    q, sf = mx.quantize(x)
    q_ref, e_ref = mx.quantize_reference(x)
    assert torch.equal(mx.sf_to_natural(sf, M, K), e_ref)
    assert torch.equal(q.view(torch.float8_e4m3fn).float(), q_ref.float())
    # rows of the last 128-row tile beyond M carry the neutral exponent, never 0xFF
    pad = mx.sf_to_natural(sf, (M + 127) // 128 * 128, K)[M:]
    assert (pad == 127).all()


@pytest.mark.parametrize("R,C", [(128, 128), (1280, 1792), (3584, 1280)])
def test_quantize_transposed_matches_rowwise_of_transpose(R, C):
    from kohakuwullm_b200.ops import mxfp8 as mx

    torch.manual_seed(1)
    w = (torch.randn(R, C, device="cuda") * 0.05).to(torch.bfloat16)
    qt, sft = mx.quantize_transposed(w)
    q_ref, sf_ref = mx.quantize(w.t().contiguous())
    assert torch.equal(qt, q_ref)
    assert torch.equal(mx.sf_to_natural(sft, C, R), mx.sf_to_natural(sf_ref, C, R))


@pytest.mark.parametrize("M,N,K", [(128, 128, 128), (256, 384, 512), (4096, 1792, 1280), (1000, 1280, 3584)])
def test_block_scaled_gemm_matches_dequantised_product(M, N, K):
    from kohakuwullm_b200.ops import mxfp8 as mx, native

    torch.manual_seed(2)
    a = (torch.randn(M, K, device="cuda") * torch.logspace(-2, 1, K, device="cuda")).to(torch.bfloat16)
    b = (torch.randn(N, K, device="cuda") * 0.1).to(torch.bfloat16)
    aq, asf = mx.quantize(a)
    bq, bsf = mx.quantize(b)
    out = mx.gemm(aq, asf, bq, bsf, out_dtype=torch.float32)
    torch.cuda.synchronize()
    native.check_status()
    ref = (mx.dequantize(aq.view(torch.float8_e4m3fn), mx.sf_to_natural(asf, M, K))
           @ mx.dequantize(bq.view(torch.float8_e4m3fn), mx.sf_to_natural(bsf, N, K)).t())
    err = (out - ref).abs().max().item()
    assert err <= 2e-3 * ref.abs().max().item() + 1e-4, f"err {err} scale {ref.abs().max().item()}"


def test_mxfp8_linear_fwd_bwd_close_to_bf16():
    from kohakuwullm_b200.models.components.mlp import Linear
    from kohakuwullm_b200.ops import native

    torch.manual_seed(3)
    lin = Linear(1280, 1792).cuda()
    torch.nn.init.normal_(lin.weight, std=0.02)
    lin.weight.data = lin.weight.data.to(torch.bfloat16)
    x = torch.randn(512, 1280, device="cuda", dtype=torch.bfloat16)
    dy = torch.randn(512, 1792, device="cuda", dtype=torch.bfloat16)
    xa = x.clone().requires_grad_()
    ya = lin(xa)
    ya.backward(dy)
    ga, gw = xa.grad.clone(), lin.weight.grad.clone()
    lin.weight.grad = None
    lin.mxfp8 = True
    xb = x.clone().requires_grad_()
    yb = lin(xb)
    yb.backward(dy)
    torch.cuda.synchronize()
    native.check_status()
    for got, want, tol in ((yb, ya, 0.06), (xb.grad, ga, 0.06), (lin.weight.grad, gw, 0.02)):
        rel = (got.float() - want.float()).norm() / want.float().norm()
        assert rel < tol, f"relative error {rel}"


def test_producer_made_fp8_copies_equal_the_quantise_kernel():
    """RMSNorm / SwiGLU (forward and backward) writing the MXFP8 copy in the same pass give the same bytes
    and scales as quantising their stored bf16 output afterwards."""
    from kohakuwullm_b200.ops import mxfp8 as mx
    from kohakuwullm_b200.ops.elementwise import rmsnorm, swiglu

    torch.manual_seed(5)
    rows, cols, H = 512, 1280, 896
    mx.clear_prequantized()
    # RMSNorm with fused residual add
    x = (torch.randn(rows, cols, device="cuda") * 2).bfloat16().requires_grad_()
    res = torch.randn(rows, cols, device="cuda").bfloat16().requires_grad_()
    w = torch.rand(cols, device="cuda").requires_grad_()
    y, h = rmsnorm(x, w, 1e-6, False, res, emit_mx=True, emit_mx_grad=True)
    got = mx.take_quantized(y.reshape(rows, cols))
    assert got is not None
    q_ref, sf_ref = mx.quantize(y.detach().reshape(rows, cols).contiguous())
    assert torch.equal(got[0], q_ref) and torch.equal(got[1], sf_ref)
    dy = torch.randn(rows, cols, device="cuda").bfloat16()
    dh = torch.randn(rows, cols, device="cuda").bfloat16()
    # the consumer (a projection's backward) receives the gradient tensor itself, not a leaf's accumulated copy
    seen = {}
    y, h = rmsnorm(x * 1.0, w, 1e-6, False, res, emit_mx=True, emit_mx_grad=True)
    mx.take_quantized(y.reshape(rows, cols))
    y.grad_fn.next_functions[0][0].register_prehook(lambda grads: seen.update(g=grads[0]))
    torch.autograd.backward([y, h], [dy, dh])
    g = seen["g"].reshape(rows, cols)
    got = mx.take_quantized(g)
    assert got is not None
    q_ref, sf_ref = mx.quantize(g.contiguous())
    assert torch.equal(got[0], q_ref) and torch.equal(got[1], sf_ref)
    # the gradients themselves are unchanged by the emission
    x2, r2, w2 = (t.detach().clone().requires_grad_() for t in (x, res, w))
    y2, h2 = rmsnorm(x2, w2, 1e-6, False, r2)
    torch.autograd.backward([y2, h2], [dy, dh])
    assert torch.equal(x2.grad, x.grad)
    torch.testing.assert_close(w2.grad, w.grad, rtol=1e-5, atol=1e-4)   # block partials meet in fp32 atomics
    # SwiGLU
    hh = torch.randn(rows, 2 * H, device="cuda").bfloat16().requires_grad_()
    a = swiglu(hh, emit_mx=True, emit_mx_grad=True)
    got = mx.take_quantized(a)
    q_ref, sf_ref = mx.quantize(a.detach())
    assert got is not None and torch.equal(got[0], q_ref) and torch.equal(got[1], sf_ref)
    a = swiglu(hh * 1.0, emit_mx=True, emit_mx_grad=True)
    mx.take_quantized(a)
    a.grad_fn.next_functions[0][0].register_prehook(lambda grads: seen.update(gh=grads[0]))
    a.backward(torch.randn(rows, H, device="cuda").bfloat16())
    got = mx.take_quantized(seen["gh"])
    q_ref, sf_ref = mx.quantize(seen["gh"].contiguous())
    assert got is not None and torch.equal(got[0], q_ref) and torch.equal(got[1], sf_ref)


def test_training_step_identical_with_and_without_fused_quantisation():
    from kohakuwullm_b200.data.synthetic import make_packs
    from kohakuwullm_b200.models import LMBackbone, get_preset
    from kohakuwullm_b200.models.components.norm import RMSNorm
    from kohakuwullm_b200.ops import native
    from kohakuwullm_b200.training.engine import TrainEngine

    def run(fused: bool):
        torch.manual_seed(0)
        cfg = get_preset("B200-dense-546M", depth=3, vocab_size=4096)
        with torch.device("cuda"):
            model = LMBackbone(cfg)
        flags = 0
        for m in model.modules():
            if isinstance(m, RMSNorm):
                flags += int(m.emit_mx) + int(m.emit_mx_grad)
                if not fused:
                    m.emit_mx = m.emit_mx_grad = False
        assert flags >= 4 * cfg.depth - 1
        if not fused:
            from kohakuwullm_b200.ops.elementwise import swiglu

            def plain_forward(mlp):
                return lambda x: mlp.w_out(swiglu(mlp.w_in(x)))   # no fp8 emission from the activation kernel

            for blk in model.blocks:
                blk.mlp.forward = plain_forward(blk.mlp)
        eng = TrainEngine(model, lr=1e-3, param_dtype=torch.bfloat16, cuda_graphs=False)
        packs = make_packs(2, 1024, 64, 512, cfg.vocab_size, seed=9)
        outs = [float(eng.step(packs)["loss"]) for _ in range(2)]
        torch.cuda.synchronize()
        native.check_status()
        return outs, torch.cat([g.data.float().reshape(-1) for g in eng.flat.groups.values()])

    (la, pa), (lb, pb) = run(True), run(False)
    # the fp8 copies are bit-identical (previous test); the two runs still differ in the order of fp32
    # atomic partial sums (norm weight gradients, split-K), so parameters agree to rounding, not bitwise
    assert abs(la[0] - lb[0]) < 1e-6, (la, lb)        # the forward pass has no atomics: identical
    assert abs(la[1] - lb[1]) < 2e-2, (la, lb)
    assert (pa - pb).abs().max().item() < 1e-2


@pytest.mark.parametrize("M,N,K,bn", [
    (256, 1280, 256, 144), (384, 1792, 384, 208), (200, 3584, 128, 224), (128, 1280, 512, 160),
    (512, 768, 256, 192), (130, 2048, 256, 240), (256, 1296, 128, 176),
])
def test_wide_tiles_with_tile_local_weight_scales_equal_the_128_wide_kernel(M, N, K, bn):
    """A weight quantised with its scales laid out for ``bn``-wide tiles gives, through the ``bn``-wide GEMM, the
    same bytes as the plain layout through the 128-wide GEMM (same products, same fp32 summation order), also
    when the last tile hangs over the matrix edge; the transposed (dgrad) copy likewise."""
    from kohakuwullm_b200.ops import mxfp8 as mx
    from kohakuwullm_b200.ops import native

    torch.manual_seed(M + N + bn)
    a = torch.randn(M, K, device="cuda").bfloat16()
    w = (torch.randn(N, K, device="cuda") * 0.1).bfloat16()
    aq, asf = mx.quantize(a)
    wq, wsf = mx.quantize(w)
    ref = mx.gemm(aq, asf, wq, wsf)
    q2 = torch.empty(N, K, dtype=torch.uint8, device="cuda")
    sf2 = mx.alloc_weight_sf(N, K, bn, "cuda")
    mx.quantize_weight(w, q2, sf2, bn)
    assert torch.equal(q2, wq)
    out = mx.gemm(aq, asf, q2, sf2, bn=bn)
    assert torch.equal(out, ref)
    # transposed copy: W^T (K, N) as the B operand of dy (M, N) @ W -> (M, K); needs N % 128 == 0
    if N % 128 == 0:
        dy = torch.randn(M, N, device="cuda").bfloat16()
        dq, dsf = mx.quantize(dy)
        qt, sft = mx.quantize_transposed(w)
        ref_t = mx.gemm(dq, dsf, qt, sft)
        qt2 = torch.empty(K, N, dtype=torch.uint8, device="cuda")
        sft2 = mx.alloc_weight_sf(K, N, bn, "cuda")
        mx.quantize_weight_transposed(w, qt2, sft2, bn)
        assert torch.equal(qt2, qt)
        assert torch.equal(mx.gemm(dq, dsf, qt2, sft2, bn=bn), ref_t)
    native.check_status()


def test_own_mxfp8_gemm_agrees_with_the_vendor_library_on_the_same_bytes():
    """Verification layer 3: the same e4m3 bytes and the same scale buffers through cuBLASLt's block-scaled
    product (``F.scaled_mm``, ``BlockWise1x32`` scales, ``SWIZZLE_32_4_4`` layout) and through the tcgen05 kernel.
    Both accumulate exact products in fp32; they may differ in summation order only, so they agree to one unit
    in the last place of the bf16 output (measured: bit-equal) and both sit within two units of the fp64 product
    (fp32 accumulation of K products, then one rounding to bf16)."""
    from kohakuwullm_b200.bench import vendor

    if not vendor.vendor_available():
        pytest.skip("F.scaled_mm with block-wise scaling is not in this torch build")
    for M, N, K in ((256, 384, 512), (512, 768, 1024)):
        r = vendor.compare_with_vendor(M, N, K, seed=M)
        assert r["ours_vs_vendor_max_ulp"] <= 1.0, r
        assert r["bit_equal_share"] >= 0.99, r
        assert r["ours_vs_fp64_max_ulp"] <= 2.0 and r["vendor_vs_fp64_max_ulp"] <= 2.0, r


@pytest.mark.parametrize("bn", [128, 144, 160, 192, 224, 240])
@pytest.mark.parametrize("M,N,K", [(1, 128, 128), (128, 256, 256), (129, 1280, 384), (640, 1168, 1280), (1000, 200, 512)])
def test_gemm_tile_widths_and_outputs(M, N, K, bn):
    """One CTA and pairs of CTAs, whole and cut tiles in both directions, each way the result leaves the kernel. The
    oracle multiplies the dequantised operands in 64 bits. Bound: products of e4m3 values are exact in fp32, so an fp32
    sum of K of them is off by at most K * 2^-24 of the sum of magnitudes (twice that for sums that truncate); a bf16
    result by another 2^-9 of itself."""
    from kohakuwullm_b200.ops import mxfp8 as mx, native

    torch.manual_seed(M + bn)
    a = (torch.randn(M, K, device="cuda") * torch.logspace(-2, 1, K, device="cuda")).to(torch.bfloat16)
    b = (torch.randn(N, K, device="cuda") * torch.logspace(1, -1, N, device="cuda")[:, None]).to(torch.bfloat16)
    aq, asf = mx.quantize(a)
    bq, bsf_plain = mx.quantize(b)
    bsf = mx.alloc_weight_sf(N, K, bn, "cuda")
    mx.quantize_weight(b, torch.empty_like(bq), bsf, bn)
    da = mx.dequantize(aq.view(torch.float8_e4m3fn), mx.sf_to_natural(asf, M, K)).double()
    db = mx.dequantize(bq.view(torch.float8_e4m3fn), mx.sf_to_natural(bsf_plain, N, K)).double()
    ref, mag = da @ db.t(), da.abs() @ db.abs().t()
    start = torch.randn(M, N, device="cuda")
    bound = 2.0 * K * 2.0**-24 * mag + 1e-6
    for dtype in (torch.float32, torch.bfloat16):
        for accumulate in (False, True):
            out = start.to(dtype)
            want = ref * 0.5 + (out.double() if accumulate else 0.0)
            mx.gemm(aq, asf, bq, bsf, out=out, accumulate=accumulate, alpha=0.5, bn=bn)
            torch.cuda.synchronize()
            native.check_status()
            limit = bound + want.abs() * (2.0**-23 if dtype == torch.float32 else 2.0**-8)
            assert ((out.double() - want).abs() <= limit).all(), f"{dtype} accumulate {accumulate}"


@pytest.mark.parametrize("R,C,offset", [(128, 1, 0), (128, 62, 1), (256, 63, 0), (384, 130, 0), (128, 257, 3), (256, 1280, 2)])
def test_transposed_quantise_of_odd_and_unaligned_matrices(R, C, offset):
    """Pairs of columns per thread or one, by alignment: the same bytes as quantising the transposed copy."""
    from kohakuwullm_b200.ops import mxfp8 as mx

    torch.manual_seed(C)
    store = (torch.randn(R, C + 8, device="cuda") * torch.logspace(-4, 3, R, device="cuda")[:, None]).to(torch.bfloat16)
    w = store[:, offset:offset + C]
    qt, sft = mx.quantize_transposed(w)
    q_ref, e_ref = mx.quantize_reference(w.t().contiguous())
    assert torch.equal(qt.view(torch.float8_e4m3fn).float(), q_ref.float())
    assert torch.equal(mx.sf_to_natural(sft, C, R), e_ref)
