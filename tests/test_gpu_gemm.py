"""tcgen05 bf16 GEMM against an fp32 PyTorch product of the same bf16 operands."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _operands(M, N, K, a_mn, b_mn, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    b = torch.randn(N, K, device="cuda", generator=g).to(torch.bfloat16)
    ref = a.float() @ b.float().t()
    a_st = a.t().contiguous() if a_mn else a
    b_st = b.t().contiguous() if b_mn else b
    return a_st, b_st, ref


@pytest.mark.parametrize("bn", [128, 256])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("shape", [(256, 256, 128), (384, 640, 192), (200, 136, 72), (4096, 1280, 1280)])
def test_gemm_matches_fp32_reference(shape, a_mn, b_mn, bn):
    from kohakuwullm_b200.ops import native
    from kohakuwullm_b200.ops.gemm import matmul

    M, N, K = shape
    a, b, ref = _operands(M, N, K, a_mn, b_mn)
    out = matmul(a, b, a_mn=a_mn, b_mn=b_mn, bn=bn)
    torch.cuda.synchronize()
    native.check_status()
    err = (out.float() - ref).abs().max().item()
    scale = ref.abs().max().item()
    assert err <= 1e-2 * scale, f"max err {err} vs scale {scale}"


def test_gemm_fp32_accumulate_and_alpha():
    from kohakuwullm_b200.ops import native
    from kohakuwullm_b200.ops.gemm import matmul

    a, b, ref = _operands(512, 384, 256, True, True, seed=3)
    out = torch.ones(512, 384, device="cuda", dtype=torch.float32)
    matmul(a, b, a_mn=True, b_mn=True, out=out, accumulate=True, alpha=0.5)
    matmul(a, b, a_mn=True, b_mn=True, out=out, accumulate=True, alpha=0.5)
    torch.cuda.synchronize()
    native.check_status()
    torch.testing.assert_close(out, ref + 1.0, rtol=1e-4, atol=1e-3)


def test_linear_autograd_matches_torch():
    from kohakuwullm_b200.ops.gemm import linear

    torch.manual_seed(0)
    x = torch.randn(640, 512, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = torch.randn(768, 512, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    dy = torch.randn(640, 768, device="cuda", dtype=torch.bfloat16)
    y = linear(x, w)
    y.backward(dy)
    xr, wr = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    yr = xr @ wr.t()
    yr.backward(dy.float())
    for got, want in ((y, yr), (x.grad, xr.grad), (w.grad, wr.grad)):
        err = (got.float() - want).abs().max().item()
        assert err <= 1e-2 * want.abs().max().item()


@pytest.mark.parametrize("M,N,K", [(1280, 1280, 4096), (7168, 1280, 4096), (1792, 1280, 8192), (384, 1000, 1024 + 64)])
def test_stream_k_weight_gradient_accumulates_exactly_once(M, N, K):
    """fp32 C += with a long contraction is scheduled stream-K: every CTA takes an equal run of (tile, k-block)
    units and adds its partial tiles into C with vector reductions; each unit must be counted exactly once."""
    from kohakuwullm_b200.ops import native
    from kohakuwullm_b200.ops.gemm import matmul

    a, b, ref = _operands(M, N, K, True, True, seed=5)
    out = torch.full((M, N), 2.0, device="cuda", dtype=torch.float32)
    matmul(a, b, a_mn=True, b_mn=True, out=out, accumulate=True)
    torch.cuda.synchronize()
    native.check_status()
    torch.testing.assert_close(out, ref + 2.0, rtol=1e-4, atol=2e-3 * (K / 4096) ** 0.5 + 1e-3)


@pytest.mark.parametrize("bn", [64, 96, 160, 224, 1128, 1160, 1192, 1224, 1256])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("shape", [(136, 72, 72), (264, 328, 200), (520, 1064, 136)])
def test_gemm_tile_widths_and_cta_pairs(shape, a_mn, b_mn, bn):
    """Every tile width of one CTA and of a CTA pair (1000 + width), rows and columns that end inside a tile, a pair whose
    second CTA has few or no rows, a contraction that ends inside a k-block; bf16 store, fp32 store and fp32 C +=. The
    row of canaries behind the output must survive: a store box that is not cut at the edge would write there."""
    from kohakuwullm_b200.ops import native
    from kohakuwullm_b200.ops.gemm import matmul

    M, N, K = shape
    a, b, ref = _operands(M, N, K, a_mn, b_mn, seed=bn)
    for dtype, acc in ((torch.bfloat16, False), (torch.float32, False), (torch.float32, True)):
        full = torch.full((M + 1, N), 3.0, device="cuda", dtype=dtype)
        matmul(a, b, a_mn=a_mn, b_mn=b_mn, out=full[:M], accumulate=acc, bn=bn)
        torch.cuda.synchronize()
        native.check_status()
        want = ref + 3.0 if acc else ref
        # bf16: half a unit in the last place (2^-9); fp32: the order of K <= 200 sums (K * 2^-24, scaled by the largest value)
        tol = 2.0 ** -8 if dtype == torch.bfloat16 else 200 * 2.0 ** -23
        assert (full[:M].float() - want).abs().max().item() <= tol * want.abs().max().item()
        assert bool((full[M] == 3.0).all())


@pytest.mark.parametrize("vocab", [1000, 256 * 9])
def test_cross_entropy_partials_fold(vocab):
    """Column tiles that are no whole batch of the folding kernel, and rows that end inside its block."""
    from kohakuwullm_b200.ops.loss import linear_cross_entropy, linear_cross_entropy_reference

    g = torch.Generator(device="cuda").manual_seed(vocab)
    h = torch.randn(133, 128, device="cuda", generator=g).to(torch.bfloat16)
    w = (torch.randn(vocab, 128, device="cuda", generator=g) * 0.2).to(torch.bfloat16)
    labels = torch.randint(0, vocab, (133,), device="cuda", generator=g)
    ce, lse = linear_cross_entropy(h, w, labels)
    want_ce, want_lse = linear_cross_entropy_reference(h, w, labels)
    torch.testing.assert_close(lse, want_lse, rtol=1e-4, atol=1e-3)
    torch.testing.assert_close(ce, want_ce, rtol=1e-4, atol=1e-3)


@pytest.mark.parametrize("M", [1, 7, 8, 9, 16, 17])
@pytest.mark.parametrize("N,K", [(16, 8), (40, 264), (768, 768), (1000, 2056), (65536, 128)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_few_rows_against_64_bits(M, N, K, out_dtype):
    """Products of up to 16 rows (and 17, the first of the tiled kernel): cut rows of B, cut slices of the contraction,
    operands and outputs that are views. An fp32 sum of K exact products is off by at most 2 K 2^-24 of the sum of
    magnitudes, a bf16 result by another 2^-9 of itself."""
    from kohakuwullm_b200.ops import native
    from kohakuwullm_b200.ops.gemm import matmul

    torch.manual_seed(M + N)
    a = torch.randn(M, K + 8, device="cuda").bfloat16()[:, :K]
    b = torch.randn(N, K + 16, device="cuda").bfloat16()[:, 8:K + 8]
    store = torch.full((M, N + 3), 7.0, device="cuda", dtype=out_dtype)
    out = matmul(a, b, out=store[:, :N], alpha=0.5)
    torch.cuda.synchronize()
    native.check_status()
    want = 0.5 * a.double() @ b.double().t()
    limit = K * 2.0**-24 * (a.double().abs() @ b.double().abs().t()) + want.abs() * (2.0**-8 if out_dtype == torch.bfloat16 else 2.0**-23) + 1e-7
    assert ((out.double() - want).abs() <= limit).all()
    assert (store[:, N:] == 7).all()


@pytest.mark.parametrize("M,N,K", [(128, 64, 1024), (130, 264, 1096), (300, 520, 4104), (640, 1280, 8192), (4096, 1280, 2056), (2500, 2600, 1024)])
def test_input_gradient_sums_in_even_ranges(M, N, K):
    """fp32 C += A B with B contraction-major and a long contraction: fewer tiles than SMs (several ranges meet in a tile),
    about one each, and more; cut tiles and contractions. Bound: fp32 sums of K exact products, at most 2 K 2^-24 of the sum
    of magnitudes, plus the rounding of a few pieces."""
    from kohakuwullm_b200.ops import native
    from kohakuwullm_b200.ops.gemm import matmul

    torch.manual_seed(K)
    a = torch.randn(M, K, device="cuda").bfloat16()
    b = torch.randn(K, N, device="cuda").bfloat16()
    out = torch.randn(M, N, device="cuda")
    want = out.double() + a.double() @ b.double()
    limit = 2 * K * 2.0**-24 * (a.double().abs() @ b.double().abs()) + want.abs() * 2.0**-20 + 1e-5
    matmul(a, b, b_mn=True, out=out, accumulate=True)
    torch.cuda.synchronize()
    native.check_status()
    assert ((out.double() - want).abs() <= limit).all()


@pytest.mark.parametrize("tiles", [1, 31, 32, 33, 64, 65, 256])
def test_fold_of_cross_entropy_partials_around_a_batch(tiles):
    """Whole batches of partials, none and a remainder; the fold's error is a few fp32 roundings."""
    import ctypes

    from kohakuwullm_b200.ops import native

    torch.manual_seed(tiles)
    rows = 77
    part = torch.stack([torch.randn(tiles, rows, device="cuda") * 8, torch.rand(tiles, rows, device="cuda") * 50 + 1], -1).contiguous()
    lse = torch.empty(rows, device="cuda")
    rc = native.require().kwu_ce_combine(native.ptr(part), ctypes.c_int(tiles), ctypes.c_int(rows), native.ptr(lse), native.stream_ptr())
    native.check(rc, "ce_combine")
    want = torch.logsumexp(part[..., 0].double() + part[..., 1].double().log(), 0)
    assert ((lse.double() - want).abs() <= 1e-5 * want.abs() + 2e-5).all()


@pytest.mark.parametrize("M,N,K", [(1, 64, 768), (17, 64, 768), (3001, 64, 768), (8190, 64, 768), (640, 1280, 1016), (300, 64, 1000)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (True, True)])
def test_short_contractions_add_into_fp32_in_one_piece(M, N, K, a_mn, b_mn):
    """fp32 C += A B below K = 1024 has one order of summation: it is C plus the product that the same tile writes without
    accumulation, to the bit, however often it runs (gate logits of routed layers are formed like this)."""
    from kohakuwullm_b200.ops import native
    from kohakuwullm_b200.ops.gemm import matmul

    if a_mn and M % 8:
        M = (M + 7) // 8 * 8           # pitches of TMA operands
    a, b, _ = _operands(M, N, K, a_mn, b_mn, seed=K)
    start = torch.randn(M, N, device="cuda")
    # bn = 128: the plain tile kernel for every M
    product = matmul(a, b, a_mn=a_mn, b_mn=b_mn, bn=128, out_dtype=torch.float32)
    for _ in range(4):
        out = start.clone()
        matmul(a, b, a_mn=a_mn, b_mn=b_mn, out=out, accumulate=True)
        assert torch.equal(out, start + product)
    torch.cuda.synchronize()
    native.check_status()
