"""tcgen05 GEMM vs an fp32 PyTorch reference, over operand layouts, shapes and outputs."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(a, b):
    return a.float() @ b.float()


def _close(out, ref, tol=2e-2):
    err = (out.float() - ref).abs().max().item()
    scale = ref.abs().max().item() + 1e-6
    assert err / scale < tol, f"max err {err} vs scale {scale}"


@pytest.mark.parametrize("m,n,k", [(128, 128, 64), (256, 256, 256), (384, 512, 192), (200, 264, 72), (1024, 4096, 1024), (2048, 11008, 512)])
@pytest.mark.parametrize("a_t,b_t", [(False, False), (False, True), (True, False), (True, True)])
def test_gemm_layouts(m, n, k, a_t, b_t):
    from axlearn_b200.ops import cuda_ops

    torch.manual_seed(0)
    dev = "cuda"
    a = torch.randn(k, m, device=dev).bfloat16().t() if a_t else torch.randn(m, k, device=dev).bfloat16()
    b = torch.randn(n, k, device=dev).bfloat16().t() if b_t else torch.randn(k, n, device=dev).bfloat16()
    out = cuda_ops.gemm(a, b)
    torch.cuda.synchronize()
    cuda_ops.check_status()
    _close(out, _ref(a, b))


def test_gemm_fp32_out_and_accumulate():
    from axlearn_b200.ops import cuda_ops

    torch.manual_seed(1)
    a = torch.randn(256, 320, device="cuda").bfloat16()
    b = torch.randn(320, 384, device="cuda").bfloat16()
    out = cuda_ops.gemm(a, b, out_dtype=torch.float32)
    _close(out, _ref(a, b), tol=1e-3)
    base = torch.randn(256, 384, device="cuda")
    acc = base.clone()
    cuda_ops.gemm(a, b, out=acc, accumulate=True)
    _close(acc, base + _ref(a, b), tol=1e-3)
    cuda_ops.check_status()


def test_linear_autograd_matches_reference():
    from axlearn_b200.ops import cuda_ops

    torch.manual_seed(2)
    x = torch.randn(4, 96, 256, device="cuda").bfloat16().requires_grad_()
    w = torch.randn(256, 512, device="cuda").bfloat16().requires_grad_()
    wt = torch.randn(384, 256, device="cuda").bfloat16().requires_grad_()  # used as x @ wt.t()
    y = cuda_ops.linear(x, w)
    z = cuda_ops.linear(x, wt.t())
    g1, g2 = torch.randn_like(y), torch.randn_like(z)
    (y * g1).sum().backward(retain_graph=True)
    (z * g2).sum().backward()
    xf, wf, wtf = x.detach().float().requires_grad_(), w.detach().float().requires_grad_(), wt.detach().float().requires_grad_()
    yr, zr = xf @ wf, xf @ wtf.t()
    ((yr * g1.float()).sum() + (zr * g2.float()).sum()).backward()
    _close(y, yr)
    _close(z, zr)
    _close(x.grad, xf.grad)
    _close(w.grad, wf.grad)
    _close(wt.grad, wtf.grad)
    cuda_ops.check_status()


def test_gemm_deterministic():
    from axlearn_b200.ops import cuda_ops

    a = torch.randn(512, 1024, device="cuda").bfloat16()
    b = torch.randn(1024, 768, device="cuda").bfloat16()
    assert torch.equal(cuda_ops.gemm(a, b), cuda_ops.gemm(a, b))


@pytest.mark.parametrize("m,n,k", [(64, 1536, 4096), (16, 2752, 4096), (8, 4096, 1376), (128, 4096, 11008), (1, 1536, 512),
                                   (8, 12288, 4096), (16, 22016, 4096), (48, 4096, 4096), (8, 32768, 4096), (5, 9504, 2112)])
@pytest.mark.parametrize("b_t", [False, True])
def test_skinny_gemm_split_k(m, n, k, b_t):
    """Decode-shaped problems (at most 128 rows) as the kernel's own plan lays them out: K slices met in a cluster where
    it splits; bf16 and fp32 outputs, with and without accumulation, repeated."""
    from axlearn_b200.ops import cuda_ops

    torch.manual_seed(2)
    a = torch.randn(m, k, device="cuda").bfloat16()
    b = torch.randn(n, k, device="cuda").bfloat16().t() if b_t else torch.randn(k, n, device="cuda").bfloat16()
    ref = _ref(a, b)
    for _ in range(3):
        _close(cuda_ops.gemm(a, b), ref)
    _close(cuda_ops.gemm(a, b, out_dtype=torch.float32), ref, tol=1e-3)
    base = torch.randn(m, n, device="cuda").bfloat16()
    acc = base.clone()
    cuda_ops.gemm(a, b, out=acc, accumulate=True)
    _close(acc, base.float() + ref)
    torch.cuda.synchronize()
    cuda_ops.check_status()
    if n * 2 <= 148 * 64 and k >= 4096:
        assert cuda_ops.lib().axb_gemm_splitk_plan(m, n, k) > 1


@pytest.mark.parametrize("m", [1, 16, 17, 33, 64, 65, 128])
@pytest.mark.parametrize("n,k", [(8, 64), (136, 72), (1000, 8), (4096, 640), (18952, 128), (37896, 64)])
@pytest.mark.parametrize("a_t,b_t", [(False, False), (False, True), (True, True)])
def test_skinny_gemm_edges(m, n, k, a_t, b_t):
    """Row counts at the edges of the tiles, feature and K remainders, one wave of wide CTAs and one more, at the split
    of the kernel's own plan.  fp32 sums of K bf16 products: the error is a few K * 2^-24 of sum |a b|."""
    from axlearn_b200.ops import cuda_ops

    torch.manual_seed(3)
    pad = (m + 7) // 8 * 8
    a = torch.randn(k, pad, device="cuda").bfloat16()[:, :m].t() if a_t else torch.randn(m, k, device="cuda").bfloat16()
    b = torch.randn(n, k, device="cuda").bfloat16().t() if b_t else torch.randn(k, n, device="cuda").bfloat16()
    ref = a.double() @ b.double()
    bound = 4 * k * 2.0 ** -24 * (a.double().abs() @ b.double().abs()) + 1e-30
    out = cuda_ops.gemm(a, b, out_dtype=torch.float32)
    assert ((out.double() - ref).abs() <= bound).all()
    base = torch.randn(m, n, device="cuda")
    acc = base.clone()
    cuda_ops.gemm(a, b, out=acc, accumulate=True)
    assert ((acc.double() - ref - base.double()).abs() <= bound + 2.0 ** -22 * (ref.abs() + base.abs())).all()
    cuda_ops.check_status()


@pytest.mark.parametrize("m", [1, 13, 16, 50, 100, 128])
@pytest.mark.parametrize("n,k", [(8, 64), (136, 72), (264, 520), (1000, 648)])
@pytest.mark.parametrize("x_t", [False, True])
@pytest.mark.parametrize("w_t", [False, True])
def test_skinny_gemm_every_split(m, n, k, x_t, w_t):
    """Each number of K slices up to the blocks of K (slices of unequal length, row counts that it does not divide), all
    four layouts, both outputs, with and without accumulation; bounds as above, and a bf16 output half a unit more."""
    from axlearn_b200.ops import cuda_ops

    g = torch.Generator(device="cuda").manual_seed(k)
    pad = (m + 7) // 8 * 8
    x = torch.randn(k, pad, device="cuda", generator=g) if x_t else torch.randn(m, k, device="cuda", generator=g)
    w = torch.randn(n, k, device="cuda", generator=g) if w_t else torch.randn(k, n, device="cuda", generator=g)
    x, w = x.bfloat16(), w.bfloat16()
    a, b = (x[:, :m].t() if x_t else x).double(), (w.t() if w_t else w).double()
    ref, bound = a @ b, 4 * k * 2.0 ** -24 * (a.abs() @ b.abs()) + 1e-30
    base = torch.randn(m, n, device="cuda", generator=g)
    status = cuda_ops.status_word()
    for split in range(1, 9):
        for dtype in (torch.float32, torch.bfloat16):
            for accumulate in (False, True):
                start = base.to(dtype)
                out = start.clone()
                rc = cuda_ops.lib().axb_gemm_skinny(
                    x.data_ptr(), w.data_ptr(), out.data_ptr(), m, n, k, x.shape[1], w.shape[1], n, int(x_t),
                    int(not w_t), int(dtype == torch.float32), int(accumulate), split, 0, status.data_ptr(),
                    cuda_ops._stream())  # pylint: disable=protected-access
                if split > (k + 63) // 64:
                    assert rc == -15 and torch.equal(out, start)
                    continue
                want = ref + start.double() if accumulate else ref
                limit = bound + 2.0 ** -22 * (ref.abs() + start.double().abs())
                if dtype == torch.bfloat16:
                    limit = limit + 2.0 ** -8 * (want.abs() + limit)
                assert rc == 0 and ((out.double() - want).abs() <= limit).all(), (split, dtype, accumulate)
    cuda_ops.check_status()


@pytest.mark.parametrize("m", [2, 15, 17, 31, 32, 33])
@pytest.mark.parametrize("blocks", [1, 3, 22, 45])
def test_skinny_gemm_stages_of_two_blocks(m, blocks):
    """Slices of odd and even numbers of 64-deep blocks, shorter and longer than the ring of stages, with a K remainder,
    at the row counts around which partial sums change hands in another way; every split, accumulating into bf16."""
    from axlearn_b200.ops import cuda_ops

    n, k = 392, 64 * blocks - 8
    g = torch.Generator(device="cuda").manual_seed(m * 100 + blocks)
    x = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    w = torch.randn(k, n, device="cuda", generator=g).bfloat16()
    start = torch.randn(m, n, device="cuda", generator=g).bfloat16()
    want = x.double() @ w.double() + start.double()
    limit = 4 * k * 2.0 ** -24 * (x.double().abs() @ w.double().abs()) + 2.0 ** -22 * (want.abs() + start.double().abs())
    limit = limit + 2.0 ** -8 * (want.abs() + limit)
    status = cuda_ops.status_word()
    for split in range(1, min(8, blocks) + 1):
        out = start.clone()
        assert cuda_ops.lib().axb_gemm_skinny(
            x.data_ptr(), w.data_ptr(), out.data_ptr(), m, n, k, k, n, n, 0, 1, 0, 1, split, 0, status.data_ptr(),
            cuda_ops._stream()) == 0  # pylint: disable=protected-access
        assert ((out.double() - want).abs() <= limit).all(), split
    cuda_ops.check_status()


@pytest.mark.parametrize("m", [129, 333, 666])
@pytest.mark.parametrize("n", [8, 72, 128, 264, 520])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_accumulate_reads_c_by_vectors(m, n, dtype):
    """Whole and cut 32-column pieces of C, rows beyond the last tile, a C whose rows lie apart; the rest of C stays."""
    from axlearn_b200.ops import cuda_ops

    k = 192
    g = torch.Generator(device="cuda").manual_seed(m + n)
    a = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    b = torch.randn(k, n, device="cuda", generator=g).bfloat16()
    whole = torch.randn(m + 3, n + 16, device="cuda", generator=g).to(dtype)
    before = whole.clone()
    out = whole[:m, 8:n + 8]
    cuda_ops.gemm(a, b, out=out, accumulate=True)
    want = a.double() @ b.double() + before[:m, 8:n + 8].double()
    limit = 4 * k * 2.0 ** -24 * (a.double().abs() @ b.double().abs()) + 2.0 ** -22 * want.abs()
    if dtype == torch.bfloat16:
        limit = limit + 2.0 ** -8 * (want.abs() + limit)
    assert ((out.double() - want).abs() <= limit).all()
    out.copy_(before[:m, 8:n + 8])
    assert torch.equal(whole, before)
    cuda_ops.check_status()


@pytest.mark.parametrize("m,f,k", [(512, 4096, 64), (513, 4232, 136), (2304, 1096, 512), (4096, 504, 64), (8192, 136, 328),
                                   (700, 11008, 1024)])
def test_product_with_swiglu_epilogue(m, f, k):
    """The bits of the product and the pass over it, at row, column and K remainders (columns of the other half read
    beyond a tile's last one are not stored)."""
    from axlearn_b200.ops import cuda_ops, decode_ops

    g = torch.Generator(device="cuda").manual_seed(m + f)
    a = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    w = (torch.randn(k, 2 * f, device="cuda", generator=g) * 2 * k ** -0.5).bfloat16()
    out = cuda_ops.gemm_swiglu(a, w)
    assert out is not None and torch.equal(out, decode_ops.swiglu_packed(cuda_ops.gemm(a, w)))
    w[0, 3], w[0, f + 5] = float("inf"), float("nan")
    a[:, 0] = a[:, 0].abs() + 0.5
    want = decode_ops.swiglu_packed(cuda_ops.gemm(a, w))
    torch.testing.assert_close(cuda_ops.gemm_swiglu(a, w), want, rtol=0, atol=0, equal_nan=True)
    assert cuda_ops.gemm_swiglu(a[:100], w) is None and cuda_ops.gemm_swiglu(a.t().contiguous().t(), w) is None
    cuda_ops.check_status()


def _close_elementwise(out, ref, atol, rtol):
    """Per-element ``|out - ref| <= atol + rtol * |ref|`` (an error confined to small outputs or one
    tile edge cannot hide behind the largest value)."""
    diff = (out.float() - ref).abs()
    bound = atol + rtol * ref.abs()
    bad = diff > bound
    assert not bad.any(), f"{int(bad.sum())} elements off; worst {diff.max().item():.4g} at {tuple(torch.nonzero(bad)[0].tolist())}"


@pytest.mark.parametrize("variant", ["1cta", "2cta"])
@pytest.mark.parametrize("m,n,k", [(2048, 2048, 512), (4096, 4096, 256), (2304, 2816, 328), (2056, 2064, 72)])
@pytest.mark.parametrize("a_t,b_t", [(False, False), (False, True), (True, False), (True, True)])
def test_large_gemm_variants_per_element(variant, m, n, k, a_t, b_t, monkeypatch):
    from axlearn_b200.ops import cuda_ops

    monkeypatch.setattr(cuda_ops, "GEMM_VARIANT", variant)
    torch.manual_seed(2)
    a = torch.randn(k, m, device="cuda").bfloat16().t() if a_t else torch.randn(m, k, device="cuda").bfloat16()
    b = torch.randn(n, k, device="cuda").bfloat16().t() if b_t else torch.randn(k, n, device="cuda").bfloat16()
    out = cuda_ops.gemm(a, b)
    torch.cuda.synchronize()
    cuda_ops.check_status()
    # bf16 rounding of the result (2^-8 relative) plus fp32 accumulation noise.
    _close_elementwise(out, _ref(a, b), atol=0.05 * (k / 256) ** 0.5, rtol=1e-2)


def test_cta_pair_gemm_fp32_out_and_accumulate(monkeypatch):
    from axlearn_b200.ops import cuda_ops

    monkeypatch.setattr(cuda_ops, "GEMM_VARIANT", "2cta")
    torch.manual_seed(3)
    a = torch.randn(2048, 320, device="cuda").bfloat16()
    b = torch.randn(320, 2304, device="cuda").bfloat16()
    ref = _ref(a, b)
    out = cuda_ops.gemm(a, b, out_dtype=torch.float32)
    _close_elementwise(out, ref, atol=1e-3, rtol=1e-4)
    base = torch.randn(2048, 2304, device="cuda")
    acc = base.clone()
    cuda_ops.gemm(a, b, out=acc, accumulate=True)
    _close_elementwise(acc, base + ref, atol=1e-3, rtol=1e-4)
    base16 = torch.randn(2048, 2304, device="cuda").bfloat16()
    acc16 = base16.clone()
    cuda_ops.gemm(a, b, out=acc16, accumulate=True)
    _close_elementwise(acc16, base16.float() + ref, atol=0.15, rtol=1e-2)
    # A strided output (a column block of a wider matrix) goes through the same store path.
    wide = torch.zeros(2048, 4608, device="cuda", dtype=torch.bfloat16)
    cuda_ops.gemm(a, b, out=wide[:, 2304:])
    _close_elementwise(wide[:, 2304:], ref, atol=0.08, rtol=1e-2)
    assert wide[:, :2304].abs().max().item() == 0
    cuda_ops.check_status()


def test_gemm_shape_fuzz(monkeypatch):
    """Seeded random shapes, including sizes that are no multiple of any tile dimension."""
    import random

    from axlearn_b200.ops import cuda_ops

    rng = random.Random(1234)
    for case in range(24):
        variant = "2cta" if case % 2 else "1cta"
        monkeypatch.setattr(cuda_ops, "GEMM_VARIANT", variant)
        m = rng.choice([8 * rng.randint(1, 40), 128 * rng.randint(1, 24), 8 * rng.randint(250, 400)])
        n = rng.choice([8 * rng.randint(1, 40), 128 * rng.randint(1, 24), 8 * rng.randint(250, 400)])
        k = 8 * rng.randint(1, 96)
        a_t, b_t = rng.random() < 0.5, rng.random() < 0.5
        a = torch.randn(k, m, device="cuda").bfloat16().t() if a_t else torch.randn(m, k, device="cuda").bfloat16()
        b = torch.randn(n, k, device="cuda").bfloat16().t() if b_t else torch.randn(k, n, device="cuda").bfloat16()
        out = cuda_ops.gemm(a, b)
        torch.cuda.synchronize()
        cuda_ops.check_status()
        _close_elementwise(out, _ref(a, b), atol=0.05 * max(1.0, (k / 256) ** 0.5), rtol=1e-2)
