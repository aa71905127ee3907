"""sm_100a kernels against plain PyTorch fp32 references of the same op (needs a B200)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

BF16 = torch.bfloat16


def _r(*shape, seed=0, scale=1.0, dtype=BF16):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(dtype)


def _close(got, ref, tol=2e-2):
    """Three bounds, so that neither a wrong row of small magnitude nor a dropped tail tile can
    hide behind the largest element: (1) max abs error against the largest reference element,
    (2) every row (last axis) on its own: error norm <= 4 tol x that row's norm + tol x the norm
    of a typical row, (3) cosine of the flattened tensors >= 1 - tol^2."""
    got, ref = got.float(), ref.float()
    assert got.shape == ref.shape, f"shape {tuple(got.shape)} vs {tuple(ref.shape)}"
    assert torch.isfinite(got).all(), "non-finite values"
    err = (got - ref).abs().max().item()
    scale = ref.abs().max().item() + 1e-6
    assert err <= tol * scale, f"max err {err:.4g} vs scale {scale:.4g}"
    if ref.ndim >= 1 and ref.shape[-1] > 1:
        g2, r2 = got.reshape(-1, ref.shape[-1]), ref.reshape(-1, ref.shape[-1])
        row_err = (g2 - r2).norm(dim=1)
        row_ref = r2.norm(dim=1)
        typical = ref.pow(2).mean().sqrt().item() * math.sqrt(ref.shape[-1]) + 1e-6
        over = row_err - (4 * tol * row_ref + tol * typical)
        worst = int(over.argmax())
        assert over[worst].item() <= 0, (f"row {worst}: err {row_err[worst].item():.4g}, row norm "
                                         f"{row_ref[worst].item():.4g}, typical row {typical:.4g}")
    denom = got.norm().item() * ref.norm().item()
    if denom > 0:
        cos = (got * ref).sum().item() / denom
        assert cos >= 1 - tol * tol, f"cosine {cos:.6f}"


def test_kernel_library_is_loaded_in_tree():
    from prometheus_b200.ops import _lib

    _lib.load()
    assert "prometheus_b200/_lib/libpb200_kernels.so" in open("/proc/self/maps").read()


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (256, 256, 128), (384, 512, 1024),
                                   (200, 328, 264), (4096, 2048, 2048)])
def test_gemm_layouts(M, N, K, a_mn, b_mn):
    from prometheus_b200.ops import functional as ops

    if (a_mn and M % 8) or (b_mn and N % 8):
        pytest.skip("MN-major operands need the MN extent to be a multiple of 8")
    a = _r(K, M, seed=1) if a_mn else _r(M, K, seed=1)
    b = _r(K, N, seed=2) if b_mn else _r(N, K, seed=2)
    c = ops.gemm(a, b, a_mn=a_mn, b_mn=b_mn)
    ref = ops.gemm_ref(a, b, a_mn=a_mn, b_mn=b_mn)
    _close(c, ref)
    ops.check_status("cuda")


def test_gemm_batched_epilogue_variants():
    from prometheus_b200.ops import functional as ops

    a, b = _r(3, 256, 192, seed=1), _r(3, 320, 192, seed=2)
    d = _r(3, 256, 320, seed=3)
    c = ops.gemm(a, b, d=d, alpha=0.5, beta=-2.0)
    _close(c, ops.gemm_ref(a, b, d=d, alpha=0.5, beta=-2.0))
    acc = torch.randn(256, 320, device="cuda")
    ref = acc + ops.gemm_ref(a[0], b[0])
    ops.gemm(a[0], b[0], out=acc, d=acc, beta=1.0)
    _close(acc, ref)
    c32 = ops.gemm(a, b, out_dtype=torch.float32)
    assert c32.dtype == torch.float32
    _close(c32, ops.gemm_ref(a, b), tol=5e-3)
    ops.check_status("cuda")


def test_gemm_2d_forms_equal_the_batched_form():
    """The two-matrix path against the same product as a batch of one: layouts, strided operands and
    destinations, accumulation, and a thread whose first CUDA call is a product."""
    import threading

    from prometheus_b200.ops import functional as ops

    base = _r(200, 520, seed=1)
    for a_mn, b_mn in ((False, False), (False, True), (True, False), (True, True)):
        a = _r(264, 208, seed=2) if a_mn else base[:, 8:272]            # a row stride of 520
        a = a[:, :200] if a_mn else a
        b = _r(264, 328, seed=3) if b_mn else _r(328, 264, seed=3)
        kw = dict(a_mn=a_mn, b_mn=b_mn)
        want = ops.gemm(a[None], b[None], **kw)[0]
        assert torch.equal(ops.gemm(a, b, **kw), want)
        d = _r(200, 328, seed=4, dtype=torch.float32)
        acc, acc3 = d.clone(), d.clone()[None]
        ops.gemm(a, b, out=acc, d=acc, beta=1.0, **kw)
        ops.gemm(a[None], b[None], out=acc3, d=acc3, beta=1.0, **kw)
        assert torch.equal(acc, acc3[0])
        wide = torch.zeros(200, 336, dtype=BF16, device="cuda")
        ops.gemm(a, b, out=wide[:, :328], **kw)
        assert torch.equal(wide[:, :328], want) and (wide[:, 328:] == 0).all()
        assert torch.equal(ops.gemm(a, b, out=torch.empty(1, 200, 328, dtype=BF16, device="cuda"), **kw), want)
        assert torch.equal(ops.gemm(a, b.t().contiguous().t(), **kw), want)      # not row-major: copied
        got = []
        out = torch.empty_like(want)
        torch.cuda.synchronize()
        th = threading.Thread(target=lambda: got.append(ops.gemm(a, b, out=out, **kw)))
        th.start()
        th.join()
        torch.cuda.synchronize()
        assert got and torch.equal(got[0], want)


@pytest.mark.parametrize("M,N", [(200, 328), (520, 264)])
@pytest.mark.parametrize("c_f32", [False, True])
@pytest.mark.parametrize("d_f32", [False, True])
def test_gemm_c_and_d_at_any_base(M, N, c_f32, d_f32):
    """A destination or D that starts at an odd element, or whose batch entries do, is written and read element
    by element: the bits of the aligned call, and nothing next to the destination."""
    from prometheus_b200.ops import functional as ops
    from prometheus_b200.ops._lib import call

    dts = {False: BF16, True: torch.float32}

    def shifted(t, by=1):      # the same values, contiguous, `by` elements past a 16-byte boundary
        buf = torch.full((t.numel() + 16,), 7.0, dtype=t.dtype, device="cuda")
        return buf, buf[by:by + t.numel()].view(t.shape).copy_(t)

    a, b = _r(2, M, 192, seed=1), _r(2, N, 192, seed=2)
    d = _r(2, M, N, seed=3, dtype=dts[d_f32])
    try:
        for variant in (0, 8):         # single CTAs, tiles of 128 x 128 and of 128 x 256
            call("pb_gemm_set_variant", variant)
            kw = dict(out_dtype=dts[c_f32], alpha=0.5, beta=-2.0)
            want = ops.gemm(a, b, d=d, **kw)
            for off_c, off_d in ((0, 1), (1, 0), (1, 1)):
                buf, out = shifted(torch.zeros_like(want), off_c)
                got = ops.gemm(a, b, out=out, d=shifted(d, off_d)[1], **kw)
                assert torch.equal(got, want), (variant, off_c, off_d)
                assert (buf[:off_c] == 7).all() and (buf[off_c + want.numel():] == 7).all()
                buf, out = shifted(torch.zeros_like(want[0]), off_c)
                got = ops.gemm(a[0], b[0], out=out, d=shifted(d[0], off_d)[1], **kw)
                assert torch.equal(got, want[0]), (variant, off_c, off_d)
            # aligned base, batch entries an odd number of elements apart
            gap = torch.empty(2 * M * N + 1, dtype=d.dtype, device="cuda").as_strided((2, M, N), (M * N + 1, N, 1)).copy_(d)
            assert torch.equal(ops.gemm(a, b, d=gap, **kw), want)
    finally:
        call("pb_gemm_set_variant", 0)
    ops.check_status("cuda")


@pytest.mark.parametrize("M,N", [(200, 328), (456, 264), (520, 264)])     # column remainders 8, row remainders 8 and 72
@pytest.mark.parametrize("c_f32", [False, True])
@pytest.mark.parametrize("d_f32", [False, True])
def test_gemm_d_at_remainders_against_fp32(M, N, c_f32, d_f32):
    """alpha A B^T + beta D where a row's D is read partly in whole slabs ahead of the accumulator and partly by
    column chunks: every combination of the types of C and D, a contiguous D and a column slice of a wider one, on
    single CTAs with 128 x 128 and 128 x 256 tiles, alone and batched."""
    from prometheus_b200.ops import functional as ops
    from prometheus_b200.ops._lib import call

    dts = {False: BF16, True: torch.float32}
    a, b = _r(2, M, 192, seed=1), _r(2, N, 192, seed=2)
    wide = _r(2, M, N + 24, seed=3, dtype=dts[d_f32], scale=8.0)      # D as large as the product
    kw = dict(out_dtype=dts[c_f32], alpha=0.5, beta=-2.0)
    try:
        for variant in (0, 8):
            call("pb_gemm_set_variant", variant)
            for d in (wide[:, :, 8:8 + N], wide[:, :, 8:8 + N].contiguous(), wide[:, :, 1:1 + N]):
                want = ops.gemm_ref(a, b, d=d, alpha=0.5, beta=-2.0)
                tol = 1e-5 if c_f32 else 2.0 ** -8      # fp32 sums of 192 products, one rounding of the result
                for got, ref in ((ops.gemm(a, b, d=d, **kw), want), (ops.gemm(a[0], b[0], d=d[0], **kw), want[0])):
                    assert got.dtype == dts[c_f32]
                    err = (got.float() - ref).abs()
                    assert (err <= tol * ref.abs() + 1e-3).all(), (variant, float(err.max()))
    finally:
        call("pb_gemm_set_variant", 0)
    ops.check_status("cuda")


# beyond one wave of 128 x 128 tiles: the same remainders as above where CTA pairs run the product
@pytest.mark.parametrize("M,N,batch", [(200, 328, 40), (456, 264, 14), (520, 264, 26), (4296, 1288, 1)])
@pytest.mark.parametrize("c_f32", [False, True])
@pytest.mark.parametrize("d_f32", [False, True])
def test_gemm_c_and_d_on_pairs_at_remainders_and_any_base(M, N, batch, c_f32, d_f32):
    """alpha A B^T + beta D on CTA pairs at row remainders 200, 8 and column remainders 8 and 72: a contiguous D, column slices
    that start on and off 16 bytes, destinations and D's an element off, against fp32 and the aligned call."""
    from prometheus_b200.ops import functional as ops
    from prometheus_b200.ops._lib import query

    assert query("pb_gemm_on_pairs", M, N, batch) == 1 and query("pb_gemm_on_pairs", 200, 328, 2) == 0
    ty = {False: BF16, True: torch.float32}
    a, b = _r(batch, M, 192, seed=1), _r(batch, N, 192, seed=2)
    wide = _r(batch, M, N + 24, seed=3, dtype=ty[d_f32], scale=8.0)      # D as large as the product
    kw = dict(alpha=0.5, beta=-2.0)
    tol = 1e-5 if c_f32 else 2.0 ** -8      # fp32 sums of 192 products, one rounding of the result
    aligned = None
    for d in (wide[:, :, 8:8 + N], wide[:, :, 8:8 + N].contiguous(), wide[:, :, 1:1 + N]):
        ref = ops.gemm_ref(a, b, d=d, **kw)
        got = ops.gemm(a, b, d=d, out_dtype=ty[c_f32], **kw)
        assert ((got.float() - ref).abs() <= tol * ref.abs() + 1e-3).all()
        aligned = got if aligned is None else aligned
    d = wide[:, :, 8:8 + N]
    for off_c, off_d in ((0, 1), (1, 0), (1, 1)):
        buf = torch.full((batch * M * N + 16,), 7.0, dtype=ty[c_f32], device="cuda")
        out = buf[off_c:off_c + batch * M * N].view(batch, M, N)
        shifted = torch.empty(batch * M * N + 1, dtype=ty[d_f32], device="cuda")[off_d:off_d + batch * M * N].view(d.shape).copy_(d)
        assert torch.equal(ops.gemm(a, b, out=out, d=shifted, **kw), aligned), (off_c, off_d)
        assert (buf[:off_c] == 7).all() and (buf[off_c + out.numel():] == 7).all()
    ops.check_status("cuda")


def test_gemm_limited_grid_and_many_tiles():
    from prometheus_b200.ops import functional as ops

    a, b = _r(2048, 512, seed=1), _r(1536, 512, seed=2)
    _close(ops.gemm(a, b, max_ctas=16), ops.gemm_ref(a, b))
    ops.check_status("cuda")


@pytest.mark.parametrize("M,N,K,a_mn,b_mn", [
    (4096, 2560, 320, False, False),      # 16 x 10 pair tiles, K not a multiple of 64
    (2304 + 72, 2048 + 136, 512, False, False),   # ragged last row block (odd CTA all out of range) and column block
    (2048, 5632, 1024, True, True),       # weight-gradient layout
    (4096, 2048, 768, False, True),       # input-gradient layout
    (3072, 3072, 256, True, False),
])
def test_gemm_cta_pair_kernel(M, N, K, a_mn, b_mn):
    """Products with at least one full wave of 256 x 256 tiles run on the two-CTA kernel
    (tcgen05.mma.cta_group::2); same products on the single-CTA kernel for comparison."""
    from prometheus_b200.ops import functional as ops
    from prometheus_b200.ops._lib import call

    a = _r(K, M, seed=1) if a_mn else _r(M, K, seed=1)
    b = _r(K, N, seed=2) if b_mn else _r(N, K, seed=2)
    ref = ops.gemm_ref(a, b, a_mn=a_mn, b_mn=b_mn)
    c = ops.gemm(a, b, a_mn=a_mn, b_mn=b_mn)
    ops.check_status("cuda")
    _close(c, ref)
    try:
        call("pb_gemm_set_variant", 8)       # every product on the single-CTA kernel
        c1 = ops.gemm(a, b, a_mn=a_mn, b_mn=b_mn)
    finally:
        call("pb_gemm_set_variant", 0)
    _close(c, c1, 2e-3)


def test_gemm_cta_pair_batched_epilogue_variants():
    from prometheus_b200.ops import functional as ops

    a, b = _r(10, 768, 192, seed=1), _r(10, 768, 192, seed=2)       # 3 x 3 x 10 = 90 pair tiles
    d = _r(10, 768, 768, seed=3)
    c = ops.gemm(a, b, d=d, alpha=0.5, beta=-2.0)
    _close(c, ops.gemm_ref(a, b, d=d, alpha=0.5, beta=-2.0))
    c32 = ops.gemm(a, b, out_dtype=torch.float32)
    _close(c32, ops.gemm_ref(a, b), tol=5e-3)
    big_a, big_b = _r(4096, 256, seed=4), _r(2560, 256, seed=5)
    acc = torch.randn(4096, 2560, device="cuda")
    ref = acc + ops.gemm_ref(big_a, big_b)
    ops.gemm(big_a, big_b, out=acc, d=acc, beta=1.0)
    _close(acc, ref)
    # a row stride that rules out the TMA store (direct-store epilogue)
    odd = torch.empty(4096, 2563, device="cuda", dtype=torch.bfloat16)[:, :2560]
    ops.gemm(big_a, big_b, out=odd)
    _close(odd, ops.gemm_ref(big_a, big_b))
    ops.check_status("cuda")


@pytest.mark.parametrize("rows,d", [(37, 256), (1000, 2048), (64, 384), (5, 128)])
def test_rmsnorm_fwd_bwd(rows, d):
    from prometheus_b200.ops import functional as ops

    x = _r(rows, d, seed=1).requires_grad_(True)
    res = _r(rows, d, seed=2).requires_grad_(True)
    w = (1 + 0.1 * torch.randn(d, device="cuda")).requires_grad_(True)
    y, h = ops.add_rmsnorm(x, res, w)
    gy, gh = _r(rows, d, seed=3), _r(rows, d, seed=4)
    (y.float() * gy.float()).sum().add((h.float() * gh.float()).sum()).backward()
    xr, rr, wr = (t.detach().float().requires_grad_(True) for t in (x, res, w))
    yr, hr = ops.rmsnorm_ref(xr, wr, res=rr)
    # the kernel rounds h to bf16 before normalising
    _close(h, hr, 1e-2)
    _close(y, yr, 2e-2)
    ((yr * gy.float()).sum() + (hr * gh.float()).sum()).backward()
    _close(x.grad, xr.grad, 3e-2)
    _close(res.grad, rr.grad, 3e-2)
    _close(w.grad, wr.grad, 3e-2)
    y1 = ops.rmsnorm(x.detach(), w.detach())
    _close(y1, ops.rmsnorm_ref(x.detach(), w.detach()), 2e-2)


def test_rope_matches_model_and_inverts():
    from prometheus_b200 import model
    from prometheus_b200.ops import functional as ops

    B, S, H, D = 2, 300, 3, 128
    x = _r(B, S, H, D, seed=1)
    y = ops.rope_(x, seq_len=S)
    ref, _ = model.rope(x.float(), x.float(), torch.arange(S, device="cuda"), partial=False)
    _close(y, ref, 1e-2)
    xg = x.clone().requires_grad_(True)
    g = _r(B, S, H, D, seed=2)
    (ops.rope_(xg, seq_len=S).float() * g.float()).sum().backward()
    xr = x.float().requires_grad_(True)
    (model.rope(xr, xr, torch.arange(S, device="cuda"), partial=False)[0] * g.float()).sum().backward()
    _close(xg.grad, xr.grad, 1e-2)
    # large positions keep full precision (no fast-math sincos)
    pos = torch.full((B * S,), 131071, dtype=torch.int32, device="cuda")
    y2 = ops.rope_(x, seq_len=S, pos=pos)
    ref2, _ = model.rope(x.float(), x.float(), torch.full((S,), 131071.0, device="cuda"), partial=False)
    _close(y2, ref2, 1e-2)


def test_swiglu_fwd_bwd():
    from prometheus_b200.ops import functional as ops

    gu = _r(77, 2 * 512, seed=1).requires_grad_(True)
    g = _r(77, 512, seed=2)
    out = ops.swiglu(gu)
    (out.float() * g.float()).sum().backward()
    gr = gu.detach().float().requires_grad_(True)
    ref = ops.swiglu_ref(gr)
    (ref * g.float()).sum().backward()
    _close(out, ref)
    _close(gu.grad, gr.grad)


def test_l2norm_fwd_bwd():
    from prometheus_b200.ops import functional as ops

    x = _r(50, 4, 128, seed=1).requires_grad_(True)
    g = _r(50, 4, 128, seed=2)
    y = ops.l2norm(x)
    (y.float() * g.float()).sum().backward()
    xr = x.detach().float().requires_grad_(True)
    yr = xr / xr.norm(dim=-1, keepdim=True).clamp(min=1e-6)
    (yr * g.float()).sum().backward()
    _close(y, yr)
    _close(x.grad, xr.grad, 3e-2)


def test_linear_multi_and_inplace_rope_equal_the_separate_ops():
    """Three projections of one input with the input gradients summed in the GEMM epilogues, rotary
    embedding written over the projection outputs: values and all gradients against fp32."""
    from prometheus_b200 import model
    from prometheus_b200.ops import functional as ops

    T, S, d, H, Hkv, D = 600, 300, 256, 4, 2, 128
    x = _r(T, d, seed=1).requires_grad_(True)
    ws = [_r(H * D, d, seed=2, scale=0.1).requires_grad_(True), _r(Hkv * D, d, seed=3, scale=0.1).requires_grad_(True),
          _r(Hkv * D, d, seed=4, scale=0.1).requires_grad_(True)]
    gs = [_r(T, H * D, seed=5), _r(T, Hkv * D, seed=6), _r(T, Hkv * D, seed=7)]
    q, k, v = ops.linear_multi(x, ws)
    q = ops.rope2d_(q, H, seq_len=S)
    k = ops.rope2d_(k, Hkv, seq_len=S)
    sum((o.float() * g.float()).sum() for o, g in zip((q, k, v), gs)).backward()

    xr = x.detach().float().requires_grad_(True)
    wr = [w.detach().float().requires_grad_(True) for w in ws]
    pos = torch.arange(S, device="cuda")
    qr = model.rope((xr @ wr[0].t()).view(T // S, S, H, D), (xr @ wr[0].t()).view(T // S, S, H, D), pos, partial=False)[0]
    kr = model.rope((xr @ wr[1].t()).view(T // S, S, Hkv, D), (xr @ wr[1].t()).view(T // S, S, Hkv, D), pos, partial=False)[0]
    vr = xr @ wr[2].t()
    outs_r = (qr.reshape(T, H * D), kr.reshape(T, Hkv * D), vr)
    sum((o * g.float()).sum() for o, g in zip(outs_r, gs)).backward()
    for got, want in zip((q, k, v), outs_r):
        _close(got, want)
    _close(x.grad, xr.grad, 4e-2)
    for w, r in zip(ws, wr):
        _close(w.grad, r.grad, 4e-2)


def test_l2norm_inplace_over_a_projection_output():
    """The in-place form on the output of a linear layer: values and the gradients of the
    layer's input and weight equal the out-of-place composition; D = 64 takes the generic kernel."""
    from prometheus_b200.ops import functional as ops

    for heads, D in ((4, 128), (8, 64)):
        x = _r(300, 256, seed=1).requires_grad_(True)
        w = _r(heads * D, 256, seed=2, scale=0.1).requires_grad_(True)
        g = _r(300, heads, D, seed=3)
        y = ops.l2norm_(ops.linear(x, w), D).view(300, heads, D)
        (y.float() * g.float()).sum().backward()
        xr, wr = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
        pr = (xr @ wr.t()).view(300, heads, D)
        yr = pr / pr.norm(dim=-1, keepdim=True).clamp(min=1e-6)
        (yr * g.float()).sum().backward()
        _close(y, yr)
        _close(x.grad, xr.grad, 4e-2)
        _close(w.grad if w.grad is not None else w.main_grad, wr.grad, 4e-2)


@pytest.mark.parametrize("cap", [30.0, 0.0])
def test_softcap_ce_fused(cap):
    from prometheus_b200.ops import functional as ops

    rows, d, V = 300, 256, 4096
    h = _r(rows, d, seed=1).requires_grad_(True)
    U = _r(V, d, seed=2, scale=0.3).requires_grad_(True)
    tgt = torch.randint(0, V, (rows,), device="cuda", dtype=torch.int32)
    wt = (torch.rand(rows, device="cuda") > 0.2).float() / rows
    loss = ops.softcap_cross_entropy(h, U, tgt, wt, cap, chunk_rows=128)
    loss.backward()
    hr, Ur = h.detach().float().requires_grad_(True), U.detach().float().requires_grad_(True)
    ref = ops.softcap_cross_entropy_ref(hr, Ur, tgt, wt, cap)
    ref.backward()
    assert abs(loss.item() - ref.item()) <= 2e-2 * abs(ref.item())
    _close(h.grad, hr.grad, 5e-2)
    _close(U.grad, Ur.grad, 5e-2)


@pytest.mark.parametrize("n", [1, 7, 8, 2047, 2056, 100003])
def test_scale_cast(n):
    from prometheus_b200.ops._lib import call, ptr, stream_ptr

    x = _r(n, seed=n, dtype=torch.float32)
    g = torch.full((1,), 0.37, device="cuda")
    out = torch.empty(n, dtype=BF16, device="cuda")
    call("pb_scale_cast", ptr(x), ptr(g), ptr(out), n, stream_ptr())
    assert torch.equal(out, (x * g).to(BF16))


@pytest.mark.parametrize("rows,d,V", [(256, 1024, 136), (200, 2048, 1000), (512, 1544, 4104)])
@pytest.mark.parametrize("scale", [0.5, 20.0])
def test_softcap_sums_from_the_logits_product(rows, d, V, scale):
    """The row sums that the product's epilogue adds up against 64 bits over the stored logits (tanh of the
    special-function unit, 2^-11 of a capped logit's slope: up to cap 2^-11 in the exponent), and loss and
    gradients against the two-sweep kernel."""
    from prometheus_b200.ops import functional as ops
    from prometheus_b200.ops._lib import call, ptr, query, stream_ptr

    cap = 30.0
    h, U = _r(rows, d, seed=1), _r(V, d, seed=2, scale=scale / math.sqrt(d))
    assert query("pb_gemm_softcap_ok", rows, V, d) == 1 and query("pb_gemm_softcap_ok", rows, V, 512) == 0
    lg = torch.empty(rows, V, dtype=BF16, device="cuda")
    sums = torch.empty(rows, device="cuda")
    part = torch.full((2 * ((V + 255) // 256) * rows,), float("nan"), device="cuda")
    call("pb_gemm_softcap_logits", ptr(h), ptr(U), ptr(lg), rows, V, d, d, d, V, cap, ptr(part), ptr(sums),
         ptr(ops.status_word("cuda")), stream_ptr())
    assert torch.equal(lg, ops.gemm(h, U))
    want = torch.exp(cap * torch.tanh(lg.double() / cap) - cap).sum(1)
    assert ((sums.double() - want).abs() <= cap * 2.0 ** -10 * want).all()
    tgt = torch.randint(0, V, (rows,), device="cuda", dtype=torch.int32)
    wt = (torch.arange(rows, device="cuda") % 5 != 0).float() / rows

    def run(variant):
        call("pb_gemm_set_variant", variant)       # 8: no CTA pairs, so the two-sweep kernel
        try:
            hg, Ug = h.clone().requires_grad_(True), U.clone().requires_grad_(True)
            loss = ops.softcap_cross_entropy(hg, Ug, tgt, wt, cap)
            return (loss.detach(), *torch.autograd.grad(loss, (hg, Ug)))
        finally:
            call("pb_gemm_set_variant", 0)

    for a, b in zip(run(0), run(8)):
        assert (a.float() - b.float()).norm() <= 5e-3 * b.float().norm()
    ops.check_status("cuda")


@pytest.mark.parametrize("grad", [True, False])
def test_softcap_sums_over_chunks_and_without_gradients(grad):
    """The head with its row sums from the logits product against the two-sweep kernel: chunks of different row
    counts (one with a last row block of 8), a ragged vocabulary, and a loss alone. The rule that chooses it
    leaves products of few tiles to the two sweeps."""
    from prometheus_b200.ops import functional as ops
    from prometheus_b200.ops._lib import call, query

    rows, d, V, cap, chunk = 2 * 768 + 520, 1024, 65544, 30.0, 768
    for n in (768, 520):
        assert query("pb_gemm_softcap_pays", n, V, d) == 1
    for n, v in ((200, 8192), (256, 65544), (4096, 8192)):      # 32, 257 and 512 tiles
        assert query("pb_gemm_softcap_ok", n, v, d) == 1 and query("pb_gemm_softcap_pays", n, v, d) == 0
    assert query("pb_gemm_softcap_pays", 4096, 131072, 1016) == 0
    h, U = _r(rows, d, seed=1), _r(V, d, seed=2, scale=2.0 / math.sqrt(d))
    tgt = torch.randint(0, V, (rows,), device="cuda", dtype=torch.int32)
    wt = (torch.arange(rows, device="cuda") % 5 != 0).float() / rows

    def run(variant):
        call("pb_gemm_set_variant", variant)       # 8: no CTA pairs, so the two-sweep kernel
        try:
            with torch.set_grad_enabled(grad):
                hg, Ug = h.clone().requires_grad_(grad), U.clone().requires_grad_(grad)
                loss = ops.softcap_cross_entropy(hg, Ug, tgt, wt, cap, chunk_rows=chunk)
                return (loss.detach(), *(torch.autograd.grad(loss, (hg, Ug)) if grad else ()))
        finally:
            call("pb_gemm_set_variant", 0)

    got, want = run(0), run(8)
    # the same logits and exponentials, added up in another order in fp32
    assert (got[0] - want[0]).abs() <= 1e-5 * want[0].abs()
    for a, b in zip(got[1:], want[1:]):
        assert (a.float() - b.float()).norm() <= 5e-3 * b.float().norm()
    ops.check_status("cuda")


def test_softcap_ce_fresh_gradient_chunks():
    """A unembedding gradient that is not accumulated: one chunk, several, and a non-unit upstream
    gradient, against the accumulating form's buffer (fp32 sums of the same products)."""
    from prometheus_b200.ops import functional as ops

    rows, d, V, cap = 130, 128, 1032, 30.0
    h, U = _r(rows, d, seed=3), _r(V, d, seed=4, scale=0.1)
    tgt = torch.randint(0, V, (rows,), device="cuda", dtype=torch.int32)
    wt = torch.full((rows,), 1.0 / rows, device="cuda")
    for chunk in (64, 4096):
        Ug = U.clone().requires_grad_(True)
        (gU,) = torch.autograd.grad(2.5 * ops.softcap_cross_entropy(h, Ug, tgt, wt, cap, chunk_rows=chunk), (Ug,))
        Um = U.clone().requires_grad_(True)
        Um.main_grad = torch.zeros(V, d, device="cuda")
        ops.softcap_cross_entropy(h, Um, tgt, wt, cap, chunk_rows=chunk)
        assert torch.equal(gU, (Um.main_grad * 2.5).to(BF16))


@pytest.mark.parametrize("form", ["bf16", "transposed", "shifted"])
def test_softcap_ce_accumulator_from_saved_tensor_hooks(form):
    """Hooks may give the fp32 accumulator back as another type, with other strides or from a base that is
    not 16-byte aligned; the scaled gradient is then that tensor's."""
    from prometheus_b200.ops import functional as ops

    rows, d, V, cap = 64, 128, 1032, 30.0
    h, U = _r(rows, d, seed=3), _r(V, d, seed=4, scale=0.1)
    tgt = torch.randint(0, V, (rows,), device="cuda", dtype=torch.int32)
    wt = torch.full((rows,), 1.0 / rows, device="cuda")

    def unpack(t):
        if t.shape != (V, d) or t.dtype != torch.float32:
            return t
        if form == "bf16":
            return t.to(BF16)
        if form == "transposed":
            return t.t().contiguous().t()
        return torch.empty(V * d + 1, device="cuda")[1:].view(V, d).copy_(t)

    def grad(hooked):
        Ug = U.clone().requires_grad_(True)
        if not hooked:
            return torch.autograd.grad(2.5 * ops.softcap_cross_entropy(h, Ug, tgt, wt, cap), (Ug,))[0]
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
            loss = 2.5 * ops.softcap_cross_entropy(h, Ug, tgt, wt, cap)
        return torch.autograd.grad(loss, (Ug,))[0]

    got, want = grad(True), grad(False)
    if form == "bf16":       # one more rounding, of the accumulator: 2^-8 of each element
        assert ((got.float() - want.float()).abs() <= 2.0 ** -7 * want.float().abs()).all()
    else:
        assert torch.equal(got, want)


@pytest.mark.parametrize("rows,form", [(1, ""), (63, ""), (256, ""), (257, ""), (130, "h rewritten"), (130, "bf16 double"),
                                       (130, "shifted"), (130, "transposed"), (130, "batched"), (130, "graph")])
def test_softcap_ce_unembedding_gradient_in_the_backward(rows, form):
    """One chunk of at most 2 d rows (256 here): dU is a product of the backward, scaled in its epilogue. fp32 sums times
    the factor, rounded once, are bit for bit the accumulating form's buffer times the factor. The saved
    tensors in other forms, an h that was reused, and batched or differentiated upstream gradients give the same."""
    from prometheus_b200.ops import functional as ops

    d, V, cap = 128, 1032, 30.0
    h, U = _r(rows, d, seed=3), _r(V, d, seed=4, scale=0.1)
    tgt = torch.randint(0, V, (rows,), device="cuda", dtype=torch.int32)
    wt = torch.full((rows,), 1.0 / rows, device="cuda")
    Um = U.clone().requires_grad_(True)
    Um.main_grad = torch.zeros(V, d, device="cuda")
    ops.softcap_cross_entropy(h, Um, tgt, wt, cap)
    want = (Um.main_grad * 2.5).to(BF16)

    def unpack(t):
        if form == "bf16 double":
            return t.double()
        if form == "transposed":
            return t.t().contiguous().t()
        return torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")[1:].view(t.shape).copy_(t)

    Ug, hg = U.clone().requires_grad_(True), h.clone()
    hooks = form in ("bf16 double", "shifted", "transposed")
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack if hooks else (lambda t: t)):
        loss = ops.softcap_cross_entropy(hg, Ug, tgt, wt, cap)
    if form == "h rewritten":
        hg.zero_()
    if form == "batched":
        (gU,) = torch.autograd.grad(loss, (Ug,), torch.tensor([2.5, 1.0], device="cuda"), is_grads_batched=True)
        assert torch.equal(gU[1], Um.main_grad.to(BF16))
        gU = gU[0]
    else:
        (gU,) = torch.autograd.grad(2.5 * loss, (Ug,), create_graph=form == "graph")
    assert torch.equal(gU.detach(), want)


@pytest.mark.parametrize("M,N,K,batch,a_mn,b_mn,out,d", [
    (1, 8, 1024, 1, 0, 0, "bf16", ""), (129, 128, 1088, 1, 0, 0, "f32", "bf16"), (64, 1, 1032, 1, 0, 0, "bf16", "f32"),
    (72, 520, 2048, 1, 1, 1, "f32", "same"), (300, 700, 4104, 1, 0, 0, "bf16", "bf16"), (128, 264, 1024, 9, 0, 1, "bf16", "f32"),
    (1024, 1152, 1536, 1, 1, 1, "f32", "same"), (1024, 1160, 1536, 1, 1, 0, "bf16", ""), (1152, 1024, 1024, 1, 0, 0, "f32", "f32")])
def test_gemm_split_contraction(M, N, K, batch, a_mn, b_mn, out, d):
    """Products with few tiles and a long contraction, shared out over clusters of two to eight CTAs: one element, ragged
    edges and unaligned rows, contractions that do not divide evenly, batches, 72 tiles (split), 80 (not), every kind of D.
    fp32 sums: each product K u of its absolute terms, then the output's rounding. Two runs give the same bits."""
    from prometheus_b200.ops import functional as ops

    a = _r(batch, *((K, M) if a_mn else (M, K)), seed=1)
    b = _r(batch, *((K, N) if b_mn else (N, K)), seed=2)
    ty = BF16 if out == "bf16" else torch.float32
    dt = {"": None, "bf16": BF16, "f32": torch.float32, "same": ty}[d]
    dd = None if dt is None else _r(batch, M, N, seed=3).to(dt)
    runs = []
    for _ in range(2):
        c = dd.clone() if d == "same" else torch.full((batch, M, N), float("nan"), dtype=ty, device="cuda")
        add = c if d == "same" else dd
        runs.append(ops.gemm(a, b, a_mn=bool(a_mn), b_mn=bool(b_mn), out=c, d=add, alpha=0.5, beta=0.75 if d != "same" else 1.0))
    assert torch.equal(runs[0], runs[1])
    ad = a.double().transpose(1, 2) if a_mn else a.double()
    bd = b.double() if b_mn else b.double().transpose(1, 2)
    ref, slack = 0.5 * ad @ bd, 0.5 * ad.abs() @ bd.abs()
    if dd is not None:
        ref = ref + (0.75 if d != "same" else 1.0) * dd.double()
        slack = slack + dd.double().abs()
    tol = (K + 8) * 2.0 ** -24 * slack + (2.0 ** -8 if out == "bf16" else 0.0) * ref.abs()
    assert bool(((runs[0].double() - ref).abs() <= tol).all())


def test_optimizer_kernels():
    from prometheus_b200 import train
    from prometheus_b200.ops import _lib
    from prometheus_b200.ops._lib import call, ptr, stream_ptr

    n = 100_003
    g = torch.randn(n, device="cuda")
    scratch = torch.empty(_lib.query("pb_sumsq_nparts", n) + 8, device="cuda")
    out = torch.zeros(1, device="cuda")
    call("pb_sumsq_f32", ptr(g), n, ptr(scratch), ptr(out), 0, stream_ptr())
    assert out.item() == pytest.approx((g.double() ** 2).sum().item(), rel=1e-5)
    p, m, v = torch.randn(n, device="cuda"), torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    lp = torch.empty(n, dtype=BF16, device="cuda")
    gn = (g ** 2).sum().reshape(1)
    clip = 1.0
    s = clip / (gn.sqrt() + 1e-6)
    rp, rm, rv = train.adamw_update(p, g * s, m, v, lr=1e-3, beta1=0.9, beta2=0.95, eps=1e-8,
                                    wd=0.1, step=3)
    call("pb_adamw", ptr(p), ptr(g), ptr(m), ptr(v), ptr(lp), n, 1e-3, 0.9, 0.95, 1e-8, 0.1, 3,
         ptr(gn), clip, 1.0, stream_ptr())
    torch.testing.assert_close(p, rp, rtol=1e-5, atol=1e-6)
    torch.testing.assert_close(m, rm, rtol=1e-5, atol=1e-7)
    torch.testing.assert_close(v, rv, rtol=1e-5, atol=1e-9)
    torch.testing.assert_close(lp.float(), rp, rtol=1e-2, atol=1e-3)
    # Muon prepare: momentum + normalised Nesterov
    r, c = 64, 96
    gm, mom = torch.randn(r * c, device="cuda"), torch.randn(r * c, device="cuda")
    x0 = torch.empty(r * c, dtype=BF16, device="cuda")
    new_m = 0.95 * mom + gm
    nes = gm + 0.95 * new_m
    call("pb_muon_prepare", ptr(gm), ptr(mom), ptr(x0), r * c, 0.95, None, 0.0, 1.0, ptr(scratch),
         stream_ptr())
    torch.testing.assert_close(mom, new_m, rtol=1e-5, atol=1e-6)
    torch.testing.assert_close(x0.float(), nes / nes.norm(), rtol=1e-2, atol=1e-3)


def test_bounded_wait_reports_timeout_instead_of_hanging():
    """A device-side wait on a flag nobody sets returns a status code within its budget."""
    from prometheus_b200.ops import _lib
    from prometheus_b200.ops._lib import call, ptr, stream_ptr

    if not hasattr(_lib.load(), "pb_wait_flag_probe"):
        pytest.skip("probe not built")
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    call("pb_wait_flag_probe", ptr(flag), 1, 2_000_000, ptr(status), stream_ptr())
    torch.cuda.synchronize()
    assert status.item() == 2


@pytest.mark.parametrize("B,S,H", [(1, 64, 1), (1, 128, 2), (2, 448, 3), (1, 200, 2)])
def test_delta_rule_fused_matches_recurrence(B, S, H):
    from prometheus_b200 import kernels
    from prometheus_b200.ops import functional as ops

    D = 128
    q = torch.nn.functional.normalize(_r(B, S, H, D, seed=1).float(), dim=-1).to(BF16)
    k = torch.nn.functional.normalize(_r(B, S, H, D, seed=2).float(), dim=-1).to(BF16)
    v = _r(B, S, H, D, seed=3)
    beta = torch.sigmoid(_r(B, S, H, seed=4).float()).to(BF16)
    s0 = _r(B, H, D, D, seed=5, scale=0.05, dtype=torch.float32)
    go = _r(B, S, H, D, seed=6)
    leaves = [t.clone().requires_grad_(True) for t in (q, k, v, beta)]
    s0l = s0.clone().requires_grad_(True)
    out, st = kernels.chunked_delta_rule(*leaves, s0l)
    torch.cuda.synchronize()
    ops.check_status("cuda")
    (out.float() * go.float()).sum().add(st.sum() * 0.01).backward()
    ref_leaves = [t.float().clone().requires_grad_(True) for t in (q, k, v, beta)]
    s0r = s0.clone().requires_grad_(True)
    o_ref, s_ref = kernels.delta_rule_recurrent(*ref_leaves, s0r)
    (o_ref * go.float()).sum().add(s_ref.sum() * 0.01).backward()
    _close(out, o_ref, 3e-2)
    _close(st, s_ref, 3e-2)
    for name, a, b in zip("qkvb", leaves, ref_leaves):
        _close(a.grad, b.grad, 6e-2)
    _close(s0l.grad, s0r.grad, 6e-2)
    ops.check_status("cuda")


@pytest.mark.parametrize("B,S,H,seg", [(1, 1024, 2, 4), (1, 512, 1, 2), (2, 768, 1, 3)])
def test_delta_rule_segmented_walk_equals_single_pass(B, S, H, seg):
    """Sequences cut into segments (summary walk -> sequential fold -> segmented walk) against
    the single-pass walk of the same kernels and against the fp32 per-token recurrence, forward,
    final state and every gradient, with an initial state and a final-state gradient."""
    from prometheus_b200 import kernels
    from prometheus_b200.ops import functional as ops
    from prometheus_b200.ops.delta import delta_rule_fused, scan_segments

    assert scan_segments(16, 256) == 8 and scan_segments(128, 64) == 1 and scan_segments(1, 8) == 1
    assert scan_segments(64, 64) == 1 and scan_segments(32, 128) == 4
    D = 128
    q = torch.nn.functional.normalize(_r(B, S, H, D, seed=1).float(), dim=-1).to(BF16)
    k = torch.nn.functional.normalize(_r(B, S, H, D, seed=2).float(), dim=-1).to(BF16)
    v = _r(B, S, H, D, seed=3)
    beta = torch.sigmoid(_r(B, S, H, seed=4).float()).to(BF16)
    s0 = _r(B, H, D, D, seed=5, scale=0.05, dtype=torch.float32)
    go = _r(B, S, H, D, seed=6)

    def run(n_seg):
        leaves = [t.clone().requires_grad_(True) for t in (q, k, v, beta)]
        s0l = s0.clone().requires_grad_(True)
        out, st = delta_rule_fused(*leaves, s0l, n_seg=n_seg)
        (out.float() * go.float()).sum().add(st.sum() * 0.01).backward()
        torch.cuda.synchronize()
        ops.check_status("cuda")
        return [out, st] + [t.grad for t in leaves] + [s0l.grad]

    one, cut = run(1), run(seg)
    for name, a, b in zip(("out", "state", "dq", "dk", "dv", "dbeta", "ds0"), cut, one):
        err = (a.float() - b.float()).norm().item()
        assert err <= 1.5e-2 * (b.float().norm().item() + 1e-6), (name, err)
    ref_leaves = [t.float().clone().requires_grad_(True) for t in (q, k, v, beta)]
    s0r = s0.clone().requires_grad_(True)
    o_ref, s_ref = kernels.delta_rule_recurrent(*ref_leaves, s0r)
    (o_ref * go.float()).sum().add(s_ref.sum() * 0.01).backward()
    _close(cut[0], o_ref, 3e-2)
    _close(cut[1], s_ref, 3e-2)
    for a, b in zip(cut[2:6], ref_leaves):
        _close(a, b.grad, 6e-2)
    _close(cut[6], s0r.grad, 6e-2)


@pytest.mark.parametrize("B,S,H,seg", [(2, 1, 1, 1), (3, 63, 2, 1), (2, 65, 2, 1), (2, 1000, 2, 4), (1, 250, 1, 2)])
def test_delta_rule_ragged_equals_explicit_padding(B, S, H, seg):
    """A length that is not a multiple of the chunk, read in place, gives the bits of the same call
    on zero-padded tensors (batch entries follow one another without a gap, so a row too many
    would be the next entry's), without grad as with it, and from a misaligned base."""
    from prometheus_b200.ops import functional as ops
    from prometheus_b200.ops.delta import delta_rule_fused

    D = 128
    q = torch.nn.functional.normalize(_r(B, S, H, D, seed=1).float(), dim=-1).to(BF16)
    k = torch.nn.functional.normalize(_r(B, S, H, D, seed=2).float(), dim=-1).to(BF16)
    v = _r(B, S, H, D, seed=3)
    beta = torch.sigmoid(_r(B, S, H, seed=4).float()).to(BF16)
    s0 = _r(B, H, D, D, seed=5, scale=0.05, dtype=torch.float32)
    go, gs = _r(B, S, H, D, seed=6), _r(B, H, D, D, seed=7, scale=0.1, dtype=torch.float32)
    pad = (-S) % 64

    def run(ts, g):
        leaves = [t.clone().requires_grad_(True) for t in ts]
        s0l = s0.clone().requires_grad_(True)
        out, st = delta_rule_fused(*leaves, s0l, n_seg=seg)
        grads = torch.autograd.grad([out, st], leaves + [s0l], [g, gs])
        ops.check_status("cuda")
        return [out.detach(), st.detach(), *grads]

    def padded(t):
        return torch.cat([t, t.new_zeros(B, pad, *t.shape[2:])], dim=1)

    got = run((q, k, v, beta), go)
    want = run([padded(t) for t in (q, k, v, beta)], padded(go))
    for name, a, b in zip(("out", "state", "dq", "dk", "dv", "dbeta", "ds0"), got, want):
        assert torch.equal(a, b if name in ("state", "ds0") else b[:, :S]), name
    with torch.no_grad():
        out, st = delta_rule_fused(q, k, v, beta, s0, n_seg=seg)
        assert torch.equal(out, got[0]) and torch.equal(st, got[1])
        off = torch.empty(q.numel() + 1, dtype=BF16, device="cuda")[1:].view(q.shape).copy_(q)
        assert torch.equal(delta_rule_fused(off, k, v, beta, s0, n_seg=seg)[0], out)


@pytest.mark.parametrize("S,seg", [(130, 1), (512, 2)])
def test_delta_walk_column_split_equals_whole_state(S, seg):
    """More CTAs than half the GPU walk the state in one piece, fewer in two halves of its columns: a
    batch of 96 sequences against its entries one by one, with state and gradients."""
    from prometheus_b200.ops import functional as ops
    from prometheus_b200.ops.delta import delta_rule_fused

    B, H, D = 6, 16, 128
    q = torch.nn.functional.normalize(_r(B, S, H, D, seed=1).float(), dim=-1).to(BF16)
    k = torch.nn.functional.normalize(_r(B, S, H, D, seed=2).float(), dim=-1).to(BF16)
    v, go = _r(B, S, H, D, seed=3), _r(B, S, H, D, seed=6)
    beta = torch.sigmoid(_r(B, S, H, seed=4).float()).to(BF16)
    s0 = _r(B, H, D, D, seed=5, scale=0.05, dtype=torch.float32)
    gs = _r(B, H, D, D, seed=7, scale=0.1, dtype=torch.float32)

    def run(sl):
        leaves = [t[sl].clone().requires_grad_(True) for t in (q, k, v, beta, s0)]
        out = delta_rule_fused(*leaves, n_seg=seg)
        grads = torch.autograd.grad(out, leaves, (go[sl], gs[sl]))
        ops.check_status("cuda")
        return [t.detach() for t in (*out, *grads)]

    whole = run(slice(0, B))
    for i in range(B):
        for name, a, b in zip(("out", "state", "dq", "dk", "dv", "dbeta", "ds0"), run(slice(i, i + 1)), whole):
            assert torch.equal(a[0], b[i]), (name, i)


@pytest.mark.parametrize("B,S,H", [(1, 64, 1), (2, 100, 3), (5, 4096, 2)])
def test_delta_chunk_products(B, S, H):
    """The four products against batched fp32, with fewer and with more chunks than CTAs."""
    from prometheus_b200.ops import delta as dl
    from prometheus_b200.ops import functional as ops
    from prometheus_b200.ops._lib import call, ptr, stream_ptr

    n = -(-S // 64)
    G = B * H * n
    ndu, u = _r(G, 64, 128, seed=1), _r(G, 64, 128, seed=2)
    sb, dsb = _r(G, 128, 128, seed=3, scale=0.2), _r(G, 128, 128, seed=4, scale=0.2)
    d_out = _r(B, S, H, 128, seed=5)
    d_w, d_q, d_k = (torch.full_like(u, float("nan")) for _ in range(3))
    d_m = torch.full((G, 64, 64), float("nan"), dtype=BF16, device="cuda")
    call("pb_delta_chunk_products", ptr(ndu), ptr(d_out), ptr(u), ptr(sb), ptr(dsb), ptr(d_w), ptr(d_q), ptr(d_k),
         ptr(d_m), B, S, H, H * 128, ptr(ops.status_word("cuda")), stream_ptr())
    ops.check_status("cuda")
    doc = dl._to_chunks(torch.nn.functional.pad(d_out, (0, 0, 0, 0, 0, n * 64 - S)), n).float()
    _close(d_w, ndu.float() @ sb.float().transpose(1, 2), 1e-2)
    _close(d_q, doc @ sb.float().transpose(1, 2), 1e-2)
    _close(d_k, u.float() @ dsb.float().transpose(1, 2), 1e-2)
    _close(d_m, doc @ u.float().transpose(1, 2), 1e-2)


@pytest.mark.parametrize("n_seq,n_chunks,n_seg,cut", [(37, 6, 2, 0), (75, 3, 1, 0), (75, 1, 1, 0), (40, 8, 4, 0), (80, 4, 2, 27)])
def test_delta_summary_maps(n_seq, n_chunks, n_seg, cut):
    """The affine map of every segment against 64 bits, on both sides of the line where one CTA computes
    both maps (more than 74 segments on 148 SMs), and with a last chunk of 64 - ``cut`` tokens in place
    (16 heads). The images of the state and of U are bf16: each chunk adds at most 2^-9 of the state
    twice, and 2^-9 sqrt(2) of at most four chunks stays under 2e-2."""
    from prometheus_b200.ops import functional as ops
    from prometheus_b200.ops._lib import call, ptr, stream_ptr

    heads, s = (16, n_chunks * 64 - cut) if cut else (0, n_chunks * 64)
    rows = n_seq * n_chunks * 64
    w, uh = (_r(rows, 128, seed=i, scale=128 ** -0.5) for i in (1, 2))
    if heads:
        k = _r(n_seq // heads, s, heads * 128, seed=3, scale=128 ** -0.5)
        kc = torch.nn.functional.pad(k, (0, 0, 0, cut)).reshape(n_seq // heads, n_chunks * 64, heads, 128).transpose(1, 2)
    else:
        k = kc = _r(rows, 128, seed=3, scale=128 ** -0.5)
    r, p = (torch.full((n_seq * n_seg, 128, 128), float("nan"), device="cuda") for _ in range(2))
    call("pb_delta_scan_summary_fwd", ptr(w), ptr(uh), ptr(k), ptr(r), ptr(p), n_seq, n_chunks, n_seg, heads, s,
         heads * 128, ptr(ops.status_word(torch.device("cuda"))), stream_ptr())
    torch.cuda.synchronize()
    ops.check_status("cuda")
    per = n_chunks // n_seg
    wd, ud, kd = (t.reshape(n_seq * n_seg, per, 64, 128).double() for t in (w, uh, kc))
    rd = torch.zeros_like(r, dtype=torch.float64)
    pd = torch.eye(128, device="cuda").double().expand_as(rd)
    for c in range(per):
        kt = kd[:, c].transpose(1, 2)
        rd = rd + kt @ (ud[:, c] - wd[:, c] @ rd)
        pd = pd - kt @ (wd[:, c] @ pd)
    for got, ref in ((r, rd), (p, pd)):
        err = (got.double() - ref).flatten(1).norm(dim=1) / ref.flatten(1).norm(dim=1)
        assert err.max() <= 2e-2, err.max()


@pytest.mark.parametrize("H,S", [(3, 448), (37, 64), (37, 129), (37, 256), (37, 448), (74, 300)])
def test_delta_walk_stages(H, S):
    """64-column walks, which have three stages, of one chunk to more than twice as many, against the same heads among 80,
    whose walk has 128 columns (from 67 on the forward has 128 too, since it keeps the states; the backward has 64 up to 74): the columns of the state never mix and each sum is over the same terms in the same
    order, so all outputs are the same bits."""
    from prometheus_b200.ops.delta import delta_rule_fused

    q, k, v, do = (_r(1, S, 80, 128, seed=i, scale=0.08) for i in (1, 2, 3, 5))
    beta = torch.sigmoid(_r(1, S, 80, seed=4, dtype=torch.float32))

    def run(h):
        leaves = [t[:, :, :h].contiguous().requires_grad_(True) for t in (q, k, v, beta)]
        out, fin = delta_rule_fused(*leaves, None, n_seg=1)
        return [t[:, :, :H] for t in (out, *torch.autograd.grad(out, leaves, do[:, :, :h].contiguous()))] + [fin[:, :H]]

    for few, many in zip(run(H), run(80)):
        assert torch.equal(few, many)


@pytest.mark.parametrize("H,grad", [(66, True), (67, True), (74, False), (75, False)])
def test_delta_walk_columns_at_their_lines(H, grad):
    """The last sequence counts of 64-column walks and the first of 128-column ones, on 148 SMs: 66 and 67 for a forward that
    keeps the states (74 and 75 for its backward), 74 and 75 for one that keeps nothing. The same heads among 80, bit for bit."""
    from prometheus_b200.ops.delta import delta_rule_fused

    q, k, v, do = (_r(1, 300, 80, 128, seed=i, scale=0.08) for i in (1, 2, 3, 5))
    beta = torch.sigmoid(_r(1, 300, 80, seed=4, dtype=torch.float32))

    def run(h):
        leaves = [t[:, :, :h].contiguous().requires_grad_(grad) for t in (q, k, v, beta)]
        out, fin = delta_rule_fused(*leaves, None, n_seg=1)
        grads = torch.autograd.grad(out, leaves, do[:, :, :h].contiguous()) if grad else ()
        return [t[:, :, :H] for t in (out, *grads)] + [fin[:, :H]]

    for few, many in zip(run(H), run(80)):
        assert torch.equal(few, many)


def test_delta_layer_over_128_sequences_of_64_chunks():
    """The walks with 128 columns and the states kept, two stages deep over 64 chunks, as a training run at 8 x 4096 tokens and 16
    heads has them, against the fp32 scan. Images of the state and of U, W, U^, M and the gradients' operands are bf16:
    each rounds by 2^-9 of its size, about ten of them between an input and a result."""
    from prometheus_b200.ops import delta as dl

    B, S, H = 8, 4096, 16
    q, k = (torch.nn.functional.normalize(_r(B, S, H, 128, seed=i).float(), dim=-1).to(BF16) for i in (1, 2))
    v, do = _r(B, S, H, 128, seed=3), _r(B, S, H, 128, seed=5)
    beta = torch.sigmoid(_r(B, S, H, seed=4))
    leaves = [t.requires_grad_(True) for t in (q, k, v, beta)]
    out, fin = dl.delta_rule_fused(*leaves, None)
    got = [out, fin, *torch.autograd.grad(out, leaves, do)]
    for b in range(0, B, 3):
        ref = [t[b:b + 1].detach().float().requires_grad_(True) for t in leaves]
        r_out, r_fin = dl.delta_rule_scan(*ref, None)
        want = [r_out, r_fin, *torch.autograd.grad(r_out, ref, do[b:b + 1].float())]
        for g, w in zip(got, want):
            assert ((g[b:b + 1].float() - w).norm() / w.norm()).item() < 10 * 2.0 ** -9


@pytest.mark.parametrize("H", [4, 80])          # 64- and 128-column walks
def test_delta_initial_state_at_any_float(H):
    """An initial state and a final-state gradient whose storage starts 4 bytes off a 16-byte boundary
    give what aligned ones give, bit for bit (the wide reads are not taken)."""
    from prometheus_b200.ops.delta import delta_rule_fused

    q, k, v = (_r(1, 128, H, 128, seed=i, scale=0.08) for i in (1, 2, 3))
    beta = torch.sigmoid(_r(1, 128, H, seed=4, dtype=torch.float32))
    flat = _r(2 * H * 128 * 128 + 1, seed=5, scale=0.05, dtype=torch.float32)
    n = H * 128 * 128

    def run(s0, gs):
        leaf = s0.requires_grad_(True)
        out, st = delta_rule_fused(q, k, v, beta, leaf, n_seg=1)
        return out, st, torch.autograd.grad([out, st], leaf, [v, gs])[0]

    off = [flat[1 + i * n:1 + (i + 1) * n].view(1, H, 128, 128).detach() for i in (0, 1)]
    assert all(x.data_ptr() % 16 == 4 for x in off)
    for a, b in zip(run(*off), run(*(x.clone() for x in off))):
        assert torch.equal(a, b)


@pytest.mark.parametrize("n_seq,n_seg", [(1, 1), (3, 8)])
@pytest.mark.parametrize("reverse", [0, 1])
def test_delta_compose(n_seq, n_seg, reverse):
    """The fold of the segments' maps against 64 bits: 128 fp32 products a step, n_seg steps."""
    from prometheus_b200.ops._lib import call, ptr, stream_ptr

    p = _r(n_seq, n_seg, 128, 128, seed=1, scale=0.08, dtype=torch.float32)
    r = _r(n_seq, n_seg, 128, 128, seed=2, dtype=torch.float32)
    s0 = _r(n_seq, 128, 128, seed=3, dtype=torch.float32)
    s_in, s_fin, p_tot = torch.empty_like(r), torch.empty_like(s0), torch.empty_like(s0)
    for start in (s0, None):
        call("pb_delta_compose", ptr(p), ptr(r), ptr(start), ptr(s_in), ptr(s_fin), None if reverse else ptr(p_tot),
             n_seq, n_seg, reverse, stream_ptr())
        cur = torch.zeros_like(s0).double() if start is None else start.double()
        tot = torch.eye(128, device="cuda").double().expand(n_seq, 128, 128)
        for j in reversed(range(n_seg)) if reverse else range(n_seg):
            assert (s_in[:, j].double() - cur).norm() <= 1e-5 * (cur.norm() + 1e-6)
            m = p[:, j].double()
            cur = (m.transpose(1, 2) if reverse else m) @ cur + r[:, j].double()
            tot = m @ tot
        assert (s_fin.double() - cur).norm() <= 1e-5 * cur.norm()
        if not reverse:
            assert (p_tot.double() - tot).norm() <= 1e-5 * tot.norm()


@pytest.mark.parametrize("M,N,K", [(256, 512, 64), (2048, 4096, 128)])      # one wave of 128 x 128 tiles, CTA pairs
def test_gemm_accumulates_sums_below_the_normal_range(M, N, K):
    """Four products of about 2^-126 added into one buffer by adding stores: the bits of the epilogue's addition, below the normal
    range and beside it."""
    from prometheus_b200.ops import functional as ops

    a, b = _r(K, M, seed=1), _r(K, N, seed=2)
    a[:, :M // 2] *= 2.0 ** -65
    b[:, :N // 2] *= 2.0 ** -65
    got, want = (torch.zeros(M, N, device="cuda") for _ in range(2))
    for _ in range(4):
        ops.gemm(a, b, a_mn=True, b_mn=True, out=got, d=got, beta=1.0)
        want = ops.gemm(a, b, a_mn=True, b_mn=True, out_dtype=torch.float32, d=want, beta=1.0)
    assert ((want != 0) & (want.abs() < 2.0 ** -126)).any()
    assert torch.equal(got, want)


@pytest.mark.parametrize("M,N,K,batch", [(8, 1024, 64, 1), (136, 264, 200, 1), (264, 1000, 72, 3), (1024, 1152, 136, 2), (4736, 512, 128, 1),
                                         (4744, 512, 128, 1)])
def test_gemm_accumulates_in_place_as_with_a_copy(M, N, K, batch):
    """fp32 C += A^T B by adding stores against the same product with D elsewhere, which the epilogue reads: the same
    bits, on tiles of 128 (up to 148 of them: 4736 x 512) and on pairs, with rows and columns cut off."""
    from prometheus_b200.ops import functional as ops

    a, b = _r(batch, K, M, seed=1), _r(batch, K, N, seed=2)
    c = _r(batch, M, N, seed=3, dtype=torch.float32)
    want = ops.gemm(a, b, a_mn=True, b_mn=True, out=torch.empty_like(c), d=c.clone(), beta=1.0)
    got = ops.gemm(a, b, a_mn=True, b_mn=True, out=c, d=c, beta=1.0)
    assert torch.equal(got, want)
    ref = (a.double().transpose(1, 2) @ b.double()) + _r(batch, M, N, seed=3, dtype=torch.float32).double()
    assert ((got.double() - ref).norm() / ref.norm()).item() < 1e-6


@pytest.mark.parametrize("rows,cols,nb,steps", [(64, 64, 1, 1), (128, 264, 3, 5), (264, 128, 2, 5), (256, 1024, 3, 4), (8, 1024, 2, 0)])
def test_newton_schulz_is_its_products(rows, cols, nb, steps):
    """One call against the products it stands for, bit for bit: both orientations, odd and even step counts."""
    from prometheus_b200 import train
    from prometheus_b200.ops import functional as ops

    x = _r(nb, rows, cols, seed=rows + cols, scale=(rows * cols) ** -0.5)
    m, wide = min(rows, cols), rows <= cols
    a, b, c = train._NS_A, train._NS_B, train._NS_C
    ref = x.clone()
    for _ in range(steps):
        g = ops.gemm(ref, ref) if wide else ops.gemm(ref, ref, a_mn=True, b_mn=True)
        p = ops.gemm(g, g, d=g, alpha=c, beta=b)
        ref = ops.gemm(p, ref, b_mn=True, d=ref, beta=a) if wide else ops.gemm(ref, p, d=ref, beta=a)
    g, p = (torch.empty(nb, m, m, dtype=BF16, device="cuda") for _ in range(2))
    assert torch.equal(ops.newton_schulz(x, torch.empty_like(x), g, p, steps, a, b, c), ref)


@pytest.mark.parametrize("S,close", [(1, False), (16, True), (17, True), (33, True), (64, True), (100, False), (640, True)])
def test_delta_chunk_inverse(S, close):
    """T = (I + diag(beta) tril(K K^T, -1))^-1 of every chunk, block by block, against float64. ``close``: keys that
    nearly agree, so that A is far from small. An inverse taken from the blocks' products in fp32 is off by at most
    n u |T| |I + A| |T| elementwise in each product, and T is then rounded to bf16."""
    from prometheus_b200.ops._lib import call, ptr, stream_ptr
    from prometheus_b200.ops.functional import status_word

    B, H, n = 2, 3, -(-S // 64)
    k = _r(B, S, H, 128, seed=S) + (4.0 * _r(B, 1, H, 128, seed=1) if close else 0)
    k = torch.nn.functional.normalize(k.float(), dim=-1).to(BF16).contiguous()
    beta = torch.sigmoid(_r(B, S, H, seed=2, dtype=torch.float32) + 1.0)
    q, v = _r(B, S, H, 128, seed=3), _r(B, S, H, 128, seed=4)
    g = B * H * n
    w, u = (torch.empty(g, 64, 128, dtype=BF16, device="cuda") for _ in range(2))
    m, ap, t = (torch.empty(g, 64, 64, dtype=BF16, device="cuda") for _ in range(3))
    call("pb_delta_prep_fwd", ptr(q), ptr(k), ptr(v), ptr(beta), 1, ptr(w), ptr(u), ptr(m), ptr(ap), ptr(t), B, S, H,
         H * 128, ptr(status_word(k.device)), 0, stream_ptr())
    pad = n * 64 - S
    kc = torch.nn.functional.pad(k, (0, 0, 0, 0, 0, pad)).reshape(B, n, 64, H, 128).permute(0, 3, 1, 2, 4).double()
    bc = torch.nn.functional.pad(beta, (0, 0, 0, pad)).reshape(B, n, 64, H).permute(0, 3, 1, 2).double()
    a = torch.tril(bc[..., None] * (kc @ kc.transpose(-1, -2)), -1).reshape(g, 64, 64)
    ia = torch.eye(64, dtype=torch.float64, device="cuda") + a
    ref = torch.linalg.inv(ia)
    slack = 2 * 64 * 2.0 ** -24 * (ref.abs() @ ia.abs() @ ref.abs()) + 2.0 ** -133
    err = (t.double() - ref).abs()
    assert bool((err <= 2.0 ** -8 * ref.abs() + 2 * slack).all()), (err - 2.0 ** -8 * ref.abs() - 2 * slack).max().item()
    err = (ap.double() - ref * bc.reshape(g, 1, 64)).abs()
    assert bool((err <= 2.0 ** -8 * ref.abs() + 2 * slack).all())


def test_delta_prep_bwd_kernel_matches_fp32_oracle():
    """The fused chunk-local backward against the same algebra in batched fp32 PyTorch."""
    from prometheus_b200.ops import delta as dl
    from prometheus_b200.ops import functional as ops
    from prometheus_b200.ops._lib import call, ptr, stream_ptr

    B, S, H, D = 2, 192, 3, 128
    n = S // 64
    G = B * H * n
    q = torch.nn.functional.normalize(_r(B, S, H, D, seed=1).float(), dim=-1).to(BF16)
    k = torch.nn.functional.normalize(_r(B, S, H, D, seed=2).float(), dim=-1).to(BF16)
    v = _r(B, S, H, D, seed=3)
    beta = torch.sigmoid(_r(B, S, H, seed=4).float()).to(BF16)
    w, uh = torch.empty(G, 64, 128, dtype=BF16, device="cuda"), torch.empty(G, 64, 128, dtype=BF16, device="cuda")
    m, ap, t = (torch.empty(G, 64, 64, dtype=BF16, device="cuda") for _ in range(3))
    st = ptr(ops.status_word("cuda"))
    call("pb_delta_prep_fwd", ptr(q), ptr(k), ptr(v), ptr(beta), 0, ptr(w), ptr(uh), ptr(m), ptr(ap),
         ptr(t), B, S, H, H * D, st, 0, stream_ptr())
    # forward operands against their definition
    kc, vc, qc = (dl._to_chunks(x, n).float() for x in (k, v, q))
    bc = beta.float().reshape(B, n, 64, H).permute(0, 3, 1, 2).reshape(G, 64)
    a = torch.tril(kc @ kc.transpose(-1, -2), diagonal=-1) * bc[:, :, None]
    eye = torch.eye(64, device="cuda")
    t_ref = torch.linalg.solve_triangular(eye + a, eye.expand(G, 64, 64).contiguous(), upper=False)
    _close(t, t_ref, 2e-2)
    _close(ap, t_ref * bc[:, None, :], 2e-2)
    _close(w, (t_ref * bc[:, None, :]) @ kc, 2e-2)
    _close(uh, (t_ref * bc[:, None, :]) @ vc, 2e-2)
    _close(m, torch.tril(qc @ kc.transpose(-1, -2)), 2e-2)
    d_w, ndu, d_qs, d_ks = (_r(G, 64, 128, seed=10 + i, scale=0.5) for i in range(4))
    d_m = _r(G, 64, 64, seed=20, scale=0.5)
    dq, dk, dv = torch.empty_like(q), torch.empty_like(q), torch.empty_like(q)
    db = torch.empty_like(beta)
    call("pb_delta_prep_bwd", ptr(q), ptr(k), ptr(v), ptr(beta), 0, ptr(ap), ptr(t), ptr(d_w),
         ptr(ndu), ptr(d_m), ptr(d_qs), ptr(d_ks), ptr(dq), ptr(dk), ptr(dv), ptr(db), B, S, H, H * D,
         st, 0, stream_ptr())
    torch.cuda.synchronize()
    ops.check_status("cuda")
    rq, rk, rv, rb = dl.delta_prep_backward_ref(q, k, v, beta, ap, t, d_w, ndu, d_m, d_qs, d_ks)
    _close(dq, rq, 3e-2)
    _close(dk, rk, 3e-2)
    _close(dv, rv, 3e-2)
    _close(db, rb, 3e-2)


@pytest.mark.parametrize("B,S,H,fp32", [(1, 1, 1, 1), (2, 63, 3, 0), (1, 64, 2, 1), (2, 65, 1, 0), (1, 300, 80, 0), (1, 300, 80, 1)])
def test_delta_bwd_kernel_matches_fp32_oracle(B, S, H, fp32):
    """The chunk-local backward in one kernel against its algebra in batched fp32 PyTorch: one token, the edges of a
    chunk, more chunks than SMs (400), both types of beta. dW, dM, dA', X and dG are rounded to bf16 once each and a
    result once more: 2^-9 of their largest values, through at most four products whose weights have row sums of a few
    units (|T|, |A'|, |K K^T| of 64 random unit keys), stays under 3e-2 of the result's scale."""
    from prometheus_b200.ops import delta as dl
    from prometheus_b200.ops import functional as ops
    from prometheus_b200.ops._lib import call, ptr, stream_ptr

    D, n = 128, -(-S // 64)
    G, pad = B * H * n, n * 64 - S
    q, k = (torch.nn.functional.normalize(_r(B, S, H, D, seed=i).float(), dim=-1).to(BF16) for i in (1, 2))
    v, d_out = _r(B, S, H, D, seed=3), _r(B, S, H, D, seed=5, scale=0.5)
    beta = torch.sigmoid(_r(B, S, H, seed=4).float()).to(torch.float32 if fp32 else BF16)
    ap, t = (torch.empty(G, 64, 64, dtype=BF16, device="cuda") for _ in range(2))
    w, uh = (torch.empty(G, 64, D, dtype=BF16, device="cuda") for _ in range(2))
    m, st = torch.empty_like(ap), ptr(ops.status_word("cuda"))
    call("pb_delta_prep_fwd", ptr(q), ptr(k), ptr(v), ptr(beta), fp32, ptr(w), ptr(uh), ptr(m), ptr(ap), ptr(t), B, S, H,
         H * D, st, 0, stream_ptr())
    ndu, u = _r(G, 64, D, seed=11, scale=0.5), _r(G, 64, D, seed=12, scale=0.5)
    sb, dsb = _r(G, D, D, seed=13, scale=0.1), _r(G, D, D, seed=14, scale=0.1)
    dq, dk, dv = (torch.full_like(q, float("nan")) for _ in range(3))
    db = torch.full_like(beta, float("nan"))
    call("pb_delta_bwd", ptr(q), ptr(k), ptr(v), ptr(beta), fp32, ptr(ap), ptr(t), ptr(ndu), ptr(d_out), ptr(u), ptr(sb),
         ptr(dsb), ptr(dq), ptr(dk), ptr(dv), ptr(db), B, S, H, H * D, st, stream_ptr())
    torch.cuda.synchronize()
    ops.check_status("cuda")
    full = lambda x: torch.nn.functional.pad(x, (0, 0) * (x.dim() - 2) + (0, pad))
    doc = dl._to_chunks(full(d_out), n).float()
    d_w, d_m = ndu.float() @ sb.float().transpose(1, 2), doc @ u.float().transpose(1, 2)
    d_qs, d_ks = doc @ sb.float().transpose(1, 2), u.float() @ dsb.float().transpose(1, 2)
    want = dl.delta_prep_backward_ref(full(q), full(k), full(v), full(beta), ap, t, d_w, ndu, d_m, d_qs, d_ks)
    for got, ref in zip((dq, dk, dv, db), want):
        _close(got, ref[:, :S], 3e-2)
    # and against the two kernels that do it in parts, which round dW, dM and the state products to bf16 in between
    d_w, d_qs, d_ks = (torch.empty_like(u) for _ in range(3))
    d_m, parts = torch.empty_like(ap), [torch.empty_like(q) for _ in range(3)] + [torch.empty_like(beta)]
    call("pb_delta_chunk_products", ptr(ndu), ptr(d_out), ptr(u), ptr(sb), ptr(dsb), ptr(d_w), ptr(d_qs), ptr(d_ks), ptr(d_m),
         B, S, H, H * D, st, stream_ptr())
    call("pb_delta_prep_bwd", ptr(q), ptr(k), ptr(v), ptr(beta), fp32, ptr(ap), ptr(t), ptr(d_w), ptr(ndu), ptr(d_m), ptr(d_qs),
         ptr(d_ks), *(ptr(x) for x in parts), B, S, H, H * D, st, 0, stream_ptr())
    for got, ref in zip((dq, dk, dv, db), parts):
        _close(got, ref, 2.0 ** -7)
    ops.check_status("cuda")


def test_debug_bounds_build_records_and_skips_a_bad_index():
    """The -DPB_DEBUG_BOUNDS library: an index that comes from data and leaves its range is
    recorded as (kernel, index, limit) and the access is skipped; the kernel finishes and the
    context stays usable. Both injected indices stay inside real allocations, so nothing could
    fault even without the check. Runs in a child interpreter (the library is chosen at load)."""
    import os
    import subprocess
    import sys
    from pathlib import Path

    code = r'''
import torch
from prometheus_b200.ops import _lib, functional as ops
from prometheus_b200.ops._lib import call, ptr, stream_ptr
assert _lib.load().pb_debug_bounds_enabled() == 1
assert _lib.debug_bounds_read() is None
# 1. soft-cap CE: a target outside the vocabulary (row 0 of 4: the element it names is in row 1)
V, rows = 1024, 4
logits = torch.randn(rows, V, device="cuda").bfloat16()
targets = torch.tensor([V + 3, 5, 6, 7], dtype=torch.int32, device="cuda")
wt = torch.ones(rows, device="cuda")
loss = torch.empty(rows, device="cuda")
call("pb_softcap_ce", ptr(logits), ptr(targets), ptr(wt), ptr(loss), None, rows, V, 30.0, 0, stream_ptr())
rec = _lib.debug_bounds_read()
assert rec["hits"] >= 1                                      # every thread of the row's block saw it
assert {k: rec[k] for k in ("file", "kernel", "index", "limit")} == \
    {"file": "elementwise", "kernel": 1, "index": V + 3, "limit": V}, rec
assert torch.isfinite(loss).all()
assert _lib.debug_bounds_read() is None                      # reading clears the record
# 2. MoE combine: a routed row beyond the stated row count (but inside the buffer)
T, k, d = 8, 2, 64
y = torch.randn(256, d, device="cuda").bfloat16()
row_of = torch.arange(T * k, dtype=torch.int32, device="cuda")
row_of[5] = 200
gates = torch.ones(T, k, device="cuda")
out = torch.empty(T, d, device="cuda", dtype=torch.bfloat16)
call("pb_moe_combine", ptr(y), ptr(row_of), ptr(gates), None, T, k, d, ptr(out), 128, stream_ptr())
rec = _lib.debug_bounds_read()
assert rec["file"] == "moe" and rec["kernel"] == 3 and rec["index"] == 200 and rec["limit"] == 128, rec
want = y[4].float()                                          # token 2 = rows 4 and (skipped) 200
assert torch.allclose(out[2].float(), want, atol=1e-2)
# the checked library computes the same results as the normal one on valid inputs
x = torch.randn(64, 256, device="cuda").bfloat16(); w = torch.ones(256, device="cuda")
assert torch.isfinite(ops.rmsnorm(x, w).float()).all()
print("DEBUG_BOUNDS_OK")
'''
    root = Path(__file__).resolve().parent.parent
    env = dict(os.environ, PB200_DEBUG_BOUNDS="1", PYTHONPATH=str(root))
    res = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300,
                         cwd=root)
    assert res.returncode == 0 and "DEBUG_BOUNDS_OK" in res.stdout, (res.stdout + res.stderr)[-3000:]
