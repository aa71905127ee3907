"""tcgen05 causal GQA attention (forward, dQ, dK/dV) against the fp32 formula."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

BF16 = torch.bfloat16


def _rand(b, s, hq, hkv, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    q = (torch.randn(b, s, hq, 128, device="cuda", generator=g) * scale).to(BF16)
    k = (torch.randn(b, s, hkv, 128, device="cuda", generator=g) * scale).to(BF16)
    v = torch.randn(b, s, hkv, 128, device="cuda", generator=g).to(BF16)
    return q, k, v


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-20)).item()


@pytest.mark.parametrize("b,s,hq,hkv", [(1, 128, 1, 1), (2, 512, 4, 2), (1, 1024, 16, 4), (1, 320, 2, 1)])
def test_attention_forward_and_backward_match_fp32(b, s, hq, hkv):
    from prometheus_b200.ops import attention

    q, k, v = _rand(b, s, hq, hkv, 1)
    q.requires_grad_(); k.requires_grad_(); v.requires_grad_()
    out, rowmax = attention.causal_gqa(q, k, v, return_max_logit=True)
    go = torch.randn_like(out)
    dq, dk, dv = torch.autograd.grad(out, (q, k, v), go)

    qf, kf, vf = (t.detach().float().requires_grad_() for t in (q, k, v))
    ref = attention.causal_gqa_ref(qf, kf, vf)
    rq, rk, rv = torch.autograd.grad(ref, (qf, kf, vf), go.float())
    assert _rel(out, ref) < 1e-2
    assert _rel(dq, rq) < 2e-2 and _rel(dk, rk) < 2e-2 and _rel(dv, rv) < 2e-2

    kk = kf.detach().transpose(1, 2).repeat_interleave(hq // hkv, dim=1)
    logits = qf.detach().transpose(1, 2) @ kk.transpose(-1, -2) / math.sqrt(128)
    mask = torch.ones(s, s, dtype=torch.bool, device="cuda").tril()
    want_max = logits.masked_fill(~mask, float("-inf")).amax(-1)
    torch.testing.assert_close(rowmax, want_max, atol=2e-3, rtol=1e-3)


def test_attention_large_logits_exercise_the_rescale_path():
    """Scores that keep growing along the keys force the running maximum to be raised
    repeatedly (more than 2^8 between blocks), so the tensor-memory rescale of O runs."""
    from prometheus_b200.ops import attention

    b, s, hq, hkv = 1, 768, 2, 2
    q, k, v = _rand(b, s, hq, hkv, 3)
    ramp = torch.linspace(0.0, 6.0, s, device="cuda").view(1, s, 1, 1)
    k = (k.float() + ramp * q.float().mean(dim=(1,), keepdim=True).sign()).to(BF16)
    q = (q.float() * 3.0).to(BF16)
    out = attention.causal_gqa(q, k, v)
    ref = attention.causal_gqa_ref(q.float(), k.float(), v.float())
    assert torch.isfinite(out.float()).all()
    assert _rel(out, ref) < 1.5e-2


@pytest.mark.parametrize("slow", [1, 2, 4])
def test_rows_that_rescale_in_every_block_beside_rows_that_never_do(slow):
    """``slow`` of the four warps of a tile see scores that grow by 2^12 a block of keys, so they rescale O in each, and the
    others, whose scores stay small, wait for none of it. P is rounded to bf16 once (2^-9 of a value) and so is the result."""
    from prometheus_b200.ops import attention

    s, hq = 2048, 32
    q, k, v = _rand(1, s, hq, 1, 5, 0.5)
    row, head = torch.arange(s, device="cuda"), torch.arange(hq, device="cuda")
    quarter = (row[:, None] // 32 + head) % 4             # which warps are slow differs from head to head
    step = 12 * math.log(2.0) * math.sqrt(128) / 16
    q[0, ..., 0] = torch.where(quarter < slow, 16.0, 0.0).to(BF16)
    k[0, :, 0, 0] = (row // 64 * step).to(BF16)
    out, top = attention.causal_gqa(q, k, v, return_max_logit=True)
    again = attention.causal_gqa(q, k, v)
    ref = attention.causal_gqa_ref(q.float(), k.float(), v.float())
    assert torch.equal(out, again)
    assert (out.float() - ref).abs().max() <= 2.0 ** -7 * v.float().abs().max()
    assert torch.isfinite(top).all()


def test_attention_is_deterministic_and_matches_library_kernel():
    import torch.nn.functional as F

    from prometheus_b200.ops import attention

    q, k, v = _rand(2, 1024, 8, 2, 5)
    q.requires_grad_(); k.requires_grad_(); v.requires_grad_()
    go = torch.randn(2, 1024, 8, 128, device="cuda").to(BF16)
    runs = []
    for _ in range(2):
        o = attention.causal_gqa(q, k, v)
        runs.append((o,) + torch.autograd.grad(o, (q, k, v), go))
    for a, b_ in zip(*runs):
        assert torch.equal(a, b_)
    o2 = F.scaled_dot_product_attention(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2),
                                        is_causal=True, enable_gqa=True).transpose(1, 2)
    g2 = torch.autograd.grad(o2, (q, k, v), go)
    assert _rel(runs[0][0], o2) < 1e-2
    for mine, lib in zip(runs[0][1:], g2):
        assert _rel(mine, lib) < 2e-2


@pytest.mark.parametrize("q_off,s_loc,s_kv", [(512, 256, 1024), (0, 512, 640), (768, 256, 1024)])
def test_offset_attention_equals_a_slice_of_the_full_sequence(q_off, s_loc, s_kv):
    """A query slice at a global offset against the whole prefix (the context-parallel case):
    output and dq of the slice, and dk / dv of every key row (zero where nothing sees it)."""
    from prometheus_b200.ops import attention

    q, k, v = _rand(2, 1024, 4, 2, 11)
    k, v = k[:, :s_kv].contiguous(), v[:, :s_kv].contiguous()
    ql = q[:, q_off:q_off + s_loc].contiguous().requires_grad_()
    kl, vl = k.clone().requires_grad_(), v.clone().requires_grad_()
    out = attention.causal_gqa_offset(ql, kl, vl, q_off)
    go = torch.randn_like(out)
    dq, dk, dv = torch.autograd.grad(out, (ql, kl, vl), go)

    s_all = max(s_kv, q_off + s_loc)
    qf = torch.zeros(2, s_all, 4, 128, device="cuda")
    qf[:, q_off:q_off + s_loc] = q[:, q_off:q_off + s_loc].float()
    qf.requires_grad_()
    kf = torch.zeros(2, s_all, 2, 128, device="cuda"); kf[:, :s_kv] = k.float(); kf.requires_grad_()
    vf = torch.zeros(2, s_all, 2, 128, device="cuda"); vf[:, :s_kv] = v.float(); vf.requires_grad_()
    ref = attention.causal_gqa_ref(qf, kf, vf)
    gof = torch.zeros_like(ref)
    gof[:, q_off:q_off + s_loc] = go.float()
    rq, rk, rv = torch.autograd.grad(ref, (qf, kf, vf), gof)
    assert _rel(out, ref[:, q_off:q_off + s_loc]) < 1e-2
    assert _rel(dq, rq[:, q_off:q_off + s_loc]) < 2e-2
    assert _rel(dk, rk[:, :s_kv]) < 2e-2 and _rel(dv, rv[:, :s_kv]) < 2e-2
    unseen = q_off + s_loc
    if unseen < s_kv:
        assert dk[:, unseen:].abs().max() == 0 and dv[:, unseen:].abs().max() == 0
    with pytest.raises(ValueError):
        attention.causal_gqa_offset(ql, kl, vl, q_off + 128)


@pytest.mark.parametrize("B,S,hq,hkv", [(2, 1, 2, 1), (3, 63, 4, 2), (2, 129, 2, 2), (2, 300, 4, 1), (2, 1000, 4, 2)])
def test_ragged_lengths_equal_explicit_padding(B, S, hq, hkv):
    """A length that is not a multiple of a tile, read in place, gives the bits of the same call on
    tensors padded to whole tiles (batch entries follow one another without a gap, so a row too
    many would be the next entry's), and from a misaligned base."""
    from prometheus_b200.ops import attention
    from prometheus_b200.ops import functional as ops

    g = torch.Generator(device="cuda").manual_seed(S)
    q, go = (torch.randn(B, S, hq, 128, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    k, v = (torch.randn(B, S, hkv, 128, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))

    def run(ts, gout):
        leaves = [t.clone().requires_grad_(True) for t in ts]
        out, top = attention.causal_gqa(*leaves, return_max_logit=True)
        grads = torch.autograd.grad(out, leaves, gout)
        ops.check_status("cuda")
        return [out.detach(), top.transpose(1, 2), *grads]

    def padded(t):
        return torch.nn.functional.pad(t, (0, 0, 0, 0, 0, (-S) % 256))

    got, want = run((q, k, v), go), run([padded(t) for t in (q, k, v)], padded(go))
    for name, a, b in zip(("out", "max", "dq", "dk", "dv"), got, want):
        assert torch.equal(a, b[:, :S]), name
    off = torch.empty(q.numel() + 1, dtype=torch.bfloat16, device="cuda")[1:].view(q.shape).copy_(q)
    assert torch.equal(attention.causal_gqa(off, k, v), got[0])


def test_ds_is_rounded_once_with_the_scale_in_it():
    """dS = P (dP - delta) scale is one bf16 rounding of the scaled value: with 1 / sqrt(128) applied after it,
    a gradient would carry two roundings. Sequences of two tokens in which each gradient is one dS times a power
    of two: the first query has dO = 0 and the first key is zero, so dQ_1 = dS_11 k_1, dK_j = dS_1j q_1."""
    from prometheus_b200.ops import attention

    g = torch.Generator(device="cuda").manual_seed(21)
    b, h = 64, 16
    pw = lambda *s: (torch.randint(0, 2, s, device="cuda", generator=g) * 2 - 1) * 0.5 ** torch.randint(
        0, 2, s, device="cuda", generator=g)
    q, k = pw(b, 2, h, 128).to(BF16), pw(b, 2, h, 128).to(BF16)
    v, go = (torch.randn(b, 2, h, 128, device="cuda", generator=g).to(BF16) for _ in range(2))
    k[:, 0], go[:, 0] = 0, 0
    q.requires_grad_(); k.requires_grad_(); v.requires_grad_()
    out = attention.causal_gqa(q, k, v)
    dq, dk, _ = torch.autograd.grad(out, (q, k, v), go)

    q1, k1, o1, g1, vd = (t.detach().double() for t in (q[:, 1], k[:, 1], out[:, 1], go[:, 1], v))
    p1 = torch.sigmoid((q1 * k1).sum(-1) / math.sqrt(128))
    delta = (g1 * o1).sum(-1)
    ds = [(p * ((g1 * vd[:, j]).sum(-1) - delta) / math.sqrt(128)) for j, p in ((0, 1 - p1), (1, p1))]
    # fp32 arithmetic (a part in 10^6 of dS) moves a value across a bf16 rounding boundary once in some hundreds;
    # a second rounding does so for a fifth of them
    for name, got, want in (("dq", dq[:, 1] / k[:, 1], ds[1]), ("dk0", dk[:, 0] / q[:, 1], ds[0]),
                            ("dk1", dk[:, 1] / q[:, 1], ds[1])):
        assert torch.equal(got, got[..., :1].expand_as(got)), name
        assert (got[..., 0] != want.to(BF16)).float().mean() < 0.02, name


def test_more_row_blocks_than_a_second_grid_dimension_holds():
    """Gradients of 65537 key blocks (the y and z dimensions of a grid end at 65535): a short query slice against
    8.4 M keys of which it sees the first 256."""
    from prometheus_b200.ops import attention
    from prometheus_b200.ops import functional as ops

    s_kv = 65537 * 128
    q, ks, vs = _rand(1, 256, 1, 1, 31)
    k, v = (torch.zeros(1, s_kv, 1, 128, dtype=BF16, device="cuda") for _ in range(2))
    k[:, :256], v[:, :256] = ks, vs
    leaves = [t.requires_grad_() for t in (q, k, v)]
    out = attention.causal_gqa_offset(*leaves, 0)
    go = torch.randn_like(out)
    dq, dk, dv = torch.autograd.grad(out, leaves, go)
    ops.check_status("cuda")
    small = [t.detach().clone().requires_grad_() for t in (q, ks, vs)]
    want_out = attention.causal_gqa(*small)
    want = torch.autograd.grad(want_out, small, go)
    assert torch.equal(out, want_out) and torch.equal(dq, want[0])
    assert torch.equal(dk[:, :256], want[1]) and torch.equal(dv[:, :256], want[2])
    assert not dk[:, 256:].any() and not dv[:, 256:].any()
