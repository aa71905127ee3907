"""Mixture-of-experts kernels and the grouped GEMMs against fp32 PyTorch (needs a B200)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def _r(*shape, seed=0, scale=1.0, dtype=BF16):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(dtype)


def _close(got, ref, tol):
    got, ref = got.float(), ref.float()
    err = (got - ref).abs().max().item()
    scale = ref.abs().max().item() + 1e-6
    assert err <= tol * scale, f"max err {err:.4g} vs scale {scale:.4g}"


@pytest.mark.parametrize("T,E,k", [(7, 8, 2), (1000, 64, 6), (300, 40, 3)])
def test_route_and_placement(T, E, k):
    from prometheus_b200.ops import moe

    logits = _r(T, E, seed=1, dtype=torch.float32)
    logits[:, 3] = logits[:, 5]                      # ties break toward the lower index
    bias = _r(E, seed=2, scale=0.1, dtype=torch.float32)
    probs, ids, gates = moe.route(logits, bias, k)
    p_ref = torch.sigmoid(logits)
    ids_ref = torch.argsort(-(p_ref + bias), dim=-1, stable=True)[:, :k]
    assert torch.equal(ids.long(), ids_ref)
    top = torch.gather(p_ref, 1, ids_ref)
    torch.testing.assert_close(probs, p_ref, rtol=1e-5, atol=1e-6)
    torch.testing.assert_close(gates, top / top.sum(-1, keepdim=True), rtol=1e-5, atol=1e-6)
    pl = moe.place(ids, E)
    torch.cuda.synchronize()
    flat = ids.reshape(-1).long().cpu()
    counts = torch.bincount(flat, minlength=E)
    assert torch.equal(pl.totals.cpu().long(), counts)
    off = pl.expert_off.cpu().long()
    assert (off % 128 == 0).all() and off[0] == 0
    assert torch.equal(off[1:] - off[:-1], (counts + 127) // 128 * 128)
    rows = pl.row_of.cpu().long()
    assert rows.unique().numel() == rows.numel()
    for e in range(E):
        mine = rows[flat == e]
        assert torch.equal(mine, off[e] + torch.arange(mine.numel()))   # stable, dense
    mg = pl.mblk_group.cpu().long()
    used = int(off[-1]) // 128
    assert (mg[used:] == -1).all()
    for m in range(used):
        assert off[mg[m]] <= m * 128 < off[mg[m] + 1]


@pytest.mark.parametrize("d,E", [(2048, 64), (1024, 8), (2056, 160), (1024, 512)])
def test_a_token_chooses_its_experts_whatever_the_call_holds_beside_it(d, E):
    """Router logits of the first rows alone and among 8192, bit for bit: 1 to 256 tiles, contractions that an ordinary product
    shares out between 8, 2 or no CTAs, and the last of them on CTA pairs."""
    from prometheus_b200.ops import functional as ops

    x, w = _r(8192, d, seed=1), _r(E, d, seed=2, scale=d ** -0.5)
    full = ops.router_logits(x, w)
    _close(full, x.float() @ w.float().t(), 1e-4)
    for n in (1, 100, 512, 2500, 4736):
        assert torch.equal(ops.router_logits(x[:n], w), full[:n]), n
    wide = torch.zeros(100, d + 5, dtype=BF16, device="cuda")        # rows that do not start on 16 bytes
    wide[:, 3:3 + d] = x[:100]
    assert torch.equal(ops.router_logits(wide[:, 3:3 + d], w), full[:100])
    ops.check_status("cuda")


@pytest.mark.parametrize("T,E,k,skew", [(683, 64, 6, 0), (4097, 512, 1, 0), (64 * 9 + 1, 300, 8, 0), (8200, 5, 3, 0), (4160, 64, 1, 1)])
def test_placement_over_many_blocks(T, E, k, skew):
    """The three-kernel sort: one pair more than the one-block sort takes, a thread or several to an expert in the scan, shares of
    blocks that do not divide, a last block of one token, and all pairs on one expert. Rows are those of a stable sort."""
    from prometheus_b200.ops import moe

    ids = torch.randint(0, 1 if skew else E, (T, k), generator=torch.Generator().manual_seed(T), dtype=torch.int32)
    pl = moe.place(ids.cuda(), E)
    flat = ids.reshape(-1).long()
    counts = torch.bincount(flat, minlength=E)
    off = torch.cat([torch.zeros(1, dtype=torch.long), ((counts + 127) // 128 * 128).cumsum(0)])
    order = torch.argsort(flat, stable=True)
    want = torch.empty_like(flat)
    want[order] = torch.arange(flat.numel()) - (counts.cumsum(0) - counts)[flat[order]] + off[flat[order]]
    assert torch.equal(pl.row_of.cpu().long(), want)
    assert torch.equal(pl.expert_off.cpu().long(), off) and torch.equal(pl.totals.cpu().long(), counts)


def test_grouped_gemms_match_per_expert_products():
    from prometheus_b200.ops import functional as ops
    from prometheus_b200.ops import moe

    T, E, k, K, N = 700, 6, 2, 256, 320
    ids = torch.randint(0, E, (T, k), device="cuda", dtype=torch.int32)
    ids[:, 1] = (ids[:, 0] + 1 + torch.randint(0, E - 1, (T,), device="cuda", dtype=torch.int32)) % E
    ids[ids == 4] = 2                                  # expert 4 gets nothing
    ids[:, 1] = torch.where(ids[:, 1] == ids[:, 0], (ids[:, 0] + 1) % E, ids[:, 1])
    ids[ids == 4] = 5
    pl = moe.place(ids.contiguous(), E)
    x = _r(T, K, seed=1)
    xp = moe.permute(x, pl)
    w = _r(E, N, K, seed=2, scale=0.1)
    y = moe.grouped_gemm(xp, w, pl)
    wt = w.transpose(1, 2).contiguous()
    y2 = moe.grouped_gemm(xp, wt, pl, b_mn=True)
    g = _r(pl.rows, N, seed=3)
    acc = torch.full((E, N, K), 0.5, dtype=torch.float32, device="cuda")
    off, tot = pl.expert_off.cpu().tolist(), pl.totals.cpu().tolist()
    for e in range(E):                                 # zero the padding rows of g
        g[off[e] + tot[e]:off[e + 1]] = 0
    moe.grouped_wgrad(g, xp, pl, acc, True)
    torch.cuda.synchronize()
    ops.check_status("cuda")
    for e in range(E):
        seg = slice(off[e], off[e] + tot[e])
        ref = xp[seg].float() @ w[e].float().t()
        if tot[e]:
            _close(y[seg], ref, 2e-2)
            _close(y2[seg], ref, 2e-2)
        assert (xp[off[e] + tot[e]:off[e + 1]] == 0).all()
        _close(acc[e], 0.5 + g[seg].float().t() @ xp[seg].float(), 2e-2)
    assert tot[4] == 0


@pytest.mark.parametrize("T,k,E", [(1, 1, 1), (33, 1, 3), (512, 2, 8), (1024, 4, 64), (1366, 3, 512), (2048, 2, 5)])
def test_placement_one_and_three_kernels(T, k, E):
    """Rows of the pairs grouped by expert against a stable sort, on both sides of the size up to which one
    kernel does it."""
    from prometheus_b200.ops import moe

    g = torch.Generator(device="cuda").manual_seed(T)
    ids = torch.randint(0, E, (T, k), generator=g, device="cuda", dtype=torch.int32)
    if E > 3:
        ids[ids == 2] = 0                                    # an empty expert
    pl = moe.place(ids, E)
    flat = ids.reshape(-1).long()
    tot = torch.bincount(flat, minlength=E)
    off = torch.cat([torch.zeros(1, dtype=torch.long, device="cuda"), ((tot + 127) // 128 * 128).cumsum(0)])
    order = torch.argsort(flat, stable=True)
    start = tot.cumsum(0) - tot
    row = torch.empty_like(flat)
    row[order] = off[flat[order]] + torch.arange(T * k, device="cuda") - start[flat[order]]
    assert torch.equal(pl.row_of.long(), row)
    assert torch.equal(pl.expert_off.long(), off) and torch.equal(pl.totals.long(), tot)
    assert torch.equal(pl.k_len.long(), off[1:] - off[:-1])
    blocks = torch.arange(pl.rows // 128, device="cuda") * 128
    want = torch.where(blocks < off[-1], torch.searchsorted(off[:-1].contiguous(), blocks, right=True) - 1, -1)
    got = pl.mblk_group.long()
    used = blocks < off[-1]
    # empty experts share their start with the next one: any expert with rows there is the last of them
    assert torch.equal(got[~used], want[~used]) and torch.equal(got[used], want[used])


@pytest.mark.parametrize("T,k,E,d", [(1, 1, 1, 128), (300, 2, 5, 384), (130, 7, 16, 2176)])
def test_token_movement_kernels(T, k, E, d):
    """Permute (plain, scaled, quantised) and combine (gated, summed, with an addend) against index
    arithmetic in fp32, at column counts that leave remainders of their steps and with empty experts."""
    from prometheus_b200.ops import fp8, moe

    g = torch.Generator(device="cuda").manual_seed(T)
    ids = torch.stack([torch.randperm(E, generator=g, device="cuda")[:k] for _ in range(T)]).to(torch.int32).contiguous()
    if E > 4:
        ids[ids == 3] = 0                                    # expert 3 gets nothing
    pl = moe.place(ids, E)
    row = pl.row_of.view(T, k).long()
    x = _r(T, d, seed=1)
    sc = _r(T * k, seed=2, dtype=torch.float32)
    want = torch.zeros(pl.rows, d, device="cuda")
    want[row] = x.float()[:, None].expand(T, k, d)
    end = int(pl.expert_off[-1])
    xp = moe.permute(x, pl)
    assert torch.equal(xp[:end].float(), want[:end])
    scaled = moe.permute(x, pl, scale=sc)
    assert torch.equal(scaled[row], (x.float()[:, None] * sc.view(T, k, 1)).to(BF16))
    q, s = moe.permute_quantized(x, pl)
    q2, s2 = fp8.quantize_rows(xp)
    assert torch.equal(q[:end], q2[:end]) and torch.equal(s[:, :end], s2[:, :end])
    y = _r(pl.rows, d, seed=3)
    gates, add = torch.rand(T, k, device="cuda"), _r(T, d, seed=4)
    ref = (gates[..., None] * y.float()[row]).sum(1)
    _close(moe.combine(y, pl, gates, T), ref, 1e-2)
    _close(moe.combine(y, pl, None, T, add=add), y.float()[row].sum(1) + add.float(), 1e-2)


@pytest.mark.parametrize("M,N", [(128, 320), (256, 256), (384, 264), (640, 520)])
@pytest.mark.parametrize("dtype", [BF16, torch.float32])
def test_grouped_wgrad_single_and_pair_kernels(M, N, dtype):
    """Grouped weight gradient with an empty first, middle and last group and tile remainders in M and
    N, with and without accumulation, on the CTA-pair kernel and on the single-CTA one."""
    from prometheus_b200.ops import moe
    from prometheus_b200.ops._lib import call

    E, T = 5, 500
    ids = (1 + 2 * torch.randint(0, 2, (T, 1), device="cuda", dtype=torch.int32)).contiguous()   # groups 1 and 3
    pl = moe.place(ids, E)
    a, b = moe.permute(_r(T, M, seed=1), pl), moe.permute(_r(T, N, seed=2), pl)
    off, tot = pl.expert_off.cpu().tolist(), pl.totals.cpu().tolist()
    for variant in (0, 8):
        try:
            call("pb_gemm_set_variant", variant)
            fresh = moe.grouped_wgrad(a, b, pl, torch.full((E, M, N), float("nan"), dtype=dtype, device="cuda"), False)
            acc = moe.grouped_wgrad(a, b, pl, torch.full((E, M, N), 0.5, dtype=dtype, device="cuda"), True)
        finally:
            call("pb_gemm_set_variant", 0)
        for e in range(E):
            seg = slice(off[e], off[e] + tot[e])
            ref = a[seg].float().t() @ b[seg].float()
            if tot[e]:
                _close(fresh[e], ref, 2e-2)
                _close(acc[e], 0.5 + ref, 2e-2)
            else:
                assert (fresh[e] == 0).all() and (acc[e] == 0.5).all()


@pytest.mark.parametrize("n_shared", [0, 2])
def test_moe_ffn_matches_fp32_reference(n_shared):
    from prometheus_b200.ops import functional as ops
    from prometheus_b200.ops import moe

    T, d, E, h, k = 500, 256, 8, 192, 2
    x = _r(T, d, seed=1).requires_grad_(True)
    rw = _r(E, d, seed=2, scale=0.2).requires_grad_(True)
    bias = _r(E, seed=3, scale=0.05, dtype=torch.float32)
    wgu = _r(E + n_shared, 2 * h, d, seed=4, scale=0.08).requires_grad_(True)
    wd = _r(E + n_shared, d, h, seed=5, scale=0.08).requires_grad_(True)
    go = _r(T, d, seed=6)
    out, probs, ids = moe.moe_ffn(x, rw, bias, wgu, wd, k, n_shared=n_shared)
    zw = 0.3
    ((out.float() * go.float()).sum() + zw * torch.logsumexp(probs, -1).square().mean()).backward()
    torch.cuda.synchronize()
    ops.check_status("cuda")
    leaves = [t.detach().float().requires_grad_(True) for t in (x, rw, wgu, wd)]
    o_ref, p_ref, i_ref = moe.moe_ffn_ref(leaves[0], leaves[1], bias, leaves[2], leaves[3], k,
                                          n_shared=n_shared)
    ((o_ref * go.float()).sum() + zw * torch.logsumexp(p_ref, -1).square().mean()).backward()
    assert (ids == i_ref).float().mean().item() > 0.995   # bf16 logits may flip near-ties
    _close(out, o_ref, 3e-2)
    _close(probs, p_ref, 1e-2)
    for got, ref in zip((x, rw, wgu, wd), leaves):
        _close(got.grad, ref.grad, 6e-2)
