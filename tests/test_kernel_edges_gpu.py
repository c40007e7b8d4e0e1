"""The attention, router and row kernels at the sizes where their tiling can go wrong: remainders of tiles, the smallest
and largest of their ranges, both sides of every rule that picks a variant."""
import pytest
import torch
import torch.nn.functional as F

from uttt_b200 import ops
from uttt_b200.ops import functional
from uttt_b200.ops import reference as ref
from uttt_b200.ops._ext import load

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _status_ok():
    st = load(required=True).gemm_status(torch.zeros(1, device=DEV))
    assert int(st[0].item()) == 0, f"a tensor-core kernel reported a timed-out wait (code {int(st[0])})"


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30))


# One query; one tile less and more than a row block; a window that starts inside a tile, of one key, and wider than the
# keys; history that ends inside a tile; query blocks of one and of two tiles (few and many heads); unmasked with
# remainders; a negative and a zero scale.
@pytest.mark.parametrize("b,h,lq,lk,hd,window,causal,scale", [
    (1, 2, 1, 1, 64, None, True, None), (1, 3, 1, 700, 64, 256, True, None), (2, 3, 127, 127, 96, None, True, None),
    (1, 2, 129, 300, 128, 64, True, None), (1, 2, 260, 260, 64, 1, True, None), (2, 40, 300, 777, 96, 513, True, None),
    (2, 45, 256, 256, 64, 2048, True, None), (3, 30, 257, 257, 128, None, False, None), (1, 2, 100, 640, 64, None, False, None),
    (1, 2, 200, 333, 64, 128, True, -0.2), (1, 2, 200, 333, 64, 128, True, 0.0)])
def test_attention_tile_edges(b, h, lq, lk, hd, window, causal, scale):
    load(required=True)
    gen = torch.Generator(device=DEV).manual_seed(lq + lk)
    q, do = (torch.randn(b, lq, h, hd, generator=gen, device=DEV).bfloat16() for _ in range(2))
    k, v = (torch.randn(b, lk, h, hd, generator=gen, device=DEV).bfloat16() for _ in range(2))
    leaves = [t.requires_grad_() for t in (q, k, v)]
    out = ops.swa_attention(*leaves, window, causal=causal, scale=scale)
    grads = torch.autograd.grad(out, leaves, do)
    torch.cuda.synchronize()
    _status_ok()
    exact = [t.detach().double().requires_grad_() for t in leaves]
    s = torch.einsum("bqhd,bkhd->bhqk", exact[0], exact[1]) * (hd ** -0.5 if scale is None else scale)
    if causal:
        qp, kp = torch.arange(lk - lq, lk, device=DEV)[:, None], torch.arange(lk, device=DEV)[None]
        s = s.masked_fill((kp > qp) | (kp <= qp - (window or lk + 1)), float("-inf"))
    want = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s, -1), exact[2])
    want_grads = torch.autograd.grad(want, exact, do.double())
    # bf16 results and bf16 probabilities / dS between the products: 2^-9 relative each, a few of them in a row
    for name, got, ref_ in zip(("out", "dq", "dk", "dv"), (out, *grads), (want, *want_grads)):
        if float(ref_.abs().max()) < 1e-9:                       # a single visible key: dS is zero but for rounding of D
            assert float(got.float().abs().max()) < 2e-2, name
        else:
            assert _rel(got, ref_) < 1e-2, (name, _rel(got, ref_))


# 364 keys, the queries on the last 300: query tile 0 sees keys 0..191 (from 1 with the window), key 200 is seen by query 136 on;
# query 10 sees keys 11..74, so the keys from 128 on see nothing of it.
@pytest.mark.parametrize("hd", [64, 96, 128])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("window,causal", [(64, True), (None, True)])
def test_attention_masked_values_that_are_not_finite(hd, value, window, causal):
    """A NaN or an infinity stays in the tiles that see it: the products skip the masked groups of 16."""
    load(required=True)
    gen = torch.Generator(device=DEV).manual_seed(hd)
    base = [torch.randn(1, n, 2, hd, generator=gen, device=DEV).bfloat16() for n in (300, 364, 364, 300)]      # q, k, v, do

    def run(which, row):
        t = [x.clone() for x in base]
        if which is not None:
            t[which][:, row] = value
        leaves = [x.requires_grad_() for x in t[:3]]
        out = ops.swa_attention(*leaves, window, causal=causal)
        res = [out.detach(), *torch.autograd.grad(out, leaves, t[3])]
        torch.cuda.synchronize()
        _status_ok()
        return res

    clean = run(None, 0)
    for which in (1, 2):                                         # a key, a value: what its queries' tile does not reach
        got = run(which, 200)
        for i in (0, 1):
            assert bool(got[i][:, :128].isfinite().all())
            assert _rel(got[i][:, :128], clean[i][:, :128]) < 1e-3       # dQ adds in any order before it is rounded to bf16
            assert not bool(got[i][:, 199].isfinite().all())             # and the queries that see it are told
    if window is not None:
        for which in (0, 3):                                     # a query, a gradient
            got = run(which, 10)
            for i in (2, 3):
                assert torch.equal(got[i][:, 128:], clean[i][:, 128:])
                assert not bool(got[i][:, 74].isfinite().all())


# Windows shorter and longer than a tile, bands that end at the last launch's tiles, no window, no mask.
@pytest.mark.parametrize("lq,lk,window,causal", [(1100, 2100, 1, True), (1100, 2100, 300, True), (1280, 1280, 131, True),
                                                 (1100, 2100, None, True), (700, 900, None, False), (100, 100, 64, True)])
def test_attention_gradients_repeat_bit_for_bit_when_asked(lq, lk, window, causal):
    """torch.use_deterministic_algorithms gives the sums of dQ an order; the values stay what they are without it."""
    load(required=True)
    gen = torch.Generator(device=DEV).manual_seed(lq)
    q, k, v, do = (torch.randn(2, n, 8, 64, generator=gen, device=DEV).bfloat16() for n in (lq, lk, lk, lq))
    leaves = [t.requires_grad_() for t in (q, k, v)]
    out = ops.swa_attention(*leaves, window, causal=causal)
    grads = lambda: torch.autograd.grad(out, leaves, do, retain_graph=True)
    plain = grads()
    torch.use_deterministic_algorithms(True, warn_only=True)
    try:
        first = grads()
        for _ in range(6):
            assert all(torch.equal(x, y) for x, y in zip(grads(), first))
    finally:
        torch.use_deterministic_algorithms(False)
    _status_ok()
    assert torch.equal(first[1], plain[1]) and torch.equal(first[2], plain[2])
    # fp32 sums in another order, then rounded to bf16: a few elements move by one unit
    assert _rel(first[0], plain[0]) < 1e-3 or float(plain[0].float().abs().max()) < 2e-2


@pytest.mark.parametrize("bsz,e,r,rows,d", [(1, 1, 256, 128, 128), (3, 2, 384, 384, 128), (2, 3, 512, 256, 384)])
def test_momentum_and_normalisation(bsz, e, r, rows, d):
    """Values and gradients against the two separate operations, with each output used alone and both together."""
    load(required=True)
    gen = torch.Generator(device=DEV).manual_seed(r + d)
    a, z = (torch.randn(bsz, e, r, d, generator=gen, device=DEV) for _ in range(2))
    m = torch.rand(bsz, 1, 1, 1, generator=gen, device=DEV)
    gz, gd = torch.randn(a.shape, generator=gen, device=DEV), torch.randn(a.shape, generator=gen, device=DEV).bfloat16()
    for use_z, use_d in ((True, True), (True, False), (False, True)):
        res = []
        for fused in (True, False):
            t = [x.clone().requires_grad_() for x in (a, z, m)]
            if fused:
                zn, dd = ops.momentum_newton_schulz(*t, rows)
            else:
                zn = torch.addcmul(t[0], t[1], t[2])
                dd = ops.newton_schulz(zn.reshape(-1, rows, d)).reshape(a.shape)
            outs, cots = zip(*([(zn, gz)] * use_z + [(dd, gd)] * use_d))
            res.append((zn.detach(), dd.detach(), *torch.autograd.grad(outs, t, cots)))
        assert _rel(res[0][0], res[1][0]) < 1e-6
        # the orthogonalisation passes the order of the norms' sums (1e-7) through five bf16 iterations; without it the
        # gradients are fp32 products and sums
        assert _rel(res[0][1], res[1][1]) < 3e-2
        for x, y in zip(res[0][2:], res[1][2:]):
            assert _rel(x, y) < (3e-2 if use_d else 1e-5)


def _odd(t, offset):
    """The same values as a contiguous view that starts ``offset`` elements into a buffer."""
    view = t.new_empty(t.numel() + offset)[offset:].view(t.shape)
    return view.copy_(t)


# Each output alone and both, gradients that start on and off a 16-byte boundary (the backward of a concatenation hands
# out the latter); expectation from the formulas in 64 bits.
@pytest.mark.parametrize("use_z,use_x", [(True, True), (True, False), (False, True)])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
def test_momentum_gradients_at_any_alignment(use_z, use_x, offset):
    ext = load(required=True)
    gen = torch.Generator(device=DEV).manual_seed(offset)
    bsz, e, r, d, rows = 2, 3, 256, 128, 128
    n = bsz * e * r // rows
    a, z, gz = (torch.randn(bsz, e, r, d, generator=gen, device=DEV) for _ in range(3))
    m, gx = torch.rand(bsz, generator=gen, device=DEV), torch.randn(a.shape, generator=gen, device=DEV).bfloat16()
    z_new, x, sumsq = ext.momentum_normalize_fwd(a, z, m, n, 1e-7)
    da, dz, dm = ext.momentum_normalize_bwd(z_new, z, m, sumsq, _odd(gz, offset) if use_z else None,
                                            _odd(gx, offset) if use_x else None, 1e-7, True, True)
    t = [v.double().requires_grad_() for v in (a, z, m)]
    zn = t[0] + t[2].view(-1, 1, 1, 1) * t[1]
    xn = (zn.view(n, -1) / (zn.view(n, -1).norm(dim=1, keepdim=True) + 1e-7)).view(a.shape)
    outs, cots = zip(*([(zn, gz.double())] * use_z + [(xn, gx.double())] * use_x))
    assert _rel(z_new, zn) < 1e-6 and _rel(sumsq, zn.view(n, -1).pow(2).sum(1)) < 1e-5
    assert _rel(x, xn) < 2 ** -8                                 # bf16
    for got, want in zip((da, dz, dm), torch.autograd.grad(outs, t, cots)):
        assert _rel(got, want) < 1e-5                            # fp32 products and sums of 1e5 of them


def test_momentum_gradients_refuse_other_sizes():
    ext = load(required=True)
    a, m = torch.randn(1, 1, 128, 128, device=DEV), torch.rand(1, device=DEV)
    z_new, _, sumsq = ext.momentum_normalize_fwd(a, a, m, 1, 1e-7)
    for bad in ((a[:, :, :64], None), (None, a[:, :, :64].bfloat16())):
        with pytest.raises(RuntimeError):
            ext.momentum_normalize_bwd(z_new, a, m, sumsq, *bad, 1e-7, True, True)
    with pytest.raises(RuntimeError):
        ext.momentum_normalize_bwd(z_new, a[:, :, :64], m, sumsq, a, None, 1e-7, True, True)


def test_momentum_gradients_repeat_bit_for_bit():
    load(required=True)
    gen = torch.Generator(device=DEV).manual_seed(4)
    t = [torch.randn(2, 4, 768, 384, generator=gen, device=DEV).requires_grad_() for _ in range(2)]
    t.append(torch.rand(2, 1, 1, 1, generator=gen, device=DEV).requires_grad_())
    z_new, _ = ops.momentum_newton_schulz(*t, 384)
    g = torch.randn(z_new.shape, generator=gen, device=DEV)
    first = torch.autograd.grad(z_new, t, g, retain_graph=True)
    for _ in range(8):
        assert all(torch.equal(x, y) for x, y in zip(torch.autograd.grad(z_new, t, g, retain_graph=True), first))


def test_momentum_gradient_through_a_concatenation():
    load(required=True)
    gen = torch.Generator(device=DEV).manual_seed(9)
    a, z = (torch.randn(1, 2, 256, 128, generator=gen, device=DEV).requires_grad_() for _ in range(2))
    m, w = torch.rand(1, 1, 1, 1, generator=gen, device=DEV), torch.randn(1 + a.numel(), generator=gen, device=DEV)
    z_new, _ = ops.momentum_newton_schulz(a, z, m, 256)
    da, dz = torch.autograd.grad((torch.cat([a.new_zeros(1), z_new.flatten()]) * w).sum(), (a, z))
    assert torch.equal(da.flatten(), w[1:]) and _rel(dz.flatten(), w[1:].double() * m.double().item()) < 1e-6


@pytest.mark.parametrize("d", [4, 512, 516, 1536, 2048])
@pytest.mark.parametrize("renorm", ["restore", "unit", "none"])
@pytest.mark.parametrize("rows", [1, 3, 700])
def test_pool_step_row_widths(d, renorm, rows):
    """One and four warps to a row."""
    load(required=True)
    gen = torch.Generator(device=DEV).manual_seed(d + rows)
    m, dd, gn = (torch.randn(rows, d, generator=gen, device=DEV) for _ in range(3))
    t = [x.clone().requires_grad_() for x in (m, dd)]
    n, w = ops.pool_step(*t, 0.3, renorm)
    x = [v.double().requires_grad_() for v in (m, dd)]
    u = x[0] + x[1] * 0.3
    want = {"restore": lambda: u / (u.norm(dim=-1, keepdim=True) + 1e-5) * x[0].norm(dim=-1, keepdim=True),
            "unit": lambda: F.normalize(u, dim=-1), "none": lambda: u}[renorm]()
    assert _rel(n, want) < 1e-6 and torch.equal(w, n.bfloat16())
    for a, b in zip(torch.autograd.grad(n, t, gn), torch.autograd.grad(want, x, gn.double())):
        assert _rel(a, b) < 1e-5


# Rows of 1 to 33 and more 16-byte vectors: every lane-group width and the remainders on both sides, row counts that leave
# groups of the last warp without a row.
@pytest.mark.parametrize("d", [8, 32, 40, 64, 72, 128, 136, 192, 256, 264, 384])
@pytest.mark.parametrize("rows", [1, 7, 1001])
def test_row_kernels_lane_groups(d, rows):
    load(required=True)
    gen = torch.Generator(device=DEV).manual_seed(d + rows)
    x, g, delta = (torch.randn(rows, d, generator=gen, device=DEV) for _ in range(3))
    weight, gate = torch.rand(d, generator=gen, device=DEV) + 0.5, torch.rand(rows, generator=gen, device=DEV)
    leaves = [t.clone().requires_grad_() for t in (x, weight, gate, delta)]
    exact = [t.double().requires_grad_() for t in (x, weight, gate, delta)]

    def norm(t, w):
        return t * torch.rsqrt(t.pow(2).mean(-1, keepdim=True) + 1e-5) * w

    y = ops.rms_norm(leaves[0], leaves[1], 1e-5) + ops.rms_norm_gated(leaves[0], leaves[1], leaves[2], 1e-5)
    s, z = ops.add_rms_norm(leaves[0], leaves[3], leaves[1], 1e-5)
    want = norm(exact[0], exact[1]) * (1 + exact[2][:, None])
    ws = exact[0] + exact[3]
    got = torch.autograd.grad([y, s, z], leaves, [g, g, g])
    expect = torch.autograd.grad([want, ws, norm(ws, exact[1])], exact, [g.double()] * 3)
    for a, b in zip((y, s, z, *got), (want, ws, norm(ws, exact[1]), *expect)):
        assert _rel(a, b) < 1e-5                                 # fp32 throughout
    # scatter into the padded layout and back
    plan = ops.build_group_plan(torch.randint(0, 3, (1, rows, 2), generator=gen, device=DEV), 3)
    wts = torch.rand(rows, 2, generator=gen, device=DEV).requires_grad_()
    xp = ops.permute_rows(leaves[0], plan)
    back = ops.unpermute_rows(xp, plan, wts)
    dx, dw = torch.autograd.grad(back, [leaves[0], wts], g)
    total = wts.detach().sum(1, keepdim=True)
    assert _rel(back, x * total) < 1e-6 and _rel(dx, g * total) < 1e-6
    assert _rel(dw, (x * g).sum(1, keepdim=True).expand(-1, 2)) < 1e-4


@pytest.mark.parametrize("heads,head,rope", [(8, 16, 0), (3, 64, 0), (8, 64, 32), (2, 192, 64), (4, 192, 192), (1, 512, 0), (1, 1024, 128)])
@pytest.mark.parametrize("rows", [1, 37])
def test_qk_prep_lane_groups(heads, head, rope, rows):
    load(required=True)
    gen = torch.Generator(device=DEV).manual_seed(heads * head + rows)
    x, g = (torch.randn(2, rows, heads * head, generator=gen, device=DEV) for _ in range(2))
    scale, shift = torch.rand(heads * head, generator=gen, device=DEV) + 0.5, torch.randn(heads * head, generator=gen, device=DEV) * 0.1
    for affine in (True, False):
        mine = [t.clone().requires_grad_() for t in (x, scale, shift)]
        theirs = [t.clone().requires_grad_() for t in (x, scale, shift)]
        run = [(fn(t[0], t[1] if affine else None, t[2] if affine else None, heads, rope, 1e4, 5, True, "l2"), t)
               for fn, t in ((ops.fw_qk_prep, mine), (ref.fw_qk_prep, theirs))]
        assert _rel(run[0][0], run[1][0]) < 1e-5
        grads = [torch.autograd.grad(y, t if affine else t[:1], g) for y, t in run]
        for a, b in zip(*grads):
            assert _rel(a, b) < 1e-4                             # sums over all rows, fast exponentials


@pytest.mark.parametrize("bsz,n,e,k", [(1, 1, 1, 1), (5, 300, 256, 2), (2, 9000, 64, 1), (1, 20000, 16, 2)])
def test_group_plan_scan(bsz, n, e, k):
    """More groups than the scan's block has threads, and more blocks of entries than it fetches at a time."""
    load(required=True)
    idx = torch.randint(0, e, (bsz, n, k), generator=torch.Generator().manual_seed(n)).to(DEV)
    plan = ops.build_group_plan(idx, e)
    dest, offsets, sizes, tile_group, rows = ref.build_group_plan(idx, e)
    for a, b in ((plan.dest, dest), (plan.offsets, offsets), (plan.sizes, sizes), (plan.tile_group, tile_group)):
        assert torch.equal(a.cpu().long(), b.cpu().long())
    assert plan.rows_padded == rows


# Expert counts of every accumulator width, one slab and several, the largest pair that fits and one that does not
# (general kernel), fewer rows than a tile, sequences that end inside a tile.
@pytest.mark.parametrize("e,d", [(16, 64), (16, 512), (32, 192), (48, 384), (48, 512), (64, 64), (64, 192), (64, 512), (24, 128)])
@pytest.mark.parametrize("kind", ["softmax", "norm_softmax", "norm_relu"])
@pytest.mark.parametrize("bsz,n,topk", [(1, 5, 1), (3, 1003, 4)])
def test_router_matches_double_precision(e, d, kind, bsz, n, topk):
    load(required=True)
    gen = torch.Generator(device=DEV).manual_seed(e + d + n)
    rows = torch.randn(bsz, n, d, generator=gen, device=DEV).bfloat16()
    router = torch.randn(e, d, generator=gen, device=DEV) * d ** -0.5
    bias = torch.randn(e, generator=gen, device=DEV) * 0.02
    idx, w, psum = ops.route_topk(rows, router, bias, topk, 0.7, False, False, kind, 0.0, 1e-6)
    _status_ok()
    sel, probs = ref.route_scores(rows.double() @ router.double().t(), kind, 0.0, 1e-6)
    score = sel + bias.double()
    top = torch.topk(score, topk + 1, dim=-1).values
    gap = 1e-4                                                   # fp32 sums of d products of size one
    clear = top[..., topk - 1] - top[..., topk] > gap
    chosen = torch.zeros(bsz, n, e, device=DEV, dtype=torch.bool).scatter_(2, idx.long(), True)
    assert bool((chosen.sum(-1) == topk).all())
    assert bool(((score >= top[..., topk - 1:topk] - gap) | ~chosen).all())
    assert bool((chosen == (score >= top[..., topk - 1:topk]))[clear].all())
    # fp32 logits: d 2^-24 of their size at most; __expf adds 2^-21 of its argument
    torch.testing.assert_close(w.view(bsz, n, topk).double(), probs.gather(-1, idx.long()) * 0.7, atol=2e-6, rtol=1e-4)
    torch.testing.assert_close(psum.double(), probs.sum(1), atol=1e-4, rtol=1e-4)


# One accumulator for all slabs is 1.1e-6 off at 384 columns and a router in two bf16 parts (16 of its 24 bits) 2.4e-6; the
# three parts with an accumulator per slab stay near 1e-7.  The general kernel, which takes 24 experts, adds D products in
# fp32 one after the other: 4e-7 at 512.
@pytest.mark.parametrize("e,d", [(16, 64), (16, 512), (32, 192), (32, 384), (48, 256), (64, 64), (64, 256), (24, 512)])
@pytest.mark.parametrize("with_bias", [False, True])
def test_router_logits_are_fp32(e, d, with_bias):
    ext = load(required=True)
    gen = torch.Generator(device=DEV).manual_seed(e * d)
    rows = torch.randn(1000, d, generator=gen, device=DEV).bfloat16()
    router = torch.randn(e, d, generator=gen, device=DEV) * d ** -0.5
    bias = torch.randn(e, generator=gen, device=DEV) * 0.1 if with_bias else None
    want = rows.double() @ router.double().t() + (bias.double() if with_bias else 0.0)
    for mode in (1, 2):                                          # the modes that hand out the raw logits
        logits = ext.router_fwd(rows, router, bias, 2, 1000, 1.0, True, False, mode, 4.0, 1e-6)[4]
        assert _rel(logits, want) < (3e-7 if e % 16 == 0 else 1e-6)
    _status_ok()


# Both variants, both row types; a router off a 16-byte boundary goes to the general kernel.
@pytest.mark.parametrize("e,d,dtype", [(16, 64, torch.bfloat16), (24, 128, torch.bfloat16), (16, 64, torch.float32)])
@pytest.mark.parametrize("rows_off,router_off", [(1, 0), (0, 1), (3, 2)])
def test_router_operands_at_any_alignment(e, d, dtype, rows_off, router_off):
    load(required=True)
    gen = torch.Generator(device=DEV).manual_seed(e + d)
    rows = torch.randn(2, 300, d, generator=gen, device=DEV).to(dtype)
    router = torch.randn(e, d, generator=gen, device=DEV) * d ** -0.5
    gw = torch.randn(600, 2, generator=gen, device=DEV)
    res = []
    for r, w in ((rows, router), (_odd(rows, rows_off), _odd(router, router_off))):
        leaves = [r.requires_grad_(), w.requires_grad_()]
        idx, wts, psum = ops.route_topk(*leaves, None, 2)
        res.append((wts.detach(), psum.detach(), *torch.autograd.grad(wts, leaves, gw)))
    _status_ok()
    for got, want in zip(res[1], res[0]):
        assert _rel(got, want) < (1e-5 if got.dtype == torch.float32 else 2 ** -8)


def _alignment_cases(gen):
    """name -> (function of the leaves, leaves): every op whose kernel moves 16 bytes at a time."""
    rnd = lambda *shape: torch.randn(*shape, generator=gen, device=DEV)
    plan = ops.build_group_plan(torch.randint(0, 3, (1, 37, 2), generator=gen, device=DEV), 3)
    rows, ids = plan.rows_padded, torch.randint(0, 50, (2, 9), generator=gen, device=DEV)
    weight = rnd(37, 2).abs()
    return {
        "rms_norm": (lambda x, w: ops.rms_norm(x, w), (rnd(37, 64), rnd(64))),
        "rms_norm_gated": (lambda x, w, g: ops.rms_norm_gated(x, w, g), (rnd(37, 64), rnd(64), rnd(37))),
        "add_rms_norm": (lambda x, y, w: torch.cat(ops.add_rms_norm(x, y, w)), (rnd(37, 64), rnd(37, 64), rnd(64))),
        "rope": (lambda x: ops.rope(x, 3, 1e4), (rnd(2, 9, 2, 32),)),
        "fw_qk_prep": (lambda x, a, b: ops.fw_qk_prep(x, a, b, 2, 32, 1e4, 5, True, "l2"), (rnd(2, 9, 64), rnd(64), rnd(64))),
        "swiglu": (lambda y: ops.swiglu(y), (rnd(37, 64),)),
        "fw_write_pointwise": (lambda y, d, r: torch.cat(functional.fw_write_pointwise(y, d, r), 1), (rnd(37, 64), rnd(37, 32), rnd(37, 3))),
        "permute": (lambda x: ops.permute_rows(x, plan)[plan.dest.flatten()], (rnd(37, 64),)),
        # (its gradient is defined for the rows that hold a copy)
        "unpermute": (lambda y: ops.unpermute_rows(y, plan, weight), (rnd(rows, 64),), plan.dest.flatten()),
        "embedding": (lambda t: ops.embedding(ids, t), (rnd(50, 64),)),
        "pool_step": (lambda m, d: ops.pool_step(m, d, 0.3)[0], (rnd(37, 64), rnd(37, 64))),
        "normalise": (lambda g: functional._FrobNormalize.apply(g, 1e-7), (rnd(2, 8, 16),)),
    }


@pytest.mark.parametrize("name", [
    "rms_norm", "rms_norm_gated", "add_rms_norm", "rope", "fw_qk_prep", "swiglu", "fw_write_pointwise", "permute",
    "unpermute", "embedding", "pool_step", "normalise"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_operands_at_any_alignment(name, dtype):
    """Values and gradients do not depend on where a contiguous operand or gradient starts."""
    load(required=True)
    gen = torch.Generator(device=DEV).manual_seed(7)
    fn, leaves, *defined = _alignment_cases(gen)[name]
    if name != "pool_step":                                      # fp32 masters only
        leaves = [t.to(dtype) for t in leaves]
    res, gout = [], None
    for offset in (0, 1, 3):
        t = [_odd(x, offset).requires_grad_() for x in leaves]
        out = fn(*t)
        gout = torch.randn(out.shape, generator=gen, device=DEV).to(out.dtype) if gout is None else gout
        grads = torch.autograd.grad(out, t, _odd(gout, offset))
        res.append((out.detach(), *(g[defined[0]] if defined else g for g in grads)))
    torch.cuda.synchronize()
    for other in res[1:]:
        for a, b in zip(other, res[0]):
            assert _rel(a, b) < 1e-6 or torch.equal(a, b)        # the sums over rows may be added in another order
