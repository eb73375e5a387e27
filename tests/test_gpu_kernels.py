r"""GPU tier: every sm_100a kernel against a plain PyTorch fp32 restatement of the same op."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _native():
    from fastmoe_b200.ops import native
    return native.get()


def _offs(counts):
    o = torch.zeros(len(counts) + 1, dtype=torch.int32)
    o[1:] = torch.cumsum(torch.tensor(counts), 0)
    return o.to(DEV)


def _segments(counts):
    base = 0
    for e, n in enumerate(counts):
        yield e, base, base + n
        base += n


def _tiled(pre, offs, groups):
    r"""Tile-blocked copy of a row-major pre-activation: the inverse of ``gg.untile_pre``."""
    from fastmoe_b200.ops import grouped_gemm as gg
    rows, n = pre.shape
    buf = gg.pre_buffer(rows, n, groups, pre.dtype, pre.device).zero_()
    blocks = buf.view(-1, 2, 4, 4, 4, 32, 8)     # tile, half, part, chunk, piece, lane, v
    o = [int(v) for v in offs.tolist()]
    n_tiles = (n + gg.TILE_N - 1) // gg.TILE_N
    tile = 0
    for e in range(groups):
        for m in range((o[e + 1] - o[e] + gg.TILE_M - 1) // gg.TILE_M):
            for nt in range(n_tiles):
                full = torch.zeros(gg.TILE_M, gg.TILE_N, dtype=pre.dtype, device=pre.device)
                r0, c0 = o[e] + m * gg.TILE_M, nt * gg.TILE_N
                nr, nc = min(gg.TILE_M, o[e + 1] - r0), min(gg.TILE_N, n - c0)
                full[:nr, :nc] = pre[r0:r0 + nr, c0:c0 + nc]
                blocks[tile] = full.view(4, 32, 2, 4, 4, 8).permute(2, 0, 3, 4, 1, 5)
                tile += 1
    return buf


def _tol(dtype, k):
    # bf16 has 8 bits of mantissa: inputs are exact in fp32, the only error is the output rounding.
    return (2e-2 if dtype == torch.bfloat16 else 4e-3)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("counts,k,n", [
    ([100, 200], 64, 32),
    ([128, 0, 257, 5], 128, 256),
    ([300, 1, 511], 256, 320),
    ([1000, 24], 1024, 512),
    ([513, 130], 4096, 96),
])
def test_grouped_gemm_forward(dtype, counts, k, n):
    from fastmoe_b200.ops import grouped_gemm as gg
    torch.manual_seed(0)
    rows = sum(counts)
    pad = 7  # rows past the last segment must stay untouched
    x = torch.randn(rows + pad, k, device=DEV, dtype=dtype)
    w = (torch.randn(len(counts), n, k, device=DEV) / k ** 0.5).to(dtype)
    b = torch.randn(len(counts), n, device=DEV).to(dtype)
    offs = _offs(counts)
    out, pre = gg.forward(x, w, offs, b, act="gelu", want_pre=True)
    if pre.dim() == 1:
        pre = gg.untile_pre(pre, offs, n, x.shape[0])
    for e, lo, hi in _segments(counts):
        ref_pre = x[lo:hi].float() @ w[e].float().t() + b[e].float()
        ref = torch.nn.functional.gelu(ref_pre)
        assert torch.allclose(pre[lo:hi].float(), ref_pre, atol=_tol(dtype, k), rtol=2e-2)
        assert torch.allclose(out[lo:hi].float(), ref, atol=_tol(dtype, k), rtol=2e-2)
    assert _native().read_status(0) == 0


@pytest.mark.parametrize("act", [None, "relu", "gelu_tanh"])
@pytest.mark.parametrize("counts,k,n", [([70, 300, 129], 192, 448), ([2048, 2048], 4096, 1024)])
def test_grouped_gemm_epilogues(act, counts, k, n):
    r"""The other fused epilogues, forward and input gradient, including a span of columns that
    is not a multiple of the 256-column tile and a K of 4096."""
    from fastmoe_b200.ops import grouped_gemm as gg
    torch.manual_seed(5)
    dtype = torch.bfloat16
    rows = sum(counts)
    x = torch.randn(rows, k, device=DEV, dtype=dtype)
    w = (torch.randn(len(counts), n, k, device=DEV) / k ** 0.5).to(dtype)
    b = torch.randn(len(counts), n, device=DEV).to(dtype)
    offs = _offs(counts)
    out, pre = gg.forward(x, w, offs, b, act=act, want_pre=True)
    if pre.dim() == 1:
        pre = gg.untile_pre(pre, offs, n, rows)
    fn = {None: lambda t: t, "relu": torch.relu,
          "gelu_tanh": lambda t: torch.nn.functional.gelu(t, approximate="tanh")}[act]
    dy = torch.randn(rows, n, device=DEV, dtype=dtype)
    wt = (torch.randn(len(counts), n, k, device=DEV) / n ** 0.5).to(dtype)   # [E, k(out)=n, n(in)=k]
    pre_in = torch.randn(rows, k, device=DEV, dtype=dtype)
    dx = gg.dgrad(dy, wt, offs, pre=_tiled(pre_in, offs, len(counts)) if act else None, act=act)
    p32 = pre_in.float().requires_grad_(True)
    fn(p32).sum().backward()
    for e, lo, hi in _segments(counts):
        ref_pre = x[lo:hi].float() @ w[e].float().t() + b[e].float()
        assert torch.allclose(pre[lo:hi].float(), ref_pre, atol=2e-2, rtol=2e-2)
        assert torch.allclose(out[lo:hi].float(), fn(ref_pre), atol=2e-2, rtol=2e-2)
        ref_dx = dy[lo:hi].float() @ wt[e].float()
        if act:
            ref_dx = ref_dx * p32.grad[lo:hi]
        assert torch.allclose(dx[lo:hi].float(), ref_dx, atol=2e-2, rtol=2e-2)
    assert _native().read_status(0) == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("counts,k,n", [
    ([100, 200], 64, 64),
    ([128, 0, 257, 5], 256, 128),
    ([700, 324], 512, 1024),
])
def test_grouped_gemm_dgrad(dtype, counts, k, n):
    r"""dX = (dY W) * gelu'(pre) with W stored [E, k(out), n(in)]."""
    from fastmoe_b200.ops import grouped_gemm as gg
    torch.manual_seed(1)
    rows = sum(counts)
    dy = torch.randn(rows, k, device=DEV, dtype=dtype)
    w = (torch.randn(len(counts), k, n, device=DEV) / k ** 0.5).to(dtype)
    pre = torch.randn(rows, n, device=DEV, dtype=dtype)
    offs = _offs(counts)
    plain = gg.dgrad(dy, w, offs)
    fused = gg.dgrad(dy, w, offs, pre=_tiled(pre, offs, len(counts)), act="gelu")
    rowmajor = gg.dgrad(dy, w, offs, pre=pre, act="gelu")   # plain matrix: derivative as a PyTorch op
    assert torch.allclose(rowmajor[:rows].float(), fused[:rows].float(), atol=2e-2, rtol=2e-2)
    p32 = pre.float().requires_grad_(True)
    torch.nn.functional.gelu(p32).sum().backward()
    for e, lo, hi in _segments(counts):
        ref = dy[lo:hi].float() @ w[e].float()
        assert torch.allclose(plain[lo:hi].float(), ref, atol=_tol(dtype, k), rtol=2e-2)
        assert torch.allclose(fused[lo:hi].float(), ref * p32.grad[lo:hi], atol=_tol(dtype, k), rtol=2e-2)
    assert _native().read_status(0) == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("counts,m,n", [
    ([64, 128], 128, 256),
    ([100, 0, 37, 300], 64, 32),
    ([1000, 24, 513], 256, 512),
])
def test_grouped_gemm_wgrad(dtype, counts, m, n):
    from fastmoe_b200.ops import grouped_gemm as gg
    torch.manual_seed(2)
    rows = sum(counts)
    pad = 70  # garbage rows after the last segment must not leak into the last expert
    dy = torch.randn(rows + pad, m, device=DEV, dtype=dtype)
    x = torch.randn(rows + pad, n, device=DEV, dtype=dtype)
    dy[rows:] = float("nan")
    x[rows:] = float("nan")
    offs = _offs(counts)
    out = gg.wgrad(dy, x, offs, len(counts))
    for e, lo, hi in _segments(counts):
        ref = dy[lo:hi].float().t() @ x[lo:hi].float()
        scale = max(1.0, (hi - lo) ** 0.5)
        assert torch.allclose(out[e].float(), ref, atol=_tol(dtype, hi - lo) * scale, rtol=2e-2), e
    bg = gg.bias_grad(dy[:rows].contiguous(), offs)
    for e, lo, hi in _segments(counts):
        ref = dy[lo:hi].float().sum(0)
        assert torch.allclose(bg[e].float(), ref, atol=0.3, rtol=2e-2)
    # the same sums produced inside the weight-gradient kernel, with and without accumulation
    out2, bg2 = gg.wgrad(dy, x, offs, len(counts), with_bias_grad=True)
    assert torch.equal(out2, out)
    for e, lo, hi in _segments(counts):
        ref = dy[lo:hi].float().sum(0)
        assert torch.allclose(bg2[e].float(), ref, atol=0.3, rtol=2e-2), e
    if gg._tc_ok(dy, gg.MODE_WGRAD, m, n, 0, len(counts)):
        acc_w = out.clone()
        acc_b = bg2.clone()
        _native().grouped_gemm(gg.MODE_WGRAD, dy, x, offs, acc_w, None, None, None, 0, 0, True, acc_b)
        assert torch.allclose(acc_b.float(), 2 * bg2.float(), atol=0.6, rtol=3e-2)
        for e, lo, hi in _segments(counts):
            scale = max(1.0, (hi - lo) ** 0.5)
            assert torch.allclose(acc_w[e].float(), 2 * out[e].float(), atol=_tol(dtype, 0) * 2 * scale,
                                  rtol=3e-2), e
        acc32 = torch.ones(len(counts), m, n, device=DEV, dtype=torch.float32)
        _native().grouped_gemm(gg.MODE_WGRAD, dy, x, offs, acc32, None, None, None, 0, 0, True, None)
        for e, lo, hi in _segments(counts):
            ref = 1.0 + dy[lo:hi].float().t() @ x[lo:hi].float()
            assert torch.allclose(acc32[e], ref, atol=1e-2 * max(1.0, (hi - lo) ** 0.5), rtol=1e-2), e
    assert _native().read_status(0) == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("counts,k,n", [([5, 0, 9, 3], 16, 24), ([300, 65, 0, 130], 200, 150)])
def test_simt_grouped_linear(dtype, counts, k, n):
    r"""The shared-memory tiled kernel for fp32 / fp64, ragged in every dimension."""
    from fastmoe_b200.ops import grouped_gemm as gg
    torch.manual_seed(3)
    torch.backends.cuda.matmul.allow_tf32 = False
    rows = sum(counts)
    x = torch.randn(rows, k, device=DEV, dtype=dtype)
    w = torch.randn(len(counts), n, k, device=DEV, dtype=dtype)
    b = torch.randn(len(counts), n, device=DEV, dtype=dtype)
    go = torch.randn(rows, n, device=DEV, dtype=dtype)
    cnt = torch.tensor(counts)
    out = gg.linear_forward_host_counts(x, cnt, w, b)
    gi, gw, gb = gg.linear_backward_host_counts(go, x, cnt, w, b)
    for e, lo, hi in _segments(counts):
        assert torch.allclose(out[lo:hi], x[lo:hi] @ w[e].t() + b[e], atol=2e-3, rtol=1e-4)
        assert torch.allclose(gi[lo:hi], go[lo:hi] @ w[e], atol=2e-3, rtol=1e-4)
        assert torch.allclose(gw[e], go[lo:hi].t() @ x[lo:hi], atol=2e-3, rtol=1e-4)
        assert torch.allclose(gb[e], go[lo:hi].sum(0), atol=2e-3, rtol=1e-4)


@pytest.mark.parametrize("n_slots,tot", [(7, 3), (64, 4), (8192, 16), (50001, 64), (4096, 1024),
                                         (1000003, 256), (300000, 8)])
def test_route_matches_cpu(n_slots, tot):
    r"""Counts, ranks, offsets and the sorted slot list; above 32 K slots several CTAs share the
    ranking (two launches) and must reproduce the single ordered scan."""
    from fastmoe_b200.ops import torch_impl
    torch.manual_seed(4)
    idx = torch.randint(-1, tot, (n_slots,), device=DEV)
    counts, rank, offs = _native().route_offs(idx, tot)
    c2, r2, o2, pos = _native().route_pos(idx, tot)
    assert torch.equal(c2, counts) and torch.equal(r2, rank) and torch.equal(o2, offs)
    kept = int(offs[-1])
    order = torch.argsort(torch.where(idx >= 0, idx, tot).cpu(), stable=True)[:kept]
    assert torch.equal(pos[:kept].cpu().long(), order)
    ref_counts = torch_impl.expert_count(idx.cpu(), tot)
    ref_rank = torch_impl.slot_rank(idx.cpu(), tot)
    assert torch.equal(counts.cpu(), ref_counts)
    assert torch.equal(rank.cpu().long(), ref_rank)
    assert torch.equal(offs.cpu()[1:].long(), torch.cumsum(ref_counts.long(), 0))


def test_capacity_kernels_match_cpu():
    from fastmoe_b200.ops import api, torch_impl
    torch.manual_seed(5)
    n_expert, n_worker = 4, 3
    ec = torch.randint(0, 20, (n_expert * n_worker,), dtype=torch.int64)
    cap = torch.full((n_expert,), 25, dtype=torch.int32)
    ref = torch_impl.limit_by_capacity(ec.clone(), cap.clone(), n_expert, n_worker)
    cap_d = cap.to(DEV)
    got = api.limit_by_capacity(ec.to(DEV), cap_d, n_expert, n_worker)
    assert torch.equal(got.cpu(), ref)
    idx = torch.randint(-1, n_expert * n_worker, (100, 2))
    capg = torch.randint(0, 12, (n_expert * n_worker,), dtype=torch.int32)
    ref_idx = torch_impl.prune_gate_by_capacity(idx.clone(), capg.clone(), n_expert, n_worker)
    got_idx = api.prune_gate_by_capacity(idx.to(DEV), capg.to(DEV), n_expert, n_worker)
    assert torch.equal(got_idx.cpu(), ref_idx)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_scatter_combine_roundtrip(dtype):
    torch.manual_seed(6)
    nat = _native()
    n_tok, k, d, tot = 300, 2, 256, 8
    x = torch.randn(n_tok, d, device=DEV, dtype=dtype)
    idx = torch.randint(-1, tot, (n_tok * k,), device=DEV)
    score = torch.rand(n_tok * k, device=DEV).to(dtype)
    counts, rank, offs = nat.route_offs(idx, tot)
    rows = torch.full((n_tok * k, d), float("nan"), device=DEV, dtype=dtype)
    row_slot = torch.full((n_tok * k,), -1, device=DEV, dtype=torch.int32)
    nat.scatter_rows(x, idx, rank, offs, None, k, rows, row_slot)
    n_valid = int(offs[-1])
    slots = row_slot[:n_valid].long()
    assert torch.equal(rows[:n_valid], x[slots // k])
    # rows are grouped by expert, ascending slot inside an expert
    assert torch.equal(idx[slots], torch.sort(idx[idx >= 0], stable=True).values)
    out = torch.empty(n_tok, d, device=DEV, dtype=dtype)
    nat.gather_combine(rows, idx, rank, offs, score, k, out)
    w = torch.where(idx >= 0, score.float(), torch.zeros_like(score, dtype=torch.float32))
    ref = (x.float().repeat_interleave(k, 0) * w[:, None]).view(n_tok, k, d).sum(1)
    assert torch.allclose(out.float(), ref, atol=3e-2, rtol=2e-2)
    # backward of the weighted combine
    dout = torch.randn(n_tok, d, device=DEV, dtype=dtype)
    drows = torch.zeros_like(rows)
    dscore = torch.empty(n_tok * k, device=DEV, dtype=dtype)
    nat.combine_bwd(dout, rows, idx, rank, offs, score, k, drows, dscore)
    ref_ds = (dout.float().repeat_interleave(k, 0) * x.float().repeat_interleave(k, 0)).sum(1)
    ref_ds = torch.where(idx >= 0, ref_ds, torch.zeros_like(ref_ds))
    assert torch.allclose(dscore.float(), ref_ds, atol=0.25, rtol=2e-2)
    ref_dr = dout.float().repeat_interleave(k, 0)[slots] * score.float()[slots][:, None]
    assert torch.allclose(drows[:n_valid].float(), ref_dr, atol=3e-2, rtol=2e-2)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n_exp,k", [(16, 2), (4, 1), (64, 3), (200, 8)])
def test_gate_topk_softmax(dtype, n_exp, k):
    from fastmoe_b200.ops import gating
    torch.manual_seed(7)
    logits = torch.randn(500, n_exp, device=DEV, dtype=dtype).requires_grad_(True)
    idx, prob = gating.topk_softmax(logits, k)
    ref_l = logits.detach().float().requires_grad_(True)
    rv, _ri = torch.topk(ref_l, k, dim=-1)
    # Ties (frequent in bf16) may be ordered differently: compare the selected values, and
    # differentiate the reference through the kernel's own selection.
    picked = torch.gather(ref_l, 1, idx)
    assert torch.equal(picked.detach(), rv.detach())
    rp = torch.softmax(picked, -1)
    assert torch.allclose(prob.float(), rp, atol=1e-2 if dtype != torch.float32 else 1e-5)
    g = torch.randn_like(prob)
    prob.backward(g)
    rp.backward(g.float())
    assert torch.allclose(logits.grad.float(), ref_l.grad, atol=2e-2 if dtype != torch.float32 else 1e-5)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n_exp,k,d,bias", [(4, 2, 64, True), (16, 2, 1024, True), (13, 3, 200, False),
                                            (32, 1, 512, True), (64, 4, 256, True)])
def test_gate_linear_topk_softmax(dtype, n_exp, k, d, bias):
    r"""Single-pass linear gate against fp32 ``linear`` → ``topk`` → ``softmax``, forward and backward,
    with gradients arriving through the probabilities and through the logits."""
    from fastmoe_b200.ops import gating
    torch.manual_seed(11)
    n = 777
    x = torch.randn(n, d, device=DEV, dtype=dtype).requires_grad_(True)
    w = (torch.randn(n_exp, d, device=DEV) / d ** 0.5).to(dtype).requires_grad_(True)
    b = (torch.randn(n_exp, device=DEV) * 0.1).to(dtype).requires_grad_(True) if bias else None
    # the autograd function directly: the public wrapper only picks it for small expert counts
    logits, idx, prob = gating._LinearTopkSoftmax.apply(x, w, b, k)
    assert logits.dtype == dtype and idx.dtype == torch.int64 and prob.shape == (n, k)

    xr = x.detach().float().requires_grad_(True)
    wr = w.detach().float().requires_grad_(True)
    br = b.detach().float().requires_grad_(True) if bias else None
    lr = torch.nn.functional.linear(xr, wr, br)
    tol = 2e-2 if dtype == torch.bfloat16 else 4e-3
    assert torch.allclose(logits.float(), lr, atol=tol, rtol=tol)
    # the selection is made on the rounded logits the kernel returns
    rv, _ = torch.topk(logits.detach().float(), k, dim=-1)
    assert torch.equal(torch.gather(logits.detach().float(), 1, idx), rv)
    rp = torch.softmax(torch.gather(lr, 1, idx), -1)
    assert torch.allclose(prob.float(), rp, atol=tol)

    gp = torch.randn_like(prob)
    gl = torch.randn_like(logits) * 0.1
    torch.autograd.backward([prob, logits], [gp, gl])
    torch.autograd.backward([rp, lr], [gp.float(), gl.float()])

    def close(a, r):
        scale = r.abs().max().item() + 1e-6
        return (a.float() - r).abs().max().item() <= 2e-2 * scale

    assert close(x.grad, xr.grad)
    assert close(w.grad, wr.grad)
    if bias:
        assert close(b.grad, br.grad)

    # gradient through the probabilities only (the plain top-k gate)
    x2 = x.detach().clone().requires_grad_(True)
    _, _, p2 = gating._LinearTopkSoftmax.apply(x2, w.detach(), None if b is None else b.detach(), k)
    p2.backward(gp)
    xr2 = x.detach().float().requires_grad_(True)
    lr2 = torch.nn.functional.linear(xr2, wr.detach(), None if br is None else br.detach())
    torch.softmax(torch.gather(lr2, 1, idx), -1).backward(gp.float())
    assert close(x2.grad, xr2.grad)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n_exp,k,d,bias", [(16, 2, 1024, True), (64, 4, 512, True), (100, 8, 256, False),
                                            (256, 2, 1024, True)])
def test_gate_tensor_core_many_experts(dtype, n_exp, k, d, bias):
    r"""The linear gate above 8 experts: logits on the tcgen05 kernel (one group, expert
    dimension padded), top-k / softmax kernel, against fp32 ``linear`` -> ``topk`` -> ``softmax``,
    forward and backward through probabilities and logits."""
    from fastmoe_b200.ops import gating
    torch.manual_seed(12)
    n = 1531
    x = torch.randn(n, d, device=DEV, dtype=dtype).requires_grad_(True)
    w = (torch.randn(n_exp, d, device=DEV) / d ** 0.5).to(dtype).requires_grad_(True)
    b = (torch.randn(n_exp, device=DEV) * 0.1).to(dtype).requires_grad_(True) if bias else None
    assert gating._gate_gemm_ok(x, w, b)
    logits, idx, prob = gating.linear_topk_softmax(x, w, b, k)
    assert logits.shape == (n, n_exp) and idx.shape == (n, k) and int(idx.max()) < n_exp

    xr = x.detach().float().requires_grad_(True)
    wr = w.detach().float().requires_grad_(True)
    br = b.detach().float().requires_grad_(True) if bias else None
    lr = torch.nn.functional.linear(xr, wr, br)
    tol = 2e-2 if dtype == torch.bfloat16 else 4e-3
    assert torch.allclose(logits.float(), lr, atol=tol, rtol=tol)
    rv, _ = torch.topk(logits.detach().float(), k, dim=-1)
    assert torch.equal(torch.gather(logits.detach().float(), 1, idx), rv)
    rp = torch.softmax(torch.gather(lr, 1, idx), -1)
    assert torch.allclose(prob.float(), rp, atol=tol)

    gp = torch.randn_like(prob)
    gl = torch.randn(n, n_exp, device=DEV, dtype=dtype) * 0.1
    torch.autograd.backward([prob, logits], [gp, gl])
    torch.autograd.backward([rp, lr], [gp.float(), gl.float()])
    for got, ref in ((x.grad, xr.grad), (w.grad, wr.grad)) + (((b.grad, br.grad),) if bias else ()):
        scale = ref.abs().max().item() + 1e-6
        assert (got.float() - ref).abs().max().item() <= 3e-2 * scale
    assert _native().read_status(0) == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("counts,m,n", [
    ([255, 0, 257, 1], 256, 288),       # one row either side of a pair's 256-row tile, an empty expert
    ([65, 15, 16, 17, 127, 128], 72, 544),   # ragged ends around the 16-row MMA step and the K block
    ([1, 513], 264, 256),               # an output tile whose second half has 8 rows
])
def test_pair_tiles_and_ragged_ends(dtype, counts, m, n):
    r"""The paired kernel at the edges of its 256 x 256 tiles, 64-row K blocks and 16-row steps; rows
    past the last expert are NaN and must not reach any output.  Against fp64: one rounding to
    the 16-bit type (relative 2^-9 / 2^-12) plus an fp32 sum of at most 513 terms."""
    from fastmoe_b200.ops import grouped_gemm as gg
    torch.manual_seed(11)
    g, rows, k = len(counts), sum(counts), 192
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    offs = _offs(counts)

    def close(got, ref, terms):
        bound = eps * ref.abs() + 2.0 ** -22 * terms ** 0.5 * ref.abs().amax().clamp(min=1.0) + 1e-6
        return bool(((got.double() - ref).abs() <= bound).all())

    dy = torch.randn(rows + 40, m, device=DEV).to(dtype)
    q = torch.randn(rows + 40, n, device=DEV).to(dtype)
    dy[rows:] = float("nan")
    q[rows:] = float("nan")
    dw, db = gg.wgrad(dy, q, offs, g, with_bias_grad=True)
    x = torch.randn(rows, k, device=DEV).to(dtype)
    w = (torch.randn(g, n, k, device=DEV) / k ** 0.5).to(dtype)
    b = torch.randn(g, n, device=DEV).to(dtype)
    y = gg.forward(x, w, offs, b)
    go = torch.randn(rows, k, device=DEV).to(dtype)
    wn = (torch.randn(g, k, n, device=DEV) / k ** 0.5).to(dtype)
    dx = gg.dgrad(go, wn, offs)
    for e, lo, hi in _segments(counts):
        assert close(dw[e], dy[lo:hi].double().t() @ q[lo:hi].double(), max(1, hi - lo)), e
        assert close(db[e], dy[lo:hi].double().sum(0), max(1, hi - lo)), e
        if hi > lo:
            assert close(y[lo:hi], x[lo:hi].double() @ w[e].double().t() + b[e].double(), k), e
            assert close(dx[lo:hi], go[lo:hi].double() @ wn[e].double(), k), e
    assert _native().read_status(0) == 0


@pytest.mark.parametrize("counts,k,n", [([64, 0, 65, 1, 127], 20, 132), ([3], 4, 4), ([0, 0], 16, 128),
                                        ([1] * 40 + [200], 36, 260), ([130, 70], 18, 128)])
def test_fp32_tiles_tail_and_column_sums(counts, k, n):
    r"""The aligned fp32 kernel (and, with k = 18, the general one) at the edges of its 64 x 128 x 16
    tiles, with more experts than a warp has lanes, against fp64: an fp32 sum of t terms is off by
    at most t * 2^-24 times the sum of the absolute products.  Rows past the last expert come back
    zero although the buffers around them hold NaN."""
    from fastmoe_b200.ops import grouped_gemm as gg
    torch.manual_seed(12)
    g, rows = len(counts), sum(counts)
    offs = _offs(counts)
    x = torch.randn(rows + 70, k, device=DEV)
    go = torch.randn(rows + 70, n, device=DEV)
    x[rows:] = float("nan")
    go[rows:] = float("nan")
    w, b = torch.randn(g, n, k, device=DEV), torch.randn(g, n, device=DEV)
    torch.full((rows + 70, max(n, k)), float("nan"), device=DEV)   # stale bits for the allocator to hand out
    y = gg.forward(x, w, offs, b)
    dx = gg.dgrad(go, w, offs)
    dw, db = gg.wgrad(go[:rows].contiguous(), x[:rows].contiguous(), offs, g, with_bias_grad=True)
    assert not y[rows:].any() and not dx[rows:].any()

    def close(got, a, bb, extra=0.0):
        ref = a.double() @ bb.double() + extra
        bound = (a.shape[1] + 2) * 2.0 ** -24 * (a.double().abs() @ bb.double().abs() + abs(extra)) + 1e-12
        return bool(((got.double() - ref).abs() <= bound).all())

    for e, lo, hi in _segments(counts):
        if hi > lo:
            assert close(y[lo:hi], x[lo:hi], w[e].t(), b[e].double()), e
            assert close(dx[lo:hi], go[lo:hi], w[e]), e
        assert close(dw[e], go[lo:hi].t(), x[lo:hi]), e
        assert close(db[e][None], torch.ones(1, hi - lo, device=DEV), go[lo:hi]), e


@pytest.mark.parametrize("n_slots,tot", [(1024, 8), (1025, 8), (22528, 8), (16384, 2), (16385, 64), (65536, 1),
                                         (65537, 3), (40000, 1024), (40000, 1025), (1, 1), (5000, 20000)])
def test_route_at_the_lines_between_cta_cluster_and_grid(n_slots, tot):
    r"""Counts, ranks, offsets and slot list where the routing kernel changes its split of the work,
    with a third of the slots dropped and one expert holding most of the others."""
    torch.manual_seed(14)
    idx = torch.randint(0, tot, (n_slots,))
    idx[torch.rand(n_slots) < 0.5] = tot // 2
    idx[torch.rand(n_slots) < 0.3] = -1
    counts, rank, offs, pos = (t.cpu().long() for t in _native().route_pos(idx.to(DEV), tot))
    kept = idx >= 0
    want = torch.bincount(idx[kept], minlength=tot)
    assert torch.equal(counts, want)
    assert torch.equal(offs, torch.cat([torch.zeros(1, dtype=torch.long), want.cumsum(0)]))
    order = torch.argsort(torch.where(kept, idx, tot), stable=True)[:int(kept.sum())]
    assert torch.equal(pos[:order.numel()], order)
    want_rank = torch.full((n_slots,), -1)
    want_rank[order] = torch.arange(order.numel()) - offs[idx[order]]
    assert torch.equal(rank, want_rank)


@pytest.mark.parametrize("n_slots,tot,launches", [(32768, 1025, 1), (32769, 1025, 2), (65536, 5000, 2), (65536, 1024, 1),
                                                  (65537, 1024, 2)])
def test_route_launches(n_slots, tot, launches):
    r"""One launch while a cluster, or with more than 1024 experts a CTA, holds the slots; then two on
    many CTAs."""
    idx = torch.zeros(n_slots, dtype=torch.int64, device=DEV)
    before = _native().launch_count()
    _native().route_pos(idx, tot)
    assert _native().launch_count() - before == launches


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,tot,k,d", [(2367, 8, 2, 136), (2368, 7, 7, 264), (2369, 2, 1, 128), (4735, 3, 2, 64),
                                          (4736, 8, 2, 1024), (4739, 2, 2, 512), (9001, 5, 4, 520), (1, 1, 1, 8)])
def test_gate_rows_per_warp(dtype, rows, tot, k, d):
    r"""The fused gate on both sides of the lines where a warp takes one, two or four tokens, against
    fp64 on the same 16-bit inputs: logits to one rounding plus an fp32 sum of d terms, ids by the
    returned logits (ties to the lower id), gradients to one rounding plus a sum of tot, k or rows
    terms."""
    from fastmoe_b200.ops import gating
    torch.manual_seed(15)
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    x = torch.randn(rows, d, device=DEV).to(dtype).requires_grad_(True)
    w = (torch.randn(tot, d, device=DEV) / d ** 0.5).to(dtype).requires_grad_(True)
    b = torch.randn(tot, device=DEV).to(dtype).requires_grad_(True)
    logits, idx, prob = gating.linear_topk_softmax(x, w, b, k)
    ref = x.double() @ w.double().t() + b.double()
    assert ((logits.double() - ref).abs() <= eps * ref.abs() + d * 2.0 ** -23).all()
    assert torch.equal(idx, logits.double().sort(dim=1, descending=True, stable=True).indices[:, :k])
    gl, gp = torch.randn_like(logits), torch.randn_like(prob)
    torch.autograd.backward([logits, prob], [gl, gp])
    p64, g64 = prob.detach().double(), gp.double()
    dl = gl.double().scatter_add(1, idx, p64 * (g64 - (p64 * g64).sum(1, keepdim=True)))

    def close(got, a, m):
        r = a @ m
        return bool(((got.double() - r).abs() <= eps * r.abs() + (a.shape[1] + 16) * 2.0 ** -22 * (a.abs() @ m.abs()) + 1e-7).all())

    assert close(x.grad, dl, w.detach().double())
    assert close(w.grad, dl.t(), x.detach().double())
    assert close(b.grad[None], torch.ones(1, rows, device=DEV, dtype=torch.float64), dl)


@pytest.mark.parametrize("rows,tot,k", [(5, 2, 1), (5, 8, 2), (2400, 3, 2), (2400, 7, 7), (4800, 8, 4), (4800, 2, 2)])
def test_gate_with_nan_logits(rows, tot, k):
    r"""NaN in one expert's weights, or in some tokens, with one, two and four tokens per warp: the
    choice is that of k scans in which only a greater logit replaces the first expert left, and a
    chosen NaN makes all scores of its token NaN."""
    from fastmoe_b200.ops import gating
    torch.manual_seed(23)
    nan = float("nan")
    for bad in range(-1, tot):
        x = torch.randn(rows, 64, device=DEV).bfloat16()
        w = torch.randn(tot, 64, device=DEV).bfloat16()
        if bad < 0:
            x[::3] = nan
        else:
            w[bad] = nan
        logits, idx, prob = (t.cpu() for t in gating.linear_topk_softmax(x, w, None, k))
        v = logits.double()
        left = torch.ones(rows, tot, dtype=torch.bool)
        for j in range(k):
            first = left.double().argmax(1, keepdim=True)       # the lowest id left
            seen = torch.where(left, v, -float("inf")).nan_to_num(nan=-float("inf"))
            best = seen.argmax(1, keepdim=True)                 # the greatest, the lowest id of equals
            choice = torch.where(v.gather(1, first).isnan(), first, best)
            assert torch.equal(idx[:, j:j + 1], choice), (bad, j)
            left.scatter_(1, choice, False)
        want = torch.softmax(v.gather(1, idx), 1)
        assert torch.equal(prob.isnan(), want.isnan())
        assert torch.allclose(prob.double().nan_to_num(), want.nan_to_num(), atol=2.0 ** -8)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("kind", ["gshard", "switch"])
@pytest.mark.parametrize("n,tot", [(1, 2), (127, 3), (129, 64), (5000, 8), (40000, 2)])
def test_balanced_gates_native_loss(dtype, kind, n, tot, monkeypatch):
    r"""Whole gates: ids, scores, loss and parameter gradients of the capacity-limited gates with the
    balance-loss kernels against the same gate as PyTorch operations in the layer's type, with a
    gradient arriving through the scores and from the loss together.  (The scores' part is the
    larger one: the tests that follow take the loss by itself.)"""
    from fastmoe_b200.gates import GShardGate, SwitchGate
    from fastmoe_b200.ops import gating
    torch.manual_seed(16)
    d = 64
    gate = (GShardGate(d, tot, 1, random_routing=False) if kind == "gshard" else
            SwitchGate(d, tot, 1, switch_eps=0.0)).to(DEV).to(dtype)
    x = torch.randn(n, d, device=DEV).to(dtype)
    idx, score = gate(x)
    loss = gate.get_loss()
    gs = torch.randn_like(score)
    torch.autograd.backward([score, loss], [gs, None])
    grads = [p.grad.double() for p in gate.parameters()]
    eps = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -20}[dtype]

    gate.zero_grad()
    monkeypatch.setattr(gating, "balance_native", lambda logits: False)
    want_idx, want_score = gate(x)
    want_loss = gate.get_loss()
    assert torch.equal(idx, want_idx)
    assert torch.allclose(score.double(), want_score.double(), rtol=2 * eps, atol=1e-6)
    assert loss.dim() == 0 and loss.dtype == want_loss.dtype
    # GShard's reference rounds the probabilities and their mean to the layer's type
    assert torch.allclose(loss.double(), want_loss.double(), rtol=4 * eps + 1e-5)
    torch.autograd.backward([want_score, want_loss], [gs, None])
    for g, p in zip(grads, gate.parameters()):
        scale = p.grad.double().abs().max().clamp(min=1e-6)
        assert ((g - p.grad.double()).abs() <= (4 * eps + 1e-5 * n ** 0.5) * scale).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("n,tot", [(1, 2), (127, 3), (1000, 2), (4096, 2), (5000, 8), (9001, 64)])
def test_gshard_loss_rounds_like_its_operations(dtype, n, tot):
    r"""GShard's loss by itself: the PyTorch operations hold the probabilities, their mean and the
    gradients of both in the logits' type, and so do the kernels.  The same fp32 values are rounded,
    up to a few units of fp32, so that about 2^-11 (fp16) or 2^-14 (bf16) of the roundings go the
    other way: one element in a hundred may differ, by a few units of the type of the largest term
    of its sum.  Unrounded, a fifth to a half of them would."""
    from fastmoe_b200.gates.gshard_gate import gshard_balance_loss
    from fastmoe_b200.ops import gating
    torch.manual_seed(19)
    eps = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -22}[dtype]
    wide = torch.randn(n, tot + 6, device=DEV).to(dtype)   # rows with a pitch, as the padded gate has them
    ids = wide[:, :tot].topk(2, dim=1).indices
    ref = lambda l, i: gshard_balance_loss(l, i[:, 0], tot, tot)   # noqa: E731
    losses, grads = [], []
    for fn in (lambda l: gating.gshard_loss(l, ids, tot ** 2, ref), lambda l: ref(l, ids)):
        w = wide.clone().requires_grad_(True)
        loss = fn(w[:, :tot])
        losses.append(loss.detach())
        grads.append(torch.autograd.grad(loss, w, torch.full_like(loss, 3.0))[0][:, :tot].double())
    assert losses[0].dtype == losses[1].dtype and losses[0].shape == losses[1].shape
    assert torch.allclose(losses[0], losses[1], rtol=eps + 1e-5)
    p = torch.softmax(wide[:, :tot].double(), 1)
    c = torch.bincount(ids[:, 0], minlength=tot).double() / n
    term = 3.0 * tot / n * c * p
    bound = 4 * eps * (term + p * term.sum(1, keepdim=True)) + (2.0 ** -23 if dtype == torch.float16 else 1e-12)
    assert ((grads[0] - grads[1]).abs() <= bound).all()
    if dtype != torch.float32 and n > 1:
        assert (grads[0] != grads[1]).double().mean() <= 0.01


@pytest.mark.parametrize("rows", [9, 300, 777])
def test_wide_gate_first_called_under_capture(rows):
    r"""The tensor-core gate (12 experts) called for a row count first inside a graph that has not
    been replayed, then eagerly, on another stream, and by the replay: nothing of one call is
    left for the next.  9 rows take the narrow kernel and, in backward, the single-CTA one."""
    from fastmoe_b200.ops import gating
    torch.manual_seed(20)
    dtype, eps = torch.bfloat16, 2.0 ** -8

    def make(n):
        x = torch.randn(n, 128, device=DEV).to(dtype).requires_grad_(True)
        w = (torch.randn(12, 128, device=DEV) / 128 ** 0.5).to(dtype).requires_grad_(True)
        return x, w, torch.randn(12, device=DEV).to(dtype).requires_grad_(True)

    def close(got, ref):
        return bool(((got.double() - ref).abs() <= eps * ref.abs() + 1e-4 * ref.abs().max()).all())

    gating.linear_topk_softmax(*make(64), 2)   # the library's own lazy set-up, for another row count
    xg, wg, bg = (t.detach() for t in make(rows))
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        captured = gating.linear_topk_softmax(xg, wg, bg, 2)[0]
    for stream in (torch.cuda.current_stream(), torch.cuda.Stream()):
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            x, w, b = make(rows)
            logits, _idx, _prob = gating.linear_topk_softmax(x, w, b, 2)
            gl = torch.randn_like(logits)
            logits.backward(gl)
        torch.cuda.synchronize()
        x64, w64, g64 = x.detach().double(), w.detach().double(), gl.double()
        assert close(logits, x64 @ w64.t() + b.detach().double())
        assert close(x.grad, g64 @ w64) and close(w.grad, g64.t() @ x64) and close(b.grad, g64.sum(0))
    graph.replay()
    torch.cuda.synchronize()
    assert close(captured, xg.double() @ wg.double().t() + bg.double())


def test_switch_gate_with_its_own_loss():
    r"""A subclass, or an instance, with another balance loss is asked for it."""
    from fastmoe_b200.gates import SwitchGate

    class Summed(SwitchGate):
        def _balance_loss(self, prob, winner):
            return prob.sum() + (winner >= 0).sum()

    x = torch.randn(40, 64, device=DEV)
    patched = SwitchGate(64, 4, 1).to(DEV)
    patched._balance_loss = lambda prob, winner: prob.sum() + (winner >= 0).sum()
    for gate in (Summed(64, 4, 1).to(DEV), patched):
        idx, _score = gate(x)
        assert abs(float(gate.get_loss()) - 40 - int((idx >= 0).sum())) < 1e-3


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_switch_gate_in_forward_mode(dtype):
    r"""Directional derivatives of Switch's scores and loss, in 64 bits up to the type's rounding (the
    derivative of a softmax over 4 entries is a sum of 4 products of numbers of order one)."""
    import torch.autograd.forward_ad as forward_ad
    from fastmoe_b200.gates import SwitchGate
    torch.manual_seed(24)
    gate = SwitchGate(64, 4, 1).to(DEV).to(dtype).eval()
    x, dx = (torch.randn(50, 64, device=DEV).to(dtype) for _ in range(2))
    with forward_ad.dual_level():
        idx, score = gate(forward_ad.make_dual(x, dx))
        dscore = forward_ad.unpack_dual(score).tangent
        dloss = forward_ad.unpack_dual(gate.get_loss()).tangent
        logits, tangent = forward_ad.unpack_dual(gate.gate(forward_ad.make_dual(x, dx)))
    assert (idx >= 0).all()   # nothing is dropped at 2.4 times the even share
    l64 = logits.detach().double().requires_grad_(True)
    p = torch.softmax(l64, 1)
    share = torch.bincount(idx.view(-1), minlength=4).double() / 50

    def along(y):   # d y of every row, or of all
        return (torch.autograd.grad(y.sum(), l64, retain_graph=True)[0] * tangent.double()).sum(1)

    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20
    want = along(p.gather(1, idx))
    assert torch.allclose(dscore.double().view(-1), want, atol=8 * eps)
    assert torch.allclose(dloss.double(), along(4 * (share * p.sum(0) / 50).sum()).sum(), atol=8 * 2.0 ** -20)


@pytest.mark.parametrize("kind", ["GShardGate", "SwitchGate"])
def test_gate_with_an_unread_loss_is_freed_at_once(kind):
    r"""The loss a gate holds does not hold the gate: no cycle that waits for the collector with the
    graph of the last pass."""
    import gc
    import weakref
    from fastmoe_b200 import gates
    gate = getattr(gates, kind)(64, 4, 1).to(DEV)
    gate(torch.randn(8, 64, device=DEV))
    assert gate.has_loss
    gone = weakref.ref(gate)
    gc.collect()
    gc.disable()
    try:
        del gate
        assert gone() is None
    finally:
        gc.enable()


def test_switch_ids_belong_to_the_caller():
    r"""Ids changed in place between forward and backward (by a gate hook, say) do not matter to the
    gradients, of first or second order."""
    from fastmoe_b200.gates import SwitchGate
    torch.manual_seed(25)
    gate = SwitchGate(64, 4, 1, switch_eps=0.0, capacity=(0.7, 0.7)).to(DEV)
    x = torch.randn(30, 64, device=DEV)
    grads = []
    for change in (False, True):
        idx, score = gate(x)
        loss = gate.get_loss() + score.square().sum()
        assert (idx < 0).any() and (idx >= 0).any()
        if change:
            idx.fill_(1)
        first = torch.autograd.grad(loss, gate.gate.weight, retain_graph=True)[0]
        again = torch.autograd.grad(loss, gate.gate.weight, create_graph=True)[0]
        grads.append((first, torch.autograd.grad(again.square().sum(), gate.gate.weight)[0]))
    for a, b in zip(*grads):
        assert torch.allclose(a, b, rtol=1e-4, atol=1e-6)   # scatter_add_ of the operations is unordered


@pytest.mark.parametrize("tot", [2, 8, 16, 33, 64])
def test_fp32_switch_scores_and_gradients_are_no_further_off(tot):
    r"""Distance of Switch's fp32 scores, loss and logit gradients from 64 bits, root of the mean square,
    against that of the PyTorch operations: equal up to what 60000 draws leave to chance."""
    from fastmoe_b200.gates.switch_gate import switch_score_and_loss
    from fastmoe_b200.ops import gating
    torch.manual_seed(26)
    n = 60000
    logits = (torch.randn(n, tot, device=DEV) * 2).requires_grad_(True)
    gs = torch.randn(n, 1, device=DEV)
    ids, score, loss = gating.switch_route(logits, n, switch_score_and_loss)
    outs = [(score, loss, torch.autograd.grad([score, loss], logits, [gs, None])[0])]
    for dtype in (torch.float32, torch.float64):
        x = logits.detach().to(dtype).requires_grad_(True)
        prob = torch.softmax(x, 1)
        share = torch.bincount(ids.view(-1), minlength=tot).to(dtype)
        s, l = prob.gather(1, ids), tot * ((share / n) * (prob.sum(0) / n)).sum()
        outs.append((s, l, torch.autograd.grad([s, l], x, [gs.to(dtype), None])[0]))
    for name, native, ops, exact in zip(("score", "loss", "gradient"), *outs):
        off = [float((t.detach().double() - exact.detach()).square().mean().sqrt()) for t in (native, ops)]
        assert off[0] <= 1.05 * off[1] + (2.0 ** -23 * abs(float(exact)) if name == "loss" else 0.0), (name, off)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("n,tot,cap", [(1, 2, 9), (127, 3, 30), (1000, 2, 600), (5000, 8, 700), (9001, 64, 100)])
def test_switch_loss_alone_in_64_bits(dtype, n, tot, cap):
    r"""Switch's loss and the logit gradient that comes from it alone, some tokens beyond the capacity,
    against 64 bits on the same logits.  The kernels hold everything in fp32: the loss is a sum of n
    terms, the gradient the difference of two numbers that are each right to a few units of fp32
    (softmax, weight, sum over 64 experts: below 2^-18), rounded once to the logits' type (relative
    error 2^-8 with the 8 significant bits of bf16, 2^-11 with the 11 of fp16)."""
    from fastmoe_b200.gates.switch_gate import switch_score_and_loss
    from fastmoe_b200.ops import gating
    torch.manual_seed(29)
    eps = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -24}[dtype]
    tiny = 2.0 ** -25 if dtype == torch.float16 else 0.0   # half a unit of fp16's smallest numbers
    logits = torch.randn(n, tot, device=DEV).to(dtype).requires_grad_(True)
    kept, _score, loss = gating.switch_route(logits, cap, switch_score_and_loss)
    (got,) = torch.autograd.grad(loss, logits, torch.full_like(loss, 3.0))
    x = logits.detach().double().requires_grad_(True)
    prob = torch.softmax(x, 1)
    ids = kept.view(-1)[kept.view(-1) >= 0]
    share, n_kept = torch.bincount(ids, minlength=tot).double(), max(1, ids.numel())
    want_loss = tot * ((share / n_kept) * (prob.sum(0) / n_kept)).sum()
    (want,) = torch.autograd.grad(3.0 * want_loss, x)
    assert torch.allclose(loss.double(), want_loss, rtol=1e-5)
    term = prob.detach() * (3.0 * tot / n_kept ** 2 * share)
    bound = eps * want.abs() + 2.0 ** -18 * (term + prob.detach() * term.sum(1, keepdim=True)) + tiny
    assert ((got.double() - want).abs() <= bound).all()


def test_balance_loss_second_derivative():
    r"""A gradient of the gradient goes through the PyTorch operations; the first one, where no second
    is wanted, comes from the kernel and is the same."""
    from fastmoe_b200.gates.gshard_gate import gshard_balance_loss
    from fastmoe_b200.ops import gating
    torch.manual_seed(17)
    logits = torch.randn(50, 4, device=DEV, requires_grad=True)
    ids = torch.randint(0, 4, (50, 2), device=DEV)
    ref = lambda l, i: gshard_balance_loss(l, i[:, 0], 4, 4)   # noqa: E731
    got = []
    native = gating.gshard_loss(logits, ids, 16, ref)
    (first,) = torch.autograd.grad(native, logits, retain_graph=True)
    assert torch.allclose(first, torch.autograd.grad(ref(logits, ids), logits)[0], rtol=1e-4, atol=1e-9)
    for loss in (native, ref(logits, ids)):
        (g,) = torch.autograd.grad(loss, logits, create_graph=True)
        got.append((g, torch.autograd.grad(g.pow(2).sum(), logits)[0]))
    for a, b in zip(*got):
        assert torch.allclose(a, b, rtol=1e-4, atol=1e-9)


@pytest.mark.parametrize("counts,want_pre", [([200, 0, 130], True), ([200, 0, 130], False), ([3, 0, 5], True),
                                             ([3, 0, 5], False)])
def test_fused_relu_of_nan_and_infinities(counts, want_pre):
    r"""The fused ReLU and its derivative treat NaN and infinities as torch.relu does, in the paired
    kernel, the single-CTA kernel (few rows, pre-activation kept) and the narrow one: NaN is not
    hidden, and a gradient, whatever it is, does not pass where the input is not positive."""
    from fastmoe_b200.ops import grouped_gemm as gg
    torch.manual_seed(27)
    nan, inf = float("nan"), float("inf")
    g, rows, k, n = len(counts), sum(counts), 64, 96
    offs = _offs(counts)
    x = torch.randn(rows, k, device=DEV).bfloat16()
    x[1] = nan
    w = torch.randn(g, n, k, device=DEV).bfloat16()
    b = torch.randn(g, n, device=DEV).bfloat16()
    b[:, 3], b[:, 40], b[:, 70] = nan, inf, -inf
    y = gg.forward(x, w, offs, b, act="relu", want_pre=want_pre)
    if want_pre:
        y, blocked = y
        plain = gg.forward(x, w, offs, b)
        dy = torch.randn(rows, k, device=DEV).bfloat16()
        dy[2] = inf
        dx = gg.dgrad(dy, w.transpose(1, 2).contiguous(), offs, pre=blocked, act="relu")
    for e, lo, hi in _segments(counts):
        if hi == lo:
            continue
        pre = x[lo:hi].double() @ w[e].double().t() + b[e].double()
        ref = torch.relu(pre)
        assert torch.equal(y[lo:hi].isnan(), ref.isnan()) and torch.equal(y[lo:hi].isinf(), ref.isinf())
        assert torch.allclose(y[lo:hi].double(), ref, rtol=2.0 ** -8, atol=1e-4, equal_nan=True)
        if want_pre:
            # (an infinite sum of the fp32 accumulators has no 64-bit counterpart: compare what is chosen)
            ungated = dy[lo:hi].double() @ w[e].double().t()
            off = plain[lo:hi].double() <= 0
            assert (dx[lo:hi][off] == 0).all()
            got, want = dx[lo:hi][~off].double(), ungated[~off]
            assert torch.equal(got.isfinite(), want.isfinite())
            keep = want.isfinite()
            assert torch.allclose(got[keep], want[keep], rtol=2.0 ** -8, atol=1e-3)
    assert _native().read_status(0) == 0


def test_inert_dropout_is_fused_and_live_dropout_is_not():
    from fastmoe_b200.transformer import activation_kind
    seq = torch.nn.Sequential(torch.nn.ReLU(), torch.nn.Dropout(0.5))
    assert activation_kind(seq) is None and activation_kind(seq.eval()) == "relu"
    assert activation_kind(torch.nn.Sequential(torch.nn.ReLU(), torch.nn.Dropout(0.0))) == "relu"
    assert activation_kind(torch.nn.Sequential(torch.nn.ReLU(), torch.nn.Tanh()).eval()) is None
    seq[0].register_forward_hook(lambda *a: None)
    assert activation_kind(seq) is None


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("act", [None, "gelu", "relu", "gelu_tanh"])
@pytest.mark.parametrize("counts,k,n", [
    ([1, 0, 2, 0, 0, 0], 64, 32),              # one K block, a quarter of a tile's columns
    ([0] * 6 + [32, 0], 128, 288),             # exactly one tile of rows, a ragged last column tile
    ([33, 0, 0, 31] + [0] * 60, 1024, 416),    # a second row tile with one row, ring longer than the K blocks
    ([65] + [0] * 9, 4096, 128),               # three row tiles of one expert
])
def test_narrow_kernel(dtype, act, counts, k, n):
    r"""A handful of rows per expert, nothing saved: against fp64, one rounding to the 16-bit type, an
    fp32 sum of k terms and, for the tanh form, the hardware tanh (2^-10.9)."""
    from fastmoe_b200.ops import grouped_gemm as gg
    torch.manual_seed(18)
    g, rows = len(counts), sum(counts)
    assert rows <= 16 * g
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    offs = _offs(counts)
    x = torch.randn(rows, k, device=DEV).to(dtype)
    w = (torch.randn(g, n, k, device=DEV) / k ** 0.5).to(dtype)
    b = torch.randn(g, n, device=DEV).to(dtype)
    fn = {None: lambda t: t, "relu": torch.relu, "gelu": torch.nn.functional.gelu,
          "gelu_tanh": lambda t: torch.nn.functional.gelu(t, approximate="tanh")}[act]
    for bias in (b, None):
        y = gg.forward(x, w, offs, bias, act=act)
        for e, lo, hi in _segments(counts):
            pre = x[lo:hi].double() @ w[e].double().t() + (0 if bias is None else bias[e].double())
            ref = fn(pre)
            bound = eps * ref.abs() + 2.0 ** -22 * k ** 0.5 * 8 + (2.0 ** -11 * pre.abs() if act == "gelu_tanh" else 0) + 1e-6
            assert ((y[lo:hi].double() - ref).abs() <= bound).all(), e
    assert _native().read_status(0) == 0
