r"""GPU tier: the grouped GEMM with the token rows on the N side, at the edges of its tiles, and the rule
that chooses among the row-mode kernels."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"
ACTS = {None: lambda x: x, "relu": torch.relu, "gelu": torch.nn.functional.gelu,
        "gelu_tanh": lambda x: torch.nn.functional.gelu(x, approximate="tanh")}


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("act", [None, "relu", "gelu", "gelu_tanh"])
@pytest.mark.parametrize("counts,k,n", [
    ([1, 0, 31], 64, 32),                          # one 64-row step, half of a pair's first quarter
    ([33, 63, 64, 65], 192, 96),                   # either side of a step; columns that are no multiple of 64
    ([127, 128, 129, 0, 191, 192, 193], 128, 256),  # 128, 192 and 256 rows in the MMA
    ([255, 256, 257, 300, 1], 64, 544),            # a second tile of one step; a third column tile
    ([20] * 70, 64, 288),                          # more tiles than pairs
    ([3] * 40, 64, 64),                            # up to 16 rows per expert
    ([1300, 5, 900], 128, 288),                    # many rows: the derivative in the 256-row tiles
])
def test_row_modes_at_tile_edges(dtype, act, counts, k, n):
    r"""Against fp64 on the same 16-bit inputs: a rounding to the 16-bit type (the derivative takes the
    rounded pre-activation), an fp32 sum of k terms, and the activation's own error of a few 2^-22 (tanh:
    2^-10).  The rows behind the last expert are NaN and reach nothing; outputs there stay as they are."""
    from fastmoe_b200.ops import grouped_gemm as gg, native
    torch.manual_seed(len(counts) + k + n)
    rows, groups, tail = sum(counts), len(counts), 3
    offs = gg.offsets_from_counts(counts, DEV)
    x = torch.randn(rows + tail, k, device=DEV, dtype=dtype)
    x[rows:] = float("nan")
    w = (torch.randn(groups, n, k, device=DEV) / k ** 0.5).to(dtype)
    wt = (torch.randn(groups, k, n, device=DEV) / k ** 0.5).to(dtype)
    b = torch.randn(groups, n, device=DEV).to(dtype)
    y, pre = gg.forward(x, w, offs, b, act=act, want_pre=True)
    plain = gg.forward(x, w, offs, b, act=act)
    flat = pre if act is None else gg.untile_pre(pre, offs, n, rows + tail)
    dx = gg.dgrad(x, wt, offs, pre=pre if act else None, act=act)
    eps, tanh = torch.finfo(dtype).eps, 2.0 ** -9 if act == "gelu_tanh" else 0.0
    base = 0
    for e, c in enumerate(counts):
        s = slice(base, base + c)
        base += c
        X = x[s].double()
        ref = X @ w[e].double().t() + b[e].double()
        size = X.abs() @ w[e].double().abs().t() + b[e].double().abs()
        err = k * 2.0 ** -24 * size
        assert bool(((flat[s].double() - ref).abs() <= eps * ref.abs() + err + 1e-7).all())
        want = ACTS[act](ref)
        assert bool(((y[s].double() - want).abs() <= eps * want.abs() + 1.2 * err + (2.0 ** -21 + tanh) * (1 + ref.abs())).all())
        assert torch.equal(plain[s], y[s])
        g = X @ wt[e].double()
        size = X.abs() @ wt[e].double().abs()
        p = flat[s].double().requires_grad_(True)
        ACTS[act](p).sum().backward()
        d = p.grad
        bound = eps * (g * d).abs() + 1.2 * k * 2.0 ** -24 * size + (2.0 ** -20 + 4 * tanh) * g.abs() + 1e-7
        assert bool(((dx[s].double() - g * d).abs() <= bound).all())
    assert native.get().read_status(0) == 0


def test_single_group_without_offsets():
    from fastmoe_b200.ops import grouped_gemm as gg
    torch.manual_seed(0)
    x = torch.randn(333, 128, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(1, 64, 128, device=DEV, dtype=torch.bfloat16) * 0.1
    ref = x.double() @ w[0].double().t()
    assert (gg.forward(x, w, None).double() - ref).abs().max() <= 2.0 ** -8 * ref.abs().max()
    ref = x[:, :64].double() @ w[0].double()
    assert (gg.dgrad(x[:, :64].contiguous(), w, None).double() - ref).abs().max() <= 2.0 ** -8 * ref.abs().max()


# the last MMA step of 16 rows full, all but full, of one row, alone; sums by the side warps and, where those
# would take longer than the tiles (12 experts), by the epilogue; widths that end inside a tile, a 64-wide box and a block of 32 columns
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("counts", [[1], [15, 0, 16, 17, 31], [63, 64, 65, 2, 81], [375] * 6, [300] * 12, [2047, 2048, 2049, 5], [0, 0, 7]])
@pytest.mark.parametrize("m,n", [(8, 32), (264, 96), (520, 288), (1024, 256)])
def test_weight_gradient_of_ragged_experts(dtype, counts, m, n):
    r"""Against 64 bits: one rounding to the type and fp32 sums of `rows` products; the neighbours' rows, infinite
    here, take no part."""
    from fastmoe_b200.ops import grouped_gemm as gg
    torch.manual_seed(len(counts) + m)
    rows = sum(counts)
    dy = torch.randn(rows + 20, m, device=DEV, dtype=dtype)
    x = torch.randn(rows + 20, n, device=DEV, dtype=dtype)
    dy[rows:], x[rows:] = float("inf"), float("nan")   # past the last expert
    offs = gg.offsets_from_counts(counts, DEV)
    starts = [sum(counts[:e]) for e in range(len(counts))]
    poisoned = max(range(len(counts)), key=lambda e: (counts[e] > 0, e))
    dy[starts[poisoned], 0] = float("inf")
    dw, db = gg.wgrad(dy, x, offs, len(counts), with_bias_grad=True)
    grown = torch.ones_like(dw)
    gg.wgrad(dy, x, offs, len(counts), out=grown, accumulate=True)
    eps, u = torch.finfo(dtype).eps, 2.0 ** -24
    for e, c in enumerate(counts):
        p, q = dy[starts[e]:starts[e] + c].double(), x[starts[e]:starts[e] + c].double()
        if e == poisoned:
            p = p[:, 1:]
        ref, size = p.t() @ q, p.abs().t() @ q.abs()
        got, more, sums = (t[e].double()[1:] if e == poisoned else t[e].double() for t in (dw, grown, db))
        assert bool(((got - ref).abs() <= eps * ref.abs() + (c + 1) * u * size + 1e-7).all()), e
        assert bool(((more - 1 - ref).abs() <= eps * (ref.abs() + 1) + (c + 2) * u * (size + 1)).all()), e
        assert bool(((sums - p.sum(0)).abs() <= eps * p.sum(0).abs() + (c + 1) * u * p.abs().sum(0) + 1e-7).all()), e
