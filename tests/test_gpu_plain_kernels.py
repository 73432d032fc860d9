"""The kernels of the 32-bit path at the edges of their tiles, against float64, and bit for bit between their forms.

A product's tile follows the number of rows (4, 16, 32, 64 rows), the way its operands are loaded their alignment; a row's
attention may be shared by a cluster of blocks. None of that may move a bit of a row's result."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from jllm_serve_b200.csrc import ops as o
    o.require_device()
    return o


def rnd(*shape, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(DEV)


@pytest.mark.parametrize("N,K", [(1, 1), (63, 12), (65, 36), (127, 515), (129, 1028), (300, 4096), (72, 12292)])
def test_product_of_every_tile_and_loader(ops, N, K):
    """Rows 1 to 150 run through all four tiles; the same operands in rows of another stride through the other loader."""
    a, w, bias = rnd(150, K), rnd(N, K, seed=1), rnd(N, seed=2)
    want = a.double() @ w.double().T + bias.double()
    # two chains of K / 8 rounded products and sums per group, five more sums: |error| <= (K / 8 + 7) 2^-24 sum |a| |w|
    bound = (K / 8 + 7) * 2.0 ** -24 * (a.abs().double() @ w.abs().double().T + bias.abs().double())
    full = torch.empty(150, N, device=DEV)
    ops.gemm_plain(a, w, full, bias)
    assert bool(((full.double() - want).abs() <= bound).all())
    for M in (1, 3, 4, 5, 16, 17, 32, 33, 64, 65, 96, 97, 128, 129):
        out = torch.full((M + 1, N + 3), 7.0, device=DEV)
        ops.gemm_plain(a[150 - M:], w, out[:M, :N], bias)
        assert torch.equal(out[:M, :N], full[150 - M:]), M
        assert float((out[M] - 7).abs().max()) == 0 and float((out[:, N:] - 7).abs().max()) == 0
    odd_a, odd_w = torch.zeros(150, K + 1, device=DEV), torch.zeros(N, K + 3, device=DEV)
    odd_a[:, :K], odd_w[:, :K] = a, w
    for M in (2, 16, 30, 150):
        out = torch.empty(M, N, device=DEV)
        ops.gemm_plain(odd_a[:M, :K], odd_w[:, :K], out, bias)
        assert torch.equal(out, full[:M]), M


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N,K", [(100, 1), (100, 7), (129, 32), (3, 100), (100, 128), (130, 129)])
def test_product_of_a_short_k(ops, dtype, N, K):
    """Groups of few or no k; products whose 16-row tiles are on the SMs at once (70 rows) and larger ones (2,560). Bias, residual,
    bfloat16 results, operands in rows of another stride: a row has the same bits in all of them."""
    M, few = 16 * 160, 70
    a, w, bias = rnd(M, K).to(dtype), rnd(N, K, seed=1).to(dtype), rnd(N, seed=2)
    base = rnd(M, N, seed=3)
    full, part = base.clone(), torch.full((few + 1, N + 3), 7.0, device=DEV)
    part[:few, :N] = base[:few]
    ops.gemm_plain(a, w, full, bias, accumulate=True)
    ops.gemm_plain(a[:few], w, part[:few, :N], bias, accumulate=True)
    assert torch.equal(part[:few, :N], full[:few]) and bool((part[few] == 7).all()) and bool((part[:, N:] == 7).all())
    want = a.double() @ w.double().T + bias.double() + base.double()
    bound = (K / 8 + 8) * 2.0 ** -24 * (a.abs().double() @ w.abs().double().T + bias.abs().double() + base.abs().double())
    assert bool(((full.double() - want).abs() <= bound).all())
    odd_a, odd_w = torch.zeros(M, K + 1, device=DEV, dtype=dtype), torch.zeros(N, K + 3, device=DEV, dtype=dtype)
    odd_a[:, :K], odd_w[:, :K] = a, w
    for rows in (1, few, M):
        out = base[:rows].clone()
        ops.gemm_plain(odd_a[:rows, :K], odd_w[:, :K], out, bias, accumulate=True)
        assert torch.equal(out, full[:rows]), rows
    if dtype == torch.bfloat16:
        out, many = torch.empty(few, N, device=DEV, dtype=dtype), torch.empty(M, N, device=DEV, dtype=dtype)
        ops.gemm_plain(a[:few], w, out)
        ops.gemm_plain(a, w, many)
        assert torch.equal(out, many[:few])


@pytest.mark.parametrize("N,K", [(65, 515), (129, 1028), (300, 333)])
def test_product_of_bfloat16_operands(ops, N, K):
    """The loader by way of registers, four values at a time and value by value, in all tiles: the bits of the float32 loader."""
    a, w = rnd(150, K).bfloat16(), rnd(N, K, seed=1).bfloat16()
    odd_a, odd_w = torch.zeros(150, K + 1, device=DEV, dtype=torch.bfloat16), torch.zeros(N, K + 3, device=DEV, dtype=torch.bfloat16)
    odd_a[:, :K], odd_w[:, :K] = a, w
    want = torch.empty(150, N, device=DEV)
    ops.gemm_plain(a.float(), w.float(), want)
    for M in (1, 4, 5, 16, 17, 33, 64, 97, 150):
        out, odd = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
        ops.gemm_plain(a[:M], w, out)
        ops.gemm_plain(odd_a[:M, :K], odd_w[:, :K], odd)
        assert torch.equal(out, want[:M]) and torch.equal(odd, want[:M]), M


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,dk,dv,window,keep", [(4, 4, 16, 16, 0, 0), (8, 2, 128, 128, 0, 0), (6, 1, 50, 140, 0, 0), (5, 1, 260, 300, 0, 0),
                                                   (6, 3, 72, 64, 70, 9), (4, 1, 64, 64, -96, 0)])
def test_attention_of_shared_rows(ops, dtype, H, G, dk, dv, window, keep):
    """Lengths around a chunk of 64 keys and around the eight that a cluster takes at a time; one row alone (a cluster to a
    row) has the bits it has among many (a block to a row)."""
    page, width, scale = 8, max(dk, dv), 1.0 / math.sqrt(dk)
    lens = [1, 63, 64, 65, 511, 512, 513, 700]
    blocks = -(-max(lens) // page)
    pool = len(lens) * blocks
    order = torch.randperm(pool, generator=torch.Generator().manual_seed(5)).int()
    tables = order.view(len(lens), blocks).to(DEV)
    k, v = rnd(pool, G, page, width, seed=1).to(dtype), rnd(pool, G, page, width, seed=2).to(dtype)
    sink = rnd(H, seed=3) if keep else None
    rows = [(s, p) for s, n in enumerate(lens) for p in sorted({n - 1, max(0, n - 7)})] * 24
    q = rnd(len(rows), H * dk, seed=4).to(dtype)
    seg = torch.tensor([s for s, _ in rows], dtype=torch.int32, device=DEV)
    pos = torch.tensor([p for _, p in rows], dtype=torch.int32, device=DEV)

    def run(lo, hi):
        out = torch.full((hi - lo, H * dv), float("nan"), dtype=dtype, device=DEV)
        ops.attention_plain(q[lo:hi], H * dk, k, v, out, seg[lo:hi], pos[lo:hi], tables, hi - lo, H, G, dk, page, window, scale, dv,
                            keep, sink)
        return out

    full = run(0, len(rows))
    for i, (s, p) in enumerate(rows[:len(rows) // 24]):
        assert torch.equal(run(i, i + 1)[0], full[i]), (s, p)
        at = torch.arange(p + 1, device=DEV)
        first = max(0, p + 1 - window) if window > 0 else p - p % -window if window < 0 else 0
        at = at[(at >= first) | (at < keep)]
        keys, values = (t[tables[s][at // page].long(), :, at % page].double() for t in (k[..., :dk], v[..., :dv]))
        x = torch.einsum("hd,jhd->hj", q[i].double().view(H, dk), keys.repeat_interleave(H // G, dim=1)) * scale
        if sink is not None:
            x = torch.cat([x, sink.double()[:, None]], dim=1)
        want = torch.einsum("hj,jhd->hd", torch.softmax(x, dim=1)[:, :len(at)], values.repeat_interleave(H // G, dim=1))
        # scores within about dk 2^-24 |q||k| scale, exponentials within a few 2^-24 of themselves, sums of 64 products
        tol = 2e-5 if dtype == torch.float32 else 2.0 ** -8
        assert float((full[i].double().view(H, dv) - want).abs().max()) <= tol * float(values.abs().max()), (s, p)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("copies", [1, 160])
@pytest.mark.parametrize("with_sink", [False, True])
def test_attention_keeps_what_is_not_a_number(ops, dtype, copies, with_sink):
    """A row of 65 keys, so that key 64 is a chunk of its own, in a cluster's form (one row) and in a block's (160 rows): a key that is
    NaN makes the row's heads NaN, a query head that is NaN itself alone (beside a sink too), and a key whose score is -inf only
    drops out: the result is, bit for bit, that of a score far below the others."""
    H, G, d, page, n = 4, 2, 64, 16, 65
    k, v = rnd(5, G, page, d, seed=1).to(dtype), rnd(5, G, page, d, seed=2).to(dtype)
    q = rnd(1, H * d, seed=3).abs().to(dtype)
    table = torch.arange(5, dtype=torch.int32, device=DEV).view(1, 5)
    seg, pos = torch.zeros(copies, dtype=torch.int32, device=DEV), torch.full((copies,), n - 1, dtype=torch.int32, device=DEV)
    sink = rnd(H, seed=4) if with_sink else None

    def run(q, k):
        out = torch.full((copies, H * d), 7.0, dtype=dtype, device=DEV)
        ops.attention_plain(q.expand(copies, -1).contiguous(), H * d, k, v, out, seg, pos, table, copies, H, G, d, page, 0, 0.125, sink=sink)
        assert bool((out == out[:1]).all() or (out.isnan() == out[:1].isnan()).all())
        return out[0].view(H, d)

    whole = run(q, k)
    assert bool(whole.isfinite().all())
    bad = k.clone()
    bad[4, 0, 0] = float("nan")                    # key 64 of the first kv head
    got = run(q, bad)
    assert bool(got[:2].isnan().all()) and torch.equal(got[2:], whole[2:])
    bad[4, 0, 0], bad[4, 0, 0, 5] = k[4, 0, 0], float("-inf")
    low = k.clone()
    low[4, 0, 0] = -1e4
    got, want = run(q, bad), run(q, low)
    assert bool(want.isfinite().all()) and torch.equal(got, want)
    bad_q = q.clone()
    bad_q[0, d + 3] = float("nan")                 # the second head
    got = run(bad_q, k)
    assert bool(got[1].isnan().all()) and torch.equal(got[[0, 2, 3]], whole[[0, 2, 3]])
