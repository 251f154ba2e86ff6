"""Each kernel alone against a plain float32 reference of the same operation, at sizes that are
not the engine's: widths and vocabularies that are no power of two, head sizes in steps of 16,
odd numbers of heads and groups, rows that do not fill a tile."""

import math

import numpy as np
import pytest
import torch

from plain import plain_llama

pytestmark = pytest.mark.gpu

DTYPES = [torch.float32, torch.bfloat16]


def tol(dtype):
    return 2e-6 if dtype == torch.float32 else 1e-2


def close(actual, expected, dtype, scale=None):
    actual, expected = actual.double().cpu(), expected.double().cpu()
    bound = tol(dtype) * (scale if scale is not None else float(expected.abs().max().clamp_min(1e-30)))
    worst = float((actual - expected).abs().max())
    assert worst <= bound, f"max abs error {worst} > {bound}"


@pytest.mark.parametrize("dtype", DTYPES)
def test_embed_gather(cuda_device, dtype):
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(0)
    table = torch.randn(203, 72, generator=g).to(dtype)
    tokens = torch.tensor([0, 202, 5, 5, 17], dtype=torch.int32)
    out = ops.embed_gather(table.cuda(), tokens.cuda(), scale=1.5)
    assert out.dtype == torch.float32
    close(out, table.float()[tokens.long()] * 1.5, torch.float32)


@pytest.mark.parametrize("out_dtype", DTYPES)
@pytest.mark.parametrize("width,count", [(72, 7), (2048, 7), (5000, 7), (72, 300), (264, 300), (1028, 261), (2048, 300),
                                         (3080, 259), (4096, 257), (5000, 260)])
def test_add_rmsnorm(cuda_device, out_dtype, width, count):
    """Few rows: a block per row; from 256 rows on, a warp per row (widths up to 4,096)."""
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(1)
    x = torch.randn(count, width, generator=g) * 3
    delta = (torch.randn(count, width, generator=g)).to(out_dtype)
    weight = 1 + 0.1 * torch.randn(width, generator=g)
    eps = 3e-6
    xd = x.cuda()
    out = ops.add_rmsnorm(xd, delta.cuda(), weight.cuda(), eps, out_dtype)
    summed = x + delta.float()
    close(xd, summed, torch.float32)
    close(out, plain_llama.rms_norm(summed, weight, eps), out_dtype)
    # without a delta, on chosen rows, x untouched
    rows = torch.tensor([6, 0, 3], dtype=torch.int32) if count < 256 else torch.randperm(count, generator=g)[:257].int()
    before = xd.clone()
    out = ops.add_rmsnorm(xd, None, weight.cuda(), eps, out_dtype, rows=rows.cuda())
    assert torch.equal(before, xd)
    close(out, plain_llama.rms_norm(summed[rows.long()], weight, eps), out_dtype)
    # a delta on chosen rows is added for the norm only
    out = ops.add_rmsnorm(xd, delta.cuda(), weight.cuda(), eps, out_dtype, rows=rows.cuda())
    assert torch.equal(before, xd)
    close(out, plain_llama.rms_norm((summed + delta.float())[rows.long()], weight, eps), out_dtype)


@pytest.mark.parametrize("m,n,k", [(1, 72, 40), (5, 203, 136), (70, 130, 97), (130, 64, 256)])
def test_gemm_f32(cuda_device, m, n, k):
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(2)
    a, w = torch.randn(m, k, generator=g), torch.randn(n, k, generator=g)
    expected = (a.double() @ w.double().t())
    outs = []
    for invariant in (True, False):
        out = ops.gemm_f32(a.cuda(), w.cuda(), row_invariant=invariant)
        close(out, expected, torch.float32, scale=float(expected.abs().max()) * 4)
        outs.append(out)
    assert torch.equal(*outs)  # every product is row-invariant
    # a row's result does not depend on the other rows of the call
    alone = ops.gemm_f32(a[:1].cuda(), w.cuda(), row_invariant=True)
    together = ops.gemm_f32(a.cuda(), w.cuda(), row_invariant=True)
    assert torch.equal(alone[0], together[0])


@pytest.mark.parametrize("m,n,k", [(1, 68, 32), (3, 8200, 260), (8, 64, 1024), (9, 130, 1028), (33, 2052, 2044), (65, 8200, 516), (130, 20000, 512)])
def test_gemm_f32_rows_of_pieces(cuda_device, m, n, k):
    """Rows of whole 16-byte pieces: parts of K, edges of tiles, few rows; row strides beyond the rows."""
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(12)
    a, w = torch.randn(m, k + 4, generator=g).cuda()[:, :k], torch.randn(n, k + 8, generator=g).cuda()[:, :k]
    out = ops.gemm_f32(a, w)
    # what test_gemm_f32_sums_of_one_sign derives is below this for every k here
    bound = 2.0 ** -24 * k * (a.abs().double() @ w.abs().double().t())
    assert bool(((out.double() - a.double() @ w.double().t()).abs() <= bound).all())
    for rows in (1, 3, 9, 33):
        if rows < m:
            assert torch.equal(ops.gemm_f32(a[:rows], w), out[:rows])  # whichever kernel and tile a row meets


@pytest.mark.parametrize("weights", ["floats", "bfloat16", "mixed"])
@pytest.mark.parametrize("m,n,k", [(161, 129, 640), (321, 65, 63), (200, 5000, 576), (2049, 130, 1088)])
def test_gemm_f32_gives_a_row_the_same_bits_in_every_kernel(cuda_device, weights, m, n, k):
    """Up to 4 rows, up to 32, and tiles of 64 to 160; more rows than are split at once; weights whose smaller parts are zero, are
    not, and are in some tiles."""
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(m + n)
    a, w = torch.randn(m, k, generator=g).cuda(), torch.randn(n, k, generator=g).cuda()
    if weights != "floats":
        rounded = w.bfloat16().float()
        w = rounded if weights == "bfloat16" else torch.where(torch.arange(n, device=cuda_device)[:, None] == 70 % n, w, rounded)
    out = ops.gemm_f32(a, w)
    exact = a.double() @ w.double().t()
    # the sums of the roundings' products and their float additions; what is dropped (2^-24) and what the small products' sum loses
    # (2^-31 k at most, see test_gemm_f32_sums_of_one_sign) is far from all of one sign here
    bound = (2.0 ** -21 + (k / 64 + 8) * 2.0 ** -24) * (a.abs().double() @ w.abs().double().t())
    assert bool(((out.double() - exact).abs() <= bound).all())
    for rows in (1, 4, 5, 32, 33, 65, 97, 129, 160, 161):
        for first in {0, m - rows}:
            if 0 <= first:
                assert torch.equal(ops.gemm_f32(a[first:first + rows], w), out[first:first + rows])
    assert ops.gemm_f32_status() == 0


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3.4e38])
@pytest.mark.parametrize("m", [3, 20, 70, 200])
def test_gemm_f32_keeps_rows_that_are_not_finite_apart(cuda_device, m, value):
    """A float without three finite parts, in a row of A and in one of W: their results are those of the floats, all others stay."""
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(m)
    a, w = torch.randn(m, 1088, generator=g).cuda(), (torch.randn(200, 1088, generator=g) * 0.01).cuda()
    a[:, 3] *= 0.1  # (so that products with the largest value stay within the floats)
    before = ops.gemm_f32(a, w)
    a2, w2 = a.clone(), w.clone()
    a2[2, 700] = value
    w2[130, 3] = value
    w2[17, 700] = 0.0
    before[:, 17] = ops.gemm_f32(a, w2)[:, 17]
    got, want = ops.gemm_f32(a2, w2).cpu(), (a2.double() @ w2.double().t()).cpu()
    rows, columns = torch.arange(m) == 2, torch.arange(200) == 130
    hit = rows[:, None] | columns[None]
    assert torch.equal(got[~hit], before.cpu()[~hit])
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    for x, y in zip(got[hit].tolist(), want[hit].tolist()):
        if abs(y) == float("inf"):
            assert x == y
        elif y == y:
            assert abs(x - y) <= 1e-5 * abs(y) + 1e-4


@pytest.mark.parametrize("m", [3, 20, 70, 200])
def test_gemm_f32_overflows_as_floats_do(cuda_device, m):
    """Finite operands whose products pass the largest float by far: infinite where the float sum is, whatever signs the smaller parts have."""
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(m)
    a, w = torch.randn(m, 1088, generator=g), torch.randn(200, 1088, generator=g)
    a[2, 700], w[:, 700] = 2.5e30, 3.1e30 * (1 + torch.rand(200, generator=g))
    w[100:, 700] *= -1
    a[1, 30], w[150:, 30] = -2.2e25, 1.7e25  # (other results stay finite beside them)
    got, want = ops.gemm_f32(a.cuda(), w.cuda()).cpu(), (a.double() @ w.double().t()).float()
    assert torch.equal(got[2], want[2]) and bool(torch.isinf(want[2]).all())
    assert torch.equal(torch.isinf(got), torch.isinf(want)) and torch.equal(got[torch.isinf(want)], want[torch.isinf(want)])
    assert bool(torch.isfinite(got[torch.isfinite(want)]).all())
    assert bool(((got.double() - want.double()).abs() <= 1e-5 * (a.abs().double() @ w.abs().double().t()))[torch.isfinite(want)].all())


@pytest.mark.parametrize("value", [1e36, 1.5e37, 5e37])
@pytest.mark.parametrize("side", ["a", "w"])
def test_gemm_f32_gives_rows_of_large_floats_the_same_bits(cuda_device, side, value):
    """Whether results are computed anew from the floats is decided by the results, which are the same in every kernel."""
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(17)
    a, w = torch.randn(161, 1088, generator=g).cuda(), torch.randn(200, 1088, generator=g).cuda()
    large, small = (a, w) if side == "a" else (w, a)
    large[0] = value
    large[3] = value * torch.rand(1088, generator=g).cuda()
    large[:, 8:16] = value  # eight neighbours of every row
    small *= 1e-4
    out = ops.gemm_f32(a, w)
    assert bool(torch.isfinite(out).all())
    for rows in (1, 4, 5, 8, 32, 33, 64, 160):
        assert torch.equal(ops.gemm_f32(a[:rows], w), out[:rows])


@pytest.mark.parametrize("size", [1e-33, 1e-36, 1e-37, 1e-41])
@pytest.mark.parametrize("m", [3, 20, 70])
def test_gemm_f32_multiplies_every_bit_of_small_floats(cuda_device, m, size):
    """Operands down to those below the normal floats beside large ones: the bound of test_gemm_f32_gives_a_row_the_same_bits_in_every_kernel."""
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(m)
    for small in (0, 1):
        a, w = torch.randn(m, 640, generator=g), torch.randn(130, 640, generator=g)
        (a, w)[small].mul_(size)
        (a, w)[1 - small].mul_(1e25)
        exact = a.double() @ w.double().t()
        bound = (2.0 ** -21 + (640 / 64 + 8) * 2.0 ** -24) * (a.abs().double() @ w.abs().double().t())
        assert bool(((ops.gemm_f32(a.cuda(), w.cuda()).double().cpu() - exact).abs() <= bound).all())


@pytest.mark.parametrize("m", [3, 7, 20, 70])
@pytest.mark.parametrize("k", [4, 32, 36, 60, 68, 132, 164, 1100])
def test_gemm_f32_rows_that_end_within_a_stage(cuda_device, m, k):
    """What lies behind the last column is not a number, and so is a float of one row: neither reaches another result."""
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(k)
    wide_a, wide_w = torch.full((m, k + 64), float("nan")), torch.full((200, k + 64), float("nan"))
    wide_a[:, :k], wide_w[:, :k] = torch.randn(m, k, generator=g), torch.randn(200, k, generator=g)
    a, w = wide_a.cuda()[:, :k], wide_w.cuda()[:, :k]
    exact = wide_a[:, :k].double() @ wide_w[:, :k].double().t()
    bound = (2.0 ** -21 + (k / 64 + 8) * 2.0 ** -24) * (wide_a[:, :k].abs().double() @ wide_w[:, :k].abs().double().t())
    out = ops.gemm_f32(a, w)
    assert bool(((out.double().cpu() - exact).abs() <= bound).all())
    w[5, k // 2], w[9, 0] = float("nan"), float("inf")
    again = ops.gemm_f32(a, w)
    others = [i for i in range(200) if i not in (5, 9)]
    assert torch.equal(again[:, others], out[:, others]) and bool(torch.isnan(again[:, 5]).all()) and bool(torch.isinf(again[:, 9]).all())


@pytest.mark.parametrize("weights", ["the float that loses most", "near one"])
@pytest.mark.parametrize("m,n,k", [(2, 130, 2048), (20, 130, 2048), (70, 9480, 8192)])
def test_gemm_f32_sums_of_one_sign(cuda_device, weights, m, n, k):
    """The bound of the split products where nothing cancels.  A float's second part is up to 2^-8 of it, its third up to 2^-17, so that the
    three products left out are up to 2^-24 of the whole; sums of 64 columns of the roundings' products are cut off four times (2^-23
    each) and added with k / 64 + 8 roundings (2^-24 each); the five small products, 2^-7 of the whole together, stay in one sum that is
    cut off 20 times a stage (20 / 64 k 2^-30)."""
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(k)
    if weights == "near one":
        a, w = 1 + torch.rand(m, k, generator=g) * 2.0 ** -7, 1 + torch.rand(n, k, generator=g) * 2.0 ** -7
    else:
        worst = torch.tensor([0x3F807FC0], dtype=torch.int32).view(torch.float32)  # 1 + 2^-8 - 2^-17: parts 1, 2^-8 and -2^-17
        a, w = worst.expand(m, k).contiguous(), worst.expand(n, k).contiguous()
    exact = a.cuda().double() @ w.cuda().double().t()
    bound = 2.0 ** -24 + 2.0 ** -21 + (k / 64 + 8) * 2.0 ** -24 + k * 2.0 ** -31
    assert bool(((ops.gemm_f32(a.cuda(), w.cuda()).double() - exact).abs() <= bound * exact).all())


@pytest.mark.parametrize("n,k", [(5, 64), (300, 100), (2048, 2048), (3076, 2048), (9480, 512), (4100, 516), (9480, 4100), (15000, 132), (40000, 260), (40000, 1900), (37, 8192)])
def test_gemm_f32_few_rows(cuda_device, n, k):
    """Up to eight rows: tiles of W that do and do not fill blocks of 4, 8 and 16 warps, one after another where there are more tiles than
    warps, one to four parts of K, A's parts that leave room for fewer stages; the bits of the kernel that many rows take."""
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(n)
    a, w = torch.randn(40, k, generator=g).cuda(), torch.randn(n, k, generator=g).cuda()
    out = ops.gemm_f32(a, w)
    exact = a.double() @ w.double().t()
    bound = (2.0 ** -21 + (k / 64 + 8) * 2.0 ** -24) * (a.abs().double() @ w.abs().double().t())
    assert bool(((out.double() - exact).abs() <= bound).all())
    for rows in range(1, 9):
        assert torch.equal(ops.gemm_f32(a[:rows], w), out[:rows])
    rounded = w.bfloat16().float()  # (weights with two parts of zeros)
    out = ops.gemm_f32(a, rounded)
    for rows in (1, 4, 8):
        assert torch.equal(ops.gemm_f32(a[:rows], rounded, weights_ready=True), out[:rows])


@pytest.mark.parametrize("m,n,k", [(1, 72, 2048), (5, 200, 260), (40, 130, 1028), (70, 8200, 516), (130, 64, 2048)])
def test_gemm_f32_gives_the_same_bits_off_its_alignment(cuda_device, m, n, k):
    """Operands whose rows do not start on 16 bytes are loaded float by float: the same sums over the same parts of K."""
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(13)
    a, w = torch.randn(m, k, generator=g).cuda(), torch.randn(n, k, generator=g).cuda()
    aligned = ops.gemm_f32(a, w)
    for shifts in ((1, 0), (0, 3), (2, 1)):
        moved = [torch.empty(t.shape[0], k + 4, device=cuda_device)[:, by:by + k] for t, by in zip((a, w), shifts)]
        for to, t in zip(moved, (a, w)):
            to.copy_(t)
        assert torch.equal(ops.gemm_f32(*moved), aligned)


@pytest.mark.parametrize("m,n,k", [(3, 2048, 2048), (20, 2048, 2048), (200, 512, 1088)])
def test_gemm_f32_takes_the_result_of_the_product_before(cuda_device, m, n, k):
    """Products queued one after another, captured, whose second operand is what the one before writes."""
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(m)
    x, z = torch.randn(m, n, generator=g).cuda(), torch.randn(n, k, generator=g).cuda()
    ys = [torch.randn(n, k, generator=g).cuda() for _ in range(3)]
    want = [ops.gemm_f32(x, w) for w in [(torch.cuda.synchronize(), ops.gemm_f32(y, z), torch.cuda.synchronize())[1] for y in ys]]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = [ops.gemm_f32(x, ops.gemm_f32(y, z)) for y in ys]
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype", DTYPES)
def test_swiglu_and_bias(cuda_device, dtype):
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(3)
    gate_up = (torch.randn(5, 2 * 136, generator=g) * 4).to(dtype)
    out = ops.swiglu(gate_up.cuda())
    f = gate_up.float()
    close(out, plain_llama.swiglu(f[:, :136], f[:, 136:]), dtype)
    x = torch.randn(5, 203, generator=g).to(dtype)
    bias = torch.randn(203, generator=g)
    got = ops.bias_add(x.cuda().clone(), bias.cuda())
    close(got, x.float() + bias, dtype)


def _pools(pages, kv_heads, page_size, head_dim, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    k = (torch.randn(pages, kv_heads, page_size, head_dim, generator=g)).to(dtype)
    v = (torch.randn(pages, kv_heads, page_size, head_dim, generator=g)).to(dtype)
    return k, v


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("pairing", ["half", "interleaved"])
@pytest.mark.parametrize("head_dim,rotary_dim", [(16, 16), (48, 48), (64, 32)])
def test_rope_cache_write(cuda_device, dtype, pairing, head_dim, rotary_dim):
    from models_b200.kernels import ops

    heads, kv_heads, page = 3, 2, 64
    tokens = 9
    g = torch.Generator().manual_seed(4)
    width = (heads + 2 * kv_heads) * head_dim
    qkv = torch.randn(tokens, width + 8, generator=g).to(dtype)  # wider rows: the stride is honoured
    positions = torch.tensor([0, 1, 2, 63, 64, 65, 130, 7, 8], dtype=torch.int32)
    freqs = plain_llama.rope_pair_frequencies(rotary_dim, 12345.0)
    cos, sin = plain_llama.rope_cos_sin(torch.arange(200), freqs, None)
    pages = 5
    k_pool, v_pool = _pools(pages, kv_heads, page, head_dim, dtype, 5)
    slot_mapping = torch.tensor([64 * 1 + 0, 64 * 1 + 1, 64 * 1 + 2, 64 * 1 + 63, 64 * 3 + 0, 64 * 3 + 1, 64 * 4 + 2, -1,
                                 64 * 2 + 8], dtype=torch.int32)
    qkv_d, k_d, v_d = qkv.cuda(), k_pool.cuda(), v_pool.cuda()
    view = qkv_d[:, :width]
    ops.rope_cache_write(view, positions.cuda(), cos.cuda(), sin.cuda(), k_d, v_d, slot_mapping.cuda(), heads, kv_heads,
                         head_dim, rotary_dim, pairing == "interleaved", page, True)

    def rotate(x, pos):  # x [T, h, hd] float
        c, s = cos[pos.long()], sin[pos.long()]
        if pairing == "half":
            return plain_llama.rope_rotate_split_half(x, c, s)
        pairs = rotary_dim // 2
        x0, x1 = x[..., 0:rotary_dim:2], x[..., 1:rotary_dim:2]
        r0, r1 = x0 * c[:, None, :] - x1 * s[:, None, :], x0 * s[:, None, :] + x1 * c[:, None, :]
        out = x.clone()
        out[..., 0:rotary_dim:2], out[..., 1:rotary_dim:2] = r0, r1
        return out

    f = qkv.float()[:, :width]
    q = f[:, : heads * head_dim].reshape(tokens, heads, head_dim)
    k = f[:, heads * head_dim:(heads + kv_heads) * head_dim].reshape(tokens, kv_heads, head_dim)
    v = f[:, (heads + kv_heads) * head_dim:].reshape(tokens, kv_heads, head_dim)
    close(qkv_d[:, : heads * head_dim], rotate(q, positions).reshape(tokens, -1), dtype)
    assert torch.equal(qkv_d[:, width:].cpu(), qkv[:, width:])  # columns beyond the heads are untouched
    ek, ev = k_pool.float().clone(), v_pool.float().clone()
    rk = rotate(k, positions)
    for t in range(tokens):
        s = int(slot_mapping[t])
        if s < 0:
            continue
        ek[s // page, :, s % page, :] = rk[t]
        ev[s // page, :, s % page, :] = v[t]
    close(k_d, ek, dtype)
    close(v_d, ev, dtype)


def _reference_attention(q, k_pool, v_pool, block_table, q_lens, kv_lens, heads, kv_heads, head_dim, window, scale):
    """q [T, heads*hd] float; whole-sequence plain attention per sequence, keys gathered from the pages."""
    page = k_pool.shape[2]
    out = torch.zeros(q.shape[0], heads * head_dim)
    row = 0
    for b, (n, total) in enumerate(zip(q_lens, kv_lens)):
        pos = torch.arange(total)
        pages = block_table[b][pos // page].long()
        k = k_pool.float()[pages, :, pos % page, :]  # [total, kv, hd]
        v = v_pool.float()[pages, :, pos % page, :]
        qfull = torch.zeros(total, heads, head_dim)
        qfull[total - n:] = q[row:row + n].reshape(n, heads, head_dim)
        full = plain_llama.causal_gqa_attention(qfull * (scale * math.sqrt(head_dim)), k, v, window)
        out[row:row + n] = full[total - n:]
        row += n
    return out


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads,kv_heads,head_dim,window", [(4, 2, 16, None), (3, 1, 32, None), (6, 3, 48, None),
                                                            (8, 2, 128, None), (5, 5, 80, 37), (4, 1, 64, 64)])
def test_paged_attention_rows(cuda_device, dtype, heads, kv_heads, head_dim, window):
    from models_b200.kernels import ops

    page = 64
    q_lens = [1, 70, 5, 1]
    kv_lens = [1, 70, 133, 200]
    pages_needed = [-(-n // page) for n in kv_lens]
    total_pages = sum(pages_needed) + 1
    k_pool, v_pool = _pools(total_pages, kv_heads, page, head_dim, dtype, 6)
    order = torch.randperm(total_pages - 1, generator=torch.Generator().manual_seed(7)) + 1
    block_table = torch.zeros(len(q_lens), max(pages_needed), dtype=torch.int32)
    at = 0
    for b, n in enumerate(pages_needed):
        block_table[b, :n] = order[at:at + n].int()
        at += n
    T = sum(q_lens)
    g = torch.Generator().manual_seed(8)
    q = torch.randn(T, heads * head_dim + 16, generator=g).to(dtype)
    cu_q = torch.tensor([0] + list(np.cumsum(q_lens)), dtype=torch.int32)
    out = torch.zeros(T, heads * head_dim, dtype=dtype, device="cuda")
    scale = 0.7 / math.sqrt(head_dim)
    ops.paged_attention_rows(q.cuda()[:, : heads * head_dim], out, k_pool.cuda(), v_pool.cuda(), block_table.cuda(),
                             cu_q.cuda(), torch.tensor(kv_lens, dtype=torch.int32).cuda(), max(q_lens), heads, kv_heads,
                             head_dim, window, scale)
    expected = _reference_attention(q.float()[:, : heads * head_dim], k_pool, v_pool, block_table, q_lens, kv_lens, heads,
                                    kv_heads, head_dim, window, scale)
    close(out, expected, dtype)


@pytest.mark.parametrize("heads,kv_heads,head_dim,window", [(8, 2, 64, None), (3, 1, 64, None), (40, 1, 64, 37), (2, 2, 128, None), (6, 2, 128, 70)])
def test_prompt_rows_of_floats_are_the_single_tokens_bits(cuda_device, heads, kv_heads, head_dim, window):
    """Prompts in tiles of 16 rows (heads that do not fill or do not divide one, windows that end in a chunk, cached positions before) against the
    kernel of a warp a row, which single tokens take: the same bits, also beside a later position whose key and value are not finite."""
    from models_b200.kernels import ops

    page = 64
    q_lens, kv_lens = [1, 70, 5, 33], [1, 70, 133, 200]
    pages_needed = [-(-n // page) for n in kv_lens]
    k_pool, v_pool = (t.cuda() for t in _pools(sum(pages_needed) + 1, kv_heads, page, head_dim, torch.float32, 6))
    table, at = torch.zeros(len(q_lens), max(pages_needed), dtype=torch.int32), 1
    for b, n in enumerate(pages_needed):
        table[b, :n] = torch.arange(at, at + n, dtype=torch.int32)
        at += n
    k_pool[1, :, 1:], v_pool[1, :, 1:] = float("nan"), float("nan")  # behind the first sequence's end
    last = int(table[1, 69 // page])
    v_pool[last, :, 69 % page] = float("inf")  # the second sequence's last position: only its last token sees it
    q = torch.randn(sum(q_lens), heads * head_dim, generator=torch.Generator().manual_seed(8)).cuda()
    cu_q = torch.tensor([0] + list(np.cumsum(q_lens)), dtype=torch.int32).cuda()
    out = torch.zeros_like(q)
    ops.paged_attention_rows(q, out, k_pool, v_pool, table.cuda(), cu_q, torch.tensor(kv_lens, dtype=torch.int32).cuda(), max(q_lens), heads,
                             kv_heads, head_dim, window, 0.1)
    singles = [(b, kv_lens[b] - q_lens[b] + i + 1) for b in range(len(q_lens)) for i in range(q_lens[b])]
    alone = torch.zeros_like(q)
    ops.paged_attention_rows(q, alone, k_pool, v_pool, table[[b for b, _ in singles]].contiguous().cuda(),
                             torch.arange(len(singles) + 1, dtype=torch.int32).cuda(),
                             torch.tensor([n for _, n in singles], dtype=torch.int32).cuda(), 1, heads, kv_heads, head_dim, window, 0.1)
    assert torch.equal(out.nan_to_num(nan=7.0), alone.nan_to_num(nan=7.0))
    assert bool(torch.isfinite(out[:70]).all()) and not bool(torch.isfinite(out[70]).all())


@pytest.mark.parametrize("heads,kv_heads,head_dim,window", [(4, 2, 16, None), (3, 1, 32, None), (6, 3, 48, None),
                                                            (32, 8, 64, None), (8, 2, 128, None), (5, 5, 80, 37),
                                                            (4, 1, 64, 64), (40, 2, 64, None), (2, 1, 256, 100)])
def test_tensor_core_attention(cuda_device, heads, kv_heads, head_dim, window):
    """Prefill (unequal new-token counts on top of unequal cached lengths) and decode (one token each,
    with 1, 3 and 16 splits of the keys) against the plain attention."""
    from models_b200.kernels import ops

    dtype, page = torch.bfloat16, 64
    for q_lens, kv_lens in (([1, 70, 5, 64, 130], [1, 70, 133, 200, 130]), ([1, 1, 1, 1], [1, 64, 65, 300])):
        pages_needed = [-(-n // page) for n in kv_lens]
        total_pages = sum(pages_needed) + 1
        k_pool, v_pool = _pools(total_pages, kv_heads, page, head_dim, dtype, 6)
        order = torch.randperm(total_pages - 1, generator=torch.Generator().manual_seed(7)) + 1
        block_table = torch.zeros(len(q_lens), max(pages_needed) + 2, dtype=torch.int32)
        at = 0
        for b, n in enumerate(pages_needed):
            block_table[b, :n] = order[at:at + n].int()
            at += n
        T = sum(q_lens)
        q = torch.randn(T, heads * head_dim + 16, generator=torch.Generator().manual_seed(8)).to(dtype)
        cu_q = torch.tensor([0] + list(np.cumsum(q_lens)), dtype=torch.int32)
        scale = 0.7 / math.sqrt(head_dim)
        expected = _reference_attention(q.float()[:, : heads * head_dim], k_pool, v_pool, block_table, q_lens, kv_lens,
                                        heads, kv_heads, head_dim, window, scale)
        common = (k_pool.cuda(), v_pool.cuda(), block_table.cuda(), cu_q.cuda(), torch.tensor(kv_lens, dtype=torch.int32).cuda())
        qd = q.cuda()[:, : heads * head_dim]
        if max(q_lens) > 1:
            for kernel in ("mma", "tcgen05") if head_dim in (64, 128) else ("mma",):
                out = torch.zeros(T, heads * head_dim, dtype=dtype, device="cuda")
                ops.prefill_attention(qd, out, *common, max(q_lens), heads, kv_heads, head_dim, window, scale, kernel=kernel)
                close(out, expected, dtype)
        else:
            for splits, use_scratch in ((1, False), (2, False), (4, False), (8, False), (3, False), (16, False), (4, True)):
                out = torch.zeros(T, heads * head_dim, dtype=dtype, device="cuda")
                ops.decode_attention(qd, out, *common, heads, kv_heads, head_dim, window, scale, splits, use_scratch)
                close(out, expected, dtype)


@pytest.mark.parametrize("heads,kv_heads,head_dim,window", [(8, 2, 64, None), (3, 3, 128, None), (4, 1, 64, 100),
                                                            (2, 1, 128, 257), (12, 4, 64, 64)])
def test_tcgen05_prefill_attention(cuda_device, heads, kv_heads, head_dim, window):
    """The tcgen05 kernel alone at sizes that turn its rings over several times: many pages per
    block, several 128-row blocks per sequence, new tokens on top of cached ones, a sequence of one
    token beside long ones, pages scattered over the pool."""
    from models_b200.kernels import ops

    dtype, page = torch.bfloat16, 64
    q_lens = [300, 1, 129, 700, 64, 128]
    kv_lens = [300, 50, 500, 700, 449, 128]
    pages_needed = [-(-n // page) for n in kv_lens]
    total_pages = sum(pages_needed) + 3
    k_pool, v_pool = _pools(total_pages, kv_heads, page, head_dim, dtype, 16)
    order = torch.randperm(total_pages - 1, generator=torch.Generator().manual_seed(17)) + 1
    block_table = torch.zeros(len(q_lens), max(pages_needed) + 1, dtype=torch.int32)
    at = 0
    for b, n in enumerate(pages_needed):
        block_table[b, :n] = order[at:at + n].int()
        at += n
    T = sum(q_lens)
    q = torch.randn(T, heads * head_dim + 24, generator=torch.Generator().manual_seed(18)).to(dtype)
    cu_q = torch.tensor([0] + list(np.cumsum(q_lens)), dtype=torch.int32)
    scale = 1.3 / math.sqrt(head_dim)
    expected = _reference_attention(q.float()[:, : heads * head_dim], k_pool, v_pool, block_table, q_lens, kv_lens,
                                    heads, kv_heads, head_dim, window, scale)
    out = torch.full((T, heads * head_dim), 7.0, dtype=dtype, device="cuda")
    ops.prefill_attention(q.cuda()[:, : heads * head_dim], out, k_pool.cuda(), v_pool.cuda(), block_table.cuda(), cu_q.cuda(),
                          torch.tensor(kv_lens, dtype=torch.int32).cuda(), max(q_lens), heads, kv_heads, head_dim, window,
                          scale, kernel="tcgen05")
    torch.cuda.synchronize()
    assert ops.prefill_attention_tcgen05_status(head_dim) == 0
    close(out, expected, dtype)


@pytest.mark.parametrize("head_dim", [64, 128])
def test_tcgen05_prefill_attention_finds_one_far_key(cuda_device, head_dim):
    """One key among 600 stands out.  Every query row at or after it must return that key's value
    row; every row before it sees equal scores and must return the mean of the values it can see."""
    from models_b200.kernels import ops

    heads, kv_heads, page, total, new = 2, 1, 64, 600, 250
    for far in (0, 349, 350, 383, 384, 511, 599):
        k_pool = torch.zeros(11, kv_heads, page, head_dim)
        v_pool = torch.randn(11, kv_heads, page, head_dim, generator=torch.Generator().manual_seed(far))
        table = torch.tensor([[5, 2, 10, 1, 3, 9, 7, 4, 8, 6]], dtype=torch.int32)
        k_pool[table[0, far // page], 0, far % page, :] = 10.0
        q = torch.ones(new, heads * head_dim).bfloat16()
        out = torch.zeros(new, heads * head_dim, device="cuda", dtype=torch.bfloat16)
        ops.prefill_attention(q.cuda(), out, k_pool.bfloat16().cuda(), v_pool.bfloat16().cuda(), table.cuda(),
                              torch.tensor([0, new], dtype=torch.int32).cuda(), torch.tensor([total], dtype=torch.int32).cuda(),
                              new, heads, kv_heads, head_dim, None, 1.0, kernel="tcgen05")
        values = v_pool.bfloat16().float()
        flat = torch.stack([values[table[0, p // page], 0, p % page, :] for p in range(total)])  # [total, hd]
        for row in range(new):
            pos = total - new + row
            want = flat[far] if pos >= far else flat[: pos + 1].mean(dim=0)
            for h in range(heads):
                got = out[row, h * head_dim:(h + 1) * head_dim].float().cpu()
                assert torch.allclose(got, want, atol=2e-2), (far, row, h, float((got - want).abs().max()))


def test_window_edge_and_stale_pages_do_not_leak(cuda_device):
    """The key just outside the window, the positions beyond a sequence's length in its last page, and
    a page that belongs to nobody are all made to attract the query; none may be seen."""
    from models_b200.kernels import ops

    heads, kv_heads, head_dim, page, window = 4, 1, 64, 64, 50
    kv_len = 150
    loud = 30.0
    k_pool = torch.zeros(5, kv_heads, page, head_dim)
    v_pool = torch.zeros(5, kv_heads, page, head_dim)
    k_pool[:] = loud  # every key attracts ...
    v_pool[:] = 1000.0  # ... and would wreck the output
    table = torch.tensor([[2, 4, 1, 0]], dtype=torch.int32)
    first = kv_len - window  # the decode query sits at 149 and sees 100..149
    for p in range(first, kv_len):  # the visible keys are quiet and carry the value 1
        k_pool[table[0, p // page], 0, p % page, :] = 0.0
        v_pool[table[0, p // page], 0, p % page, :] = 1.0
    q = torch.ones(1, heads * head_dim)
    for dtype in (torch.bfloat16, torch.float32):
        args = (k_pool.to(dtype).cuda(), v_pool.to(dtype).cuda(), table.cuda(), torch.tensor([0, 1], dtype=torch.int32).cuda(),
                torch.tensor([kv_len], dtype=torch.int32).cuda())
        out = torch.zeros(1, heads * head_dim, dtype=dtype, device="cuda")
        ops.paged_attention_rows(q.to(dtype).cuda(), out, *args, 1, heads, kv_heads, head_dim, window, 1.0)
        assert torch.allclose(out.float().cpu(), torch.ones(1, heads * head_dim)), dtype
        if dtype == torch.bfloat16:
            for splits in (1, 2, 4):
                out = torch.zeros(1, heads * head_dim, dtype=dtype, device="cuda")
                ops.decode_attention(q.to(dtype).cuda(), out, *args, heads, kv_heads, head_dim, window, 1.0, splits)
                assert torch.allclose(out.float().cpu(), torch.ones(1, heads * head_dim)), splits
            # prefill of the last 3 tokens: each sees its own 50 positions; make 97..99 quiet for them
            for p in range(first - 2, first):
                k_pool[table[0, p // page], 0, p % page, :] = 0.0
                v_pool[table[0, p // page], 0, p % page, :] = 1.0
            args = (k_pool.to(dtype).cuda(), v_pool.to(dtype).cuda()) + args[2:3] + (
                torch.tensor([0, 3], dtype=torch.int32).cuda(), args[4])
            out = torch.zeros(3, heads * head_dim, dtype=dtype, device="cuda")
            ops.prefill_attention(q.to(dtype).cuda().expand(3, -1).contiguous(), out, *args, 3, heads, kv_heads, head_dim,
                                  window, 1.0)
            assert torch.allclose(out.float().cpu(), torch.ones(3, heads * head_dim))


def test_attention_finds_one_far_key(cuda_device):
    """One key among hundreds is made to stand out; the output must be that key's value row."""
    from models_b200.kernels import ops

    heads, kv_heads, head_dim, page = 2, 1, 32, 64
    total = 300
    for far in (0, 63, 64, 191, 299):
        k_pool = torch.zeros(6, kv_heads, page, head_dim)
        v_pool = torch.randn(6, kv_heads, page, head_dim, generator=torch.Generator().manual_seed(far))
        table = torch.tensor([[5, 2, 4, 1, 3]], dtype=torch.int32)
        k_pool[table[0, far // page], 0, far % page, :] = 10.0
        q = torch.ones(1, heads * head_dim)
        out = torch.zeros(1, heads * head_dim, device="cuda")
        ops.paged_attention_rows(q.cuda(), out, k_pool.cuda(), v_pool.cuda(), table.cuda(),
                                 torch.tensor([0, 1], dtype=torch.int32).cuda(),
                                 torch.tensor([total], dtype=torch.int32).cuda(), 1, heads, kv_heads, head_dim, None, 1.0)
        expected = v_pool[table[0, far // page], 0, far % page, :]
        for h in range(heads):
            assert torch.allclose(out[0, h * head_dim:(h + 1) * head_dim].cpu(), expected, atol=1e-5), far
        for splits in (1, 5):
            out16 = torch.zeros(1, heads * head_dim, device="cuda", dtype=torch.bfloat16)
            ops.decode_attention(q.bfloat16().cuda(), out16, k_pool.bfloat16().cuda(), v_pool.bfloat16().cuda(), table.cuda(),
                                 torch.tensor([0, 1], dtype=torch.int32).cuda(),
                                 torch.tensor([total], dtype=torch.int32).cuda(), heads, kv_heads, head_dim, None, 1.0, splits)
            for h in range(heads):
                assert torch.allclose(out16[0, h * head_dim:(h + 1) * head_dim].float().cpu(), expected.bfloat16().float(),
                                      atol=1e-2), (far, splits)


def test_decode_attention_finds_one_far_key_in_a_long_context(cuda_device):
    """5,000 cached positions split over 16 to 64 blocks (partial results through scratch memory): the one
    key that stands out may lie in any split, also the first and the last, and in a split's last page."""
    from models_b200.kernels import ops

    heads, kv_heads, head_dim, page = 8, 2, 64, 64
    total = 5000
    pages = -(-total // page)
    order = torch.randperm(pages, generator=torch.Generator().manual_seed(3)).to(torch.int32) + 1
    table = order.reshape(1, pages)
    for far in (0, 63, 2047, 2048, 3333, 4992, 4999):
        k_pool = torch.zeros(pages + 1, kv_heads, page, head_dim)
        v_pool = torch.randn(pages + 1, kv_heads, page, head_dim, generator=torch.Generator().manual_seed(far))
        k_pool[table[0, far // page], :, far % page, :] = 4.0
        q = torch.ones(1, heads * head_dim)
        for splits in (16, 32, 64):
            assert ops.decode_splits(1, heads, kv_heads, head_dim, total) > 8  # what the engine would choose is of this kind
            out = torch.zeros(1, heads * head_dim, device="cuda", dtype=torch.bfloat16)
            ops.decode_attention(q.bfloat16().cuda(), out, k_pool.bfloat16().cuda(), v_pool.bfloat16().cuda(), table.cuda(),
                                 torch.tensor([0, 1], dtype=torch.int32).cuda(),
                                 torch.tensor([total], dtype=torch.int32).cuda(), heads, kv_heads, head_dim, None, 1.0, splits)
            for h in range(heads):
                expected = v_pool[table[0, far // page], h // (heads // kv_heads), far % page, :]
                assert torch.allclose(out[0, h * head_dim:(h + 1) * head_dim].float().cpu(), expected.bfloat16().float(),
                                      atol=1e-2), (far, splits, h)


def test_decode_splits_follow_the_context_class(cuda_device):
    """Short contexts: the split depends on the batch size alone and stays within a cluster.  Long ones:
    more blocks for few sequences, the same count for every length of a class."""
    from models_b200.kernels import ops

    short = ops.decode_splits(1, 32, 8, 64)
    assert short <= 8 and short == ops.decode_splits(1, 32, 8, 64, 1) == ops.decode_splits(1, 32, 8, 64, ops.LONG_KEYS)
    assert ops.decode_span(ops.LONG_KEYS) == 0 and ops.decode_span(ops.LONG_KEYS + 1) == 2 * ops.LONG_KEYS
    assert ops.decode_span(5000) == 8192 and ops.decode_span(8192) == 8192
    for keys in (4097, 5000, 8192):
        assert ops.decode_splits(1, 32, 8, 64, keys) == ops.decode_splits(1, 32, 8, 64, 8192) > 8
    assert ops.decode_splits(1, 32, 8, 64, 32768) == 32
    assert ops.decode_splits(8, 32, 8, 64, 65536) == 32  # 2,048 blocks at most
    assert ops.decode_splits(64, 32, 8, 64, 16384) <= 8
    assert ops.decode_splits(1, 32, 8, 64, 32768, window=512) == short  # a window's few pages need no more blocks


def test_argmax_first_maximum(cuda_device):
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(9)
    logits = torch.randn(5, 5003, generator=g)
    logits[1, 4000] = logits[1, 77] = 50.0  # a tie: the lower id wins
    logits[2, 0] = 60.0
    logits[3, 5002] = 60.0
    got = ops.argmax_rows(logits.cuda()).cpu().tolist()
    assert got == [plain_llama.plain_argmax(row) for row in logits]
    assert got[1] == 77


@pytest.mark.parametrize("batch", [1, 3, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("n,k", [(48, 64), (203, 136), (3072, 2048), (130, 8192)])
def test_skinny_gemm_all_prologues_and_epilogues(cuda_device, batch, n, k):
    """The decode matrix product against float64: plain, with the folded RMSNorm (and a row gather),
    with the residual add, and with the gated activation, at widths that do not fill its tiles."""
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(batch * 1000 + n)
    w = (torch.randn(n, k, generator=g) * 0.05).bfloat16()
    x = torch.randn(batch, k, generator=g).bfloat16()
    wd, xd = w.cuda(), x.cuda()
    exact = x.double() @ w.double().t()
    scale = float(exact.abs().max())
    out = ops.skinny_gemm(wd, ops.EPI_F32, x=xd)
    assert float((out.double().cpu() - exact).abs().max()) < 2e-5 * scale * math.sqrt(k)
    out = ops.skinny_gemm(wd, ops.EPI_BF16, x=xd)
    assert out.dtype == torch.bfloat16 and float((out.double().cpu() - exact).abs().max()) < 1e-2 * scale
    residual = torch.randn(batch, n, generator=g)
    rd = residual.cuda()
    ops.skinny_gemm(wd, ops.EPI_RESIDUAL, x=xd, out=rd)
    assert float((rd.double().cpu() - (residual.double() + exact)).abs().max()) < 2e-5 * (scale + 4) * math.sqrt(k)
    if n % 2 == 0:
        gated = ops.skinny_gemm(wd, ops.EPI_SWIGLU, x=xd)
        want = plain_llama.swiglu(exact[:, : n // 2], exact[:, n // 2:])
        assert gated.shape == (batch, n // 2)
        assert float((gated.double().cpu() - want).abs().max()) < 1e-2 * float(want.abs().max())
    if batch <= 16:
        rows_total = batch + 3
        xf = torch.randn(rows_total, k, generator=g) * 2
        gain = 1 + 0.1 * torch.randn(k, generator=g)
        pick = torch.randperm(rows_total, generator=g)[:batch].int()
        eps = 1e-5
        normed = plain_llama.rms_norm(xf.double(), gain.double(), eps)[pick.long()]
        want = normed @ w.double().t()
        got = ops.skinny_gemm(wd, ops.EPI_F32, xf=xf.cuda(), gain=gain.cuda(), eps=eps, rows=pick.cuda())
        # the normalised rows are rounded to bfloat16 before the product
        assert float((got.double().cpu() - want).abs().max()) < 1e-2 * float(want.abs().max())
        if n % 2 == 0:
            got = ops.skinny_gemm(wd, ops.EPI_SWIGLU, xf=xf.cuda()[:batch].contiguous(), gain=gain.cuda(), eps=eps)
            full = plain_llama.rms_norm(xf.double()[:batch], gain.double(), eps) @ w.double().t()
            want = plain_llama.swiglu(full[:, : n // 2], full[:, n // 2:])
            assert float((got.double().cpu() - want).abs().max()) < 2e-2 * float(want.abs().max())
    else:
        with pytest.raises(ops.KernelError):
            ops.skinny_gemm(wd, ops.EPI_F32, xf=x.float().cuda(), gain=torch.ones(k).cuda(), eps=1e-5)
    with pytest.raises(ops.KernelError):
        ops.skinny_gemm(wd, ops.EPI_F32, x=torch.zeros(33, k, dtype=torch.bfloat16, device="cuda"))


@pytest.mark.parametrize("batch", [1, 5, 16])
@pytest.mark.parametrize("heads,kv_heads,head_dim,hidden", [(4, 2, 16, 64), (3, 1, 32, 96), (32, 8, 64, 2048), (6, 3, 48, 72)])
@pytest.mark.parametrize("prepared", [False, True])
def test_skinny_qkv_with_norm_rotation_and_cache_write(cuda_device, batch, heads, kv_heads, head_dim, hidden, prepared):
    """The folded decode kernel (norm, q/k/v product, rotation, cache write) against the plain parts.
    `prepared`: the rows arrive as x times the gain in bfloat16 with parts of their sums of squares (as the
    product before leaves them) instead of as float32 rows that the kernel normalises itself."""
    from models_b200.kernels import ops

    page = 64
    g = torch.Generator().manual_seed(batch + head_dim)
    n = (heads + 2 * kv_heads) * head_dim
    w = (torch.randn(n, hidden, generator=g) * 0.05).bfloat16()
    xf = torch.randn(batch, hidden, generator=g) * 2
    gain = 1 + 0.1 * torch.randn(hidden, generator=g)
    eps = 1e-5
    positions = torch.randint(0, 300, (batch,), generator=g).int()
    cos, sin = plain_llama.rope_cos_sin(torch.arange(300), plain_llama.rope_pair_frequencies(head_dim, 50000.0), None)
    pages = batch + 2
    k_pool, v_pool = _pools(pages, kv_heads, page, head_dim, torch.bfloat16, 3)
    slots = (torch.randperm(pages - 1, generator=g)[:batch] + 1) * page + torch.randint(0, page, (batch,), generator=g)
    slots = slots.int()
    if batch > 1:
        slots[1] = -1  # a padding row stores nothing
    kd, vd = k_pool.cuda(), v_pool.cuda()
    if prepared:
        squares = (xf.double() ** 2).sum(1)
        share = torch.rand(5, batch, generator=g).double()
        ssq = torch.zeros(7, ops.SSQ_COLUMNS)  # five parts that add up to the rows' sums of squares, two that do not count
        ssq[:5, :batch] = (share / share.sum(0) * squares).float()
        ssq[5:] = 1e6
        q = ops.skinny_qkv_rope(w.cuda(), None, None, 0.0, heads, kv_heads, head_dim, positions.cuda(), cos.cuda(), sin.cuda(),
                                kd, vd, slots.cuda(), x=(xf * gain).bfloat16().cuda(), norm_parts=(ssq.cuda(), 5, hidden, eps))
    else:
        q = ops.skinny_qkv_rope(w.cuda(), xf.cuda(), gain.cuda(), eps, heads, kv_heads, head_dim, positions.cuda(), cos.cuda(),
                                sin.cuda(), kd, vd, slots.cuda())
    qkv = plain_llama.rms_norm(xf, gain, eps) @ w.float().t()
    c, s_ = cos[positions.long()], sin[positions.long()]
    want_q = plain_llama.rope_rotate_split_half(qkv[:, : heads * head_dim].reshape(batch, heads, head_dim), c, s_)
    want_k = plain_llama.rope_rotate_split_half(
        qkv[:, heads * head_dim:(heads + kv_heads) * head_dim].reshape(batch, kv_heads, head_dim), c, s_)
    want_v = qkv[:, (heads + kv_heads) * head_dim:].reshape(batch, kv_heads, head_dim)
    scale = float(qkv.abs().max())
    assert float((q.float().cpu() - want_q.reshape(batch, -1)).abs().max()) < 2e-2 * scale
    ek, ev = k_pool.float().clone(), v_pool.float().clone()
    for b in range(batch):
        slot = int(slots[b])
        if slot >= 0:
            ek[slot // page, :, slot % page, :] = want_k[b]
            ev[slot // page, :, slot % page, :] = want_v[b]
    assert float((kd.float().cpu() - ek).abs().max()) < 2e-2 * max(scale, 4.0)
    assert float((vd.float().cpu() - ev).abs().max()) < 2e-2 * max(scale, 4.0)
    untouched = torch.ones(pages, dtype=torch.bool)
    untouched[[int(x) // page for x in slots if x >= 0]] = False
    assert torch.equal(kd.cpu()[untouched], k_pool[untouched])  # pages of other sequences are left alone


@pytest.mark.parametrize("rows,heads,kv_heads,head_dim,hidden", [(129, 8, 2, 64, 512), (300, 3, 3, 128, 264), (700, 5, 1, 64, 328),
                                                               (257, 2, 2, 128, 1024), (1500, 28, 4, 64, 136)])
def test_tcgen05_qkv_product_with_rotation_and_cache_write(cuda_device, rows, heads, kv_heads, head_dim, hidden):
    """The prefill q/k/v product with rotation and paged cache write in its epilogue against the plain
    parts: head counts that leave the last tile partly empty, rows that do not fill the last row tile,
    padding rows that must store nothing, positions scattered over the table."""
    from models_b200.kernels import ops

    page = 64
    g = torch.Generator().manual_seed(rows + head_dim)
    n = (heads + 2 * kv_heads) * head_dim
    w = (torch.randn(n, hidden, generator=g) * 0.05).bfloat16()
    a = torch.randn(rows, hidden, generator=g).bfloat16()
    positions = torch.randint(0, 900, (rows,), generator=g).int()
    cos, sin = plain_llama.rope_cos_sin(torch.arange(900), plain_llama.rope_pair_frequencies(head_dim, 50000.0), None)
    pages = -(-rows // page) + 3
    k_pool, v_pool = _pools(pages, kv_heads, page, head_dim, torch.bfloat16, 3)
    slots = (torch.randperm((pages - 1) * page, generator=g)[:rows] + page).int()  # distinct cache positions, none in page 0
    slots[1] = -1  # padding rows store nothing
    slots[rows - 1] = -1
    kd, vd = k_pool.cuda(), v_pool.cuda()
    q = ops.gemm_tcgen05_qkv_rope(a.cuda(), w.cuda(), heads, kv_heads, head_dim, positions.cuda(), cos.cuda(), sin.cuda(), kd, vd,
                                  slots.cuda())
    torch.cuda.synchronize()
    assert ops.gemm_tcgen05_status() == 0
    qkv = (a.float() @ w.float().t()).bfloat16().float()  # the product passes through bfloat16 before the rotation
    c, s_ = cos[positions.long()], sin[positions.long()]
    want_q = plain_llama.rope_rotate_split_half(qkv[:, : heads * head_dim].reshape(rows, heads, head_dim), c, s_)
    want_k = plain_llama.rope_rotate_split_half(
        qkv[:, heads * head_dim:(heads + kv_heads) * head_dim].reshape(rows, kv_heads, head_dim), c, s_)
    want_v = qkv[:, (heads + kv_heads) * head_dim:].reshape(rows, kv_heads, head_dim)
    scale = float(qkv.abs().max())
    assert q.shape == (rows, heads * head_dim)
    assert float((q.float().cpu() - want_q.reshape(rows, -1)).abs().max()) < 1.5e-2 * scale
    ek, ev = k_pool.float().clone(), v_pool.float().clone()
    for b in range(rows):
        slot = int(slots[b])
        if slot >= 0:
            ek[slot // page, :, slot % page, :] = want_k[b]
            ev[slot // page, :, slot % page, :] = want_v[b]
    assert float((kd.float().cpu() - ek).abs().max()) < 1.5e-2 * max(scale, 4.0)
    assert float((vd.float().cpu() - ev).abs().max()) < 1.5e-2 * max(scale, 4.0)
    written = torch.zeros(pages * page, dtype=torch.bool)
    written[slots[slots >= 0].long()] = True
    untouched = ~written.reshape(pages, page)
    assert torch.equal(kd.cpu().permute(0, 2, 1, 3)[untouched], k_pool.permute(0, 2, 1, 3)[untouched])  # nothing else was stored
    assert torch.equal(vd.cpu().permute(0, 2, 1, 3)[untouched], v_pool.permute(0, 2, 1, 3)[untouched])
    with pytest.raises(ops.KernelError):
        ops.gemm_tcgen05_qkv_rope(a.cuda(), w.cuda(), heads, kv_heads, 48, positions.cuda(), cos.cuda(), sin.cuda(), kd, vd, slots.cuda())


@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (70, 144, 136), (300, 272, 200), (1, 512, 2048), (513, 1040, 328),
                                   (2100, 5136, 264), (200, 528, 4136), (520, 272, 1288)])
def test_tcgen05_gemm_all_epilogues(cuda_device, m, n, k):
    """The prefill matrix product (TMA, tcgen05.mma, accumulator in tensor memory) against float64,
    at sizes that do not fill its 128 x 256 x 64 tiles; no bounded wait may have given up.  With few
    tiles and a long K the residual epilogue splits K over blocks (the last part shorter than the rest)."""
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(m + n + k)
    a = torch.randn(m, k, generator=g).bfloat16()
    w = (torch.randn(n, k, generator=g) * 0.05).bfloat16()
    exact = a.double() @ w.double().t()
    scale = float(exact.abs().max())
    # the launcher's choice; both tile widths of single blocks by name; pairs of blocks (cta_group::2)
    for tile_width, pair in ((0, 0), (128, 1), (256, 1), (0, 2)):
        out = ops.gemm_tcgen05(a.cuda(), w.cuda(), ops.EPI_F32, tile_width=tile_width, pair=pair)
        assert float((out.double().cpu() - exact).abs().max()) < 2e-5 * scale * math.sqrt(k)
        out = ops.gemm_tcgen05(a.cuda(), w.cuda(), ops.EPI_BF16, tile_width=tile_width, pair=pair)
        assert out.dtype == torch.bfloat16 and float((out.double().cpu() - exact).abs().max()) < 1e-2 * scale
        residual = torch.randn(m, n, generator=g)
        rd = residual.cuda()
        ops.gemm_tcgen05(a.cuda(), w.cuda(), ops.EPI_RESIDUAL, out=rd, tile_width=tile_width, pair=pair)
        assert float((rd.double().cpu() - (residual.double() + exact)).abs().max()) < 2e-5 * (scale + 4) * math.sqrt(k)
    with pytest.raises(ops.KernelError, match="256"):
        ops.gemm_tcgen05(a.cuda(), w.cuda(), ops.EPI_SWIGLU, tile_width=128)
    want = plain_llama.swiglu(exact[:, : n // 2], exact[:, n // 2:])
    for pair in (1, 2):
        gated = ops.gemm_tcgen05(a.cuda(), w.cuda(), ops.EPI_SWIGLU, pair=pair)
        assert gated.shape == (m, n // 2)
        assert float((gated.double().cpu() - want).abs().max()) < 1e-2 * float(want.abs().max())
    # a strided view of wider activations is taken as it is
    wide = torch.randn(m, k + 24, generator=g).bfloat16().cuda()
    out = ops.gemm_tcgen05(wide[:, 8:8 + k], w.cuda(), ops.EPI_F32)
    want = wide[:, 8:8 + k].double().cpu() @ w.double().t()
    assert float((out.double().cpu() - want).abs().max()) < 2e-5 * float(want.abs().max()) * math.sqrt(k)
    assert ops.gemm_tcgen05_status() == 0
    with pytest.raises(ops.KernelError):
        ops.gemm_tcgen05(a.cuda(), torch.zeros(n + 4, k, dtype=torch.bfloat16, device="cuda"), ops.EPI_BF16)


@pytest.mark.parametrize("batch", [9, 17, 33, 64, 100, 128])
@pytest.mark.parametrize("n,k", [(144, 136), (2048, 2048), (272, 8192), (1040, 328)])
def test_wide_decode_gemm_all_epilogues(cuda_device, batch, n, k):
    """The wide decode product (weights as the 128-row tcgen05 operand, K split over the blocks of a
    cluster whose sums meet in distributed shared memory) against float64; a second call gives the
    same bits."""
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(batch + n + k)
    a = torch.randn(batch, k, generator=g).bfloat16()
    w = (torch.randn(n, k, generator=g) * 0.05).bfloat16()
    ad, wd = a.cuda(), w.cuda()
    exact = a.double() @ w.double().t()
    scale = float(exact.abs().max())
    out = ops.wide_gemm(ad, wd, ops.EPI_F32)
    assert float((out.double().cpu() - exact).abs().max()) < 2e-5 * scale * math.sqrt(k)
    assert torch.equal(out, ops.wide_gemm(ad, wd, ops.EPI_F32))
    out = ops.wide_gemm(ad, wd, ops.EPI_BF16)
    assert out.dtype == torch.bfloat16 and float((out.double().cpu() - exact).abs().max()) < 1e-2 * scale
    residual = torch.randn(batch, n, generator=g)
    rd = residual.cuda()
    ops.wide_gemm(ad, wd, ops.EPI_RESIDUAL, out=rd)
    assert float((rd.double().cpu() - (residual.double() + exact)).abs().max()) < 2e-5 * (scale + 4) * math.sqrt(k)
    gated = ops.wide_gemm(ad, wd, ops.EPI_SWIGLU)
    want = plain_llama.swiglu(exact[:, : n // 2], exact[:, n // 2:])
    assert gated.shape == (batch, n // 2)
    assert float((gated.double().cpu() - want).abs().max()) < 1e-2 * float(want.abs().max())
    assert ops.gemm_tcgen05_status() == 0


@pytest.mark.parametrize("rows", [1, 5, 8, 9, 33, 64, 100, 128])
@pytest.mark.parametrize("width,inner", [(264, 520), (2048, 2048), (272, 4136), (3088, 264), (1040, 8200)])
def test_the_norm_rides_in_the_products_around_it(cuda_device, rows, width, inner):
    """x = x + h . Wd^T with the next RMSNorm half done in the same kernel (x * gain as bfloat16, and parts of
    every row's sum of squares), then a product that divides by the root mean square in its own epilogue:
    against float64 of the same steps (y = x / sqrt(mean(x^2) + eps) * gain, integrallis/models,
    backend-java/.../ops/TensorOps.java:45-58).  These are the decode products (the narrow ones up to 8 rows, the
    wide ones from 9 to 128); over more rows the norms keep kernels of their own, and the products say so."""
    from models_b200.kernels import ops

    def product(a, w, epilogue, **more):
        if rows <= ops.SKINNY_PAYS_ROWS:
            return ops.skinny_gemm(w, epilogue, x=a, **more)
        return ops.tensor_core_gemm(a, w, epilogue, **more)

    g = torch.Generator().manual_seed(rows + width + inner)
    eps = 3e-5
    h = torch.randn(rows, inner, generator=g).bfloat16()
    w_down = (torch.randn(width, inner, generator=g) * 0.05).bfloat16()
    w_next = (torch.randn(144, width, generator=g) * 0.05).bfloat16()
    gain = (1.0 + 0.2 * torch.randn(width, generator=g)).float()
    x = (3.0 * torch.randn(rows, width, generator=g)).float()
    xd = x.cuda()
    out, gained, ssq, count = product(h.cuda(), w_down.cuda(), ops.EPI_RESIDUAL, out=xd, emit_gain=gain.cuda())
    assert out is xd and gained.shape == (rows, width) and gained.dtype == torch.bfloat16
    exact_x = x.double() + h.double() @ w_down.double().t()
    scale = float(exact_x.abs().max())
    assert float((xd.double().cpu() - exact_x).abs().max()) < 2e-5 * scale * math.sqrt(inner)
    # the gained rows are the kernel's own new x times the gain, rounded once
    assert torch.equal(gained.cpu(), (xd.cpu() * gain).bfloat16())
    squares = ssq[:count, :rows].double().sum(0).cpu()
    want_squares = (xd.double().cpu() ** 2).sum(1)
    assert float(((squares - want_squares) / want_squares).abs().max()) < 1e-5
    parts = (ssq, count, width, eps)
    inv_rms = 1.0 / torch.sqrt(want_squares / width + eps)
    normed = gained.double().cpu() * inv_rms[:, None]
    exact = normed @ w_next.double().t()
    got = product(gained, w_next.cuda(), ops.EPI_F32, norm_parts=parts)
    assert float((got.double().cpu() - exact).abs().max()) < 2e-5 * float(exact.abs().max()) * math.sqrt(width)
    got = product(gained, w_next.cuda(), ops.EPI_SWIGLU, norm_parts=parts)
    want = plain_llama.swiglu(exact[:, :72], exact[:, 72:])
    assert float((got.double().cpu() - want).abs().max()) < 1e-2 * float(want.abs().max())
    # the same bits in a second run (ordered sums everywhere)
    xd2 = x.cuda()
    _, gained2, ssq2, count2 = product(h.cuda(), w_down.cuda(), ops.EPI_RESIDUAL, out=xd2, emit_gain=gain.cuda())
    assert torch.equal(xd, xd2) and torch.equal(gained, gained2) and count == count2 and torch.equal(ssq[:count, :rows], ssq2[:count, :rows])
    assert ops.gemm_tcgen05_status() == 0
    with pytest.raises(ops.KernelError, match="128 rows"):
        ops.tensor_core_gemm(torch.zeros(129, width, dtype=torch.bfloat16, device="cuda"), w_next.cuda(), ops.EPI_F32, norm_parts=parts)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("count", [1, 3, 4, 1001, 262147])
def test_random_weights_are_the_same_bits_on_host_and_device(cuda_device, dtype, count):
    """The counter-based normal generator of random-weights mode: the device kernel and its numpy twin
    evaluate the same polynomials with the same roundings."""
    from models_b200.weights.philox_normal import normal_float32, tensor_key

    from models_b200.kernels import ops

    torch_dtype = dtype
    for mean, std, name in ((0.0, 0.02, "a.weight"), (1.0, 0.1, "b.weight"), (0.0, 1.0, "c")):
        key = tensor_key(count, name)
        device = ops.random_normal(torch.empty(count, dtype=torch_dtype, device="cuda"), key, mean, std)
        host = torch.from_numpy(normal_float32(count, key, mean, std)).to(torch_dtype)
        assert torch.equal(device.cpu(), host), (count, name)


def test_a_random_model_is_the_same_from_a_file_and_on_the_device(cuda_device, tmp_path):
    """`engine_from_config` (weights drawn on the GPU) and `write_random_model` (drawn on the host, written,
    read back) give one model: the same tensors, so the same logits."""
    from models_b200.config import config_from_dict
    from models_b200.engine import StepEntry
    from models_b200.engine.loading import engine_from_config, engine_from_folder
    from tiny import TINY_B, make_folder, random_tokens

    folder = make_folder(TINY_B, 9, tmp_path)
    from_file = engine_from_folder(folder, "bfloat16", 256)
    on_device = engine_from_config(config_from_dict(TINY_B), 9, "bfloat16", 256)
    assert torch.equal(from_file.model.embedding.weight, on_device.model.embedding.weight)
    assert torch.equal(from_file.model.head.weight, on_device.model.head.weight)
    assert torch.equal(from_file.model.final_norm.weight, on_device.model.final_norm.weight)
    for a, b in zip(from_file.model.blocks, on_device.model.blocks):
        assert torch.equal(a.mixer.w_qkv, b.mixer.w_qkv) and torch.equal(a.feed_forward.w_down, b.feed_forward.w_down)
        assert torch.equal(a.mixer_norm.weight, b.mixer_norm.weight)
    tokens = random_tokens(TINY_B["vocab_size"], 50, 1)
    outs = []
    for engine in (from_file, on_device):
        slot = engine.open_slot()
        outs.append(engine.step([StepEntry(slot, tokens, [49])]))
    assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("activation", ["silu", "gelu_tanh"])
def test_gated_products_take_their_activation_as_an_argument(cuda_device, activation):
    """act(gate) * up with the gate's activation as an argument of every kernel that applies it: the
    stand-alone kernel (float32 and bfloat16), the decode product (with and without the folded norm),
    the wide tcgen05 product and the prefill tcgen05 product."""
    from models_b200.kernels import ops

    act = {"silu": P_swiglu, "gelu_tanh": plain_llama.gelu_glu}[activation]
    g = torch.Generator().manual_seed(5)
    n, k = 272, 264
    w = (torch.randn(2 * n, k, generator=g) * 0.2).to(torch.bfloat16)
    gain = 1.0 + 0.1 * torch.randn(k, generator=g)
    for dtype in DTYPES:
        both = (torch.randn(37, 2 * 203, generator=g) * 2).to(dtype)
        expected = act(both[:, :203].float(), both[:, 203:].float())
        close(ops.swiglu(both.cuda(), activation), expected, dtype)
    code = ops.gated_epilogue(activation)
    for rows in (5, 16, 64, 300):
        x = (torch.randn(rows, k, generator=g)).to(torch.bfloat16)
        product = x.float() @ w.float().t()
        expected = act(product[:, :n], product[:, n:])
        if rows <= 32:
            close(ops.skinny_gemm(w.cuda(), code, x=x.cuda()), expected, torch.bfloat16)
        if rows <= 16:
            xf = torch.randn(rows, k, generator=g)
            normed = plain_llama.rms_norm(xf, gain, 1e-5).to(torch.bfloat16).float() @ w.float().t()
            got = ops.skinny_gemm(w.cuda(), code, xf=xf.cuda(), gain=gain.cuda(), eps=1e-5)
            want = act(normed[:, :n], normed[:, n:])
            # as for silu in the test of all epilogues: two roundings to bfloat16 (rows, result) around a product of two sums
            assert float((got.double().cpu() - want.double()).abs().max()) < 2e-2 * float(want.abs().max())
        if rows <= 128:
            close(ops.wide_gemm(x.cuda(), w.cuda(), code), expected, torch.bfloat16)
        close(ops.gemm_tcgen05(x.cuda(), w.cuda(), code), expected, torch.bfloat16)
    with pytest.raises(ops.KernelError, match="not built"):
        ops.gated_epilogue("relu")
    assert ops.gemm_tcgen05_status() == 0


def P_swiglu(gate, up):
    return plain_llama.swiglu(gate, up)


def test_logit_epilogue(cuda_device):
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(9)
    logits = torch.randn(5, 203, generator=g) * 3
    wide = torch.zeros(5, 256)
    wide[:, :203] = logits
    view = wide.cuda()[:, :203]  # rows wider than the vocabulary: the stride is an argument
    close(ops.logit_epilogue(view, 2.0, 5.0), plain_llama.softcap_logits(logits * 2.0, 5.0), torch.float32)
    close(ops.logit_epilogue(logits.clone().cuda(), 0.5, 0.0), logits * 0.5, torch.float32)


def test_split_k_residual_product_is_the_same_bits_every_time(cuda_device):
    """Few tiles and a long K: the residual product splits K over blocks.  The parts are summed in their
    order, so ten runs give one result, bit for bit, and it is the plain product; letting the parts add
    in as they finish is still there as an option and gives the same numbers within rounding."""
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(11)
    for m, n, k in ((256, 2048, 8192), (200, 520, 4096), (129, 264, 2048)):
        a = torch.randn(m, k, generator=g).to(torch.bfloat16).cuda()
        w = (torch.randn(n, k, generator=g) * 0.05).to(torch.bfloat16).cuda()
        x0 = torch.randn(m, n, generator=g).cuda()
        expected = x0.double().cpu() + a.double().cpu() @ w.double().cpu().t()
        results = []
        for _ in range(10):
            x = x0.clone()
            ops.gemm_tcgen05(a, w, ops.EPI_RESIDUAL, out=x)
            results.append(x)
        for other in results[1:]:
            assert torch.equal(results[0], other), (m, n, k)
        close(results[0], expected, torch.float32, scale=float(expected.abs().max()) * 1e3)  # bfloat16 inputs, float sums
        loose = ops.gemm_tcgen05(a, w, ops.EPI_RESIDUAL, out=x0.clone(), arrival_order=True)
        close(loose, expected, torch.float32, scale=float(expected.abs().max()) * 1e3)
    tickets = ops._split_tickets[torch.cuda.current_device()]
    assert int(tickets.abs().sum()) == 0  # every launch leaves them as it found them
    assert ops.gemm_tcgen05_status() == 0


@pytest.mark.parametrize("batch", [9, 40, 64, 128])
@pytest.mark.parametrize("heads,kv_heads,head_dim,hidden", [(4, 2, 16, 64), (3, 1, 32, 96), (32, 8, 64, 2048), (6, 3, 128, 264)])
@pytest.mark.parametrize("normed", [False, True])
def test_wide_qkv_product_with_rotation_and_cache_write(cuda_device, batch, heads, kv_heads, head_dim, hidden, normed):
    """The q/k/v product of a decode step of 9 to 128 sequences with rotation and cache write folded in,
    against the plain functions: queries rotated by each row's own position, keys rotated and values
    as they are at each row's cache position, rows without a position of their own storing nothing.
    `normed`: the division by the rows' root mean square happens in the product's epilogue, from parts
    of their sums of squares."""
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(batch * 7 + head_dim)
    rows_w = (heads + 2 * kv_heads) * head_dim
    w = (torch.randn(rows_w, hidden, generator=g) * 0.05).bfloat16()
    x = torch.randn(batch, hidden, generator=g).bfloat16()
    positions = torch.randint(0, 300, (batch,), generator=g).int()
    freqs = plain_llama.rope_pair_frequencies(head_dim, 10000.0)
    cos, sin = plain_llama.rope_cos_sin(torch.arange(300), freqs, None)
    pages, page = 2 * batch + 1, 64
    k_pool = torch.zeros(pages, kv_heads, page, head_dim, dtype=torch.bfloat16)
    v_pool = torch.zeros_like(k_pool)
    slots = torch.randperm(pages * page - page, generator=g)[:batch].int() + page
    slots[batch // 2] = -1  # a padding row: nothing is stored for it
    kd, vd = k_pool.cuda(), v_pool.cuda()
    parts, inv_rms = None, torch.ones(batch, dtype=torch.float64)
    if normed:
        ssq = torch.rand(7, ops.SSQ_COLUMNS, generator=g) * hidden  # (two more parts than are counted)
        parts = (ssq.cuda(), 5, hidden, 2e-5)
        inv_rms = 1.0 / torch.sqrt(ssq[:5, :batch].double().sum(0) / hidden + 2e-5)
    q = ops.wide_qkv_rope(x.cuda(), w.cuda(), heads, kv_heads, head_dim, positions.cuda(), cos.cuda(), sin.cuda(), kd, vd, slots.cuda(),
                          norm_parts=parts)
    full = ((x.double() @ w.double().t()) * inv_rms[:, None]).float()
    qe = full[:, : heads * head_dim].bfloat16().float().reshape(batch, heads, head_dim)
    ke = full[:, heads * head_dim:(heads + kv_heads) * head_dim].bfloat16().float().reshape(batch, kv_heads, head_dim)
    ve = full[:, (heads + kv_heads) * head_dim:].reshape(batch, kv_heads, head_dim)
    c, s = cos[positions.long()], sin[positions.long()]
    qe, ke = plain_llama.rope_rotate_split_half(qe, c, s), plain_llama.rope_rotate_split_half(ke, c, s)
    close(q.reshape(batch, heads, head_dim), qe, torch.bfloat16)
    kflat, vflat = kd.cpu().permute(0, 2, 1, 3).reshape(-1, kv_heads, head_dim), vd.cpu().permute(0, 2, 1, 3).reshape(-1, kv_heads, head_dim)
    for b in range(batch):
        if slots[b] < 0:
            continue
        close(kflat[slots[b]], ke[b], torch.bfloat16, scale=float(ke.abs().max()))
        close(vflat[slots[b]], ve[b], torch.bfloat16, scale=float(ve.abs().max()))
    stored = (kflat.abs().sum(dim=(1, 2)) > 0).sum()
    assert int(stored) == batch - 1  # exactly the rows with a cache position wrote
    assert ops.gemm_tcgen05_status() == 0


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("vdim", [64, 128])
@pytest.mark.parametrize("lengths", [[64], [1, 127, 64], [65, 0, 200, 63]])
def test_gated_delta_chunks(cuda_device, monkeypatch, dtype, vdim, lengths):
    """Chunks of 64 against the walk token by token and against the recurrence in 64 bits, from states that are not zero."""
    from models_b200.kernels import ops

    monkeypatch.setattr(ops, "DELTA_CHUNK_MIN_MEAN", 1)  # (sequences of edge lengths, not of lengths that are worth it)
    heads, kv_heads, dim = 4, 2, 64
    g = torch.Generator().manual_seed(21)
    tokens, width = sum(lengths), 2 * kv_heads * dim + heads * vdim
    conv = torch.randn(tokens, width, generator=g).cuda()
    wide = torch.randn(tokens, 2 * heads + heads * vdim, generator=g).to(dtype).cuda()
    a_in, b_in, gate = wide[:, :heads], wide[:, heads:2 * heads], wide[:, 2 * heads:]
    decay = -torch.tensor([0.01, 0.5, 4.0, 16.0]).cuda()
    dt_bias, gain = torch.randn(heads, generator=g).cuda(), (1 + 0.1 * torch.randn(vdim, generator=g)).cuda()
    state0 = torch.randn(len(lengths) + 1, heads * dim * vdim + 5, generator=g).cuda()
    slots = torch.arange(len(lengths), dtype=torch.int32).flip(0).contiguous().cuda()
    cu_q = torch.tensor([0] + torch.tensor(lengths).cumsum(0).tolist(), dtype=torch.int32).cuda()
    found = []
    for most in (0, max(lengths)):
        state, out = state0.clone(), torch.zeros(tokens, heads * vdim, dtype=dtype).cuda()
        ops.gated_delta_scan(conv.clone(), 0, kv_heads * dim, 2 * kv_heads * dim, a_in, b_in, gate, decay, dt_bias, gain, 1e-6, 1e-6, state, 3,
                             slots, cu_q, heads, kv_heads, dim, vdim, out, 0.5, max_q_len=most)
        found.append((out.float(), state))
    (out, state), (chunk_out, chunk_state) = found
    assert ops.gated_delta_chunks_takes(conv, gate, gain, out.to(dtype), dim, vdim, (0, kv_heads * dim, 2 * kv_heads * dim), max(lengths),
                                        len(lengths))
    # sums of at most 64 + 64 products a token either way; the states' numbers are of size one to ten
    assert torch.allclose(chunk_state, state, rtol=1e-4, atol=1e-4)
    assert torch.equal(chunk_state[:, :3], state0[:, :3]) and torch.equal(chunk_state[-1], state0[-1])
    close(chunk_out, out, dtype, scale=4.0)
    # A chunk adds a number up over some 64 + 64 products, whose roundings of 2^-24 grow like the root of their count: 2^-20.5, and what
    # the gates' functions and the chunks before bring, four times that in all.  (Measured: 1.3e-7.  Operands of two bfloat16
    # parts would be off by 2^-17.)
    bound = 2.0 ** -18.5
    q, k, v = (t.double().cpu().view(tokens, n, -1) for t, n in zip(conv.split([kv_heads * dim, kv_heads * dim, heads * vdim], 1), (kv_heads, kv_heads, heads)))
    q, k = (t.repeat_interleave(heads // kv_heads, 1) / (t.repeat_interleave(heads // kv_heads, 1).square().sum(-1, keepdim=True) + 1e-6).sqrt() for t in (q, k))
    forget = torch.exp(decay.double() * torch.nn.functional.softplus(a_in.double() + dt_bias.double())).cpu()
    beta, results = torch.sigmoid(b_in.double()).cpu(), torch.empty(tokens, heads, vdim, dtype=torch.float64)
    for i, n in enumerate(lengths):
        mine = slice(3, 3 + heads * dim * vdim)
        S = state0[slots[i], mine].double().cpu().view(heads, dim, vdim)
        for t in range(int(cu_q[i]), int(cu_q[i]) + n):
            S = S * forget[t, :, None, None]
            S = S + k[t, :, :, None] * (beta[t, :, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t])))[:, None, :]
            results[t] = torch.einsum("hdv,hd->hv", S, q[t]) / 8.0
        got = chunk_state[slots[i], mine].double().cpu().view(heads, dim, vdim)
        assert float((got - S).norm()) <= bound * float(S.norm())
    results = 0.5 * results / (results.square().mean(-1, keepdim=True) + 1e-6).sqrt() * gain.double().cpu()
    results = results.flatten(1) * torch.nn.functional.silu(gate.double().cpu())
    bound = bound if dtype == torch.float32 else 2.0 ** -8  # (a result's own rounding)
    assert float((chunk_out.double().cpu() - results).norm()) <= bound * float(results.norm())


def _delta_call(lengths, heads, kv_heads, vdim, dtype, seed, unit_eps=1e-6, spoil=None):
    """The gated delta rule over sequences of these lengths, from states that are not zero, as a function of max_q_len: (results, states)
    by the walk (0) or in chunks.  `spoil` changes the convolved rows."""
    from models_b200.kernels import ops

    dim, g = 64, torch.Generator().manual_seed(seed)
    tokens = sum(lengths)
    conv = torch.randn(tokens, 2 * kv_heads * dim + heads * vdim, generator=g)
    if spoil is not None:
        spoil(conv)
    conv, wide = conv.cuda(), torch.randn(tokens, 2 * heads + heads * vdim, generator=g).to(dtype).cuda()
    decay = -torch.tensor([(0.01, 0.5, 4.0, 16.0)[h % 4] for h in range(heads)]).cuda()
    dt_bias, gain = torch.randn(heads, generator=g).cuda(), (1 + 0.1 * torch.randn(vdim, generator=g)).cuda()
    state0 = torch.randn(len(lengths), heads * dim * vdim, generator=g).cuda()
    slots = torch.arange(len(lengths), dtype=torch.int32).cuda()
    cu_q = torch.tensor([0] + torch.tensor(lengths).cumsum(0).tolist(), dtype=torch.int32).cuda()

    def call(max_q_len):
        state, out = state0.clone(), torch.zeros(tokens, heads * vdim, dtype=dtype).cuda()
        ops.gated_delta_scan(conv.clone(), 0, kv_heads * dim, 2 * kv_heads * dim, wide[:, :heads], wide[:, heads:2 * heads], wide[:, 2 * heads:], decay,
                             dt_bias, gain, unit_eps, 1e-6, state, 0, slots, cu_q, heads, kv_heads, dim, vdim, out, 0.5, max_q_len=max_q_len)
        return out.float(), state

    return call


@pytest.mark.parametrize("vdim", [64, 128])
@pytest.mark.parametrize("lengths", [[128], [192, 129], [449, 640]])
def test_gated_delta_chunks_carry_through_their_ring(cuda_device, vdim, lengths):
    """Two to ten chunks of a sequence through three places in shared memory, the last ones not full."""
    from models_b200.kernels import ops

    call = _delta_call(lengths, 4, 2, vdim, torch.float32, 11)
    (out, state), (chunk_out, chunk_state) = call(0), call(max(lengths))
    # the bounds of test_gated_delta_chunks, and the same bits once more
    assert torch.allclose(chunk_state, state, rtol=1e-4, atol=1e-4)
    close(chunk_out, out, torch.float32, scale=4.0)
    again = call(max(lengths))
    assert torch.equal(again[0], chunk_out) and torch.equal(again[1], chunk_state)
    assert ops.waits_given_up() == {}


@pytest.mark.parametrize("lengths", [[65], [100, 64, 3]])
def test_gated_delta_chunks_without_an_epsilon(cuda_device, monkeypatch, lengths):
    """Keys that are divided by their own length alone: the empty rows of a chunk that is not full have none."""
    from models_b200.kernels import ops

    monkeypatch.setattr(ops, "DELTA_CHUNK_MIN_MEAN", 1)
    call = _delta_call(lengths, 4, 2, 64, torch.float32, 5, unit_eps=0.0)
    (out, state), (chunk_out, chunk_state) = call(0), call(max(lengths))
    # the bounds of the test above
    assert bool(out.isfinite().all()) and torch.allclose(chunk_state, state, rtol=1e-4, atol=1e-4)
    close(chunk_out, out, torch.float32, scale=4.0)


def test_gated_delta_steps_beyond_the_scratch_bound_are_walked(cuda_device, monkeypatch):
    from models_b200.kernels import ops

    call = _delta_call([130, 70], 2, 1, 128, torch.bfloat16, 7)
    # three chunks of one sequence and two of the other: what the launcher asks for
    assert ops.gated_delta_chunk_floats(200, 2, 2, 128) == 5 * 2 * (2 * 64 * 128 + 3 * 64 * 64 + 128)
    walked, chunks = call(0), call(130)
    assert not torch.equal(walked[1], chunks[1])
    monkeypatch.setattr(ops, "DELTA_CHUNK_BYTES", 4 * ops.gated_delta_chunk_floats(200, 2, 2, 128) - 1)
    assert all(torch.equal(a, b) for a, b in zip(call(130), walked))


@pytest.mark.parametrize("lengths,most,chunks", [([96], 96, True), ([95], 95, False), ([130, 62], 130, True), ([130, 61], 130, False), ([8] * 8, 64, False),
                                                 ([24] * 8, 192, False), ([96, 96], 192, True)])
def test_gated_delta_steps_of_short_sequences_are_walked(cuda_device, lengths, most, chunks):
    """Either side of the line, and steps that say no more than how many tokens they have in all: as captured ones do."""
    call = _delta_call(lengths, 2, 1, 64, torch.float32, 8)
    assert torch.equal(call(most)[1], call(0)[1]) != chunks


SPOILED = [("v", 5), ("v", 77), ("v", 90), ("k", 66), ("k", 127), ("q", 20)]  # a row that is not finite: within its 16 tokens, chunk and sequence


@pytest.mark.parametrize("vdim", [64, 128])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("part,at", SPOILED)
def test_gated_delta_chunks_keep_earlier_tokens_apart(cuda_device, vdim, value, part, at):
    """A row that is not finite spoils its own sequence from its token on, as in the walk; earlier tokens and other sequences give what they
    give without it."""
    lengths = [130, 70]

    def spoil(conv):
        conv[at, {"q": 3, "k": 64 + 7, "v": 128 + vdim + 9}[part]] = value

    clean, clean_state = _delta_call(lengths, 2, 1, vdim, torch.float32, 6)(130)
    out, state = _delta_call(lengths, 2, 1, vdim, torch.float32, 6, spoil=spoil)(130)
    # (a chunk that holds such a row is added up in another order)
    close(out[:at], clean[:at], torch.float32, scale=4.0)
    assert torch.equal(out[130:], clean[130:]) and torch.equal(state[1], clean_state[1])
    assert not bool(out[at].isfinite().all())


@pytest.mark.parametrize("vdim", [64, 128])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("part,at", SPOILED)
def test_retention_chunks_keep_earlier_tokens_apart(cuda_device, vdim, value, part, at):
    """The same of retention; in its raw results a value that is not finite spoils its own column alone."""
    from models_b200.kernels import ops

    heads, dim, lengths = 2, 64, [130, 70]
    g = torch.Generator().manual_seed(23)
    proj = torch.randn(sum(lengths), heads * (2 * dim + 2 * vdim), generator=g).bfloat16()
    decay, state0 = torch.tensor([0.97, 0.5]).cuda(), torch.randn(2, heads, dim, vdim, generator=g).cuda()
    slots, cu_q, positions = (torch.tensor(v, dtype=torch.int32).cuda() for v in ([0, 1], [0, 130, 200], [0] * 200))
    found = []
    for spoiled in (False, True):
        rows = proj.clone()
        if spoiled:
            rows[at, {"q": 3, "k": heads * dim + 7, "v": 2 * heads * dim + 9}[part]] = value
        q, k, v, _ = rows.cuda().split([heads * dim, heads * dim, heads * vdim, heads * vdim], dim=1)
        state, raw = state0.clone(), torch.zeros(200, heads * vdim).cuda()
        ops.retention_scan(q, k, v, None, positions, None, None, 0, decay, 0.3, 1e-6, state, slots, cu_q, heads, dim, vdim, None, 0.5, 130, raw_out=raw)
        found.append((raw, state))
    (clean, clean_state), (raw, state) = found
    touched = torch.zeros_like(clean, dtype=torch.bool)
    touched[at:130, :vdim] = True
    if part == "v":
        touched[:, :9] = touched[:, 10:] = False
    close(torch.where(touched, clean, raw), clean, torch.float32, scale=4.0 * float(clean.abs().max()))
    assert torch.equal(raw[130:], clean[130:]) and torch.equal(state[1], clean_state[1])
    assert not bool(raw[at, :vdim].isfinite().all())


@pytest.mark.parametrize("vdim", [64, 128])
@pytest.mark.parametrize("lengths", [[64], [1, 127, 64], [65, 0, 200, 63]])
@pytest.mark.parametrize("whole", [True, False])
def test_retention_chunks(cuda_device, vdim, lengths, whole):
    """Chunks of 64 on the tensor cores against the walk, from states that are not zero: raw results of activated projections, and
    rotated ones with the head's norm and gate."""
    from models_b200.kernels import ops

    heads, dim = 3, 64
    g = torch.Generator().manual_seed(22)
    tokens = sum(lengths)
    proj = torch.randn(tokens, heads * (2 * dim + 2 * vdim), generator=g).bfloat16().cuda()
    q, k, v, gate = proj.split([heads * dim, heads * dim, heads * vdim, heads * vdim], dim=1)
    decay = torch.tensor([0.97, 0.5, 0.0]).cuda()
    state0 = torch.randn(len(lengths) + 1, heads, dim, vdim, generator=g).cuda()
    slots = torch.arange(len(lengths), dtype=torch.int32).flip(0).contiguous().cuda()
    cu_q = torch.tensor([0] + torch.tensor(lengths).cumsum(0).tolist(), dtype=torch.int32).cuda()
    starts = [5, 0, 11, 2][:len(lengths)]
    positions = torch.cat([torch.arange(s, s + n) for s, n in zip(starts, lengths)]).to(torch.int32).cuda()
    angle = torch.rand(300, 24, generator=g) * 6
    cos, sin = angle.cos().cuda(), angle.sin().cuda()
    found = []
    for run_length in (0, None):  # the walk, and what the dispatch picks
        state = state0.clone()
        raw = torch.zeros(tokens, heads * vdim).cuda() if whole else None
        out = None if whole else torch.zeros(tokens, heads * vdim).bfloat16().cuda()
        ops.retention_scan(q, k, v, None if whole else gate, positions, None if whole else cos, None if whole else sin, 0 if whole else 48, decay,
                           0.3, 1e-6, state, slots, cu_q, heads, dim, vdim, out, 0.5, max(lengths), run_length=run_length,
                           input_activation="silu" if whole else None, raw_out=raw)
        found.append(((raw if whole else out).float(), state))
    (out, state), (chunk_out, chunk_state) = found
    assert ops.retention_chunks_takes(q, k, v, None if whole else gate, None if whole else out.bfloat16(), out if whole else None, state, dim, vdim, max(lengths),
                                      len(lengths))
    # three parts hold a float's 24 bits; either side adds up to 200 floats in some order, each addition off by up to 2^-23 of a sum that
    # is no larger than a few times its result: 2^-23 times the root of 200 additions, times four
    assert torch.equal(chunk_state[-1], state0[-1])
    assert float((chunk_state - state).norm() / state.norm()) < 2.0 ** -17
    if whole:
        assert float((chunk_out - out).norm() / out.norm()) < 2.0 ** -17
    else:
        close(chunk_out, out, torch.bfloat16)


@pytest.mark.parametrize("vdim", [64, 128])
@pytest.mark.parametrize("activation", [None, "silu", "gelu_tanh", "relu2"])
def test_retention_chunks_rotated_by_nothing(cuda_device, vdim, activation):
    """Rows that are rotated and rows that are not are activated by two pieces of code: one bit pattern, also where the activations' divisions are
    unusual ones (gates below -40 and beyond 2^60)."""
    from models_b200.kernels import ops

    heads, dim, lengths = 2, 64, [100, 64, 33]
    tokens = sum(lengths)
    g = torch.Generator().manual_seed(vdim)
    proj = torch.randn(tokens, heads * (2 * dim + vdim), generator=g) * 3
    proj[::5, ::9] = -torch.rand(proj[::5, ::9].shape, generator=g) * 100
    proj[7, heads * dim + 3], proj[90, heads * dim + 70], proj[120, 5], proj[130, -2] = 2.0 ** 61, 2.0 ** 60, 2.0 ** 40, -2.0 ** 61
    q, k, v = proj.bfloat16().cuda().split([heads * dim, heads * dim, heads * vdim], dim=1)
    decay, state0 = torch.tensor([0.97, 0.5]).cuda(), torch.randn(3, heads, dim, vdim, generator=g).cuda()
    slots = torch.arange(3, dtype=torch.int32).cuda()
    cu_q = torch.tensor([0] + torch.tensor(lengths).cumsum(0).tolist(), dtype=torch.int32).cuda()
    positions = torch.cat([torch.arange(n) for n in lengths]).to(torch.int32).cuda()
    found = []
    for rotary in (0, 48, 64):
        cos, sin = torch.ones(100, max(rotary, 2) // 2).cuda(), torch.zeros(100, max(rotary, 2) // 2).cuda()
        state, raw = state0.clone(), torch.zeros(tokens, heads * vdim).cuda()
        ops.retention_scan(q, k, v, None, positions, cos if rotary else None, sin if rotary else None, rotary, decay, 2.0 ** -70, 1e-6, state, slots, cu_q,
                           heads, dim, vdim, None, 0.5, max(lengths), input_activation=activation, raw_out=raw)
        found.append((raw, state))
    assert bool(found[0][0].isfinite().all()) and bool(found[0][1].isfinite().all())
    for raw, state in found[1:]:
        assert torch.equal(raw, found[0][0]) and torch.equal(state, found[0][1])


@pytest.mark.parametrize("lengths,most,chunks", [([64], 64, True), ([33, 31], 64, True), ([33, 30], 64, False), ([8] * 8, 64, False), ([16] * 8, 128, False),
                                                 ([16] * 8, 129, True)])
def test_retention_steps_of_short_sequences_are_walked(cuda_device, lengths, most, chunks):
    """Either side of the line, and steps that say no more than how many tokens they have in all: as captured ones do."""
    from models_b200.kernels import ops

    heads, dim, tokens = 2, 64, sum(lengths)
    g = torch.Generator().manual_seed(24)
    q, k, v = torch.randn(tokens, 3 * heads * dim, generator=g).bfloat16().cuda().split(heads * dim, dim=1)
    decay, state0 = torch.tensor([0.97, 0.5]).cuda(), torch.randn(len(lengths), heads, dim, dim, generator=g).cuda()
    slots, positions = (torch.arange(n, dtype=torch.int32).cuda() for n in (len(lengths), tokens))
    cu_q = torch.tensor([0] + torch.tensor(lengths).cumsum(0).tolist(), dtype=torch.int32).cuda()
    found = []
    for run_length in (0 if most <= 128 else 64, None):
        state, raw = state0.clone(), torch.zeros(tokens, heads * dim).cuda()
        ops.retention_scan(q, k, v, None, positions, None, None, 0, decay, 0.3, 1e-6, state, slots, cu_q, heads, dim, dim, None, 0.5, most,
                           run_length=run_length, raw_out=raw)
        found.append(raw)
    assert torch.equal(*found) != chunks


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width", [8, 2040, 2048, 2056, 8192, 8200])
@pytest.mark.parametrize("shift", [0, 1])
def test_group_norm_gate_in_eights(cuda_device, dtype, width, shift):
    """Rows at the edges of the form in eights and off its alignment, against 64 bits."""
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(width)
    raw, gain = torch.randn(3, width + 8, generator=g)[:, shift:shift + width], 1 + 0.1 * torch.randn(width, generator=g)
    gate = torch.randn(3, width + 8, generator=g).to(dtype)[:, shift:shift + width]
    for name in ("sigmoid", "silu"):
        rows = torch.full((3, width + 8), 7.0, dtype=dtype, device=cuda_device)
        moved = [torch.empty(3, width + 8, dtype=t.dtype, device=cuda_device)[:, shift:shift + width] for t in (raw, gate)]
        for to, t in zip(moved, (raw, gate)):
            to.copy_(t)
        ops.group_norm_gate(moved[0], gain.cuda(), moved[1], rows[:, shift:shift + width], 1e-5, name)
        x, z = raw.double(), gate.double()
        want = x / (x.pow(2).mean(1, keepdim=True) + 1e-5).sqrt() * gain.double() * torch.sigmoid(z) * (z if name == "silu" else 1)
        close(rows[:, shift:shift + width].float(), want.float(), dtype)
        assert bool((rows[:, :shift] == 7).all()) and bool((rows[:, shift + width:] == 7).all())


@pytest.mark.parametrize("heads,kv_heads,dim,vdim,rotary,value_rotary", [(16, 4, 64, 128, 64, 128), (3, 1, 8, 8, 8, 0), (5, 5, 256, 24, 0, 8),
                                                                         (32, 8, 128, 128, 40, 16)])
@pytest.mark.parametrize("unit", [True, False])
def test_rotate_norm_store_in_eights(cuda_device, heads, kv_heads, dim, vdim, rotary, value_rotary, unit):
    """The form in eights against the general one, which rows that start off its alignment take: rotations that end within a head, a
    token without a slot, more pieces than a block has threads."""
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(dim + vdim)
    tokens, page, widths = 5, 64, (heads * dim, kv_heads * dim, kv_heads * vdim)
    rows = [torch.randn(tokens, w, generator=g).bfloat16().cuda() for w in widths]
    positions = torch.tensor([0, 1, 77, 150, 2], dtype=torch.int32).cuda()
    slots = torch.tensor([64, 130, -1, 191, 65], dtype=torch.int32).cuda()
    angle, value_angle = torch.rand(200, max(rotary, 2) // 2, generator=g) * 6, torch.rand(200, max(value_rotary, 2) // 2, generator=g) * 6
    tables = [t.cuda() for a in (angle, value_angle) for t in (a.cos(), a.sin())]
    found = []
    for shift in (0, 2):  # (pairs stay aligned, eights do not)
        wide = [torch.zeros(tokens, w + 8, dtype=torch.bfloat16, device=cuda_device) for w in widths]
        q, k, v = (t[:, shift:shift + w] for t, w in zip(wide, widths))
        for to, t in zip((q, k, v), rows):
            to.copy_(t)
        pools = [torch.zeros(3, kv_heads, page, d, dtype=torch.bfloat16, device=cuda_device) for d in (dim, vdim)]
        ops.rotate_norm_store(q, k, v, positions, tables[0], tables[1], rotary, True, unit, 1e-5, tables[2], tables[3], value_rotary, *pools, slots,
                              heads, kv_heads, dim, vdim)
        found.append([q.float()] + [pool.float() for pool in pools])
        assert all(bool((t[:, :shift] == 0).all()) and bool((t[:, shift + w:] == 0).all()) for t, w in zip(wide, widths))
    # the same floats but for the order of a head's squares: a rounding to bfloat16 may fall to the other side
    for here, there in zip(*found):
        assert torch.allclose(here, there, rtol=2.0 ** -7, atol=0)
        assert float((here != there).float().mean()) < 0.01


@pytest.mark.parametrize("activation", ["silu", "gelu_tanh"])
@pytest.mark.parametrize("rows", [129, 300, 512])
def test_gated_prompt_product_with_rows_of_zeros(cuda_device, activation, rows):
    """Rows of nothing but zeros within a piece of other rows, as whole pieces and at the end: their results are
    zero, and the other rows' what they are without them."""
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(rows)
    a, w = torch.randn(rows, 256, generator=g).bfloat16().cuda(), (torch.randn(1024, 256, generator=g) * 0.05).bfloat16().cuda()
    epilogue = ops.EPI_SWIGLU | ops.activation_code(activation) << 8  # (the epilogue carries its activation above its code)
    want = ops.gemm_tcgen05(a, w, epilogue)
    empty = torch.zeros(rows, dtype=torch.bool)
    empty[[5, 40, rows - 1]] = True
    empty[64:100] = True
    zeroed = a.clone()
    zeroed[empty.cuda()] = 0
    got = ops.gemm_tcgen05(zeroed, w, epilogue)
    assert bool((got[empty.cuda()] == 0).all()) and torch.equal(got[~empty.cuda()], want[~empty.cuda()])


@pytest.mark.parametrize("clamp", [None, (7.0, 1.702, 1.0)])
def test_gated_prompt_product_of_unusual_gates(cuda_device, clamp):
    """Gates whose exponential overflows, vanishes or is at the edge of either: within the rounding to bfloat16 (eight bits: 2^-8), the float
    operations before it (below 2^-18) and what a float that small holds of a quotient by more than 2^126."""
    from models_b200.kernels import ops

    gates = torch.tensor([0.0, 1e-30, 1.0, -1.0, -20.0, 20.0, -85.0, -87.5, -88.5, -90.0, -104.0, 104.0, -1e4, 1e4, -3e38, 3e38] * 8)
    n = gates.numel()
    a = torch.zeros(130, 2 * n, dtype=torch.bfloat16)
    a[:, :n] = torch.diag(gates.bfloat16().float())[torch.arange(130) % n].bfloat16()  # row r: gate r alone, and up 0.5
    a[:, n] = 1.0
    w = torch.zeros(2 * n, 2 * n, dtype=torch.bfloat16)
    w[:n, :n] = torch.eye(n)
    w[n:, n] = 0.5
    gate = (a.double() @ w.double().t())[:, :n]
    if clamp is None:
        want = gate / (1 + torch.exp(-gate)) * 0.5
        got = ops.gemm_tcgen05(a.cuda(), w.cuda(), ops.EPI_SWIGLU)
    else:
        g = gate.clamp(max=clamp[0])
        want = g / (1 + torch.exp(-clamp[1] * g)) * (0.5 + clamp[2])
        got = ops.gemm_tcgen05(a.cuda(), w.cuda(), ops.EPI_CLAMPED, clamp=clamp)
    error = (got.double().cpu() - want).abs()
    assert bool((error <= want.abs() * (2.0 ** -8 + 2.0 ** -18) + 90.0 * 2.0 ** -126).all())


@pytest.mark.parametrize("clamp", [None, (7.0, 1.702, 1.0), (7.0, -0.5, 1.0), (1e30, 2.0 ** -31, 0.0)])
def test_prompts_gate_with_the_bits_of_decode(cuda_device, clamp):
    """Gates of 24 bits beside a million ups: the quotients of prompts, which are made without a division, are those of decode's division.
    (Sums of three parts and a zero are exact in either product.)"""
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(31)
    n, rows = 4096, 256
    gates = torch.randn(n, generator=g) * torch.exp(torch.rand(n, generator=g) * 8 - 5)
    gates[:64] = torch.tensor([0.0, -0.0, 1e-30, -1e-38, 39.9, -39.9, -40.1, -87.5, -89.0, -104.0, 104.0, 1e17, 2e18, -2e18, 3e38, -3e38]).repeat(4)
    w = torch.zeros(2 * n, 64, dtype=torch.bfloat16)
    left = gates.clone()
    for part in range(3):
        w[:n, part] = left.bfloat16()
        left = left - w[:n, part].float()
    w[n:, 3] = torch.randn(n, generator=g).bfloat16()
    a = torch.zeros(rows, 64, dtype=torch.bfloat16)
    a[:, :3] = 1.0
    a[:, 3] = torch.randn(rows, generator=g).bfloat16()
    epilogue = ops.EPI_SWIGLU if clamp is None else ops.EPI_CLAMPED
    a, w = a.cuda(), w.cuda()
    got = ops.gemm_tcgen05(a, w, epilogue, clamp=clamp)
    decoded = torch.cat([ops.skinny_gemm(w, epilogue, x=a[i:i + 8].contiguous(), clamp=clamp) for i in range(0, rows, 8)])
    assert torch.equal(got.view(torch.int16), decoded.view(torch.int16))


@pytest.mark.parametrize("batch", [1, 3, 8])
@pytest.mark.parametrize("n,k", [(2048, 4104), (37, 5000), (16, 8192), (2360, 8192)])
def test_skinny_gemm_streams_activations(cuda_device, batch, n, k):
    """One row tile a block and a long K: the shortest one, one that ends within a step, rows that end within a tile, and 148 tiles."""
    from models_b200.kernels import ops

    g = torch.Generator().manual_seed(n + k)
    w, x = (torch.randn(n, k, generator=g) * 0.05).bfloat16(), torch.randn(batch, k, generator=g).bfloat16()
    exact = x.double() @ w.double().t()
    scale, wd = float(exact.abs().max()), w.cuda()
    xd = torch.full((batch, k + 8), 9.0, dtype=torch.bfloat16, device=cuda_device)[:, :k]
    xd.copy_(x)
    # k float additions of products that are exact, the eight warps' sums among them
    assert float((ops.skinny_gemm(wd, ops.EPI_F32, x=xd).double().cpu() - exact).abs().max()) < 2.0 ** -23 * scale * math.sqrt(k) * 4
    out = torch.randn(batch, n, generator=g)
    got = ops.skinny_gemm(wd, ops.EPI_RESIDUAL, x=xd, out=out.cuda())
    assert float((got.double().cpu() - out.double() - exact).abs().max()) < 2.0 ** -23 * (scale + 4) * math.sqrt(k) * 4


@pytest.mark.parametrize("dim,vdim", [(64, 128), (128, 64)])
@pytest.mark.parametrize("cap,sink,turned", [(5.0, True, True), (0.0, True, False), (30.0, False, True)])
def test_shaped_scores_on_tcgen05(cuda_device, dim, vdim, cap, sink, turned):
    """Prompts at the edges of query tiles and pages, some on top of cached positions, with factors of either sign on the scores, against
    the kernel with a warp per row."""
    from models_b200.kernels import ops

    heads, kv_heads, page = 4, 2, 64
    g = torch.Generator().manual_seed(31)
    q_lens, past = [33, 64, 129, 1, 70], [0, 100, 64, 5, 0]
    lens = [a + b for a, b in zip(q_lens, past)]
    pages = [-(-n // page) for n in lens]
    table = torch.zeros(len(lens), max(pages), dtype=torch.int32)
    order = (torch.randperm(sum(pages), generator=g) + 1).to(torch.int32)
    at = 0
    for i, n in enumerate(pages):
        table[i, :n] = order[at:at + n]
        at += n
    k_pool, v_pool = (torch.randn(sum(pages) + 1, kv_heads, page, d, generator=g).bfloat16() for d in (dim, vdim))
    for i, n in enumerate(lens):  # what lies behind a sequence's end belongs to nobody
        if n % page:
            k_pool[table[i, n // page], :, n % page:] = v_pool[table[i, n // page], :, n % page:] = float("nan")
    T = sum(q_lens)
    q = torch.randn(T, heads * dim, generator=g).bfloat16().cuda()
    head_scale = torch.tensor([1.0, -0.7, 2.0, 0.0]).cuda()
    angle = torch.rand(max(lens), vdim // 2, generator=g) * 6
    turn = (angle.cos().cuda(), angle.sin().cuda()) if turned else (None, None)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32).cuda()  # noqa: E731
    outs = []
    for kernel in (None, "rows"):
        out = torch.full((T, heads * vdim), float("nan")).bfloat16().cuda()
        with ops.recording() as names:
            ops.gated_attention(q, out, k_pool.cuda(), v_pool.cuda(), table.cuda(), i32(np.concatenate([[0], np.cumsum(q_lens)]).tolist()), i32(lens),
                                max(q_lens), heads, kv_heads, dim, vdim, "softmax", dim ** -0.5, head_scale=head_scale, softcap=cap, sink=sink,
                                turn_cos=turn[0], turn_sin=turn[1], kernel=kernel)
        assert names == ["gated_attention"]
        assert ops.float_weight_attention_takes(q, out, k_pool.cuda(), v_pool.cuda(), dim, vdim, max(q_lens))
        outs.append(out.float())
    # float weights either way: what differs is a rounding to bfloat16 of the result here and there
    assert float((outs[0] - outs[1]).abs().max()) <= 2.0 ** -7 * float(outs[1].abs().max())
    assert float((outs[0] - outs[1]).norm()) <= 2.0 ** -9 * float(outs[1].norm())


@pytest.mark.parametrize("cap", [50.0, 8.0])
@pytest.mark.parametrize("size", [0.3, 1.0, 2.2, 6.0])
def test_bounded_scores_small_and_large(cuda_device, cap, size):
    """Scores without a word on their size, from small ones to far beyond the bound, in the same rows and in rows of their own, against 64 bits: the
    weights' two bfloat16 parts (2^-16), the score's float arithmetic and the result's rounding (eight bits: up to 2^-8 of it)."""
    from models_b200.kernels import ops

    heads, dim, vdim, lens = 2, 64, 128, [200, 65]
    g = torch.Generator().manual_seed(int(cap))
    k_pool, v_pool = (torch.randn(7, 1, 64, d, generator=g).bfloat16() for d in (dim, vdim))
    k_pool[2] *= 5.0  # positions 64 to 127 of the first sequence
    table = torch.tensor([[1, 2, 3, 4], [5, 6, 0, 0]], dtype=torch.int32)
    T = sum(lens)
    q = (torch.randn(T, heads * dim, generator=g) * size).bfloat16()
    q[100:140] *= 0.05
    i32 = lambda v: torch.tensor(v, dtype=torch.int32).cuda()  # noqa: E731
    out = torch.zeros(T, heads * vdim, dtype=torch.bfloat16, device=cuda_device)
    ops.gated_attention(q.cuda(), out, k_pool.cuda(), v_pool.cuda(), table.cuda(), i32([0, 200, 265]), i32(lens), 200, heads, 1, dim, vdim, "softmax",
                        0.125, softcap=cap, sink=True)
    at = 0
    for i, n in enumerate(lens):
        k, v = (torch.cat([p[t, 0] for t in table[i]])[:n].double() for p in (k_pool, v_pool))
        for h in range(heads):
            s = cap * torch.tanh(q[at:at + n, h * dim:(h + 1) * dim].double() @ k.t() * 0.125 / cap)
            s = s.masked_fill(torch.ones(n, n, dtype=torch.bool).triu(1), -math.inf)
            top = s.amax(1, keepdim=True).clamp(min=0)
            w = torch.exp(s - top)
            want = w / (w.sum(1, keepdim=True) + torch.exp(-top)) @ v
            error = (out[at:at + n, h * vdim:(h + 1) * vdim].double().cpu() - want).abs()
            assert bool((error <= 2.0 ** -8 * want.abs() + 2.0 ** -14 * v.abs().max()).all())
        at += n


@pytest.mark.parametrize("sequences,tokens,most,tcgen05", [(8, 40, 40, True), (8, 64, 512, True), (16, 40, 640, False)])
def test_shaped_scores_of_mostly_empty_tiles(cuda_device, sequences, tokens, most, tcgen05):
    """A step that says that one sequence may hold all of its tokens (a captured one does) takes the mma.sync kernel where most tiles would be
    empty."""
    from models_b200.kernels import ops

    heads, dim, vdim, rows = 2, 64, 128, sequences * tokens
    g = torch.Generator().manual_seed(33)
    k_pool, v_pool = (torch.randn(sequences + 1, 1, 64, d, generator=g).bfloat16().cuda() for d in (dim, vdim))
    q = torch.randn(rows, heads * dim, generator=g).bfloat16().cuda()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32).cuda()  # noqa: E731
    outs = []
    for kernel in (None, "tc"):
        outs.append(torch.zeros(rows, heads * vdim, dtype=torch.bfloat16, device=cuda_device))
        ops.gated_attention(q, outs[-1], k_pool, v_pool, i32([[i + 1] for i in range(sequences)]), i32([i * tokens for i in range(sequences + 1)]),
                            i32([tokens] * sequences), most, heads, 1, dim, vdim, "softmax", 0.125, softcap=20.0, sink=True, kernel=kernel)
    assert torch.equal(*outs) != tcgen05
    assert torch.allclose(outs[0].float(), outs[1].float(), rtol=2.0 ** -7, atol=2.0 ** -9)


@pytest.mark.parametrize("cap", [50.0, 8.0])
@pytest.mark.parametrize("size,word", [(0.05, True), (0.2, True), (0.3, False), (2.2, False), (6.0, False)])
@pytest.mark.parametrize("window", [0, 70])
def test_bounded_scores_of_what_a_row_does_not_see(cuda_device, cap, size, word, window):
    """A row's bits follow from what it sees: not from what an earlier sequence left in the last page, not from keys and queries of later
    tokens, of other rows of its warp or before its window, with and without a word on the scores."""
    from models_b200.kernels import ops

    heads, dim, vdim, past, lens = 2, 64, 128, [70, 0, 10], [200, 65, 128]
    g = torch.Generator().manual_seed(int(cap))
    ends = [a + b for a, b in zip(past, lens)]
    pages = [-(-n // 64) for n in ends]
    table, at = torch.zeros(3, max(pages), dtype=torch.int32), 1
    for i, n in enumerate(pages):
        table[i, :n], at = torch.arange(at, at + n), at + n
    k, v = ([torch.randn(n * 64, d, generator=g).bfloat16() for n in pages] for d in (dim, vdim))
    q = [(torch.randn(n, heads * dim, generator=g) * size).bfloat16() for n in lens]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32).cuda()  # noqa: E731
    bound = max(float((a.float().view(-1, heads, dim) @ b.float().t()).abs().max()) for a, b in zip(q, k)) if word else 0.0
    assert not word or bound * 0.125 <= 0.5 * cap  # (the polynomial's reach)

    def run(k, v, q):
        pools = [torch.cat([torch.zeros(64, x[0].shape[1]).bfloat16(), *x]).view(-1, 1, 64, x[0].shape[1]).cuda() for x in (k, v)]
        out = torch.zeros(sum(lens), heads * vdim, dtype=torch.bfloat16, device=cuda_device)
        ops.gated_attention(torch.cat(q).cuda(), out, *pools, table.cuda(), i32(np.concatenate([[0], np.cumsum(lens)]).tolist()), i32(ends), max(lens), heads, 1,
                            dim, vdim, "softmax", 0.125, softcap=cap, sink=True, window=window, score_bound=bound)
        return list(out.view(torch.int16).split(lens))

    want = run(k, v, q)
    for left in (0.0, 3.0, 3e4, -3e38, float("nan")):  # behind the sequences' ends
        stale = [[torch.cat([x[:n], torch.full_like(x[n:], left)]) for x, n in zip(xs, ends)] for xs in (k, v)]
        assert all(torch.equal(a, b) for a, b in zip(run(*stale, q), want))
    for keep in (40, 64, 100):  # rows from there on, queries and keys, become loud or still
        for factor in (0.0, 30.0):
            changed = [[torch.cat([x[:b + min(keep, n)], x[b + min(keep, n):] * factor]) for x, b, n in zip(k, past, lens)],
                       [torch.cat([x[:keep], x[keep:] * factor]) for x in q]]
            assert all(torch.equal(a[:keep], b[:keep]) for a, b in zip(run(changed[0], v, changed[1]), want))
    if window:  # positions that the rows from 100 on do not see any more
        changed = [torch.cat([x[:b + 100 - window] * 30.0, x[b + 100 - window:]]) if n > 100 else x for x, b, n in zip(k, past, lens)]
        assert all(torch.equal(a[100:], b[100:]) for a, b in zip(run(changed, v, q), want))


@pytest.mark.parametrize("cap", [50.0, 8.0])
@pytest.mark.parametrize("dim,vdim", [(64, 128), (128, 64)])
@pytest.mark.parametrize("lens,past,window", [([200, 65], [0, 100], 0), ([128, 33], [64, 0], 0), ([300], [10], 70), ([129], [0], 1)])
def test_small_bounded_scores_by_the_callers_word(cuda_device, cap, dim, vdim, lens, past, window):
    """Scores that fill the polynomial's reach, heads of either sign, one whose scores the word does not keep small and one of factor 0, against
    64 bits: the score's float arithmetic (2^-22 of at most cap / 2), the weights' two bfloat16 parts (2^-16) and the result's rounding
    (2^-8).  The general form stays within the same, and what is not covered by the word gives its bits."""
    from models_b200.kernels import ops

    heads, ends = 4, [a + b for a, b in zip(past, lens)]
    g = torch.Generator().manual_seed(int(cap) + dim)
    pages = [-(-n // 64) for n in ends]
    table, at = torch.zeros(len(lens), max(pages), dtype=torch.int32), 0
    for i, n in enumerate(pages):
        table[i, :n], at = torch.arange(at, at + n), at + n
    unit = lambda x: (x / x.square().mean(-1, keepdim=True).sqrt()).bfloat16()  # noqa: E731
    k_pool, v_pool = unit(torch.randn(at, 1, 64, dim, generator=g)), torch.randn(at, 1, 64, vdim, generator=g).bfloat16()
    q = unit(torch.randn(sum(lens), heads, dim, generator=g))
    q[::7] = k_pool[table[0, 0], 0, 3]  # (the largest score there is)
    scale = dim ** -0.5
    whole = 0.5 * cap / (1.01 * dim * scale)  # the factor that fills the reach
    factors = torch.tensor([whole, -whole, 3.0 * whole, 0.0]).float()
    factors[0] = factors[0] * (1 - 2.0 ** -20)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32).cuda()  # noqa: E731
    outs = []
    for bound in (1.01 * dim * (1 - 2.0 ** -20), 0.0):
        out = torch.zeros(sum(lens), heads * vdim, dtype=torch.bfloat16, device=cuda_device)
        ops.gated_attention(q.view(sum(lens), -1).cuda(), out, k_pool.cuda(), v_pool.cuda(), table.cuda(), i32(np.concatenate([[0], np.cumsum(lens)]).tolist()),
                            i32(ends), max(lens), heads, 1, dim, vdim, "softmax", scale, head_scale=factors.cuda(), softcap=cap, sink=True, window=window,
                            score_bound=bound)
        outs.append(out.view(-1, heads, vdim))
    assert torch.equal(outs[0][:, 2].view(torch.int16), outs[1][:, 2].view(torch.int16))
    at = 0
    for i, (n, before) in enumerate(zip(lens, past)):
        k, v = (torch.cat([p[t, 0] for t in table[i]])[:before + n].double() for p in (k_pool, v_pool))
        i_at, j_at = torch.arange(before, before + n)[:, None], torch.arange(before + n)[None]
        unseen = (j_at > i_at) | ((i_at - j_at >= window) if window else False)
        for h in range(heads):
            s = (cap * torch.tanh(q[at:at + n, h].double() @ k.t() * scale * float(factors[h]) / cap)).masked_fill(unseen, -math.inf)
            top = s.amax(1, keepdim=True).clamp(min=0)
            w = torch.exp(s - top)
            w = w / (w.sum(1, keepdim=True) + torch.exp(-top))
            for out in outs:
                error = (out[at:at + n, h].double().cpu() - w @ v).abs()
                assert bool((error <= 2.0 ** -8 * (w @ v).abs() + (cap * 2.0 ** -21 + 2.0 ** -15) * (w @ v.abs()) + 1e-30).all())
        at += n


@pytest.mark.parametrize("bound", [-1.0, math.inf, math.nan])
def test_a_word_that_is_no_bound_is_refused(cuda_device, bound):
    from models_b200.kernels import ops

    q, out = (torch.zeros(64, 2 * 64, dtype=torch.bfloat16, device=cuda_device) for _ in range(2))
    pools = [torch.zeros(2, 1, 64, 64, dtype=torch.bfloat16, device=cuda_device) for _ in range(2)]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda_device)  # noqa: E731
    with pytest.raises(ops.KernelError, match="scores bounded by"):
        ops.gated_attention(q, out, *pools, i32([[1]]), i32([0, 64]), i32([64]), 64, 2, 1, 64, 64, "softmax", 0.125, softcap=5.0, score_bound=bound)


@pytest.mark.parametrize("max_q_len,kernel", [(1, None), (64, None), (64, "tc"), (64, "rows")])
def test_a_negative_bound_on_scores_is_refused(cuda_device, max_q_len, kernel):
    """Whichever kernel a call meets."""
    from models_b200.kernels import ops

    q, out = (torch.zeros(max_q_len, 2 * 64, dtype=torch.bfloat16, device=cuda_device) for _ in range(2))
    pools = [torch.zeros(2, 1, 64, 64, dtype=torch.bfloat16, device=cuda_device) for _ in range(2)]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda_device)  # noqa: E731
    with pytest.raises(ops.KernelError, match="softcap -1"):
        ops.gated_attention(q, out, *pools, i32([[1]]), i32([0, max_q_len]), i32([max_q_len]), max_q_len, 2, 1, 64, 64, "softmax", 0.125, softcap=-1.0,
                            kernel=kernel)


@pytest.mark.parametrize("query_latent,gate_kind,window,turned", [(128, "element", 0, 64), (0, "head", 90, 32), (128, None, 64, 0)])
@pytest.mark.parametrize("q_lens,past", [([70, 200], [0, 0]), ([150, 64, 129], [100, 0, 37]), ([33], [31])])
def test_latent_prompts_expand_the_rows_they_see(cuda_device, monkeypatch, query_latent, gate_kind, window, turned, q_lens, past):
    """A prompt whose rows are expanded into keys and values, from a sequence's start and on top of cached positions, gives what the
    attention in the latent space gives."""
    from models_b200.cache import KvCache
    from models_b200.config.specs import LatentAttentionSpec, RopeSpec
    from models_b200.engine.batch import build_step_batch
    from models_b200.parts import RunContext, Runtime, build_part, latent_attention

    monkeypatch.setattr(latent_attention, "EXPANDED_TOKENS", 0)
    width, heads, dim, vdim, rank = 256, 4, 64, 128, 128
    g = torch.Generator().manual_seed(41)
    roles = ["down_q", "down_q_norm", "up_q", "q", "down", "down_norm", "up_k", "up_v", "gate", "o"]
    spec = LatentAttentionSpec(hidden_size=width, num_heads=heads, head_dim=dim, value_dim=vdim, latent_dim=rank, scale=(dim + turned) ** -0.5, eps=1e-6,
                               gated=gate_kind is not None, weights={r: r for r in roles}, query_latent=query_latent,
                               position=RopeSpec(turned, 1e4, "half") if turned else None, window=window or None, gate_kind=gate_kind or "head")
    outs, ways, plain = [], [], latent_attention.ops.prompt_attention
    monkeypatch.setattr(latent_attention.ops, "prompt_attention", lambda *args, **kwargs: (ways.append("expanded"), plain(*args, **kwargs))[1])
    for expanded in (True, False):
        ways.append("step")
        mixer = build_part("mixer", spec, Runtime(torch.device("cuda:0"), "bfloat16", max_positions=512))
        draw = torch.Generator().manual_seed(5)
        mixer.load({p.name: (torch.randn(p.shape, generator=draw) * p.shape[-1] ** -0.5).bfloat16() if len(p.shape) > 1
                    else 1 + 0.1 * torch.randn(p.shape, generator=draw) for p in mixer.parameters()})
        assert mixer.expand is not None
        if not expanded:
            mixer.expand = None
        cache = KvCache([mixer.kv_request()], [None], 64 * 20, len(q_lens))
        cache.allocate_storage(lambda shape: torch.full(shape, float("nan"), dtype=torch.bfloat16, device="cuda:0"))
        run = RunContext(run=0)
        run.group, run.k_pool, run.v_pool = cache.pools(0)
        slots = [cache.open_slot() for _ in q_lens]
        rows = torch.Generator().manual_seed(6)
        for counts in (past, q_lens):
            entries = [(s, n) for s, n in zip(slots, counts) if n]
            if entries:
                cache.append(entries)
                batch = build_step_batch(cache, [(s, [0] * n, []) for s, n in entries], torch.device("cuda:0"))
                cache.commit(entries)
                out = mixer.forward(torch.randn(sum(n for _, n in entries), width, generator=rows).bfloat16().cuda(), batch, run)
        outs.append(out.float())
    assert ways[-2:] == ["expanded", "step"]  # the first mixer's last step, and none of the second's
    # keys, values and queries pass through bfloat16 at other places: four roundings' worth
    assert float((outs[0] - outs[1]).norm()) <= 4 * 2.0 ** -8 * float(outs[1].norm())


@pytest.mark.parametrize("query_latent,window,value_dim", [(0, 0, 64), (128, 0, 64), (0, 64, 64), (0, 0, 40)])
@pytest.mark.parametrize("q_lens", [[129, 160, 192], [160] * 40, [600]])
def test_latent_prompts_without_a_position_gated_by_elements(cuda_device, monkeypatch, query_latent, window, value_dim, q_lens):
    """Heads of 64 with no rotated part keep three tiles in flight: prompts whose last tiles see three pages, and all of a window's."""
    from models_b200.cache import KvCache
    from models_b200.config.specs import LatentAttentionSpec
    from models_b200.engine.batch import build_step_batch
    from models_b200.parts import RunContext, Runtime, build_part, latent_attention

    monkeypatch.setattr(latent_attention, "EXPANDED_TOKENS", 0)
    width, heads, dim, rank = 256, 4, 64, 128
    roles = ["down_q", "down_q_norm", "up_q", "q", "down", "down_norm", "up_k", "up_v", "gate", "o"]
    spec = LatentAttentionSpec(hidden_size=width, num_heads=heads, head_dim=dim, value_dim=value_dim, latent_dim=rank, scale=dim ** -0.5, eps=1e-6,
                               gated=True, weights={r: r for r in roles}, query_latent=query_latent, position=None, window=window or None,
                               gate_kind="element")
    outs = []
    for expanded in (True, False):
        mixer = build_part("mixer", spec, Runtime(torch.device("cuda:0"), "bfloat16", max_positions=1024))
        draw = torch.Generator().manual_seed(5)
        mixer.load({p.name: (torch.randn(p.shape, generator=draw) * p.shape[-1] ** -0.5).bfloat16() if len(p.shape) > 1
                    else 1 + 0.1 * torch.randn(p.shape, generator=draw) for p in mixer.parameters()})
        assert mixer.expand is not None
        if not expanded:
            mixer.expand = None
        cache = KvCache([mixer.kv_request()], [None], sum(q_lens) + 64 * 2 * len(q_lens), len(q_lens))
        cache.allocate_storage(lambda shape: torch.full(shape, float("nan"), dtype=torch.bfloat16, device="cuda:0"))
        run = RunContext(run=0)
        run.group, run.k_pool, run.v_pool = cache.pools(0)
        entries = [(cache.open_slot(), n) for n in q_lens]
        cache.append(entries)
        batch = build_step_batch(cache, [(s, [0] * n, []) for s, n in entries], torch.device("cuda:0"))
        cache.commit(entries)
        x = torch.randn(sum(q_lens), width, generator=torch.Generator().manual_seed(6)).bfloat16().cuda()
        outs.append(mixer.forward(x, batch, run).float())
    # keys, values and queries pass through bfloat16 at other places: four roundings' worth
    assert float((outs[0] - outs[1]).norm()) <= 4 * 2.0 ** -8 * float(outs[1].norm())


@pytest.mark.parametrize("window,past,q_lens", [(90, [300, 40], [150, 129]), (64, [127, 641], [33, 65]), (1, [200, 0], [70, 64])])
def test_latent_prompts_expand_only_what_their_window_sees(cuda_device, monkeypatch, window, past, q_lens):
    """On top of a cache that gave pages back: the rows gathered begin at the window's first page, and what lies before it (not a number here)
    is not touched; beyond the workspace's bound a step stays in the latent space."""
    from models_b200.cache import KvCache
    from models_b200.config.specs import LatentAttentionSpec, RopeSpec
    from models_b200.engine.batch import build_step_batch
    from models_b200.kernels import ops
    from models_b200.parts import RunContext, Runtime, build_part, latent_attention

    monkeypatch.setattr(latent_attention, "EXPANDED_TOKENS", 0)
    width, heads, dim, vdim, rank, turned = 256, 4, 64, 128, 128, 64
    roles = ["down_q", "down_q_norm", "up_q", "down", "down_norm", "up_k", "up_v", "o"]
    spec = LatentAttentionSpec(hidden_size=width, num_heads=heads, head_dim=dim, value_dim=vdim, latent_dim=rank, scale=(dim + turned) ** -0.5, eps=1e-6,
                               gated=False, weights={r: r for r in roles}, query_latent=128, position=RopeSpec(turned, 1e4, "half"), window=window)
    outs, gathered, plain_gather = [], [], ops.latent_gather

    def gather(*args):
        rows = plain_gather(*args)
        gathered.append((args[5], rows))
        return rows

    monkeypatch.setattr(ops, "latent_gather", gather)
    for most in (latent_attention.EXPANDED_BYTES, 0):
        monkeypatch.setattr(latent_attention, "EXPANDED_BYTES", most)
        mixer = build_part("mixer", spec, Runtime(torch.device("cuda:0"), "bfloat16", max_positions=1024))
        draw = torch.Generator().manual_seed(5)
        mixer.load({p.name: (torch.randn(p.shape, generator=draw) * p.shape[-1] ** -0.5).bfloat16() if len(p.shape) > 1
                    else 1 + 0.1 * torch.randn(p.shape, generator=draw) for p in mixer.parameters()})
        cache = KvCache([mixer.kv_request()], [None], 64 * 30, len(q_lens))
        cache.allocate_storage(lambda shape: torch.full(shape, float("nan"), dtype=torch.bfloat16, device="cuda:0"))
        run = RunContext(run=0)
        run.group, run.k_pool, run.v_pool = cache.pools(0)
        slots = [cache.open_slot() for _ in q_lens]
        rows = torch.Generator().manual_seed(6)
        for counts in (past, q_lens):
            entries = [(s, n) for s, n in zip(slots, counts) if n]
            cache.append(entries)
            batch = build_step_batch(cache, [(s, [0] * n, []) for s, n in entries], torch.device("cuda:0"))
            cache.commit(entries)
            out = mixer.forward(torch.randn(sum(n for _, n in entries), width, generator=rows).bfloat16().cuda(), batch, run)
        outs.append(out.float())
    assert len(gathered) == 1  # (the second mixer's steps stay in the latent space)
    per, (latents, tails) = gathered[0]
    assert per % 64 == 0 and per <= max(64, min(-(-max(a + b for a, b in zip(past, q_lens)) // 64) * 64, window + max(q_lens) + 126))
    for i, (before, n) in enumerate(zip(past, q_lens)):
        first = max(0, before - window + 1) // 64 * 64
        for kept in (latents, tails):
            assert bool(kept[i * per:i * per + before + n - first].isfinite().all())
    assert bool(outs[0].isfinite().all()) and float((outs[0] - outs[1]).norm()) <= 4 * 2.0 ** -8 * float(outs[1].norm())
