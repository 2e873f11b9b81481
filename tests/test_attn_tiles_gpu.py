"""Paged attention of calls of a few rows on tcgen05 tiles (prompt_attn_kernel over ranges of the keys) against float64: head sizes and groups, row counts
around a tile, contexts around a chunk and shorter than the ranges, a batch of uneven contexts, a cache that holds NaN wherever nothing was stored."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,hd", [(64, 8, 128), (32, 8, 64), (16, 1, 128), (8, 2, 64), (4, 4, 128)])
@pytest.mark.parametrize("q_len,ctx", [(7, [1500, 64, 1, 700]), (8, [3000]), (5, [2047, 2048, 2049]), (3, [60, 130, 4000]), (40, [300, 0]), (17, [1000, 63, 65])])
def test_against_float64(heads, kv_heads, hd, q_len, ctx):
    """A probability and the output are rounded to bf16, and a weight moves with its score's error: 2^-7 + 2^-10 of sum p |v| (as derived for
    whole prompts); each range's sums are joined with weights of their own in fp32 (below 2^-20)."""
    from ssd_b200 import ops
    G, B, bs = heads // kv_heads, len(ctx), 64
    g = torch.Generator(device="cuda").manual_seed(heads * 1000 + q_len)
    pages = -(-(max(ctx) + q_len) // bs)
    order = torch.randperm(B * pages + 3, generator=torch.Generator().manual_seed(1))[:B * pages].to(torch.int32).view(B, pages).cuda()
    q = torch.randn(B * q_len, heads, hd, generator=g, device="cuda").to(torch.bfloat16)
    kc, vc = (torch.full((B * pages + 3, bs, kv_heads, hd), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    kv = []
    for b, n0 in enumerate(ctx):
        n = n0 + q_len
        k, v = (torch.randn(n, kv_heads, hd, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
        at = torch.arange(n, device="cuda")
        slots = order[b, at // bs].long() * bs + at % bs
        kc.view(-1, kv_heads, hd)[slots], vc.view(-1, kv_heads, hd)[slots] = k, v
        kv.append((k.double(), v.double()))
    lens = torch.tensor([n + q_len for n in ctx], dtype=torch.int32, device="cuda")
    out = ops.paged_attention(q, kc, vc, order.contiguous(), lens, q_len, hd ** -0.5).view(B, q_len, heads, hd).double()
    for b, n0 in enumerate(ctx):
        k, v = kv[b]
        hidden = torch.arange(n0 + q_len, device="cuda")[None, :] > torch.arange(n0, n0 + q_len, device="cuda")[:, None]
        for h in range(0, heads, max(1, heads // 8)):
            s = (q.view(B, q_len, heads, hd)[b, :, h].double() @ k[:, h // G].T) * hd ** -0.5
            p = torch.softmax(s.masked_fill(hidden, float("-inf")), -1)
            bound = (2.0 ** -7 + 2.0 ** -10) * (p @ v[:, h // G].abs())
            off = (out[b, :, h] - p @ v[:, h // G]).abs() / bound
            assert torch.isfinite(off).all() and off.max().item() < 1, (b, h, off.max().item())


@pytest.mark.parametrize("heads,kv_heads,hd,q_len,ctx", [(64, 8, 128, 7, [1500, 64, 1, 700]), (32, 8, 64, 16, [300, 2, 900, 40]), (16, 1, 128, 3, [60, 130, 4000, 7, 1000, 2, 300, 64]),
                                                         (32, 32, 128, 100, [50, 400]),
                                                         (32, 8, 64, 16, [100, 2500, 30, 700, 64, 9, 1, 333]), (64, 8, 128, 8, [700, 128, 63, 4, 2000, 1, 40, 350]), (64, 8, 128, 7, [90, 500, 3, 1700, 57, 58, 2, 250]),
                                                         (64, 8, 128, 4, [40, 300] * 8), (64, 8, 128, 3, [77] * 32)])
@pytest.mark.parametrize("table", [2048, 8192])   # (long tables: the low pieces in rows of their own)
def test_weights_keep_sixteen_bits(heads, kv_heads, hd, q_len, ctx, table):
    """The output is rounded to bf16 (eight significant bits: 2^-8 of it at most); weights are not (two pieces: 2^-17), and fp32 sums of scores and products move them
    by less than 2^-15: together 2^-14 of sum p |v|.  Weights of one bf16 piece are off by up to 2^-8 each, which short contexts show."""
    from ssd_b200 import ops
    G, B, bs = heads // kv_heads, len(ctx), 64
    g = torch.Generator(device="cuda").manual_seed(heads * 1000 + q_len)
    pages = -(-(max(ctx) + q_len) // bs)
    tables = torch.full((B, max(pages, table // bs)), -1, dtype=torch.int32, device="cuda")   # (its capacity takes the call to the tiles)
    tables[:, :pages] = torch.arange(B * pages, dtype=torch.int32, device="cuda").view(B, pages)
    q = torch.randn(B * q_len, heads, hd, generator=g, device="cuda").to(torch.bfloat16)
    kc, vc = (torch.randn(B * pages, bs, kv_heads, hd, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    lens = torch.tensor([n + q_len for n in ctx], dtype=torch.int32, device="cuda")
    out = ops.paged_attention(q, kc, vc, tables, lens, q_len, hd ** -0.5).view(B, q_len, heads, hd).double()
    for b, n0 in enumerate(ctx):
        k, v = (c.view(B, pages * bs, kv_heads, hd)[b, :n0 + q_len].double() for c in (kc, vc))
        hidden = torch.arange(n0 + q_len, device="cuda")[None, :] > torch.arange(n0, n0 + q_len, device="cuda")[:, None]
        for h in range(0, heads, max(1, heads // 8)):
            s = (q.view(B, q_len, heads, hd)[b, :, h].double() @ k[:, h // G].T) * hd ** -0.5
            p = torch.softmax(s.masked_fill(hidden, float("-inf")), -1)
            y = p @ v[:, h // G]
            bound = 2.0 ** -8 * y.abs() + 2.0 ** -14 * (p @ v[:, h // G].abs())
            assert ((out[b, :, h] - y).abs() <= bound).all(), (b, h, ((out[b, :, h] - y).abs() / bound).max().item())


def test_pages_that_a_table_does_not_name_count_as_zero_keys():
    """As in the tiles that this form takes over from: a chunk behind a table entry of -1 scores 0 and has no value."""
    from ssd_b200 import ops
    heads, kv_heads, hd, bs, n = 32, 4, 128, 64, 640
    g = torch.Generator(device="cuda").manual_seed(5)
    q = torch.randn(7, heads, hd, generator=g, device="cuda").to(torch.bfloat16)
    kc, vc = (torch.randn(40, bs, kv_heads, hd, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    tables = torch.arange(40, dtype=torch.int32, device="cuda").view(1, 40).clone()
    lens = torch.tensor([n], dtype=torch.int32, device="cuda")
    holes = tables.clone()
    holes[0, 3], holes[0, 7] = -1, -1
    kz, vz = kc.clone(), vc.clone()
    kz[[3, 7]], vz[[3, 7]] = 0, 0
    assert torch.equal(ops.paged_attention(q, kc, vc, holes, lens, 7, hd ** -0.5), ops.paged_attention(q, kz, vz, tables, lens, 7, hd ** -0.5))
