"""Sparse MLA decode kernel against the fp32 PyTorch statement of the same op."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(B, ctx, topk, seed, frac_invalid=0.0):
    from umdk_b200.ops.attention import DIM, HEADS, PAGE
    g = torch.Generator().manual_seed(seed)
    pages_per_seq = (ctx + PAGE - 1) // PAGE
    num_pages = B * pages_per_seq + 3
    kv = (torch.randn(num_pages, PAGE, DIM, generator=g) * 0.5).to(torch.bfloat16)
    perm = torch.randperm(num_pages, generator=g)[:B * pages_per_seq]
    bt = perm.reshape(B, pages_per_seq).to(torch.int32)
    q = (torch.randn(B, HEADS, DIM, generator=g) * 0.5).to(torch.bfloat16)
    idx = torch.stack([torch.randperm(ctx, generator=g)[:topk] for _ in range(B)]).to(torch.int32)
    if frac_invalid > 0:
        m = torch.rand(B, topk, generator=g) < frac_invalid
        idx[m] = -1
    return q, kv, bt, idx


@pytest.mark.parametrize("B,ctx,topk,splits,inv", [
    (1, 64, 64, 1, 0.0),
    (2, 512, 128, 1, 0.1),
    (3, 1000, 200, 1, 0.3),
    (2, 4096, 512, 2, 0.0),
    (4, 8192, 2048, 1, 0.0),
    (2, 8192, 2048, 4, 0.05),
    (2, 32768, 2048, 1, 0.0),      # the serving benchmark's context and key count
    (1, 8192, 4096, 1, 0.02),      # more keys than one CTA pair resolves: the wrapper raises the split count
    (3, 300, 50, 3, 0.0),          # splits with no keys at all
])
def test_sparse_mla_decode(B, ctx, topk, splits, inv):
    from umdk_b200.ops.attention import ref_sparse_mla_decode, sparse_mla_decode
    q, kv, bt, idx = _case(B, ctx, topk, seed=B * 7 + topk, frac_invalid=inv)
    scale = 576 ** -0.5
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    out, lse = sparse_mla_decode(q.cuda(), kv.cuda(), bt.cuda(), idx.cuda(), scale, num_splits=splits, status=status)
    torch.cuda.synchronize()
    assert status.tolist()[0] == 0, status.tolist()
    want, want_lse = ref_sparse_mla_decode(q, kv, bt, idx, scale)
    err = (out.float().cpu() - want).abs().max().item()
    rel = ((out.float().cpu() - want).norm() / want.norm()).item()
    assert rel < 2e-2, (err, rel)
    assert torch.allclose(lse.cpu(), want_lse, atol=2e-2, rtol=1e-3)


@pytest.mark.parametrize("B,topk,splits", [
    (1, 1, 1), (2, 23, 1), (2, 25, 1), (1, 47, 1), (1, 49, 1), (2, 97, 2),   # around a set's 24 and a chunk's 48 keys
    (1, 2064, 1),                                                            # all the rows one CTA pair resolves
    (1, 480, 8), (1, 480, 9), (2, 1152, 24),                                 # the merge takes eight splits at a time
])
@pytest.mark.parametrize("kind", ["plain", "half_chunks", "growing"])
def test_sparse_mla_decode_chunk_edges(B, topk, splits, kind):
    """Chunk and set remainders; chunks in which one set's keys, or all keys, are masked; scores that grow along the key
    list, so that the running maximum is raised and O rescaled in the middle of it."""
    from umdk_b200.ops.attention import ref_sparse_mla_decode, sparse_mla_decode
    q, kv, bt, idx = _case(B, 4096, topk, seed=topk + splits)
    if kind == "half_chunks":
        pos = torch.arange(topk)
        idx[:, (pos // 24) % 4 == 0] = -1
        idx[:, (pos // 48) % 4 == 1] = -1
    if kind == "growing":   # every key is a multiple of the mean query: scores rise by some 30 (in log2 units) over the list
        flat = kv.view(-1, 576)
        mean = q.float().mean(1)
        for b in range(B):
            rows = bt[b].long()[idx[b].long() // 64] * 64 + idx[b].long() % 64
            ramp = torch.linspace(0.0, 1.0, topk)[:, None] * 20.0 / mean[b].norm() ** 2 * 24
            flat[rows] = (flat[rows].float() * 0.1 + ramp * mean[b]).to(torch.bfloat16)
    scale = 576 ** -0.5
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    out, lse = sparse_mla_decode(q.cuda(), kv.cuda(), bt.cuda(), idx.cuda(), scale, num_splits=splits, status=status)
    torch.cuda.synchronize()
    assert status.tolist()[0] == 0, status.tolist()
    want, want_lse = ref_sparse_mla_decode(q, kv, bt, idx, scale)
    # P and the result are rounded to bf16 once each (2^-9 relative); the scores are exact fp32 sums of bf16 products
    assert ((out.float().cpu() - want).norm() / want.norm().clamp_min(1e-9)).item() < 2e-2
    assert torch.equal(torch.isinf(lse.cpu()), torch.isinf(want_lse))
    ok = ~torch.isinf(want_lse)
    assert torch.allclose(lse.cpu()[ok], want_lse[ok], atol=2e-2, rtol=1e-3)


# chunks around the stages of the ring: the first stages, those in the memory that Q leaves, and their second use
@pytest.mark.parametrize("topk", [144, 145, 192, 193, 240, 241, 288, 481, 529])
@pytest.mark.parametrize("kind", ["plain", "growing"])
def test_sparse_mla_decode_stage_edges(topk, kind):
    test_sparse_mla_decode_chunk_edges(2, topk, 1, kind)


@pytest.mark.parametrize("B,topk,splits,live", [(2, 1000, 10, 7), (1, 100, 13000, 3), (2, 40, 4, 1)])
def test_sparse_mla_decode_splits_without_keys(B, topk, splits, live):
    """Splits take whole chunks of keys, so the last ones may have none: their part of the scratch is neither needed nor read,
    however many there are, and the result is that of the splits which have keys."""
    from umdk_b200.ops.attention import DIM_V, HEADS, sparse_mla_decode
    q, kv, bt, idx = (t.cuda() for t in _case(B, 4096, topk, seed=topk))
    scale = 576 ** -0.5

    def run(n, ws):
        return sparse_mla_decode(q, kv, bt, idx, scale, num_splits=n, workspace=ws)

    ws = (torch.full((B, splits, HEADS, DIM_V), float("nan"), device="cuda"),
          torch.full((B, splits, HEADS), float("nan"), device="cuda"))
    out, lse = run(splits, ws)
    want, want_lse = run(live, None)
    torch.cuda.synchronize()
    if live > 1:
        assert torch.equal(out, want) and torch.equal(lse, want_lse)
    else:   # one split alone rounds its sum to bf16 directly, without the detour over a weight of one
        assert torch.allclose(out.float(), want.float(), rtol=2 ** -7, atol=1e-6) and torch.allclose(lse, want_lse, rtol=1e-5)
    assert bool(torch.isnan(ws[0][:, live:]).all()) and not bool(torch.isnan(ws[0][:, :live]).any())


# the last groups of 16 keys, one and several chunks behind them; quads of keys with none, one and all masked; the merge's ways
@pytest.mark.parametrize("B,topk,splits", [(1, 16, 1), (2, 17, 1), (1, 32, 1), (2, 33, 1), (1, 64, 1), (3, 65, 1), (1, 81, 1), (1, 800, 17),
                                           (2, 800, 17), (1, 384, 8)])
@pytest.mark.parametrize("first", [0, 3, 4])
def test_sparse_mla_decode_last_keys_and_masked_quads(B, topk, splits, first):
    from umdk_b200.ops.attention import ref_sparse_mla_decode, sparse_mla_decode
    q, kv, bt, idx = _case(B, 4096, topk, seed=topk + splits)
    pos = torch.arange(topk)
    idx[:, (pos % 16 >= 4) & (pos % 16 < 4 + first)] = -1
    idx[:, pos % 7 == 3] = -1
    scale = 576 ** -0.5
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    out, lse = sparse_mla_decode(q.cuda(), kv.cuda(), bt.cuda(), idx.cuda(), scale, num_splits=splits, status=status)
    torch.cuda.synchronize()
    assert status.tolist()[0] == 0, status.tolist()
    want, want_lse = ref_sparse_mla_decode(q, kv, bt, idx, scale)
    # P and the result are rounded to bf16 once each (2^-9 relative); the scores are exact fp32 sums of bf16 products
    assert ((out.float().cpu() - want).norm() / want.norm()).item() < 2e-2
    assert torch.allclose(lse.cpu(), want_lse, atol=2e-2, rtol=1e-3)
