"""Kernel variants at the edges of their ranges: the sizes where a launch changes shape, remainders of its
tiles, and the smallest and largest of what it takes, against the oracle."""
import numpy as np
import pytest
import torch

from oracle import adamas_ref as ref
from test_gpu_parity import DEV, State, _assert_attn_close, _mods, _randn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hq,hk", [(32, 32), (28, 4), (3, 1)])
@pytest.mark.parametrize("seq", [1, 2, 4735, 4737, 4739])   # several tokens per block from 4736 on, with remainders
def test_rope_token_groups(seq, hq, hk):
    _, K, U = _mods()
    q, k = _randn((seq, hq, 128), 1 + seq, torch.float16), _randn((seq, hk, 128), 2 + seq, torch.float16)
    qd, kd = q.to(DEV), k.to(DEV)
    U.apply_rope_in_place(qd, kd, 100, rope_scale=8.0)
    # the reference's tolerance for this operator (adamas/tests/test_rope.py:10-15)
    torch.testing.assert_close(qd.cpu().float(), ref.rope(q, 100, 8.0).float(), rtol=5e-3, atol=5e-3)
    torch.testing.assert_close(kd.cpu().float(), ref.rope(k, 100, 8.0).float(), rtol=5e-3, atol=5e-3)


@pytest.mark.parametrize("hq,hkv,L,ps", [
    (32, 32, 1, 16), (32, 32, 17, 16), (4, 4, 63, 1),     # single tile, tile remainders
    (8, 8, 700, 7),                                       # blocks share a row evenly
    (32, 32, 2500, 16),                                   # the line of tiles is cut over the grid
    (32, 8, 9473, 16), (28, 4, 16001, 32),                # grouped queries in one part, line cut inside rows
    (12, 1, 333, 16), (32, 2, 5000, 16), (9, 1, 20000, 1),   # groups of more than 8: several parts
    (1, 1, 20001, 16), (2, 1, 9000, 16),                  # many parts of one and of two query heads: merged by all warps
])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_dense_decode_shapes(hq, hkv, L, ps, dtype):
    """Attention over every token (one page list for all heads) at the edges of the tiles and of the two ways
    in which the work is cut, all query heads of a cache head together."""
    _, K, _ = _mods()
    pages = (L + ps - 1) // ps
    perm = torch.randperm(pages, generator=torch.Generator().manual_seed(L))
    kv = _randn((pages, 2, ps, hkv, 128), 7 + L, dtype)
    q = _randn((1, hq, 128), 8 + L, dtype)
    last = L - (pages - 1) * ps
    w = K.BatchDecodeWithPagedKVCachePyTorchWrapper(0)
    w.begin_forward(torch.tensor([0, pages], dtype=torch.int32), hq, hkv, 128, ps, torch.empty(0, dtype=dtype))
    table = perm.to(torch.int32).to(DEV)
    o, lse = torch.empty_like(q.to(DEV)), torch.zeros(hq, dtype=torch.float32, device=DEV)
    for _ in range(2):      # (the counters are back at zero after a launch)
        w.forward(q.to(DEV), o, kv.to(DEV), table[: pages - 1].unsqueeze(0).expand(hq, pages - 1), None, last, int(perm[-1]), lse=lse)
    t = torch.arange(L)
    k_all, v_all = (ref.repeat_kv(kv[perm[t // ps], i, t % ps], hq // hkv) for i in (0, 1))
    want = ref.sparse_attention(q[0], k_all, v_all, np.tile(np.arange(L), (hq, 1)))
    _assert_attn_close(o[0], want)
    s = torch.einsum("hd,lhd->hl", q[0].float(), k_all.float()) / np.sqrt(128.0)
    torch.testing.assert_close(lse.cpu(), torch.logsumexp(s, 1) / np.log(2.0), rtol=1e-4, atol=1e-3)


def test_sparse_decode_list_with_holes():
    """Negative list entries are skipped: whole tiles of them, single ones, and a list of nothing else."""
    _, K, _ = _mods()
    H, L, ps, n = 4, 900, 16, 130
    pages = (L + ps - 1) // ps
    kv = _randn((pages, 2, ps, H, 128), 3, torch.float16)
    q = _randn((1, H, 128), 4, torch.float16)
    idx = torch.stack([torch.randperm(L - 1, generator=torch.Generator().manual_seed(h))[:n] for h in range(H)]).to(torch.int32)
    idx[0, 16:64] = -1
    idx[1, ::3] = -1
    idx[2, :] = -1
    w = K.BatchDecodeWithPagedKVCachePyTorchWrapper(0)
    w.begin_forward(torch.tensor([0, n], dtype=torch.int32), H, H, 128, ps, torch.empty(0, dtype=torch.float16))
    o = torch.empty_like(q.to(DEV))
    w.forward(q.to(DEV), o, kv.to(DEV), idx.to(DEV), None, (L - 1) % ps + 1, pages - 1, token_granular=True)
    flat = kv.permute(0, 2, 1, 3, 4).reshape(pages * ps, 2, H, 128)
    for h in range(H):
        sel = np.append(idx[h][idx[h] >= 0].numpy(), L - 1)
        want = ref.sparse_attention(q[0, h:h + 1], flat[:, 0, h:h + 1], flat[:, 1, h:h + 1], sel[None])
        _assert_attn_close(o[0, h:h + 1], want)


@pytest.mark.parametrize("H,Hq", [(1, 1), (2, 2), (3, 9), (4, 4), (5, 5), (8, 64), (4, 28), (2, 32), (12, 12), (28, 28), (40, 40), (6, 48), (96, 96)])
@pytest.mark.parametrize("L,ps", [(2, 16), (33, 1), (130, 16), (257, 7), (5000, 32), (40001, 16)])
def test_estimate_items_shapes(H, Hq, L, ps):
    """The estimate for any head count: remainders of its items, one item, several per warp, counts in shared memory and, with few
    tokens a block, in global memory; distances and per-slice counts exact, grouped queries included."""
    _, K, _ = _mods()
    if Hq * L > 1 << 22:
        pytest.skip("larger than the range this is about")
    g = torch.Generator().manual_seed(L + H)
    pages = (L + ps - 1) // ps
    perm = torch.randperm(pages, generator=g)
    codes = torch.randint(-32768, 32768, (pages, 1, ps, H, 16), generator=g, dtype=torch.int32).to(torch.int16)
    q = torch.randint(-32768, 32768, (1, Hq, 16), generator=g, dtype=torch.int32).to(torch.int16)
    n = L - 1
    slices = 5
    store = torch.zeros(Hq, (n + 7) // 8 * 8, dtype=torch.int16, device=DEV)
    hist = K.histogram_scratch(Hq, DEV)
    K.estimate_attn_score(q.to(DEV), store[:, :n], codes.to(DEV), perm.to(torch.int32).to(DEV), None, L - (pages - 1) * ps, 0, 0,
                          hist=hist, hist_slices=slices)
    t = torch.arange(n)
    kc = codes[perm[t // ps], 0, t % ps]                                  # [n, H, 16]
    want = torch.empty(Hq, n, dtype=torch.int64)
    def bits(x):
        x = x.to(torch.int32) & 0xffff
        return torch.stack([(x >> (2 * i)) & 3 for i in range(8)], -1).flatten(-2).to(torch.int8)
    qb, group = bits(q[0]), Hq // H
    for h in range(H):
        kb = bits(kc[:, h])
        for r in range(h * group, (h + 1) * group):
            want[r] = (kb - qb[r]).abs().sum(1, dtype=torch.int64)
    got = store[:, :n].cpu().to(torch.int64)
    assert torch.equal(got, want)
    per = ((((n + 7) // 8 + slices - 1) // slices + 3) // 4 * 4) * 8      # tokens per slice
    counts = K.histogram_counts(hist).cpu()
    for r in (0, Hq // 2, Hq - 1):
        for sl in range(slices):
            assert torch.equal(counts[r, sl].to(torch.int64), torch.bincount(want[r, sl * per:(sl + 1) * per], minlength=512))


# (The line between the kernels has moved since the lengths of the next two tests were chosen: with counts they are all in the item kernel.  The
# tests of short rows behind them stand on it.)
@pytest.mark.parametrize("H,L", [(16, 65536), (16, 65537), (32, 49152), (32, 49153), (64, 24576), (64, 24577)])
def test_estimate_on_both_sides_of_the_kernels_line(H, L):
    """16, 32 and 64 heads: the last length of the tile pipeline and the first one of the item kernel; exact."""
    test_estimate_items_shapes(H, H, L, 16)


@pytest.mark.parametrize("H,L,dtype", [(16, 65536, torch.float16), (16, 65537, torch.bfloat16), (32, 49152, torch.float16), (32, 49153, torch.bfloat16),
                                       (64, 24576, torch.float16), (64, 24577, torch.float16), (151, 6000, torch.float16)])
def test_step_on_both_sides_of_the_kernels_line(H, L, dtype):
    """The fused step (append, rotation and counts inside the estimate) selects what the separate operators do, at the last length of the
    tile pipeline and the first one of the item kernel; 151 heads: more pieces than half of the blocks."""
    _, K, U = _mods()
    budget, ps, rope = 256, 16, (8.0, 1e4)
    gen = torch.Generator(device=DEV).manual_seed(L)
    rand = lambda n: torch.randn(n, H, 128, device=DEV, generator=gen).to(dtype)
    k, v = rand(L), rand(L)
    q, k1, v1 = rand(1), rand(1), rand(1)
    found = []
    for fused in (True, False):
        c = U.InferenceController(1, H, 128, ps, budget // ps, L + 1, dtype, DEV)
        c.prepare_hadamard(L)
        c.begin_forward(L)
        U.append_kvh(k, v, None, c, 0)
        c.end_forward()
        c.prepare_hadamard(1)
        c.begin_forward(1)
        qd, kd = q.clone(), k1.clone()
        if fused:
            U.decode_step(qd, kd, v1, c, 0, rope=rope)
        else:
            U.decode_topk(U.decode_estimate(U.append_qkv_fused(qd, kd, v1, c, 0, rope=rope), c, 0), c)
        code = c.hadamard_cache.buf_layer(0)[c.hadamard_cache.indicies[-1], 0, L % ps].view(torch.int16)
        found.append((c.topk_dindices_buffer.sort(1).values, qd.view(torch.int16), kd.view(torch.int16), code.clone()))
        c.end_forward()
    for a, b in zip(*found):
        assert torch.equal(a, b)


@pytest.mark.parametrize("H,L", [(16, 3585), (16, 3586), (32, 3585), (32, 3586), (64, 1500)])
def test_estimate_of_short_rows_on_both_sides_of_the_kernels_line(H, L):
    """16 and 32 heads with counts: the last length of the tile pipeline (3584 tokens in front of the newest) and the first one of the item
    kernel; 64 heads, in the item kernel; exact."""
    test_estimate_items_shapes(H, H, L, 16)


@pytest.mark.parametrize("H,n", [(16, 65535), (16, 65536), (32, 65536), (64, 30000)])
def test_estimate_without_counts_on_both_sides_of_the_kernels_line(H, n):
    """16 heads without counts: the last length of the tile pipeline and the first one of the item kernel; 32 and 64: the tile pipeline.
    The distances are those of the same call with counts."""
    _, K, _ = _mods()
    ps = 16
    pages = n // ps + 1
    g = torch.Generator(device=DEV).manual_seed(n)
    codes = torch.randint(-32768, 32768, (pages, 1, ps, H, 16), generator=g, device=DEV).to(torch.int16)
    q = torch.randint(-32768, 32768, (1, H, 16), generator=g, device=DEV).to(torch.int16)
    table = torch.randperm(pages, generator=g, device=DEV).to(torch.int32)
    stores = [torch.zeros(H, (n + 7) // 8 * 8, dtype=torch.int16, device=DEV) for _ in range(2)]
    last = n + 1 - (pages - 1) * ps
    K.estimate_attn_score(q, stores[0][:, :n], codes, table, None, last, 0, 0)
    K.estimate_attn_score(q, stores[1][:, :n], codes, table, None, last, 0, 0, hist=K.histogram_scratch(H, DEV), hist_slices=8)
    assert torch.equal(stores[0], stores[1]) and int(stores[0].max()) > 0


@pytest.mark.parametrize("H,L,rope,dtype", [
    (16, 3584, None, torch.float16), (16, 3585, None, torch.float16), (32, 3584, None, torch.bfloat16), (32, 3585, None, torch.bfloat16),
    (16, 600, (8.0, 1e4), torch.bfloat16), (32, 600, (8.0, 1e4), torch.float16)])
def test_step_of_short_rows_on_both_sides_of_the_kernels_line(H, L, rope, dtype):
    """The fused step (append, rotation and counts inside the estimate) selects what the separate operators do, without rotation at the
    last length of the tile pipeline and the first one of the item kernel, with it in the item kernel."""
    _, K, U = _mods()
    budget, ps = 256, 16
    gen = torch.Generator(device=DEV).manual_seed(L)
    rand = lambda n: torch.randn(n, H, 128, device=DEV, generator=gen).to(dtype)
    k, v = rand(L), rand(L)
    q, k1, v1 = rand(1), rand(1), rand(1)
    found = []
    for fused in (True, False):
        c = U.InferenceController(1, H, 128, ps, budget // ps, L + 1, dtype, DEV)
        c.prepare_hadamard(L)
        c.begin_forward(L)
        U.append_kvh(k, v, None, c, 0)
        c.end_forward()
        c.prepare_hadamard(1)
        c.begin_forward(1)
        qd, kd = q.clone(), k1.clone()
        if fused:
            U.decode_step(qd, kd, v1, c, 0, rope=rope)
        else:
            U.decode_topk(U.decode_estimate(U.append_qkv_fused(qd, kd, v1, c, 0, rope=rope), c, 0), c)
        code = c.hadamard_cache.buf_layer(0)[c.hadamard_cache.indicies[-1], 0, L % ps].view(torch.int16)
        found.append((c.topk_dindices_buffer.sort(1).values, qd.view(torch.int16), kd.view(torch.int16), code.clone()))
        c.end_forward()
    for a, b in zip(*found):
        assert torch.equal(a, b)


@pytest.mark.parametrize("H,Hq", [(40, 40), (8, 64), (4, 4), (1000, 1000)])   # (1000: more pieces than blocks)
def test_estimate_leaves_half_of_every_sm(H, Hq):
    """One estimate block per SM as the setting: the same distances and counts, from half of the SM's registers and shared
    memory.  (How many blocks a launch has is checked by the CPU test of the cuts.)"""
    _, K, _ = _mods()
    L, ps = 9001 if H < 1000 else 1100, 16
    g = torch.Generator().manual_seed(H)
    pages = (L + ps - 1) // ps
    codes = torch.randint(-32768, 32768, (pages, 1, ps, H, 16), generator=g, dtype=torch.int32).to(torch.int16).to(DEV)
    q = torch.randint(-32768, 32768, (1, Hq, 16), generator=g, dtype=torch.int32).to(torch.int16).to(DEV)
    table = torch.randperm(pages, generator=g).to(torch.int32).to(DEV)
    results = []
    for blocks in (2, 1):
        K.set_estimate_blocks_per_sm(blocks)
        try:
            out = torch.zeros(Hq, L - 1, dtype=torch.int16, device=DEV)
            hist = K.histogram_scratch(Hq, DEV)
            K.estimate_attn_score(q, out, codes, table, None, L - (pages - 1) * ps, 0, 0, hist=hist, hist_slices=4)
            results.append((out, K.histogram_counts(hist)))
        finally:
            K.set_estimate_blocks_per_sm(2)
    for a, b in zip(*results):
        assert torch.equal(a, b)


def _blocks_per_head(hist):
    """Thread blocks per head of the last select_attend launch with this scratch table (zeroed before): the slots of partial
    results that hold a sum (a single block leaves none)."""
    slots = hist.view(hist.size(0), -1)[:, 16 * 512:].view(hist.size(0), 16, 132)
    return max(1, int((slots[:, :, 129] != 0).sum(1).max()))


@pytest.mark.parametrize("n,k,H,ps,blocks,slices", [
    (1, 1, 3, 16, 1, 1), (9, 9, 4, 1, 1, 1),           # fewer granules than threads; everything wins
    (2047, 72, 32, 16, 1, 1), (2049, 73, 32, 16, 2, 2),   # one block per head / two; winners around the rows of its tiles
    (2047, 96, 32, 16, 2, 2), (2049, 97, 32, 16, 2, 2),
    (30000, 1023, 32, 16, 16, 8), (32768, 2047, 8, 1, 16, 8),   # two blocks share a histogram slice; page numbers not staged (page size 1)
    (40001, 4000, 4, 7, 16, 16),                       # several rounds per warp, a page size that is no power of two
    # (20000 distances per block: nearly as many as are staged)
    (100000, 63, 100, 32, 5, 5),                       # few blocks per row: distances beyond the staged ones
    (30000, 63, 600, 16, 1, 1), (30001, 700, 592, 16, 1, 1), (400003, 1000, 2, 16, 16, 16),   # ... and beyond the 21824 that are staged per block
])
@pytest.mark.parametrize("ties", [False, True])
def test_select_attend_shapes(n, k, H, ps, blocks, slices, ties):
    """Selection (exact, ties to the lower position) and attention at the edges of the launch shapes."""
    _, K, _ = _mods()
    g = torch.Generator().manual_seed(n + k)
    dist = torch.randint(180, 183, (H, n), generator=g) if ties else (torch.randn(H, n, generator=g) * 12 + 190).round().clamp(0, 384).long()
    store = torch.zeros(H, (n + 7) // 8 * 8, dtype=torch.int16, device=DEV)
    store[:, :n] = dist.to(torch.int16).to(DEV)
    pages = (n + ps - 1) // ps
    perm = torch.randperm(pages, generator=g)
    kv = torch.empty(pages, 2, ps, 1, 128, dtype=torch.float16, device=DEV).normal_(generator=torch.Generator(device=DEV).manual_seed(n))
    q = _randn((1, H, 128), 5, torch.float16)
    idx = torch.full((H, k), -1, dtype=torch.int32, device=DEV)
    o = torch.empty_like(q.to(DEV))
    hist = K.histogram_scratch(H, DEV)
    for _ in range(2):
        K.select_attend(store[:, :n], k, q.to(DEV), o, kv, perm.to(torch.int32).to(DEV), 0, 0, indices_out=idx, hist=hist)
    # (with ties all winners are at the front: blocks without any leave no sum)
    assert K.select_attend_slices(n, k, H) == slices and (ties or _blocks_per_head(hist) == blocks)
    order = torch.argsort(dist * (n + 1) + torch.arange(n), 1)[:, :k].sort(1).values          # ascending positions of the winners
    slots = (perm[order // ps] * ps + order % ps).to(torch.int32)
    assert torch.equal(idx.cpu(), slots)
    assert int(K.histogram_counts(hist).abs().sum().item()) == 0
    flat = kv.permute(0, 2, 1, 3, 4).reshape(pages * ps, 2, 128).cpu()
    for h in (0, H // 2, H - 1):
        rows = flat[slots[h].long()]
        want = ref.sparse_attention(q[0, h:h + 1], rows[:, 0:1], rows[:, 1:2], np.arange(k)[None])
        _assert_attn_close(o[0, h:h + 1], want)


@pytest.mark.parametrize("H", [16, 32, 64])
@pytest.mark.parametrize("L", [2, 33, 34, 148 * 32 + 1, 295 * 32 + 1, 296 * 32 + 1, 297 * 32 + 1, 2 * 296 * 32 + 1, 20001])
def test_append_estimate_tiles(H, L):
    """Estimate with the append inside, where the appending block has tiles of its own and where it has none: the
    same bits as the separate append and estimate."""
    _, K, _ = _mods()
    ps, n = 16, L - 1
    pages = (L + ps - 1) // ps
    g = torch.Generator().manual_seed(L + H)
    table = torch.randperm(pages, generator=g).to(torch.int32).to(DEV)
    codes = torch.randint(-32768, 32768, (pages, 1, ps, H, 16), generator=g, dtype=torch.int32).to(torch.int16)
    q, k, v = (_randn((1, H, 128), s + L, torch.float16) for s in (1, 2, 3))
    results = []
    for inside in (False, True):
        qd, kd, vd = q.to(DEV), k.to(DEV), v.to(DEV)
        code_cache, kv_cache = codes.to(DEV), torch.zeros(pages, 2, ps, H, 128, dtype=torch.float16, device=DEV)
        q_code = torch.zeros(1, H, 16, dtype=torch.int16, device=DEV)
        dist = torch.zeros(H, (n + 7) // 8 * 8, dtype=torch.int16, device=DEV)
        last = L - (pages - 1) * ps
        if inside:
            K.append_estimate(qd, kd, vd, q_code, kv_cache, table, last, code_cache, table, last, dist[:, :n], scale=1.0)
        else:
            K.append_kv_cache_decode_fused(qd, kd, vd, q_code, kv_cache, table, last, code_cache, table, last, 0, scale=1.0)
            K.estimate_attn_score(q_code, dist[:, :n], code_cache, table, None, last, 0, 0)
        results.append([t.cpu() for t in (kv_cache, code_cache, q_code, dist)])
    for a, b in zip(*results):
        assert torch.equal(a, b)


# (All four are in the item kernel by now; the tile pipeline is in the test behind this one.)
@pytest.mark.parametrize("H,L", [(16, 70001), (32, 50001), (64, 26001), (32, 20001)])
def test_query_codes_on_any_16_bit_word(H, L):
    """Estimate with the append inside for 16, 32 and 64 heads, at lengths of the item kernel and (the last one) of the tiles: the
    query codes may start on any 16-bit word."""
    _, K, _ = _mods()
    ps, n = 16, L - 1
    pages = (L + ps - 1) // ps
    gen = torch.Generator(device=DEV).manual_seed(L)
    table = torch.randperm(pages, device=DEV, generator=gen).to(torch.int32)
    codes = torch.randint(-32768, 32768, (pages, 1, ps, H, 16), device=DEV, generator=gen).to(torch.int16)
    q, k, v = (torch.randn(1, H, 128, device=DEV, generator=gen).to(torch.float16) for _ in range(3))
    results = []
    for off in (0, 1, 2):
        code_cache, kv_cache = codes.clone(), torch.zeros(pages, 2, ps, H, 128, dtype=torch.float16, device=DEV)
        store = torch.zeros(H * 16 + 8, dtype=torch.int16, device=DEV)
        q_code = store[off:off + H * 16].view(1, H, 16)
        dist = torch.zeros(H, (n + 7) // 8 * 8, dtype=torch.int16, device=DEV)
        hist = K.histogram_scratch(H, DEV)
        last = L - (pages - 1) * ps
        K.append_estimate(q, k, v, q_code, kv_cache, table, last, code_cache, table, last, dist[:, :n], scale=1.0, hist=hist, hist_slices=8)
        assert int(store[:off].abs().sum()) == 0 and int(store[off + H * 16:].abs().sum()) == 0
        results.append([q_code.clone(), dist, code_cache, kv_cache, hist])
    for other in results[1:]:
        for a, b in zip(results[0], other):
            assert torch.equal(a, b)


@pytest.mark.parametrize("H,L", [(16, 3000), (32, 3000), (64, 700)])
def test_query_codes_of_short_rows_on_any_16_bit_word(H, L):
    """The same in the tile pipeline (16 and 32 heads at 3000 tokens) and for a short row of 64 heads."""
    test_query_codes_on_any_16_bit_word(H, L)


def _kernels_of(run):
    """Names of this library's kernels that `run` launches, and how often."""
    from collections import Counter
    from torch.profiler import ProfilerActivity, profile
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        run()
        torch.cuda.synchronize()
    names = Counter(e.name for e in p.events() if "adamas::" in e.name)
    assert names, "the profiler saw no kernel"
    return names


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("H,lengths,rope", [(32, [9000, 8000, 8999], None), (64, [3000, 2000], (8.0, 1e4)), (16, [900, 700, 300], (8.0, 1e4)), (32, [500, 300], (8.0, 1e4)), (64, [300 - 10 * i for i in range(19)], (8.0, 1e4)),
                                            (32, [700, 300], None)])
def test_step_with_query_codes_on_any_16_bit_word(H, lengths, rope, dtype):
    """A batch whose query codes start on any 16-bit word: the same kernels as with aligned ones, and the same bits."""
    _, K, U = _mods()
    B, budget, ps = len(lengths), 64, 16
    gen = torch.Generator(device=DEV).manual_seed(H)
    rand = lambda *shape: torch.randn(*shape, device=DEV, generator=gen).to(dtype)
    cs = [U.InferenceController(1, H, 128, ps, budget // ps, max(lengths) + 16, dtype, DEV) for _ in lengths]
    for c, L in zip(cs, lengths):
        c.prepare_hadamard(L - 1)
        c.begin_forward(L - 1)
        U.append_kvh(rand(L - 1, H, 128), rand(L - 1, H, 128), None, c, 0)
        c.end_forward()
    batch = U.SequenceBatch(cs)
    batch.prepare(1)
    batch.sync_seq_lens()
    q, k, v = rand(B, H, 128), rand(B, H, 128), rand(B, H, 128)
    found = []
    for off in (0, 1, 2, 8):
        store = torch.zeros(B * H * 16 + 16, dtype=dtype, device=DEV)
        batch._q_code = store[off:off + B * H * 16].view(B, H, 16)
        idx = torch.full((B * H, budget - 1), -1, dtype=torch.int32, device=DEV)
        qd, kd, o = q.clone(), k.clone(), torch.zeros_like(q)
        names = _kernels_of(lambda: batch.decode_step_dev(qd, kd, v, 0, out=o, rope=rope, indices_out=idx))
        words = store.view(torch.int16)
        assert int(words[:off].abs().sum()) == 0 and int(words[off + B * H * 16:].abs().sum()) == 0
        found.append((names, batch._q_code.view(torch.int16).clone(), qd, kd, o, idx))
    for other in found[1:]:
        assert other[0] == found[0][0]
        for a, b in zip(found[0][1:], other[1:]):
            assert torch.equal(a, b)


@pytest.mark.parametrize("H", [4, 40])
def test_query_codes_of_other_heads_start_on_16_bytes(H):
    """Other head counts refuse a query code that is not 16-byte aligned; the caches and the distances stay as they are."""
    _, K, _ = _mods()
    ps, L = 16, 200
    pages = (L + ps - 1) // ps
    table = torch.arange(pages, dtype=torch.int32, device=DEV)
    q, k, v = (_randn((1, H, 128), s, torch.float16).to(DEV) for s in (1, 2, 3))
    codes = torch.zeros(pages, 1, ps, H, 16, dtype=torch.int16, device=DEV)
    kv = torch.zeros(pages, 2, ps, H, 128, dtype=torch.float16, device=DEV)
    dist = torch.zeros(H, 200, dtype=torch.int16, device=DEV)
    store = torch.zeros(H * 16 + 8, dtype=torch.int16, device=DEV)
    with pytest.raises(Exception, match="16-byte aligned"):
        K.append_estimate(q, k, v, store[1:1 + H * 16].view(1, H, 16), kv, table, L - (pages - 1) * ps, codes, table, L - (pages - 1) * ps, dist[:, :L - 1], scale=1.0)
    assert not any(bool(t.any()) for t in (kv, codes, dist, store))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("thresholds", [(-10.0, 0.0, 10.0), (-1.0001, 0.10007, 3.14159), (float("-inf"), 0.0, float("inf")), (-1e6, 70000.0, 1e30),
                                        (0.5, float("nan"), 0.25)])
def test_prefill_codes_at_any_thresholds(thresholds, dtype):
    """The fused prefill append compares in the storage type with thresholds rounded down: the codes are those of a comparison in fp32,
    for thresholds that the type does not have, beyond its range, infinite and in any order, and values up to infinities."""
    from adamas_b200 import hadamard_transform
    _, K, _ = _mods()
    N, H, ps = 37, 3, 16
    k = _randn((N, H, 128), 5, dtype)
    k[:5] *= 3000.0
    k[5] = 60000.0   # (the first coefficient overflows fp16)
    pages = (N + ps - 1) // ps
    kd, table = k.to(DEV), torch.arange(pages, dtype=torch.int32, device=DEV)
    kv = torch.zeros(pages, 2, ps, H, 128, dtype=dtype, device=DEV)
    codes = torch.zeros(pages, 1, ps, H, 16, dtype=torch.int16, device=DEV)
    last = (N - 1) % ps + 1
    K.append_kv_cache_prefill(kd, kd, None, kv, table, None, last, 0, codes, table, None, last, 0, 0, None, thresholds)
    h = hadamard_transform(kd).float().cpu()
    bucket = sum((h > torch.tensor(t)).to(torch.int32) for t in thresholds).view(N, H, 16, 8)
    want = sum(bucket[..., i] << (2 * i) for i in range(8)).to(torch.int16)
    assert torch.equal(codes.view(pages * ps, H, 16)[:N].cpu(), want)
    assert torch.equal(kv.permute(0, 2, 1, 3, 4).reshape(pages * ps, 2, H, 128)[:N].cpu().view(torch.int16),
                       torch.stack([k, k], 1).view(torch.int16))


@pytest.mark.parametrize("given", [False, True])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("N,H,past", [(1, 1, 0), (15, 1, 3), (16, 1, 0), (17, 1, 5), (3, 5, 16), (11, 3, 2), (31, 33, 1)])
def test_prefill_around_a_block_of_rows(N, H, past, dtype, given):
    """Prompts of a few rows, sixteen to a block, behind `past` cached tokens: every row has its codes and its K and V, and no other place of
    the caches is written."""
    from adamas_b200 import hadamard_transform
    _, K, _ = _mods()
    ps, total = 4, N + past
    k, v = _randn((N, H, 128), 5, dtype).to(DEV), _randn((N, H, 128), 6, dtype).to(DEV)
    pages = (total + ps - 1) // ps
    table = torch.arange(pages - 1, -1, -1, dtype=torch.int32, device=DEV)
    kv = torch.zeros(pages + 1, 2, ps, H, 128, dtype=dtype, device=DEV)
    codes = torch.zeros(pages + 1, 1, ps, H, 16, dtype=torch.int16, device=DEV)
    last = (total - 1) % ps + 1
    h = hadamard_transform(k)
    K.append_kv_cache_prefill(k, v, h if given else None, kv, table, None, last, 0, codes, table, None, last, 0, 0, None, (-10.0, 0.0, 10.0))
    bucket = sum((h.float() > t).to(torch.int32) for t in (-10.0, 0.0, 10.0)).view(N, H, 16, 8)
    want = sum(bucket[..., i] << (2 * i) for i in range(8)).to(torch.int16)
    order = table.long()
    got = codes[order].reshape(pages * ps, H, 16)
    rows = kv[order].permute(0, 2, 1, 3, 4).reshape(pages * ps, 2, H, 128).view(torch.int16)
    assert torch.equal(got[past:total], want)
    assert torch.equal(rows[past:total], torch.stack([k, v], 1).view(torch.int16))
    for t in (got[:past], got[total:], rows[:past], rows[total:], kv[pages], codes[pages]):
        assert not bool(t.any())


@pytest.mark.parametrize("H,L", [(1, 18944), (1, 18945), (2, 9472), (2, 9473), (28, 672), (28, 673), (33, 512), (33, 513), (40, 3136), (40, 3137)])
def test_estimate_with_given_codes_around_a_tile_per_sm(H, L):
    """Given codes: the last length with a block to a tile (148 of them on the chip) and the first one with a tile per warp; 40 heads, the last one
    of those and the first one behind it."""
    test_estimate_items_shapes(H, H, L, 16)


@pytest.mark.parametrize("H,L", [(16, 5121), (16, 5122), (32, 12289), (32, 12290), (64, 4097), (64, 4098), (64, 12289), (64, 12290)])
def test_estimate_with_given_codes_on_both_sides_of_the_kernels_line(H, L):
    """Given codes and counts: the lengths on both sides of the line between the kernels; exact."""
    test_estimate_items_shapes(H, H, L, 16)
