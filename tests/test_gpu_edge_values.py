"""Arguments and values at the edge of what the operators take."""
import math

import pytest
import torch

from test_gpu_parity import DEV, _mods

pytestmark = pytest.mark.gpu


def test_flag_that_has_no_truth_value():
    """A flag that refuses to be a truth value raises its own error."""
    _, K, _ = _mods()
    x = torch.zeros(2, 128, dtype=torch.float16, device=DEV)
    with pytest.raises(RuntimeError, match="[Bb]oolean value"):
        K.hadamard_transform(x, inplace=torch.zeros(2))


@pytest.mark.parametrize("dtype,tol", [(torch.float16, 2.0 ** -11), (torch.bfloat16, 2.0 ** -8)])
def test_many_weights_far_below_the_largest(dtype, tol):
    """One dominating token over a flat remainder whose weights, 2^-25 of its own, make up 0.4 % of the sum: handler
    forward, 32-bit partial result and a batched dense step against 64 bits.  The dominating token's V is zero, so the
    remainder IS the result.  16-bit results may be off by one rounding (and what the partial may be off by, far less); the
    partial by 1e-5: the logits' difference of 25 is formed in 32 bits (25 * 2^-24 * ln 2 = 1e-6 relative)."""
    _, K, U = _mods()
    L, H, ps = 131072, 2, 16
    q = torch.zeros(1, H, 128, dtype=dtype)
    k, v = torch.zeros(L, H, 128, dtype=dtype), torch.ones(L, H, 128, dtype=dtype)
    v += (torch.randn(L, H, 128, generator=torch.Generator().manual_seed(1)) * 0.25).to(dtype)
    q[..., 0], k[5, :, 0], v[5] = 14.0, 14.0, 0.0      # 196 / sqrt(128) * log2(e) = 25.0
    s = torch.einsum("hd,lhd->hl", q[0].double(), k.double()) / 128.0 ** 0.5
    want = torch.einsum("hl,lhd->hd", torch.softmax(s, 1), v.double())

    pages = L // ps
    kv = torch.stack([k.view(pages, ps, H, 128), v.view(pages, ps, H, 128)], 1).to(DEV)
    table = torch.arange(pages, dtype=torch.int32, device=DEV)[: pages - 1].unsqueeze(0).expand(H, pages - 1)
    w = K.BatchDecodeWithPagedKVCachePyTorchWrapper(0)
    w.begin_forward(torch.tensor([0, pages], dtype=torch.int32), H, H, 128, ps, torch.empty(0, dtype=dtype))
    o, part, lse = torch.empty(1, H, 128, dtype=dtype, device=DEV), torch.empty(H, 128, device=DEV), torch.empty(H, device=DEV)
    w.forward(q.to(DEV), o, kv, table, None, ps, pages - 1, lse=lse)
    torch.testing.assert_close(o[0].cpu().double(), want, rtol=tol * 1.05, atol=0)
    w.forward(q.to(DEV), None, kv, table, None, ps, pages - 1, lse=lse, o_f32=part)
    torch.testing.assert_close(part.cpu().double(), want, rtol=1e-5, atol=0)
    torch.testing.assert_close(lse.cpu().double(), torch.logsumexp(s, 1) / math.log(2.0), rtol=1e-6, atol=1e-5)

    controllers = []
    for n in (L, 4096):
        c = U.InferenceController(1, H, 128, ps, 4, L, dtype, DEV)
        c.prepare_hadamard(n - 1)
        c.begin_forward(n - 1)
        U.append_kvh(k[: n - 1].to(DEV), v[: n - 1].to(DEV), None, c, 0)
        c.end_forward()
        controllers.append(c)
    batch = U.SequenceBatch(controllers)
    batch.prepare(1)
    batch.sync_seq_lens()
    row = lambda x: torch.stack([x[L - 1], x[4095]]).to(DEV)
    got = batch.decode_step_dev(q.expand(2, H, 128).contiguous().to(DEV), row(k), row(v), 0, dense=True)
    torch.testing.assert_close(got[0].cpu().double(), want, rtol=tol * 1.05, atol=0)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_long_sums_are_rounded(dtype):
    """32768 tokens of nearly equal weight and V = 2 + noise: the 32-bit result keeps to 1e-6.  A warp adds up 55 tiles one after
    the other, each sum rounded to 2^-24 of itself at most: 55 * 2^-24 = 3e-6 if all went one way, as cutting off
    would, and sqrt(55) * 2^-24 = 4e-7 as roundings go."""
    _, K, _ = _mods()
    L, H, ps = 32768, 32, 16
    g = torch.Generator(device=DEV).manual_seed(7)
    kv = torch.randn(L // ps, 2, ps, H, 128, device=DEV, generator=g)
    kv[:, 1] += 2
    kv = kv.to(dtype)
    q = (torch.randn(1, H, 128, device=DEV, generator=g) * 0.1).to(dtype)
    w = K.BatchDecodeWithPagedKVCachePyTorchWrapper(0)
    w.begin_forward(torch.tensor([0, L // ps], dtype=torch.int32), H, H, 128, ps, torch.empty(0, dtype=dtype))
    table = torch.arange(L // ps - 1, dtype=torch.int32, device=DEV).unsqueeze(0).expand(H, L // ps - 1)
    part, lse = torch.empty(H, 128, device=DEV), torch.empty(H, device=DEV)
    w.forward(q, None, kv, table, None, ps, L // ps - 1, lse=lse, o_f32=part)
    k, v = (kv[:, i].reshape(L, H, 128).double() for i in (0, 1))
    p = torch.softmax(torch.einsum("hd,lhd->hl", q[0].double(), k) / 128.0 ** 0.5, 1)
    want = torch.einsum("hl,lhd->hd", p, v)
    assert float((part.double() - want).norm() / want.norm()) < 1e-6


def test_results_at_the_alignment_of_a_word():
    """Attention writes to any buffer whose rows start on a 32-bit word; scratch that the kernels read in vectors is checked."""
    _, K, _ = _mods()
    H, ps, pages, last = 3, 16, 7, 4
    g = torch.Generator().manual_seed(1)
    kv = torch.randn(pages, 2, ps, H, 128, generator=g).half().to(DEV)
    q = torch.randn(1, H, 128, generator=g).half().to(DEV)
    table = torch.arange(pages, dtype=torch.int32, device=DEV)
    lists = table[: pages - 1].unsqueeze(0).expand(H, pages - 1)
    w = K.BatchDecodeWithPagedKVCachePyTorchWrapper(0)
    w.begin_forward(torch.tensor([0, pages], dtype=torch.int32), H, H, 128, ps, torch.empty(0, dtype=torch.float16))
    o, part, lse = torch.empty_like(q), torch.empty(H, 128, device=DEV), torch.empty(H, device=DEV)
    w.forward(q, o, kv, lists, None, last, pages - 1)
    w.forward(q, None, kv, lists, None, last, pages - 1, lse=lse, o_f32=part)
    for off in (1, 2, 3):
        o2 = torch.empty(H * 128 + 8, dtype=torch.float16, device=DEV)[2 * off: 2 * off + H * 128].view(1, H, 128)
        p2 = torch.empty(H * 128 + 4, device=DEV)[off: off + H * 128].view(H, 128)
        w.forward(q, o2, kv, lists, None, last, pages - 1)
        w.forward(q, None, kv, lists, None, last, pages - 1, lse=lse, o_f32=p2)
        assert torch.equal(o, o2) and torch.equal(part, p2)
    dist = torch.zeros(H, 104, dtype=torch.int16, device=DEV)[:, :99]
    words = K.histogram_scratch(H, DEV).numel()
    hist = torch.zeros(words + 1, dtype=torch.int32, device=DEV)[1:]
    with pytest.raises(RuntimeError, match="aligned"):
        K.select_attend(dist, 10, q, o, kv, table, last, pages - 1, hist=hist, hist_ready=True)


def _attend64(q, k, v, scale=128.0 ** -0.5):
    """Softmax attention of q [H, 128] over k, v [n, H, 128] in 64 bits; a weight of 0 takes no part, whatever its value is."""
    s = torch.einsum("hd,lhd->hl", q.double(), k.double()) * scale
    p = torch.softmax(s, 1).T[..., None]
    return torch.where(p > 0, p * v.double(), torch.zeros(())).sum(0)


@pytest.mark.parametrize("case", ["inf", "two infinities", "nan", "weight 0", "logits -inf"])
@pytest.mark.parametrize("L", [1, 7, 100, 3000])
def test_values_that_are_not_finite(case, L):
    """V rows with infinities and NaN count as weight times value does, and not at all where the weight is 0; a logit of -inf
    is a weight of 0, also where a warp sees nothing else.  Dense, by list, and select+attend (where a weight that
    underflows counts as the smallest number there is)."""
    _, K, _ = _mods()
    H, ps, dtype = 3, 16, torch.bfloat16
    g = torch.Generator().manual_seed(L)
    q, k, v = torch.randn(1, H, 128, generator=g), torch.randn(L, H, 128, generator=g), torch.randn(L, H, 128, generator=g)
    t = L // 2
    if case == "inf":
        v[t, 0, 3], v[t, 1, 70] = math.inf, -math.inf
    elif case == "two infinities":
        v[0, 0, 3], v[L - 1, 0, 3], v[L - 1, 1, 9] = math.inf, math.inf, math.inf
    elif case == "nan":
        v[t, 0, 3] = math.nan
    elif case == "weight 0":     # (all but the last token: a logit 2000 below)
        q[..., 0], k[: L - 1, :, 0] = 100.0, -300.0
        v[: L - 1, 0, 3], v[: L - 1, 1, 5] = math.inf, math.nan
    else:
        q[..., 0], k[: L - 1, :, 0] = 1.0, -math.inf
    q, k, v = q.to(dtype), k.to(dtype), v.to(dtype)
    pages = (L + ps - 1) // ps
    last = L - (pages - 1) * ps
    kv = torch.zeros(pages * ps, 2, H, 128, dtype=dtype)
    kv[:L, 0], kv[:L, 1] = k, v
    kv = kv.view(pages, ps, 2, H, 128).transpose(1, 2).contiguous().to(DEV)
    table = torch.arange(pages, dtype=torch.int32, device=DEV)
    want = _attend64(q[0], k, v)
    tol = dict(rtol=2.0 ** -7, atol=2.0 ** -7, equal_nan=True)
    o = torch.empty(1, H, 128, dtype=dtype, device=DEV)
    w = K.BatchDecodeWithPagedKVCachePyTorchWrapper(0)
    w.begin_forward(torch.tensor([0, pages], dtype=torch.int32), H, H, 128, ps, torch.empty(0, dtype=dtype))
    w.forward(q.to(DEV), o, kv, table[: pages - 1].unsqueeze(0).expand(H, pages - 1), None, last, pages - 1)
    torch.testing.assert_close(o[0].cpu().double(), want, **tol)
    idx = torch.arange(L - 1, dtype=torch.int32).repeat(H, 1).to(DEV)
    w.forward(q.to(DEV), o, kv, idx, None, last, pages - 1, token_granular=True)
    torch.testing.assert_close(o[0].cpu().double(), want, **tol)
    if L > 1 and case != "weight 0":
        dist = torch.zeros(H, (L + 6) // 8 * 8, dtype=torch.int16, device=DEV)
        K.select_attend(dist[:, : L - 1], L - 1, q.to(DEV), o, kv, table, last, pages - 1)
        torch.testing.assert_close(o[0].cpu().double(), want, **tol)
