"""Paged attention, KV append and the sampler against their dense / CPU oracles."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _pool(P, Hkv, D, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    k = torch.randn(P, 128, Hkv, D, device="cuda", generator=g).to(torch.bfloat16)
    v = torch.randn(P, 128, Hkv, D, device="cuda", generator=g).to(torch.bfloat16)
    return k, v


@pytest.mark.parametrize("Hq,Hkv,D", [(8, 1, 128), (8, 2, 128), (4, 4, 64), (16, 2, 128)])
def test_paged_attention_mixed_prefill_decode(Hq, Hkv, D):
    from easydel_b200.ops import serving as S

    P = 40
    kp, vp = _pool(P, Hkv, D, 1)
    # sequences: decode (1 new token, long context), chunked prefill over a cached prefix, fresh prefill
    q_lens = [1, 1, 200, 77, 1]
    kv_lens = [1000, 129, 456, 77, 5]
    B = len(q_lens)
    perm = torch.randperm(P, generator=torch.Generator().manual_seed(3)).tolist()
    maxp = max((L + 127) // 128 for L in kv_lens)
    table = torch.zeros(B, maxp, dtype=torch.int32)
    nxt = 0
    for b, L in enumerate(kv_lens):
        n = (L + 127) // 128
        table[b, :n] = torch.tensor(perm[nxt:nxt + n], dtype=torch.int32)
        nxt += n
    cu = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32)
    T = int(cu[-1])
    q = torch.randn(T, Hq, D, device="cuda").to(torch.bfloat16)
    o = S.paged_attention(q, kp, vp, cu.cuda(), torch.tensor(kv_lens, dtype=torch.int32).cuda(), table.cuda(),
                          max(q_lens))
    ref = S.paged_attention_reference(q.cpu(), kp.cpu(), vp.cpu(), cu, torch.tensor(kv_lens), table)
    assert torch.allclose(o.float().cpu(), ref.float(), atol=2e-2, rtol=2e-2), (o.float().cpu() - ref.float()).abs().max()


def test_kv_append_then_attend_matches_dense():
    from easydel_b200.ops import serving as S, reference as R

    Hq, Hkv, D, L = 8, 2, 128, 300
    kp, vp = torch.zeros(8, 128, Hkv, D, device="cuda", dtype=torch.bfloat16), torch.zeros(
        8, 128, Hkv, D, device="cuda", dtype=torch.bfloat16)
    q = torch.randn(L, Hq, D, device="cuda").to(torch.bfloat16)
    k = torch.randn(L, Hkv, D, device="cuda").to(torch.bfloat16)
    v = torch.randn(L, Hkv, D, device="cuda").to(torch.bfloat16)
    pages = [5, 2, 7]
    slots = torch.tensor([pages[i // 128] * 128 + i % 128 for i in range(L)], dtype=torch.int32, device="cuda")
    slots[10] = -1  # a padded token is skipped
    S.kv_append(k, v, kp, vp, slots)
    flat = kp.view(-1, Hkv, D)
    assert torch.equal(flat[pages[1] * 128 + 5], k[133]) and flat[pages[0] * 128 + 10].abs().sum() == 0
    slots[10] = pages[0] * 128 + 10
    S.kv_append(k, v, kp, vp, slots)
    table = torch.tensor([pages], dtype=torch.int32, device="cuda")
    o = S.paged_attention(q, kp, vp, torch.tensor([0, L], dtype=torch.int32, device="cuda"),
                          torch.tensor([L], dtype=torch.int32, device="cuda"), table, L)
    ref = R.attention(q[None], k[None], v[None], causal=True)[0]
    assert torch.allclose(o.float(), ref.float(), atol=2e-2, rtol=2e-2)


def test_sampler_greedy_penalties_and_topk():
    from easydel_b200.ops import serving as S

    R_, V = 9, 5000
    g = torch.Generator(device="cuda").manual_seed(0)
    logits = (torch.randn(R_, V, device="cuda", generator=g) * 3).to(torch.bfloat16)
    tok, lp = S.sample(logits, want_logprob=True)
    assert torch.equal(tok.long().cpu(), logits.float().argmax(-1).cpu())
    ref_lp = torch.log_softmax(logits.float(), -1).gather(-1, tok.long()[:, None]).squeeze(-1)
    assert torch.allclose(lp, ref_lp, atol=2e-3)
    # penalties change the arg-max the same way as the oracle
    counts = torch.zeros(R_, V, dtype=torch.int32, device="cuda")
    S.count_update(counts, tok)
    S.count_update(counts, tok)
    assert int(counts.sum()) == 2 * R_
    pres = torch.full((R_,), 0.5, device="cuda")
    freq = torch.full((R_,), 0.7, device="cuda")
    rep = torch.full((R_,), 1.3, device="cuda")
    tok2, _ = S.sample(logits, presence=pres, frequency=freq, repetition=rep, counts=counts)
    z = S.apply_penalties_reference(logits.cpu(), counts.cpu(), pres.cpu(), freq.cpu(), rep.cpu())
    assert torch.equal(tok2.long().cpu(), z.argmax(-1))
    # stochastic rows: draws stay inside the top-k / top-p set and follow the distribution
    temp = torch.full((R_,), 0.8, device="cuda")
    topk = torch.full((R_,), 5, dtype=torch.int32, device="cuda")
    topp = torch.full((R_,), 0.9, device="cuda")
    seeds = torch.arange(R_, dtype=torch.int64, device="cuda") + 100
    hist = torch.zeros(V)
    top5 = logits.float().topk(5, -1).indices.cpu()
    for step in range(200):
        steps = torch.full((R_,), step, dtype=torch.int32, device="cuda")
        t, _ = S.sample(logits, temperature=temp, top_k=topk, top_p=topp, seeds=seeds, steps=steps)
        t = t.long().cpu()
        assert all(int(t[r]) in top5[r].tolist() for r in range(R_))
        hist[t[0]] += 1
    p = torch.softmax(logits[0].float().cpu()[top5[0]] / 0.8, -1)
    assert hist[top5[0][0]] / 200 > 0.5 * float(p[0])
    # same seed and step -> same draw
    steps = torch.zeros(R_, dtype=torch.int32, device="cuda")
    a, _ = S.sample(logits, temperature=temp, top_k=topk, seeds=seeds, steps=steps)
    b, _ = S.sample(logits, temperature=temp, top_k=topk, seeds=seeds, steps=steps)
    assert torch.equal(a, b)


@pytest.mark.parametrize("splits", [2, 4, 7])
def test_split_kv_decode_matches_unsplit(splits):
    """Long contexts cut into page ranges and merged by log-sum-exp give the same output as one pass."""
    from easydel_b200.ops import serving as S

    torch.manual_seed(0)
    dev = "cuda"
    B, Hq, Hkv, D, P = 3, 8, 2, 128, 64
    k_pages = torch.randn(P, 128, Hkv, D, device=dev, dtype=torch.bfloat16)
    v_pages = torch.randn(P, 128, Hkv, D, device=dev, dtype=torch.bfloat16)
    kv_lens = torch.tensor([2000, 130, 901], dtype=torch.int32, device=dev)
    table = torch.zeros(B, 16, dtype=torch.int32, device=dev)
    perm = torch.randperm(P - 1, device=dev)[:48].to(torch.int32) + 1
    table[:, :16] = perm.view(3, 16)
    q = torch.randn(B, Hq, D, device=dev, dtype=torch.bfloat16)
    cu = torch.arange(B + 1, dtype=torch.int32, device=dev)
    sinks = torch.randn(Hq, device=dev)
    for sk in (None, sinks):
        ref = S.paged_attention_reference(q, k_pages, v_pages, cu, kv_lens, table, causal=True, sinks=sk)
        got = S.paged_attention_splitkv(q, k_pages, v_pages, kv_lens, table, splits, sinks=sk)
        assert (got.float() - ref.float()).abs().max() < 2e-2


def test_attn_combine_matches_reference():
    from easydel_b200.ops import serving as S

    torch.manual_seed(1)
    o = torch.randn(3, 5, 4, 64, device="cuda", dtype=torch.bfloat16)
    lse = torch.randn(3, 4, 5, device="cuda")
    lse[1, :, 2] = float("-inf")
    got, l = S.attn_combine(o, lse, want_lse=True)
    ref, lr = S.attn_combine(o.cpu(), lse.cpu(), want_lse=True)
    assert (got.float().cpu() - ref.float()).abs().max() < 2e-2 and (l.cpu() - lr).abs().max() < 1e-4


def test_greedy_sampler_fast_path_matches_argmax():
    from easydel_b200.ops import serving as S

    torch.manual_seed(2)
    logits = torch.randn(37, 128256, device="cuda", dtype=torch.bfloat16)
    tok, lp = S.sample(logits, want_logprob=True)
    ref = logits.float().argmax(-1)
    assert torch.equal(tok.long(), ref)
    ref_lp = torch.log_softmax(logits.float(), -1).gather(-1, ref[:, None])[:, 0]
    assert (lp - ref_lp).abs().max() < 1e-3


@pytest.mark.parametrize("Hq,Hkv,D", [(8, 1, 128), (32, 8, 128), (4, 4, 64), (16, 1, 128), (12, 4, 64)])
@pytest.mark.parametrize("splits,window", [(1, 0), (3, 0), (1, 200)])
def test_streaming_decode_attention(Hq, Hkv, D, splits, window):
    """The decode kernel (one query token per sequence, 32-key tiles streamed per warp) against the reference, with
    ragged key counts (1 key, a count inside a tile, several pages), key splits and a sliding window."""
    from easydel_b200.ops import serving as S

    P = 48
    kp, vp = _pool(P, Hkv, D, 5)
    kv_lens = [1, 31, 33, 128, 129, 777, 1500, 5]
    B = len(kv_lens)
    perm = torch.randperm(P, generator=torch.Generator().manual_seed(8)).tolist()
    maxp = max((L + 127) // 128 for L in kv_lens)
    table = torch.zeros(B, maxp, dtype=torch.int32)
    nxt = 0
    for b, L in enumerate(kv_lens):
        n = (L + 127) // 128
        table[b, :n] = torch.tensor(perm[nxt:nxt + n], dtype=torch.int32)
        nxt += n
    q = torch.randn(B, Hq, D, device="cuda").to(torch.bfloat16)
    sinks = torch.randn(Hq, device="cuda") if window == 0 and splits == 1 else None
    lens = torch.tensor(kv_lens, dtype=torch.int32)
    o = S.decode_attention(q, kp, vp, lens.cuda(), table.cuda(), window=window, sinks=sinks, num_splits=splits)
    ref = S.paged_attention_reference(q.cpu(), kp.cpu(), vp.cpu(), torch.arange(B + 1, dtype=torch.int32), lens, table,
                                      window=window, sinks=None if sinks is None else sinks.cpu())
    err = (o.float().cpu() - ref.float()).abs().max().item()
    assert torch.allclose(o.float().cpu(), ref.float(), atol=2e-2, rtol=2e-2), err


@pytest.mark.parametrize("B,H,ctx,splits", [(5, 16, [1, 31, 128, 700, 2049], 1), (3, 40, [513, 64, 900], 1),
                                            (2, 16, [3000, 33], 4)])
def test_latent_decode_attention_kernel(B, H, ctx, splits):
    """Absorbed-form latent attention for decode steps: 576-wide scores and 512-wide value sums over the same paged
    rows, against fp32 softmax attention over the gathered rows."""
    from easydel_b200.ops import serving as S

    torch.manual_seed(0)
    dev = "cuda"
    pages_per = (max(ctx) + 127) // 128
    P = B * pages_per + 1
    pages = (torch.randn(P, 128, 1, 576, device=dev) * 0.5).to(torch.bfloat16)
    perm = torch.randperm(P - 1, device=dev)[: B * pages_per] + 1
    table = perm.view(B, pages_per).to(torch.int32)
    lens = torch.tensor(ctx, dtype=torch.int32, device=dev)
    q = (torch.randn(B, H, 576, device=dev) * 0.5).to(torch.bfloat16)
    scale = 0.07
    o = S.mla_decode_attention(q, pages, lens, table, scale=scale, num_splits=splits)
    for b in range(B):
        rows = pages[table[b].long()].reshape(-1, 576)[: ctx[b]].float()
        s = (q[b].float() @ rows.t()) * scale
        ref = torch.softmax(s, -1) @ rows[:, :512]
        err = (o[b].float() - ref).abs().max() / ref.abs().max()
        assert err < 2e-2, (b, float(err))


@pytest.mark.parametrize("D,Dv,window,softcap", [(128, 128, 0, 0.0), (128, 64, 50, 0.0), (72, 128, 0, 5.0), (64, 64, 33, 0.0)])
def test_decode_attention_with_more_sequences_than_sms(D, Dv, window, softcap):
    """Enough (sequence, KV head) pairs for two CTAs per SM, which have two warps each: lengths around a tile of 32 keys and a
    round of two tiles, one key only, several pages."""
    from easydel_b200.ops import serving as S

    torch.manual_seed(0)
    lens = [1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 300] * 40
    B, Hkv, G = len(lens), 3, 4
    per = 3
    kp = torch.randn(B * per + 1, 128, Hkv, D, device="cuda").to(torch.bfloat16)
    vp = torch.randn(B * per + 1, 128, Hkv, Dv, device="cuda").to(torch.bfloat16)
    table = (torch.randperm(B * per, device="cuda") + 1).view(B, per).to(torch.int32)
    q = torch.randn(B, Hkv * G, D, device="cuda").to(torch.bfloat16)
    sinks = torch.randn(Hkv * G, device="cuda")
    kv = torch.tensor(lens, dtype=torch.int32, device="cuda")
    o = S.decode_attention(q, kp, vp, kv, table, window=window, sinks=sinks, softcap=softcap)
    k = kp[table.long()].reshape(B, -1, Hkv, D).double().repeat_interleave(G, 2)
    v = vp[table.long()].reshape(B, -1, Hkv, Dv).double().repeat_interleave(G, 2)
    s = torch.einsum("bhd,bkhd->bhk", q.double(), k) * D ** -0.5
    if softcap:
        s = softcap * torch.tanh(s / softcap)
    at = torch.arange(per * 128, device="cuda")[None]
    see = (at < kv[:, None]) & (at >= kv[:, None] - (window or per * 128))
    s = s.masked_fill(~see[:, None], float("-inf"))
    p = torch.softmax(torch.cat([s, sinks.double()[None, :, None].expand(B, -1, 1)], -1), -1)[..., :-1]
    want = torch.einsum("bhk,bkhd->bhd", p, v)
    # probabilities and outputs are rounded to bf16: 2^-9 each of the largest value of a row
    assert (o.double() - want).abs().max() <= 3 * 2.0 ** -9 * v.abs().max()


@pytest.mark.parametrize("H,L,R", [(17, 512, 64), (64, 512, 64), (128, 512, 64), (130, 512, 64), (40, 128, 64), (33, 320, 32),
                                   (20, 72, 24), (18, 504, 72), (24, 256, 0), (5, 512, 64), (64, 320, 256),
                                   (128, 384, 192), (96, 320, 136), (70, 384, 136), (64, 64, 512), (128, 128, 448), (64, 64, 384)])
@pytest.mark.parametrize("lens", [[1], [64, 65, 0, 700, 129], [33] * 20 + [2000], [190] * 90])
@pytest.mark.parametrize("window,splits", [(0, 1), (100, 1), (0, 3)])
def test_latent_decode_many_heads(H, L, R, lens, window, splits):
    """Latent decode attention by either kernel: partial tiles, empty sequences, windows, every cluster size (by the number
    of sequences), row widths that fill their last box or not and that leave a half more score columns than its ring of
    six boxes holds (seven or eight of them), maxima that grow along a sequence, sinks."""
    from easydel_b200.ops import _lib, serving as S

    torch.manual_seed(H + L)
    B, W = len(lens), L + R
    per = 40 if H > 16 else (max(lens) + 127) // 128        # the rule between the kernels goes by the table's width
    pages = (torch.randn(B * per + 1, 128, 1, W, device="cuda") * 0.5).to(torch.bfloat16)
    table = (torch.randperm(B * per, device="cuda") + 1).view(B, per).to(torch.int32)
    q = (torch.randn(B, H, W, device="cuda") * 0.5).to(torch.bfloat16)
    if lens[-1] > 1000:      # one late row that every head of the last sequence prefers by far
        pages[table[-1, lens[-1] // 128].long(), lens[-1] % 128 - 1] = q[-1].float().sum(0).to(torch.bfloat16) * 8
    sinks = torch.randn(H, device="cuda")
    scale = 0.3 * W ** -0.5 * 8
    kv = torch.tensor(lens, dtype=torch.int32, device="cuda")
    q_lat = q[..., :L].transpose(0, 1).contiguous().transpose(0, 1) if H % 2 else q[..., :L]     # both orders of heads
    o = S.latent_decode(q_lat, q[..., L:], pages, kv, table, scale=scale, window=window, sinks=sinks, num_splits=splits)
    torch.cuda.synchronize()
    _lib.check_status()
    assert o.shape == (B, H, L)
    for b, n in enumerate(lens):
        rows = pages[table[b].long()].reshape(-1, W)[max(0, n - window) if window else 0:n].double()
        s = torch.cat([q[b].double() @ rows.t() * scale, sinks.double()[:, None]], 1)
        want = torch.softmax(s, -1)[:, :-1] @ rows[:, :L]
        # probabilities, outputs (and partial outputs of the splits) are rounded to bf16: 2^-9 of the largest row each
        tol = 3 * 2.0 ** -8 * float(rows.abs().max() if n else 0)
        assert float((o[b].double() - want).abs().max()) <= tol, (b, n)


@pytest.mark.parametrize("H,splits", [(128, 1), (40, 4)])
def test_latent_decode_of_short_and_long_sequences_under_a_wide_table(H, splits):
    """A table far wider than the sequences: every sequence takes the form for its own length within one launch. Queries that
    are one row for all heads, or for all sequences, are views with a pitch of zero."""
    from easydel_b200.ops import serving as S

    torch.manual_seed(H)
    lens = [1, 50, 2500, 0, 190, 900]
    B, need = len(lens), 20
    pages = (torch.randn(B * need + 1, 128, 1, 576, device="cuda") * 0.5).to(torch.bfloat16)
    table = torch.zeros(B, 256, dtype=torch.int32, device="cuda")
    table[:, :need] = (torch.randperm(B * need, device="cuda") + 1).view(B, need)
    q = (torch.randn(B, H, 576, device="cuda") * 0.5).to(torch.bfloat16)
    kv = torch.tensor(lens, dtype=torch.int32, device="cuda")
    for qq in (q, q[:, :1].expand(B, H, 576), q[:1].expand(B, H, 576)):
        o = S.latent_decode(qq[..., :512], qq[..., 512:], pages, kv, table, scale=0.1, num_splits=splits)
        for b, n in enumerate(lens):
            rows = pages[table[b, :need].long()].reshape(-1, 576)[:n].double()
            want = torch.softmax(qq[b].double() @ rows.T * 0.1, -1) @ rows[:, :512]
            # as above: probabilities, outputs and partial outputs rounded to bf16
            assert float((o[b].double() - want).abs().max()) <= 3 * 2.0 ** -8 * float(rows.abs().max() if n else 0), (b, n)


def test_latent_view_plans_its_own_splits():
    """The step's key splits are counted for the KV heads of a cache; all heads of a latent view share its rows, so it splits
    keys by sequences and heads, and 32 sequences of 128 heads not at all."""
    from types import SimpleNamespace

    from easydel_b200.caching.paged import PagedBatchMeta, PagedLatentView

    torch.manual_seed(0)
    B, H, n = 32, 128, 700
    rnd = lambda *s: (torch.randn(*s, device="cuda") * 0.3).to(torch.bfloat16)
    mla = SimpleNamespace(kv_b_proj=SimpleNamespace(weight=rnd(H * 256, 512)), nope=128, vd=128, rope_dim=64, scale=0.07)
    table = torch.arange(B * 32, dtype=torch.int32, device="cuda").view(B, 32)
    view = PagedLatentView(rnd(B * 32, 128, 1, 576))
    meta = PagedBatchMeta(cu_q=torch.arange(B + 1, dtype=torch.int32, device="cuda"),
                          kv_lens=torch.full((B,), n, dtype=torch.int32, device="cuda"), page_table=table,
                          slot_mapping=table[:, (n - 1) // 128] * 128 + (n - 1) % 128, max_q=1, num_seqs=B)
    args = rnd(1, B, H, 128), rnd(1, B, H, 64), rnd(1, B, 512), rnd(1, B, 64)
    got = []
    for meta.num_splits in (1, 4):
        got.append(view.attend_latent(mla, *args, meta))
    assert torch.equal(*got)


@pytest.mark.parametrize("B,H,n", [(32, 128, 600), (4, 128, 2000), (100, 64, 300)])
def test_latent_decode_of_peaked_scores_keeps_the_output_s_precision(B, H, n):
    """Scores of a standard deviation of 2.25, so that a few keys carry most of a sum and maxima grow along a sequence: what is
    left of the error against 64 bits is the rounding of the output to bf16 (7 stored bits: 2^-7 / sqrt(12) of a unit, over
    mantissas that are log-uniform 0.7355 of that), and a tenth for the rest."""
    from easydel_b200.ops import serving as S

    torch.manual_seed(n)
    per = (n + 127) // 128
    pages = (torch.randn(B * per + 1, 128, 1, 576, device="cuda") * 1.5).to(torch.bfloat16)
    table = (torch.randperm(B * per, device="cuda") + 1).view(B, per).to(torch.int32)
    q = (torch.randn(B, H, 576, device="cuda") * 1.5).to(torch.bfloat16)
    kv = torch.full((B,), n, dtype=torch.int32, device="cuda")
    o = S.mla_decode_attention(q, pages, kv, table, scale=1 / 24)
    rows = pages[table.long()].reshape(B, -1, 576)[:, :n].double()
    want = torch.softmax(q.double() @ rows.mT / 24, -1) @ rows[..., :512]
    assert float((o.double() - want).norm() / want.norm()) < 1.1 * 2.0 ** -7 / 12 ** 0.5 * 0.7355


def _hash_u32(x):
    x &= 0xFFFFFFFF
    x = ((x ^ (x >> 16)) * 0x7FEB352D) & 0xFFFFFFFF
    x = ((x ^ (x >> 15)) * 0x846CA68B) & 0xFFFFFFFF
    return x ^ (x >> 16)


def _draw(z, row, t, k, tp, mp, seed, step):
    """What the sampler picks for one row of (penalised) logits, and its log-probability: the k best by (value, lowest index),
    top-p and min-p on them, a draw by the counter-based generator."""
    v, i = torch.sort(z.double(), descending=True, stable=True)
    n = int((v[:k] > -float("inf")).sum())
    p = torch.exp((v[:n] - v[0]) / t)
    share, kept = p / p.sum(), 0
    cum = 0.0
    while kept < n and (kept == 0 or (cum < tp and p[kept] >= mp * p[0])):
        cum += float(share[kept])
        kept += 1
    h = _hash_u32((seed & 0xFFFFFFFF) ^ _hash_u32((seed >> 32) + 0x9E3779B9 * (step + 1)) ^ _hash_u32(row))
    u = ((h >> 8) + 0.5) / 2 ** 24
    acc = torch.cumsum(p[:kept], 0) / p[:kept].sum()
    j = min(int((acc < u).sum()), kept - 1)
    return int(i[j]), float(torch.log_softmax(z.double() / t, -1)[i[j]]), float((acc - u).abs().min())


@pytest.mark.parametrize("R,V", [(1, 70), (3, 128256), (40, 128256), (200, 5000), (2, 50257), (1, 8192), (300, 33)])
@pytest.mark.parametrize("form", ["spread", "ties", "equal", "masked", "sorted"])
def test_sampler_draws_what_the_oracle_draws(R, V, form):
    """Rows cut into slices, rows that do not start on 16 bytes, many equal logits, rows of which few tokens are allowed and rows
    whose best tokens lie side by side: the candidates are the k best by (value, lowest index) in every case."""
    from easydel_b200.ops import serving as S

    g = torch.Generator(device="cuda").manual_seed(R * 7 + V)
    dev = "cuda"
    z = torch.randn(R, V, device=dev, generator=g) * 2.5
    if form == "ties":
        z = torch.round(z)
    elif form == "equal":
        z = torch.zeros(R, V, device=dev)
    elif form == "masked":
        keep = torch.rand(R, V, device=dev, generator=g) < 20 / V
        keep[:, V // 2] = True
        z = torch.where(keep, z, -float("inf"))
    elif form == "sorted":
        z = z.sort(-1).values
    for dtype in (torch.bfloat16, torch.float32):
        logits = z.to(dtype)
        u = lambda: torch.rand(R, device=dev, generator=g)  # noqa: E731
        temp, top_p, min_p = 0.5 + u(), 0.5 + 0.5 * u(), 0.1 * u() * (u() < 0.5)
        top_k = (u() * 70).to(torch.int32)
        seeds = torch.randint(0, 1 << 40, (R,), device=dev, generator=g)
        steps = torch.randint(0, 99, (R,), device=dev, generator=g).to(torch.int32)
        tok, lp = S.sample(logits, temperature=temp, top_k=top_k, top_p=top_p, min_p=min_p, seeds=seeds, steps=steps,
                           want_logprob=True)
        zc = logits.float().cpu()
        for r in range(0, R, max(1, R // 12)):
            k = int(top_k[r])
            if k == 1:
                assert int(tok[r]) == int(zc[r].argmax())
                continue
            want, want_lp, margin = _draw(zc[r], r, float(temp[r]), 64 if k <= 0 or k > 64 else k, float(top_p[r]),
                                          float(min_p[r]), int(seeds[r]), int(steps[r]))
            if margin < 1e-5:      # the draw falls on a boundary of the fp32 sums
                continue
            assert int(tok[r]) == want, (r, k)
            assert abs(float(lp[r]) - want_lp) < 1e-4 * max(1.0, abs(want_lp))


@pytest.mark.parametrize("V", [1000, 1003, 40000])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("penalties", [False, True])
@pytest.mark.parametrize("temperature", [0.0, 0.7])
def test_sampler_on_rows_without_a_usable_value(V, dtype, penalties, temperature):
    """Rows of minus infinities, of NaNs and of both give token 0 with log-probability minus infinity in every form of the
    kernel (16-byte loads or not, a row cut over a cluster, penalties); one finite value among them is taken."""
    from easydel_b200.ops import serving as S

    inf = float("inf")
    logits = torch.full((5, V), -inf, device="cuda")
    logits[1] = float("nan")
    logits[2, ::2] = float("nan")
    logits[3, V - 2] = -3.0
    logits[4] = float("nan")
    logits[4, 17] = 2.0
    kw = dict(temperature=torch.full((5,), temperature, device="cuda"))
    if penalties:
        kw.update(counts=torch.ones(5, V, dtype=torch.int32, device="cuda"), presence=torch.full((5,), 0.5, device="cuda"))
    tokens, logprobs = S.sample(logits.to(dtype), want_logprob=True, **kw)
    assert tokens.tolist() == [0, 0, 0, V - 2, 17]
    assert (logprobs[:3] == -inf).all() and abs(float(logprobs[3])) < 1e-5
