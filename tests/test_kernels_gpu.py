"""Each CUDA kernel alone against its plain reference, at sizes other than the engine's."""
import ctypes
import importlib
import math
import os
import random
import subprocess

import pytest
import torch

import plain_qwen3 as plain
from conftest import rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DTYPES = [torch.float32, torch.bfloat16]
KTOL = {torch.float32: 2e-6, torch.bfloat16: 8e-3}   # one rounding of the output (2^-9 = 2e-3, a few ulps)


@pytest.fixture(scope="module")
def ops(pe):
    pe.kernels.library()
    return pe.kernels.ops


def _status():
    return torch.zeros(4, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("dtype", DTYPES)
def test_embed_gather(ops, dtype):
    torch.manual_seed(0)
    table = torch.randn(515, 80, device=DEV).to(dtype)
    ids = torch.tensor([0, 514, 7, 7, 300], dtype=torch.int32, device=DEV)
    out = torch.empty(5, 80, device=DEV)
    st = _status()
    ops.embed_gather(table, ids, out, st)
    assert torch.equal(out, table.float()[ids.long()])
    assert st.tolist()[0] == 0
    bad = torch.tensor([3, 515], dtype=torch.int32, device=DEV)
    out2 = torch.empty(2, 80, device=DEV)
    ops.embed_gather(table, bad, out2, st)
    assert st.tolist()[:3] == [1, 1, 515] and float(out2[1].abs().sum()) == 0.0


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("dim", [80, 1000, 4096, 5120])
@pytest.mark.parametrize("n", [7, 100])    # a handful of rows get more threads a row than many rows do
def test_rmsnorm_with_residual(ops, dtype, dim, n):
    torch.manual_seed(1)
    res = torch.randn(n, dim, device=DEV) * 3
    delta = torch.randn(n, dim, device=DEV).to(dtype)
    w = 1 + 0.1 * torch.randn(dim, device=DEV)
    eps = 3e-6
    want_h = res + delta.float()
    want = plain.rms_norm(want_h.cpu(), w.cpu(), eps)
    # add + write back + norm
    r1, out = res.clone(), torch.empty(n, dim, device=DEV, dtype=dtype)
    ops.rmsnorm_residual(r1, delta, w, out, eps)
    assert torch.equal(r1, want_h)
    assert rel_err(out.float().cpu(), want) < KTOL[dtype]
    # no delta: the stream is left alone
    r2, out2 = res.clone(), torch.empty(n, dim, device=DEV, dtype=dtype)
    ops.rmsnorm_residual(r2, None, w, out2, eps)
    assert torch.equal(r2, res)
    assert rel_err(out2.float().cpu(), plain.rms_norm(res.cpu(), w.cpu(), eps)) < KTOL[dtype]
    # gathered rows: nothing written back
    rows = torch.tensor([5, 0, 5], dtype=torch.int32, device=DEV)
    r3, out3 = res.clone(), torch.empty(3, dim, device=DEV, dtype=dtype)
    ops.rmsnorm_residual(r3, delta, w, out3, eps, rows)
    assert torch.equal(r3, res)
    assert rel_err(out3.float().cpu(), want[[5, 0, 5]]) < KTOL[dtype]


@pytest.mark.parametrize("dtype", DTYPES)
def test_rmsnorm_plain(ops, dtype):
    torch.manual_seed(2)
    x = torch.randn(6, 5, 48, device=DEV).to(dtype)
    w = 1 + 0.1 * torch.randn(48, device=DEV)
    out = torch.empty_like(x)
    ops.rmsnorm(x, w, out, 1e-5)
    assert rel_err(out.float().cpu(), plain.rms_norm(x.float().cpu(), w.cpu(), 1e-5)) < KTOL[dtype]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n,inter", [(1, 176), (9, 200), (33, 3072)])
def test_silu_mul(ops, dtype, n, inter):
    torch.manual_seed(3)
    gu = (torch.randn(n, 2 * inter, device=DEV) * 4).to(dtype)
    out = torch.empty(n, inter, device=DEV, dtype=dtype)
    ops.silu_mul(gu, out)
    g, u = gu.float().cpu()[:, :inter], gu.float().cpu()[:, inter:]
    want = g / (1 + torch.exp(-g)) * u
    assert rel_err(out.float().cpu(), want) < KTOL[dtype]


def test_batch_expand(ops):
    qstart = torch.tensor([0, 3, 4, 4, 9], dtype=torch.int32, device=DEV)      # the third sequence brings nothing
    past = torch.tensor([10, 0, 7, 100], dtype=torch.int32, device=DEV)
    seq = torch.full((9,), -1, dtype=torch.int32, device=DEV)
    pos = torch.full((9,), -1, dtype=torch.int32, device=DEV)
    ops.batch_expand(qstart, past, 4, seq, pos)
    assert seq.tolist() == [0, 0, 0, 1, 3, 3, 3, 3, 3]
    assert pos.tolist() == [10, 11, 12, 0, 100, 101, 102, 103, 104]


class PagedSetup:
    """A batch of sequences with keys and values scattered over shuffled pages of a pool."""

    def __init__(self, lens, nkv, d, dtype, seed=0, extra_pages=5, key_scale=1.0):
        g = torch.Generator().manual_seed(seed)
        self.lens, self.nkv, self.d, self.dtype = lens, nkv, d, dtype
        B = len(lens)
        pages_per = [(L + 63) // 64 for L in lens]
        self.num_pages = sum(pages_per) + extra_pages
        order = list(range(self.num_pages))
        random.Random(seed).shuffle(order)
        self.table_width = max(pages_per) + 2
        self.slots = list(range(B - 1, -1, -1))   # slot numbers differ from batch order
        table = torch.full((B + 1, self.table_width), -1, dtype=torch.int32)
        self.k = [(torch.randn(L, nkv, d, generator=g) * key_scale).to(dtype) for L in lens]
        self.v = [torch.randn(L, nkv, d, generator=g).to(dtype) for L in lens]
        kp = torch.randn(self.num_pages, nkv, 64, d, generator=g).to(dtype)   # junk where nothing was written
        vp = torch.randn(self.num_pages, nkv, 64, d, generator=g).to(dtype)
        it = iter(order)
        for b, L in enumerate(lens):
            for lp in range(pages_per[b]):
                page = next(it)
                table[self.slots[b], lp] = page
                n = min(64, L - lp * 64)
                kp[page, :, :n] = self.k[b][lp * 64: lp * 64 + n].transpose(0, 1)
                vp[page, :, :n] = self.v[b][lp * 64: lp * 64 + n].transpose(0, 1)
        self.k_pages, self.v_pages, self.table = kp.to(DEV), vp.to(DEV), table.to(DEV)
        self.seq_slot = torch.tensor(self.slots, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("nh,nkv,d,rot", [(4, 2, 16, 16), (6, 2, 32, 32), (5, 5, 48, 48), (8, 1, 128, 64), (3, 3, 80, 80),
                                        (8, 2, 128, 128), (2, 1, 256, 256), (7, 3, 96, 96), (9, 3, 64, 64)])
@pytest.mark.parametrize("lens,q_lens", [([70, 3, 129], [6, 3, 65]), ([300, 3, 200], [230, 3, 136])])
def test_qk_norm_rope_append(ops, dtype, nh, nkv, d, rot, lens, q_lens):
    # lens: lengths after the step; q_lens: tokens this step brings (the second sequence starts here);
    # the longer step takes the 16-byte kernel where the sizes allow it
    torch.manual_seed(4)
    ps = PagedSetup(lens, nkv, d, dtype, seed=4)
    N = sum(q_lens)
    ld = (nh + 2 * nkv) * d + 16        # row stride larger than the row
    qkv = torch.randn(N, ld, device=DEV).to(dtype)
    before = qkv.clone()
    qw = 1 + 0.2 * torch.randn(d, device=DEV)
    kw = 1 + 0.2 * torch.randn(d, device=DEV)
    eps, theta, max_pos = 1e-5, 1e4, 512
    inv = plain.rope_inv_freq(rot, theta)
    ang = torch.outer(torch.arange(max_pos, dtype=torch.float32), inv)
    cos, sin = torch.cos(ang).to(DEV), torch.sin(ang).to(DEV)
    token_seq = torch.tensor(sum(([b] * n for b, n in enumerate(q_lens)), []), dtype=torch.int32, device=DEV)
    pos_list = sum(([lens[b] - q_lens[b] + i for i in range(q_lens[b])] for b in range(3)), [])
    token_pos = torch.tensor(pos_list, dtype=torch.int32, device=DEV)
    qstart = torch.tensor([0, q_lens[0], q_lens[0] + q_lens[1], N], dtype=torch.int32, device=DEV)
    k_before, v_before = ps.k_pages.clone(), ps.v_pages.clone()
    st = _status()
    ops.qk_norm_rope_append(qkv[:, : ld], N, nh, nkv, d, qw, kw, eps, cos, sin, rot, token_seq, token_pos, ps.seq_slot,
                            qstart, ps.table, ps.num_pages, ps.k_pages, ps.v_pages, True, st)
    assert st.tolist()[0] == 0
    x = before.float().cpu()
    q_in = x[:, : nh * d].view(N, nh, d)
    k_in = x[:, nh * d: (nh + nkv) * d].view(N, nkv, d)
    v_in = x[:, (nh + nkv) * d: (nh + 2 * nkv) * d].view(N, nkv, d)
    c, s = plain.rope_cos_sin(torch.tensor(pos_list), rot, theta)
    q_want = plain.rope_rotate_neox(plain.rms_norm(q_in, qw.cpu(), eps), c, s, rot)
    k_want = plain.rope_rotate_neox(plain.rms_norm(k_in, kw.cpu(), eps), c, s, rot)
    got = qkv.float().cpu()
    assert rel_err(got[:, : nh * d].view(N, nh, d), q_want) < KTOL[dtype]
    assert rel_err(got[:, nh * d: (nh + nkv) * d].view(N, nkv, d), k_want) < KTOL[dtype]
    assert torch.equal(got[:, (nh + nkv) * d:], x[:, (nh + nkv) * d:])     # v and the padding are untouched
    # the cache holds exactly the new rows, at their pages; every other row is as before
    touched = torch.zeros(ps.num_pages, 64, dtype=torch.bool)
    kp, vp = ps.k_pages.float().cpu(), ps.v_pages.float().cpu()
    for t, (b, p) in enumerate(zip(token_seq.tolist(), pos_list)):
        page = int(ps.table[ps.slots[b], p // 64])
        touched[page, p % 64] = True
        assert rel_err(kp[page, :, p % 64], k_want[t]) < KTOL[dtype]
        assert torch.equal(vp[page, :, p % 64], v_in[t])
    # the last token of each multi-token step clears the rest of its page (rows after it hold zeros);
    # every other row is as before
    cleared = torch.zeros(ps.num_pages, 64, dtype=torch.bool)
    for b in range(3):
        last = lens[b] - 1
        page = int(ps.table[ps.slots[b], last // 64])
        cleared[page, last % 64 + 1:] = True
    keep = ~touched & ~cleared
    assert torch.equal(ps.k_pages.cpu().transpose(1, 2)[keep], k_before.cpu().transpose(1, 2)[keep])
    assert torch.equal(ps.v_pages.cpu().transpose(1, 2)[keep], v_before.cpu().transpose(1, 2)[keep])
    assert float(ps.k_pages.float().cpu().transpose(1, 2)[cleared].abs().sum()) == 0.0
    assert float(ps.v_pages.float().cpu().transpose(1, 2)[cleared].abs().sum()) == 0.0
    # write_cache off: q and k are still rewritten, the cache is not
    k_now = ps.k_pages.clone()
    qkv2 = before.clone()
    ops.qk_norm_rope_append(qkv2, N, nh, nkv, d, qw, kw, eps, cos, sin, rot, token_seq, token_pos, ps.seq_slot,
                            qstart, ps.table, ps.num_pages, ps.k_pages, ps.v_pages, False, st)
    assert torch.equal(qkv2, qkv) and torch.equal(ps.k_pages, k_now)


def _plain_attention(ps, q_list, pasts, nh, scale, window):
    outs = []
    for b, q in enumerate(q_list):
        T = pasts[b] + q.shape[0]
        outs.append(plain.causal_gqa_attention(q.float(), ps.k[b][:T].float(), ps.v[b][:T].float(), scale,
                                               window=window, q_start=pasts[b]))
    return torch.cat(outs, 0)


ATT_TOL = {torch.float32: 5e-6, torch.bfloat16: 8e-3}


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("nh,nkv,d", [(4, 2, 16), (6, 2, 32), (5, 5, 48), (8, 1, 128), (4, 1, 256), (2, 2, 80)])
@pytest.mark.parametrize("window", [0, 37])
def test_attention_prefill(ops, dtype, nh, nkv, d, window):
    torch.manual_seed(5)
    lens = [200, 1, 77, 64]
    pasts = [0, 0, 50, 0]                # the third sequence continues an earlier chunk
    q_lens = [L - p for L, p in zip(lens, pasts)]
    ps = PagedSetup(lens, nkv, d, dtype, seed=5, key_scale=2.0)
    N = sum(q_lens)
    ld = nh * d + 32
    q_all = torch.randn(N, ld, device=DEV).to(dtype)
    out = torch.zeros(N, nh * d, device=DEV, dtype=dtype)
    qstart = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32, device=DEV)
    past_t = torch.tensor(pasts, dtype=torch.int32, device=DEV)
    scale = 1 / math.sqrt(d)
    st = _status()
    ops.attention_generic(False, q_all, out, len(lens), max(q_lens), nh, nkv, d, scale, window, qstart, past_t,
                          ps.seq_slot, ps.table, ps.num_pages, ps.k_pages, ps.v_pages, None, 0, 0, st)
    assert st.tolist()[0] == 0
    qs, o = [], 0
    for n in q_lens:
        qs.append(q_all[o:o + n, : nh * d].cpu().view(n, nh, d)); o += n
    want = _plain_attention(ps, qs, pasts, nh, scale, window or None)
    assert rel_err(out.float().cpu().view(N, nh, d), want) < ATT_TOL[dtype]


@pytest.mark.parametrize("nh,nkv,d", [(16, 8, 128), (3, 3, 128), (10, 2, 64), (33, 1, 64)])
@pytest.mark.parametrize("window,sink", [(0, False), (37, False), (0, True)])
def test_attention_prefill_float32_tiles(ops, nh, nkv, d, window, sink):
    """The tiled float32 kernel (head sizes 64 and 128) at the edges of its 32-row tiles and 64-key pages, against 64 bits."""
    torch.manual_seed(27)
    q_lens, pasts = [1, 15, 16, 17, 65, 200], [0, 64, 63, 128, 7, 0]
    ps = PagedSetup([a + b for a, b in zip(q_lens, pasts)], nkv, d, torch.float32, seed=27, key_scale=2.0)
    N = sum(q_lens)
    q_all = torch.randn(N, nh * d + 32, device=DEV)
    out = torch.zeros(N, nh * d, device=DEV)
    qstart = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32, device=DEV)
    past_t = torch.tensor(pasts, dtype=torch.int32, device=DEV)
    st = _status()
    ops.attention_generic_ex(False, q_all, out, len(q_lens), max(q_lens), nh, nkv, d, d, d ** -0.5, window, sink, None, None, 0,
                             False, qstart, past_t, ps.seq_slot, ps.table, ps.num_pages, ps.k_pages, ps.v_pages, None, 0, 0, st)
    assert st.tolist()[0] == 0
    o = 0
    for b, (n, past) in enumerate(zip(q_lens, pasts)):
        L = n + past
        idx = ps.table[ps.slots[b], :-(-L // 64)].long()
        k, v = (t[idx].permute(1, 0, 2, 3).reshape(nkv, -1, d)[:, :L].double().repeat_interleave(nh // nkv, 0) for t in (ps.k_pages, ps.v_pages))
        q = q_all[o:o + n, :nh * d].double().view(n, nh, d).transpose(0, 1)
        i, j = torch.arange(n, device=DEV)[:, None] + past, torch.arange(L, device=DEV)[None]
        hidden = (j > i) | ((i - j >= window) if window else False)
        s = (q @ k.transpose(1, 2) * d ** -0.5).masked_fill(hidden, -math.inf)
        if sink:
            s = torch.cat([s, torch.zeros(nh, n, 1, device=DEV, dtype=torch.float64)], -1)
        want = (torch.softmax(s, -1)[..., :L] @ v).transpose(0, 1).reshape(n, -1)
        # 2 d sums and as many roundings of the scores (which grow to about 2 * 5 here) before the exponential
        assert float((out[o:o + n].double() - want).norm() / want.norm()) < ATT_TOL[torch.float32]
        o += n


@pytest.mark.parametrize("nh,nkv,d", [(16, 8, 128), (4, 4, 64), (33, 1, 64)])
@pytest.mark.parametrize("window", [0, 37])
def test_attention_prefill_float32_tiles_leave_out_what_a_row_does_not_see(ops, nh, nkv, d, window):
    """Keys and values that are infinite or not numbers, behind a token or in front of its window, change no bit of its output."""
    torch.manual_seed(28)
    n, past = 50, 130
    ps = PagedSetup([n + past], nkv, d, torch.float32, seed=28)
    q = torch.randn(n, nh * d, device=DEV)
    qstart = torch.tensor([0, n], dtype=torch.int32, device=DEV)
    past_t = torch.tensor([past], dtype=torch.int32, device=DEV)
    at = past + 20                                          # the key that is spoilt: seen by tokens 20 .. 20 + window - 1
    page = int(ps.table[ps.slots[0], at // 64])
    outs = []
    for bad in (None, float("nan"), float("inf")):
        k, v = ps.k_pages.clone(), ps.v_pages.clone()
        if bad is not None:
            k[page, :, at % 64], v[page, :, at % 64] = bad, bad
        out, st = torch.zeros(n, nh * d, device=DEV), _status()
        ops.attention_generic(False, q, out, 1, n, nh, nkv, d, d ** -0.5, window, qstart, past_t, ps.seq_slot, ps.table, ps.num_pages,
                              k, v, None, 0, 0, st)
        assert st.tolist()[0] == 0
        outs.append(out)
    unseen = torch.tensor([i < 20 or (window > 0 and i - 20 >= window) for i in range(n)], device=DEV)
    assert bool(outs[0].isfinite().all()) and bool(outs[1][~unseen].isnan().all())
    assert torch.equal(outs[0][unseen], outs[1][unseen]) and torch.equal(outs[0][unseen], outs[2][unseen])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("nh,nkv,d", [(4, 2, 16), (6, 2, 32), (5, 5, 48), (32, 8, 128), (4, 1, 256), (16, 2, 64)])
@pytest.mark.parametrize("window", [0, 300])
def test_attention_decode(ops, dtype, nh, nkv, d, window):
    torch.manual_seed(6)
    lens = [1, 700, 256, 257, 33]        # one token, several ranges, a range's edge on both sides
    pasts = [L - 1 for L in lens]
    ps = PagedSetup(lens, nkv, d, dtype, seed=6, key_scale=2.0)
    B = len(lens)
    q_all = torch.randn(B, nh * d, device=DEV).to(dtype)
    out = torch.zeros(B, nh * d, device=DEV, dtype=dtype)
    qstart = torch.arange(B + 1, dtype=torch.int32, device=DEV)
    past_t = torch.tensor(pasts, dtype=torch.int32, device=DEV)
    scale = 1 / math.sqrt(d)
    split_keys, max_splits = 256, 4       # 4 ranges allowed although the longest needs 3
    scratch = torch.full((ops.attention_generic_scratch_floats(B, nh, d, max_splits),), float("nan"), device=DEV)
    st = _status()
    ops.attention_generic(True, q_all, out, B, 1, nh, nkv, d, scale, window, qstart, past_t, ps.seq_slot, ps.table,
                          ps.num_pages, ps.k_pages, ps.v_pages, scratch, split_keys, max_splits, st)
    assert st.tolist()[0] == 0
    qs = [q_all[b: b + 1].cpu().view(1, nh, d) for b in range(B)]
    want = _plain_attention(ps, qs, pasts, nh, scale, window or None)
    assert rel_err(out.float().cpu().view(B, nh, d), want) < ATT_TOL[dtype]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("decode", [False, True])
def test_attention_finds_a_far_key(ops, decode, dtype):
    """One key among hundreds matches the query; the output must be that key's value."""
    nh, nkv, d = 4, 2, 32
    L, far = 650, 13
    ps = PagedSetup([L], nkv, d, dtype, seed=7, key_scale=0.05)
    q = torch.zeros(1, nh * d)
    probe = torch.randn(d)
    probe = probe / probe.norm() * 12.0
    for h in range(nh):
        q[0, h * d:(h + 1) * d] = probe
    page = int(ps.table[ps.slots[0], far // 64])
    ps.k_pages[page, :, far % 64] = (probe.to(DEV) * 2.0).to(dtype)       # score 288*scale against ~0 elsewhere
    q_lens = [1]
    out = torch.zeros(1, nh * d, device=DEV, dtype=dtype)
    qstart = torch.tensor([0, 1], dtype=torch.int32, device=DEV)
    past_t = torch.tensor([L - 1], dtype=torch.int32, device=DEV)
    scratch = torch.zeros(ops.attention_generic_scratch_floats(1, nh, d, 3), device=DEV)
    ops.attention_generic(decode, q.to(DEV, dtype), out, 1, 1, nh, nkv, d, 1 / math.sqrt(d), 0, qstart, past_t, ps.seq_slot,
                          ps.table, ps.num_pages, ps.k_pages, ps.v_pages, scratch if decode else None,
                          256 if decode else 0, 3 if decode else 0, _status())
    v_far = ps.v_pages[page, :, far % 64].float().cpu()       # [nkv, d]
    got = out.float().cpu().view(nh, d)
    for h in range(nh):
        assert torch.allclose(got[h], v_far[h // 2], atol=1e-4 if dtype == torch.float32 else 2e-2)


@pytest.mark.parametrize("kernel,decode", [("generic_f32", False), ("generic_f32", True), ("generic_bf16", False),
                                           ("generic_bf16", True), ("mma", False), ("mma", True), ("umma", False)])
def test_attention_at_the_windows_edge(ops, kernel, decode):
    """Two keys match the query strongly: the last one outside the window of the last query and the
    first one inside it.  With an edge off by one either way the output changes by tens."""
    dtype = torch.float32 if kernel == "generic_f32" else torch.bfloat16
    nh, nkv, d = (8, 2, 128) if kernel in ("mma", "umma") else (4, 2, 32)
    L, W = 200, 50
    outside, inside = L - 1 - W, L - W            # positions 149 and 150 for the query at 199
    ps = PagedSetup([L], nkv, d, dtype, seed=21, key_scale=0.05)
    probe = torch.randn(d)
    probe = probe / probe.norm() * 12.0
    for pos, value in ((outside, 50.0), (inside, -30.0)):
        page = int(ps.table[ps.slots[0], pos // 64])
        ps.k_pages[page, :, pos % 64] = (probe * 2.0).to(DEV, dtype)
        ps.v_pages[page, :, pos % 64] = value
        ps.k[0][pos] = (probe * 2.0).to(dtype)
        ps.v[0][pos] = value
    n_q = 1 if decode else L
    past = L - n_q
    q = probe.repeat(n_q, nh).contiguous()          # every query matches the two keys
    ld = nh * d + 2 * nkv * d
    q_all = torch.zeros(n_q, ld)
    q_all[:, : nh * d] = q
    q_all = q_all.to(DEV, dtype)
    out = torch.zeros(n_q, nh * d, device=DEV, dtype=dtype)
    qstart = torch.tensor([0, n_q], dtype=torch.int32, device=DEV)
    past_t = torch.tensor([past], dtype=torch.int32, device=DEV)
    scale = 1 / math.sqrt(d)
    scratch = torch.zeros(ops.attention_generic_scratch_floats(1, nh, d, 4), device=DEV) if decode else None
    split = (64, 4) if decode else (0, 0)
    st = _status()
    if kernel == "umma":
        ops.attention_umma_prefill(q_all, out, 1, n_q, nh, nkv, d, scale, W, qstart, past_t, ps.seq_slot, ps.table,
                                   ps.num_pages, ps.k_pages, ps.v_pages, st)
    else:
        fn = ops.attention_mma if kernel == "mma" else ops.attention_generic
        fn(decode, q_all, out, 1, n_q, nh, nkv, d, scale, W, qstart, past_t, ps.seq_slot, ps.table, ps.num_pages,
           ps.k_pages, ps.v_pages, scratch, split[0], split[1], st)
    assert st.tolist()[0] == 0
    got = out.float().cpu().view(n_q, nh, d)
    want = plain.causal_gqa_attention(q.view(n_q, nh, d).float(), ps.k[0].float(), ps.v[0].float(), scale, window=W,
                                      q_start=past)
    tol = 1e-3 if dtype == torch.float32 else 0.3
    assert float((got - want).abs().max()) < tol
    # the last query sees the inside key only, the one before it both
    assert abs(float(got[-1].mean()) + 30.0) < 0.5
    if not decode:
        assert abs(float(got[-2].mean()) - 10.0) < 0.5


MMA_SHAPES = [(8, 2, 64), (32, 8, 128), (16, 1, 128), (3, 3, 64), (6, 2, 128), (10, 2, 64)]


@pytest.mark.parametrize("nh,nkv,d", MMA_SHAPES)
@pytest.mark.parametrize("window", [0, 37, 150])
def test_attention_mma_prefill(ops, nh, nkv, d, window):
    torch.manual_seed(15)
    dtype = torch.bfloat16
    assert ops.attention_mma_supported(dtype, d, nh, nkv)
    lens = [200, 1, 77, 64, 130]
    pasts = [0, 0, 50, 0, 127]            # the third and the last sequence continue earlier chunks
    q_lens = [L - p for L, p in zip(lens, pasts)]
    ps = PagedSetup(lens, nkv, d, dtype, seed=15, key_scale=2.0)
    N = sum(q_lens)
    ld = nh * d + 2 * nkv * d             # q rows inside a fused q|k|v buffer
    q_all = torch.randn(N, ld, device=DEV).to(dtype)
    out = torch.zeros(N, nh * d, device=DEV, dtype=dtype)
    qstart = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32, device=DEV)
    past_t = torch.tensor(pasts, dtype=torch.int32, device=DEV)
    scale = 1 / math.sqrt(d)
    st = _status()
    ops.attention_mma(False, q_all, out, len(lens), max(q_lens), nh, nkv, d, scale, window, qstart, past_t,
                      ps.seq_slot, ps.table, ps.num_pages, ps.k_pages, ps.v_pages, None, 0, 0, st)
    assert st.tolist()[0] == 0
    qs, o = [], 0
    for n in q_lens:
        qs.append(q_all[o:o + n, : nh * d].cpu().view(n, nh, d)); o += n
    want = _plain_attention(ps, qs, pasts, nh, scale, window or None)
    assert rel_err(out.float().cpu().view(N, nh, d), want) < ATT_TOL[dtype]


@pytest.mark.parametrize("nh,nkv", [(32, 8), (16, 1), (3, 3), (8, 4), (16, 2), (10, 2), (6, 2), (3, 1), (24, 1)])
@pytest.mark.parametrize("window", [0, 37, 150])
def test_attention_umma_prefill(ops, nh, nkv, window):
    """The tcgen05 prefill attention against the plain formula (head size 128; groups 4, 16, 1, 2, 8, and
    5, 3, 24, which do not divide a block's 128 rows)."""
    torch.manual_seed(25)
    d, dtype = 128, torch.bfloat16
    assert ops.attention_umma_supported(dtype, d, nh, nkv)
    lens = [300, 1, 77, 64, 130, 513]
    pasts = [0, 0, 50, 0, 127, 0]
    q_lens = [L - p for L, p in zip(lens, pasts)]
    ps = PagedSetup(lens, nkv, d, dtype, seed=25, key_scale=2.0)
    N = sum(q_lens)
    ld = nh * d + 2 * nkv * d
    q_all = torch.randn(N, ld, device=DEV).to(dtype)
    out = torch.zeros(N, nh * d, device=DEV, dtype=dtype)
    qstart = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32, device=DEV)
    past_t = torch.tensor(pasts, dtype=torch.int32, device=DEV)
    scale = 1 / math.sqrt(d)
    st = _status()
    ops.attention_umma_prefill(q_all, out, len(lens), max(q_lens), nh, nkv, d, scale, window, qstart, past_t, ps.seq_slot,
                               ps.table, ps.num_pages, ps.k_pages, ps.v_pages, st)
    torch.cuda.synchronize()
    assert st.tolist()[0] == 0, st.tolist()
    qs, o = [], 0
    for n in q_lens:
        qs.append(q_all[o:o + n, : nh * d].cpu().view(n, nh, d)); o += n
    want = _plain_attention(ps, qs, pasts, nh, scale, window or None)
    assert rel_err(out.float().cpu().view(N, nh, d), want) < ATT_TOL[dtype]


def test_attention_umma_prefill_rows_beyond_a_sequences_last(ops):
    """A tile's spare rows hold the next sequence's queries: whatever those are, the sequence's own rows do not see them."""
    torch.manual_seed(26)
    nh, nkv, d, dtype = 32, 8, 128, torch.bfloat16
    q_lens, pasts = [33, 31, 1, 40], [70, 0, 300, 128]
    ps = PagedSetup([a + b for a, b in zip(q_lens, pasts)], nkv, d, dtype, seed=26)
    N = sum(q_lens)
    q_all = torch.randn(N, (nh + 2 * nkv) * d, device=DEV).to(dtype)
    qstart = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32, device=DEV)
    past_t = torch.tensor(pasts, dtype=torch.int32, device=DEV)
    outs = []
    for bad in (None, float("nan"), float("inf")):
        q = q_all.clone()
        if bad is not None:
            q[33:64] = bad
        out = torch.zeros(N, nh * d, device=DEV, dtype=dtype)
        st = _status()
        ops.attention_umma_prefill(q, out, 4, max(q_lens), nh, nkv, d, d ** -0.5, 0, qstart, past_t, ps.seq_slot, ps.table,
                                   ps.num_pages, ps.k_pages, ps.v_pages, st)
        assert st.tolist()[0] == 0
        outs.append(torch.cat([out[:33], out[64:]]))
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


def test_attention_umma_prefill_blocks_of_two_pages_again_and_again(ops):
    """Blocks that see two or three pages only (a short window) end a few barrier phases after they
    start; a wait that names a phase by its parity must not pass because the barrier is two phases
    behind.  The same launch forty times must give the same, right result every time."""
    torch.manual_seed(27)
    nh, nkv, d, dtype, window = 8, 4, 128, torch.bfloat16, 37
    lens = [300, 77, 513, 130]
    ps = PagedSetup(lens, nkv, d, dtype, seed=27, key_scale=2.0)
    N = sum(lens)
    q_all = torch.randn(N, nh * d + 2 * nkv * d, device=DEV).to(dtype)
    qstart = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    past_t = torch.zeros(len(lens), dtype=torch.int32, device=DEV)
    scale = 1 / math.sqrt(d)
    st = _status()
    qs, o = [], 0
    for n in lens:
        qs.append(q_all[o:o + n, : nh * d].cpu().view(n, nh, d)); o += n
    want = _plain_attention(ps, qs, [0] * len(lens), nh, scale, window)
    outs = []
    for _ in range(40):
        out = torch.zeros(N, nh * d, device=DEV, dtype=dtype)
        ops.attention_umma_prefill(q_all, out, len(lens), max(lens), nh, nkv, d, scale, window, qstart, past_t, ps.seq_slot,
                                   ps.table, ps.num_pages, ps.k_pages, ps.v_pages, st)
        outs.append(out)
    torch.cuda.synchronize()
    assert st.tolist()[0] == 0
    for out in outs:
        assert torch.equal(out, outs[0])
    assert rel_err(outs[0].float().cpu().view(N, nh, d), want) < ATT_TOL[dtype]


def test_attention_umma_prefill_rescales_when_the_maximum_grows(ops):
    """Scores that grow by far more than 2^8 along the sequence: the reference of the exponentials
    must move and the accumulated output be rescaled."""
    nh, nkv, d, dtype = 4, 1, 128, torch.bfloat16
    L = 400
    ps = PagedSetup([L], nkv, d, dtype, seed=26, key_scale=0.1)
    probe = torch.randn(d)
    probe = probe / probe.norm()
    q_all = (probe * 6.0).repeat(L, nh).to(dtype).to(DEV)                 # every query points along `probe`
    for pos in range(L):                                                   # keys grow along `probe` with the position
        page = int(ps.table[ps.slots[0], pos // 64])
        ps.k_pages[page, 0, pos % 64] += (probe * (pos / 10.0)).to(dtype).to(DEV)
    ps.k[0] = torch.stack([ps.k_pages[int(ps.table[ps.slots[0], p // 64]), :, p % 64].cpu() for p in range(L)])
    out = torch.zeros(L, nh * d, device=DEV, dtype=dtype)
    qstart = torch.tensor([0, L], dtype=torch.int32, device=DEV)
    past_t = torch.zeros(1, dtype=torch.int32, device=DEV)
    scale = 1 / math.sqrt(d)
    st = _status()
    ops.attention_umma_prefill(q_all, out, 1, L, nh, nkv, d, scale, 0, qstart, past_t, ps.seq_slot, ps.table,
                               ps.num_pages, ps.k_pages, ps.v_pages, st)
    assert st.tolist()[0] == 0
    want = _plain_attention(ps, [q_all.cpu().view(L, nh, d)], [0], nh, scale, None)
    assert rel_err(out.float().cpu().view(L, nh, d), want) < ATT_TOL[dtype]


@pytest.mark.parametrize("nh,nkv,d", MMA_SHAPES)
@pytest.mark.parametrize("window", [0, 300])
# split_keys 0: even shares of each length, of at least `least` keys (spare ranges of the grid do nothing)
@pytest.mark.parametrize("split_keys,max_splits,least", [(256, 5, 0), (0, 5, 0), (0, 1, 0), (0, 23, 0), (0, 23, 128), (0, 9, 512)])
def test_attention_mma_decode(ops, nh, nkv, d, window, split_keys, max_splits, least):
    torch.manual_seed(16)
    dtype = torch.bfloat16
    lens = [1, 700, 256, 257, 33, 64, 65, 513]
    pasts = [L - 1 for L in lens]
    ps = PagedSetup(lens, nkv, d, dtype, seed=16, key_scale=2.0)
    B = len(lens)
    ld = nh * d + 2 * nkv * d
    q_all = torch.randn(B, ld, device=DEV).to(dtype)
    out = torch.zeros(B, nh * d, device=DEV, dtype=dtype)
    qstart = torch.arange(B + 1, dtype=torch.int32, device=DEV)
    past_t = torch.tensor(pasts, dtype=torch.int32, device=DEV)
    scale = 1 / math.sqrt(d)
    scratch = torch.full((ops.attention_generic_scratch_floats(B, nh, d, max_splits),), float("nan"), device=DEV)
    st = _status()
    ops.attention_mma(True, q_all, out, B, 1, nh, nkv, d, scale, window, qstart, past_t, ps.seq_slot, ps.table,
                      ps.num_pages, ps.k_pages, ps.v_pages, scratch, split_keys, max_splits, st, min_range_keys=least)
    assert st.tolist()[0] == 0
    qs = [q_all[b: b + 1, : nh * d].cpu().view(1, nh, d) for b in range(B)]
    want = _plain_attention(ps, qs, pasts, nh, scale, window or None)
    assert rel_err(out.float().cpu().view(B, nh, d), want) < ATT_TOL[dtype]


@pytest.mark.parametrize("nh,nkv,d", [(8, 4, 128), (32, 2, 64), (10, 2, 128)])
@pytest.mark.parametrize("B,splits", [(8, 1), (8, 2), (4, 3), (3, 5), (2, 8)])
@pytest.mark.parametrize("window,keep,sink", [(0, 0, False), (100, 0, True), (100, 70, False), (0, 0, True)])
def test_attention_mma_decode_clusters(ops, nh, nkv, d, B, splits, window, keep, sink):
    """The ranges of a sequence as one cluster, among them ranges that hold nothing (short sequences, keys before the window),
    against fixed ranges of a page merged by the second kernel, and against the plain formula."""
    torch.manual_seed(18)
    lens = [700, 257, 33, 513, 1, 256, 64, 65][:B]
    ps = PagedSetup(lens, nkv, d, torch.bfloat16, seed=18, key_scale=2.0)
    q = torch.randn(B, nh * d, device=DEV).to(torch.bfloat16)
    gate = torch.randn(B, nh, device=DEV).to(torch.bfloat16)
    qstart = torch.arange(B + 1, dtype=torch.int32, device=DEV)
    past = torch.tensor([L - 1 for L in lens], dtype=torch.int32, device=DEV)
    st = _status()
    outs = []
    for split_keys, n, least in ((0, splits, 64), (0, splits, 128), (64, 11, 0)):   # 700 keys: 11 pages
        out = torch.full((B, nh * d), float("nan"), device=DEV, dtype=torch.bfloat16)
        scratch = torch.full((ops.attention_generic_scratch_floats(B, nh, d, n),), float("nan"), device=DEV)
        before = ops.launch_count()
        ops.attention_mma_gated(True, q, out, B, 1, nh, nkv, d, d, d ** -0.5, window, qstart, past, ps.seq_slot, ps.table, ps.num_pages,
                                ps.k_pages, ps.v_pages, scratch, split_keys, n, st, min_range_keys=least, sink=sink, gate=gate,
                                keep_first=keep)
        assert ops.launch_count() - before == (2 if split_keys else 1)
        outs.append(out.float().cpu())
    assert st.tolist()[0] == 0
    assert rel_err(outs[0], outs[2]) < 2 * ATT_TOL[torch.bfloat16] and rel_err(outs[1], outs[2]) < 2 * ATT_TOL[torch.bfloat16]
    if not keep and not sink:
        want = _plain_attention(ps, [q[b:b + 1].cpu().view(1, nh, d) for b in range(B)], [L - 1 for L in lens], nh, d ** -0.5, window or None)
        want = want * torch.sigmoid(gate.float().cpu())[:, :, None]
        assert rel_err(outs[0].view(B, nh, d), want) < ATT_TOL[torch.bfloat16]


@pytest.mark.parametrize("M", [1, 3, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("hidden,inner", [(16, 8), (100 * 8, 40), (1024, 3072), (4104, 520), (8208, 64)])
def test_gemm_smallm_chain(ops, M, hidden, inner):
    """A product into the stream, the stream times the next norm's weight and its squares, and the product that reads them (plain and
    gated), against the norm and the products in 64 bits on the same rounded inputs."""
    torch.manual_seed(21)
    bf = torch.bfloat16
    x, w = torch.randn(M, inner, device=DEV).to(bf), (torch.randn(hidden, inner, device=DEV) / inner ** 0.5).to(bf)
    stream0, norm = torch.randn(M, hidden, device=DEV) * 3, 1 + 0.3 * torch.randn(hidden, device=DEV)
    stream, rows, squares = stream0.clone(), torch.full((M, hidden), float("nan"), device=DEV, dtype=bf), torch.full(((hidden + 15) // 16, ops.chain_rows(M)), float("nan"), device=DEV)
    ops.gemm_smallm_residual(x, w, stream, norm, rows, squares)
    want = stream0.double() + x.double() @ w.double().t()
    size = stream0.double().abs() + x.double().abs() @ w.double().abs().t()
    assert bool(((stream.double() - want).abs() <= 2.0 ** -22 * size).all())          # float32 sums of exact products
    assert bool(((rows.double() - stream.double() * norm.double()).abs() <= 2.0 ** -8 * (stream.double() * norm.double()).abs() + 1e-30).all())
    total = squares.double().sum(0)
    assert bool(((total[:M] - (stream.double() ** 2).sum(1)).abs() <= 1e-5 * (stream.double() ** 2).sum(1)).all()) and float(total[M:].abs().sum()) == 0
    again = stream0.clone()
    ops.gemm_smallm_residual(x, w, again)                                              # nobody reads the rows
    assert torch.equal(again, stream)
    eps = 1e-5
    inv = 1 / ((stream.double() ** 2).mean(1, keepdim=True) + eps).sqrt()
    for n in (40, 1000):
        gu = (torch.randn(2 * n, hidden, device=DEV) / hidden ** 0.5).to(bf)
        y = rows.double() @ gu.double().t() * inv
        room = rows.double().abs() @ gu.double().abs().t() * inv
        out = torch.empty(M, 2 * n, device=DEV, dtype=bf)
        ops.gemm_smallm_scaled(rows, gu, out, squares, eps)
        assert bool(((out.double() - y).abs() <= 2.0 ** -8 * y.abs() + 1e-5 * room).all())
        g, u = y[:, :n], y[:, n:]
        act = torch.empty(M, n, device=DEV, dtype=bf)
        ops.gemm_smallm_scaled(rows, gu, act, squares, eps, pair_offset=n)
        want = g / (1 + (-g).exp()) * u
        slack = 2e-5 * (room[:, :n] * u.abs() * 1.1 + room[:, n:] * g.abs())           # |d silu| <= 1.1
        assert bool(((act.double() - want).abs() <= 2.0 ** -8 * want.abs() + slack).all())
        bias = torch.randn(2 * n, device=DEV)
        ops.gemm_smallm_scaled(rows, gu, act, squares, eps, pair_offset=n, glu=("relu", 0.0, 1.0, bias))
        g, u = g + bias[:n].double(), u + bias[n:].double()
        want = g.clamp(min=0) * u
        slack = 2e-5 * (room[:, :n] * u.abs() + room[:, n:] * g.abs())
        assert bool(((act.double() - want).abs() <= 2.0 ** -8 * want.abs() + slack).all())


@pytest.mark.parametrize("nh,nkv,d", [(16, 8, 128), (8, 2, 64), (16, 1, 128), (16, 1, 64), (3, 3, 64)])
@pytest.mark.parametrize("blocks,least", [(0, 64), (1, 64), (5, 128), (296, 64), (296, 256)])      # 0: each sequence's ranges as one cluster
@pytest.mark.parametrize("normed,rotated,window", [(True, True, 0), (False, True, 100), (True, False, 0)])
def test_attention_mma_append(ops, nh, nkv, d, blocks, least, normed, rotated, window):
    """Norm, rotation, append and attention in one against the two kernels: outputs, cached rows, and the rest of a page that starts
    (which holds NaN before).  With the keys shared out: pairs that lie inside a block, that end in one, that span many."""
    torch.manual_seed(23)
    bf = torch.bfloat16
    lens = [1, 700, 257, 64, 65, 130][:64 // (4 * nkv) or 1] if blocks == 0 else [1, 700, 257, 64, 65, 513, 130]
    B = len(lens)
    qkv = torch.randn(B, (nh + 2 * nkv) * d + 8, device=DEV).to(bf)
    qw, kw = ((1 + 0.2 * torch.randn(d, device=DEV)) if normed else None for _ in range(2))
    angles = torch.rand(704, d // 2, device=DEV) * 6
    cos, sin = (angles.cos(), angles.sin()) if rotated else (None, None)
    qstart, past = torch.arange(B + 1, dtype=torch.int32, device=DEV), torch.tensor([L - 1 for L in lens], dtype=torch.int32, device=DEV)
    st = _status()
    outs, pages = [], []
    for fused in (True, False):
        ps = PagedSetup(lens, nkv, d, bf, seed=23, key_scale=2.0)
        for b, L in enumerate(lens):      # nothing is cached at the new position, and nothing finite behind it in a page that starts
            page = int(ps.table[ps.slots[b], (L - 1) // 64])
            ps.k_pages[page, :, (L - 1) % 64:] = ps.v_pages[page, :, (L - 1) % 64:] = float("nan") if L % 64 == 1 else 0.0
        where = (qstart, past, ps.seq_slot, ps.table, ps.num_pages, ps.k_pages, ps.v_pages)
        x, out = qkv.clone(), torch.full((B, nh * d), float("nan"), device=DEV, dtype=bf)
        if fused:
            floats = ops.attention_generic_scratch_floats(B, nh, d, 4)
            if blocks:
                floats = int(ops.library().pe_attention_mma_shared_scratch_floats(B, nh, nkv, d, blocks))
            scratch = torch.full((floats + 64,), float("nan"), device=DEV)
            ops.attention_mma_append(x, out, B, nh, nkv, d, d ** -0.5, window, qw, kw, 1e-5, cos, sin, *where, scratch, blocks, 4, least, st)
            assert torch.equal(x, qkv) and bool(scratch[floats:].isnan().all())      # inside the scratch it asked for
        else:
            t = torch.arange(B, dtype=torch.int32, device=DEV)
            ops.qk_norm_rope_append(x, B, nh, nkv, d, qw, kw, 1e-5, cos, sin, d if rotated else 0, t, past, ps.seq_slot, qstart, ps.table,
                                    ps.num_pages, ps.k_pages, ps.v_pages, True, st)
            scratch = torch.empty(ops.attention_generic_scratch_floats(B, nh, d, 11), device=DEV)
            ops.attention_mma(True, x, out, B, 1, nh, nkv, d, d ** -0.5, window, *where, scratch, 64, 11, st)
        outs.append(out.float())
        pages.append((ps.k_pages, ps.v_pages))
    assert st.tolist()[0] == 0
    assert rel_err(outs[0], outs[1]) < 2 * ATT_TOL[bf]
    assert torch.equal(pages[0][1], pages[1][1])
    # a key is one rounding of the same float32 numbers, whose sums may round differently
    k0, k1 = pages[0][0].double(), pages[1][0].double()
    assert bool(((k0 - k1).abs() <= 2.0 ** -7 * k1.abs()).all())


@pytest.mark.parametrize("nh,nkv,d", [(16, 8, 128), (6, 2, 64)])
@pytest.mark.parametrize("lens,others", [([300, 1, 64, 65, 130], [2, 512, 100, 449, 7]), ([520, 513], [576, 515]), ([2000, 1900, 2048], [1990, 2048, 1921])])
def test_attention_mma_append_takes_whole_pairs(ops, nh, nkv, d, lens, others):
    """Short sequences, or such of about the same length, are not cut: no partial results, and a sequence's output has the same bits
    whatever the others' lengths; with a block too few for that, and by the two kernels, the same within rounding."""
    torch.manual_seed(35)
    bf, B = torch.bfloat16, len(lens)
    qkv, angles = torch.randn(B, (nh + 2 * nkv) * d, device=DEV).to(bf), torch.rand(2112, d // 2, device=DEV) * 6
    t, qstart, st, outs = torch.arange(B, dtype=torch.int32, device=DEV), torch.arange(B + 1, dtype=torch.int32, device=DEV), _status(), []
    whole = PagedSetup(lens, nkv, d, bf, seed=35)
    for seen, blocks in ((lens, 296), (lens, B * nkv), (lens, B * nkv - 1), (lens, 0), ([lens[0]] + others[1:], 296)):
        ps = PagedSetup(seen, nkv, d, bf, seed=36)
        for i in range(-(-lens[0] // 64)):      # the first sequence's pages are the same in every run
            page, as_in = int(ps.table[ps.slots[0], i]), int(whole.table[whole.slots[0], i])
            ps.k_pages[page], ps.v_pages[page] = whole.k_pages[as_in], whole.v_pages[as_in]
        past = torch.tensor([L - 1 for L in seen], dtype=torch.int32, device=DEV)
        where = (qstart, past, ps.seq_slot, ps.table, ps.num_pages, ps.k_pages, ps.v_pages)
        x, out = qkv.clone(), torch.full((B, nh * d), float("nan"), device=DEV, dtype=bf)
        if blocks:
            scratch = torch.full((int(ops.library().pe_attention_mma_shared_scratch_floats(B, nh, nkv, d, blocks)),), float("nan"), device=DEV)
            ops.attention_mma_append(x, out, B, nh, nkv, d, d ** -0.5, 0, None, None, 1e-5, angles.cos(), angles.sin(), *where, scratch, blocks, 0, 128, st)
            assert bool(scratch[:(B * nkv + blocks) * (nh // nkv) * (d + 1)].isnan().all()) == (blocks >= B * nkv)
        else:
            ops.qk_norm_rope_append(x, B, nh, nkv, d, None, None, 1e-5, angles.cos(), angles.sin(), d, t, past, ps.seq_slot, qstart, ps.table,
                                    ps.num_pages, ps.k_pages, ps.v_pages, True, st)
            scratch = torch.empty(ops.attention_generic_scratch_floats(B, nh, d, 32), device=DEV)
            ops.attention_mma(True, x, out, B, 1, nh, nkv, d, d ** -0.5, 0, *where, scratch, 64, 32, st)
        outs.append(out)
    assert st.tolist()[0] == 0
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0][0], outs[4][0])
    assert all(rel_err(outs[0].float(), o.float()) < 2 * ATT_TOL[bf] for o in outs[2:4])


@pytest.mark.parametrize("B", [129, 512, 513])
def test_attention_mma_append_of_many_sequences(ops, B):
    """Batches around the number of sequences whose pages a block lists, keys shared out, against the two kernels."""
    torch.manual_seed(27)
    nh, nkv, d, bf = 4, 2, 64, torch.bfloat16
    lens = [64 * (b % 3) + 1 + b % 64 for b in range(B)]
    floats = int(ops.library().pe_attention_mma_shared_scratch_floats(B, nh, nkv, d, 444))
    assert (floats > 0) == (B <= 512)
    if not floats:
        return
    qkv, angles = torch.randn(B, (nh + 2 * nkv) * d, device=DEV).to(bf), torch.rand(256, d // 2, device=DEV) * 6
    t, qstart = torch.arange(B, dtype=torch.int32, device=DEV), torch.arange(B + 1, dtype=torch.int32, device=DEV)
    past, st, outs = torch.tensor([L - 1 for L in lens], dtype=torch.int32, device=DEV), _status(), []
    for fused in (True, False):
        ps = PagedSetup(lens, nkv, d, bf, seed=27)
        where = (qstart, past, ps.seq_slot, ps.table, ps.num_pages, ps.k_pages, ps.v_pages)
        x, out = qkv.clone(), torch.full((B, nh * d), float("nan"), device=DEV, dtype=bf)
        scratch = torch.empty(max(floats, ops.attention_generic_scratch_floats(B, nh, d, 4)), device=DEV)
        if fused:
            ops.attention_mma_append(x, out, B, nh, nkv, d, d ** -0.5, 0, None, None, 1e-5, angles.cos(), angles.sin(), *where, scratch, 444, 0, 64, st)
        else:
            ops.qk_norm_rope_append(x, B, nh, nkv, d, None, None, 1e-5, angles.cos(), angles.sin(), d, t, past, ps.seq_slot, qstart, ps.table,
                                    ps.num_pages, ps.k_pages, ps.v_pages, True, st)
            ops.attention_mma(True, x, out, B, 1, nh, nkv, d, d ** -0.5, 0, *where, scratch, 64, 4, st)
        outs.append(out.float())
    assert st.tolist()[0] == 0 and rel_err(outs[0], outs[1]) < 2 * ATT_TOL[bf]


@pytest.mark.parametrize("form", ["ranges", "clusters", 1, 5, 40])      # a number: keys shared out over so many blocks
@pytest.mark.parametrize("where,number", [("key", "nan"), ("key", "inf"), ("value", "nan"), ("value", "inf"), ("query", "nan"), ("query", "inf")])
def test_decode_attention_keeps_nan_and_infinity(ops, form, where, number):
    """One number that is none, in a cached key, value or query: outputs that it reaches are not finite, whichever range, block or warp
    it falls to, and all others have the bits they have without it."""
    torch.manual_seed(33)
    bf, nh, nkv, d, lens = torch.bfloat16, 8, 2, 64, [700, 130]
    B, st = len(lens), _status()
    qkv, t = torch.randn(B, (nh + 2 * nkv) * d, device=DEV).to(bf), torch.arange(len(lens), dtype=torch.int32, device=DEV)
    qstart, past = torch.arange(B + 1, dtype=torch.int32, device=DEV), torch.tensor([L - 1 for L in lens], dtype=torch.int32, device=DEV)

    def run(poisoned):
        ps, x = PagedSetup(lens, nkv, d, bf, seed=33), qkv.clone()
        page = int(ps.table[ps.slots[0], 300 // 64])
        if poisoned:
            {"key": ps.k_pages[page, 1, 300 % 64], "value": ps.v_pages[page, 1, 300 % 64], "query": x[0, 2 * d:3 * d]}[where][7] = float(number)
        out, blocks = torch.full((B, nh * d), 7.0, device=DEV, dtype=bf), form if isinstance(form, int) else 0
        floats = int(ops.library().pe_attention_mma_shared_scratch_floats(B, nh, nkv, d, max(blocks, 1)))
        scratch = torch.empty(max(floats, ops.attention_generic_scratch_floats(B, nh, d, 11)), device=DEV)
        where_to = (qstart, past, ps.seq_slot, ps.table, ps.num_pages, ps.k_pages, ps.v_pages)
        if form == "ranges":
            ops.qk_norm_rope_append(x, B, nh, nkv, d, None, None, 1e-5, None, None, 0, t, past, ps.seq_slot, qstart, ps.table, ps.num_pages,
                                    ps.k_pages, ps.v_pages, True, st)
            ops.attention_mma(True, x, out, B, 1, nh, nkv, d, d ** -0.5, 0, *where_to, scratch, 64, 11, st)
        else:
            ops.attention_mma_append(x, out, B, nh, nkv, d, d ** -0.5, 0, None, None, 1e-5, None, None, *where_to, scratch, blocks, 4, 64, st)
        assert st.tolist()[0] == 0
        return out.float().view(B, nh, d)

    reached = torch.zeros(B, nh, d, dtype=torch.bool, device=DEV)
    if where == "query":
        reached[0, 2] = True
    elif where == "value":
        reached[0, nh // 2:, 7] = True
    else:      # a score of minus infinity weighs nothing
        reached[0, nh // 2:] = (qkv[0, nh // 2 * d:nh * d].view(-1, d)[:, 7:8] > 0) | (number == "nan")
    got, clean = run(True), run(False)
    assert torch.equal(got.isfinite(), ~reached)
    if number == "nan":
        assert torch.equal(got[~reached], clean[~reached]) and bool(clean.isfinite().all())


class _Impatient:
    """The library, but for the entry points of one file compiled so that every bounded wait runs out at once."""

    def __init__(self, pe, folder, source):
        build, lib = pe.kernels.build, importlib.import_module("pytorch-engine_b200.kernels.lib")
        path = os.path.join(str(folder), "impatient.so")
        subprocess.run([build._find_nvcc(), *build.NVCC_FLAGS, "-DPE_WAIT_POLLS=0", "-I", build.CSRC, "-shared", os.path.join(build.CSRC, source),
                        "-o", path], check=True)
        self._usual, self._own = lib.library(), ctypes.CDLL(path)
        for name, argtypes in lib._SIGNATURES.items():
            if hasattr(self._own, name):
                getattr(self._own, name).argtypes = argtypes

    def __getattr__(self, name):
        return getattr(self._own if name == "pe_attention_mma_append" else self._usual, name)


def test_attention_mma_append_whose_waits_run_out(ops, pe, tmp_path, monkeypatch):
    """Keys shared out, and no wait ends: the step comes back with a status, every sequence's new row is in its own page and no
    other row of the cache has changed.  (Pages in the ring may then be anybody's; outputs say nothing.)"""
    torch.manual_seed(31)
    nh, nkv, d, bf, lens = 8, 2, 128, torch.bfloat16, [700, 1, 65, 64, 513]
    B, t = len(lens), torch.arange(len(lens), dtype=torch.int32, device=DEV)
    qkv, angles = torch.randn(B, (nh + 2 * nkv) * d, device=DEV).to(bf), torch.rand(704, d // 2, device=DEV) * 6
    qstart, past = torch.arange(B + 1, dtype=torch.int32, device=DEV), torch.tensor([L - 1 for L in lens], dtype=torch.int32, device=DEV)
    usual, impatient = ops.library(), _Impatient(pe, tmp_path, "attention_mma.cu")
    for blocks in (1, 3, 40):
        floats = int(usual.pe_attention_mma_shared_scratch_floats(B, nh, nkv, d, blocks))
        pages = []
        for library in (impatient, usual):
            ps, st = PagedSetup(lens, nkv, d, bf, seed=31), _status()
            scratch, out = torch.full((floats + 64,), float("nan"), device=DEV), torch.empty(B, nh * d, device=DEV, dtype=bf)
            monkeypatch.setattr(ops, "library", lambda: library)
            ops.attention_mma_append(qkv, out, B, nh, nkv, d, d ** -0.5, 0, None, None, 1e-5, angles.cos(), angles.sin(), qstart, past,
                                     ps.seq_slot, ps.table, ps.num_pages, ps.k_pages, ps.v_pages, scratch, blocks, 0, 64, st)
            assert st.tolist()[0] == (4 if library is impatient else 0)
            assert bool(scratch[floats:].isnan().all())
            pages.append((ps.k_pages, ps.v_pages))
        assert all(torch.equal(a, b) for a, b in zip(*pages))


@pytest.mark.parametrize("d,dv,kind", [(36, 96, "delta"), (64, 126, "mlstm")])
def test_recurrences_just_below_48_kb(ops, d, dv, kind):
    """Heads whose dynamic shared memory stays below 48 KB only without the kernel's static part: two tokens in one call as in two."""
    torch.manual_seed(26)
    H, B, slots = 2, 2, 3
    slot, rand = torch.tensor([2, 0], dtype=torch.int32, device=DEV), (lambda *shape: torch.randn(*shape, device=DEV))
    rows, gates, bias = rand(2 * B, H * (2 * d + 2 * dv)), rand(2 * B, 2 * H), rand(2 * H)
    S0, n0, m0, w = rand(slots, H, d, dv), rand(slots, H, d), rand(slots, H), 1 + 0.2 * rand(H * dv)

    def run(rows, gates, per, S, n, m):
        rows, gates = rows.contiguous(), gates.contiguous()
        out, st = torch.full((per * B, H * dv), float("nan"), device=DEV), _status()
        qstart = torch.arange(0, per * B + 1, per, dtype=torch.int32, device=DEV)
        q, k, v, g = (rows[:, lo:hi] for lo, hi in ((0, H * d), (H * d, 2 * H * d), (2 * H * d, H * (2 * d + dv)), (H * (2 * d + dv), rows.shape[1])))
        if kind == "delta":
            ops.delta_rule_recurrence(rows[:, :H * (2 * d + dv)].contiguous(), gates[:, :H].contiguous(), bias[:H], bias[H:], gates[:, H:].contiguous(), g, w[:dv],
                                      1e-6, d ** -0.5, out, S, slot, qstart, B, per, H, H, d, dv, st, head_decay=True)
        else:
            ops.mlstm_recurrence(q, k, v, g, gates, bias, w, 15.0, 1e-6, d ** -0.5, out, S, n, m, slot, qstart, B, per, H, d, dv, st)
        assert st.tolist()[0] == 0
        return out

    once, twice = [t.clone() for t in (S0, n0, m0)], [t.clone() for t in (S0, n0, m0)]
    whole = run(rows, gates, 2, *once)
    for i in range(2):
        assert rel_err(run(rows[i::2], gates[i::2], 1, *twice), whole[i::2]) < 2e-5
    assert all(rel_err(x, y) < 5e-6 for x, y in zip(once, twice))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("d,dv", [(128, 128), (128, 256), (64, 64), (8, 16), (100, 48), (32, 160), (36, 96)])
def test_recurrences_of_single_tokens_over_a_cluster(ops, dtype, d, dv):
    """A step of one token a sequence with a head's columns over a cluster against the same step in one block a head (which runs where
    a step says that it may bring two tokens): outputs and every part of the state; a sequence's slot out of range is left out."""
    torch.manual_seed(24)
    H, G, B, slots, f32 = 4, 2, 3, 5, torch.float32
    slot, qstart = torch.tensor([4, 0, 2], dtype=torch.int32, device=DEV), torch.arange(B + 1, dtype=torch.int32, device=DEV)
    rand = lambda *shape: torch.randn(*shape, device=DEV)  # noqa: E731
    qkv, gate = rand(B, 2 * G * d + H * dv).to(dtype), rand(B, H * dv + 8).to(dtype)[:, :H * dv]
    a, b, dt, A, nw, S0 = rand(B, H * d), rand(B, H), rand(H * d) - 2, rand(H) * 0.3, 1 + 0.2 * rand(dv), rand(slots, H, d, dv)
    tol = 2e-5 if dtype == f32 else 1e-2
    for head_decay, gate_silu in ((False, False), (True, True)):
        got = []
        for max_q in (1, 2):
            out, S, st = torch.full((B, H * dv), float("nan"), device=DEV, dtype=dtype), S0.clone(), _status()
            ops.delta_rule_recurrence(qkv, a[:, :H].contiguous() if head_decay else a, dt[:H] if head_decay else dt, A, b, gate, nw, 1e-6, d ** -0.5,
                                      out, S, slot, qstart, B, max_q, H, G, d, dv, st, head_decay=head_decay, gate_silu=gate_silu)
            assert st.tolist()[0] == 0
            got.append((out.float(), S))
        assert rel_err(got[0][0], got[1][0]) < tol and rel_err(got[0][1], got[1][1]) < 2e-6
    rows = rand(B, H * (2 * d + 2 * dv)).to(dtype)
    q, k, v, g = (rows[:, lo:hi] for lo, hi in ((0, H * d), (H * d, 2 * H * d), (2 * H * d, H * (2 * d + dv)), (H * (2 * d + dv), H * (2 * d + 2 * dv))))
    gates, bias, mw, n0, m0 = 3 * rand(B, 2 * H), rand(2 * H), 1 + 0.2 * rand(H * dv), rand(slots, H, d), rand(slots, H)
    got = []
    for max_q in (1, 2):
        out, S, n, mx, st = torch.full((B, H * dv), float("nan"), device=DEV, dtype=dtype), S0.clone(), n0.clone(), m0.clone(), _status()
        ops.mlstm_recurrence(q, k, v, g, gates, bias, mw, 15.0, 1e-6, d ** -0.5, out, S, n, mx, slot, qstart, B, max_q, H, d, dv, st)
        assert st.tolist()[0] == 0
        got.append((out.float(), S, n, mx))
    assert rel_err(got[0][0], got[1][0]) < tol
    for i in (1, 2, 3):
        assert rel_err(got[0][i], got[1][i]) < 2e-6
    S, st = S0.clone(), _status()
    ops.mlstm_recurrence(q, k, v, g, gates, bias, mw, 15.0, 1e-6, d ** -0.5, out, S, n, mx, slot + 2, qstart, B, 1, H, d, dv, st)
    assert st.tolist()[0] == 5 and torch.equal(S[[0, 1, 3]], S0[[0, 1, 3]])
    some, S, st = torch.tensor([0, 1, 1, 2], dtype=torch.int32, device=DEV), S0.clone(), _status()      # a sequence without a token
    ops.mlstm_recurrence(q, k, v, g, gates, bias, mw, 15.0, 1e-6, d ** -0.5, out, S, n, mx, slot, some, B, 1, H, d, dv, st)
    ops.delta_rule_recurrence(qkv, a, dt, A, b, gate, nw, 1e-6, d ** -0.5, out, S, slot, some, B, 1, H, G, d, dv, st)
    assert st.tolist()[0] == 0 and torch.equal(S[0], S0[0]) and not torch.equal(S[2], S0[2]) and not torch.equal(S[4], S0[4])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("taps,channels", [(2, 40), (4, 2048), (8, 129), (9, 64)])
@pytest.mark.parametrize("lengths", [(1, 1, 1), (2, 0, 1), (0, 0, 3)])
def test_short_conv_of_single_tokens(ops, dtype, taps, channels, lengths):
    """As many tokens as sequences (up to eight taps: one kernel) against the sum over the tail and the tokens, and the tail moved on."""
    torch.manual_seed(25)
    B, slots = 3, 5
    slot, ends = torch.tensor([4, 0, 2], dtype=torch.int32, device=DEV), [0, lengths[0], lengths[0] + lengths[1], B]
    qstart, of = torch.tensor(ends, dtype=torch.int32, device=DEV), [b for b in range(B) for _ in range(lengths[b])]
    x, w, bias = torch.randn(B, channels + 16, device=DEV).to(dtype), torch.randn(channels, taps, device=DEV), torch.randn(channels, device=DEV)
    tail = torch.randn(slots, taps - 1, channels, device=DEV)
    before, out, st = tail.clone(), torch.empty(B, channels, device=DEV, dtype=dtype), _status()
    ops.short_conv_silu(x, 8, w, tail, torch.tensor(of, dtype=torch.int32, device=DEV), slot, qstart, out, B, st, bias)
    want = before.clone()
    for t, s in enumerate(slot[of].tolist()):
        rows = torch.cat([want[s], x[t:t + 1, 8:8 + channels].float()])
        y = (rows.double() * w.t().double()).sum(0) + bias.double()
        assert rel_err(out[t].float(), (y / (1 + (-y).exp())).float()) < (2e-6 if dtype == torch.float32 else 1e-2)
        want[s] = rows[1:]
    assert torch.equal(tail, want) and st.tolist()[0] == 0


@pytest.mark.parametrize("nh,nkv,d,dv", [(8, 2, 128, 128), (5, 1, 128, 128), (6, 2, 192, 64)])
@pytest.mark.parametrize("parts", [2, 3, 8])
@pytest.mark.parametrize("window,sink,extra", [(0, False, ""), (200, True, "gate"), (0, True, "turn")])
def test_attention_umma_prefill_in_parts(ops, nh, nkv, d, dv, parts, window, sink, extra):
    """A row tile's pages over several blocks against one block a tile: new tokens behind a long past, tiles with fewer pages than
    parts, rows whose keys all lie in one part."""
    if extra == "turn" and (d, dv) != (128, 128):
        pytest.skip("turned outputs: heads of 128 features")
    torch.manual_seed(26)
    bf = torch.bfloat16
    q_lens, pasts = [70, 1, 33, 130], [900, 70, 0, 512]
    lens, N = [a + b for a, b in zip(q_lens, pasts)], sum(q_lens)
    kp, vp = PagedSetup(lens, nkv, d, bf, seed=26, key_scale=2.0), PagedSetup(lens, nkv, dv, bf, seed=26)
    q = torch.randn(N, (nh + nkv) * d, device=DEV).to(bf)
    gate = torch.randn(N, nh, device=DEV).to(bf) if extra == "gate" else None
    angles = torch.rand(1024, 64, device=DEV) * 6
    turn = dict(out_cos=angles.cos(), out_sin=angles.sin()) if extra == "turn" else {}
    qstart = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32, device=DEV)
    past, st = torch.tensor(pasts, dtype=torch.int32, device=DEV), _status()
    outs = []
    for n in (1, parts):
        out = torch.full((N, nh * dv), float("nan"), device=DEV, dtype=bf)
        scratch = torch.full((n * N * nh * (dv + 1) + 64,), float("nan"), device=DEV)
        ops.attention_umma_prefill(q, out, 4, max(q_lens), nh, nkv, d, d ** -0.5, window, qstart, past, kp.seq_slot, kp.table, kp.num_pages,
                                   kp.k_pages, vp.v_pages, st, sink=sink, v_dim=dv, gate=gate, parts=n, scratch=scratch, **turn)
        assert st.tolist()[0] == 0 and bool(scratch[n * N * nh * (dv + 1):].isnan().all())
        outs.append(out.float())
    assert rel_err(outs[1], outs[0]) < 2 * ATT_TOL[bf]


@pytest.mark.parametrize("parts", [3, 8])
@pytest.mark.parametrize("where,number", [("key", "nan"), ("key", "inf"), ("value", "nan"), ("value", "inf"), ("query", "nan"), ("query", "inf")])
def test_attention_umma_prefill_in_parts_keeps_nan_and_infinity(ops, parts, where, number):
    """One number that is none, in a cached key or value that every row of the first sequence sees or in one query: with parts the same
    outputs are NaN as with one block a tile, and the rows that do not see it have the bits they have without it."""
    torch.manual_seed(32)
    bf, nh, nkv, d = torch.bfloat16, 8, 2, 128
    q_lens, pasts = [70, 33], [900, 512]
    N, st = sum(q_lens), _status()
    q = torch.randn(N, (nh + nkv) * d, device=DEV).to(bf)
    qstart, past = torch.tensor([0, 70, N], dtype=torch.int32, device=DEV), torch.tensor(pasts, dtype=torch.int32, device=DEV)

    def run(n, poisoned):
        ps, x = PagedSetup([a + b for a, b in zip(q_lens, pasts)], nkv, d, bf, seed=32, key_scale=2.0), q.clone()
        page = int(ps.table[ps.slots[0], 300 // 64])
        if poisoned:
            row = {"key": ps.k_pages[page, 1, 300 % 64], "value": ps.v_pages[page, 1, 300 % 64], "query": x[5, 2 * d:3 * d]}[where]
            row[7] = float(number)
        out = torch.full((N, nh * d), 7.0, device=DEV, dtype=bf)
        scratch = torch.empty(n * N * nh * (d + 1), device=DEV)
        ops.attention_umma_prefill(x, out, 2, max(q_lens), nh, nkv, d, d ** -0.5, 0, qstart, past, ps.seq_slot, ps.table, ps.num_pages,
                                   ps.k_pages, ps.v_pages, st, parts=n, scratch=scratch)
        assert st.tolist()[0] == 0
        return out.float().view(N, nh, d)

    one, cut, clean = run(1, True), run(parts, True), run(parts, False)
    assert torch.equal(one.isfinite(), cut.isfinite()) and not bool(cut.isfinite().all())
    sees = torch.zeros(N, nh, dtype=torch.bool, device=DEV)
    if where == "query":
        sees[5, 2] = True
    else:
        sees[:70, nh // 2:] = True
    assert torch.equal(cut[~sees], clean[~sees]) and bool(clean.isfinite().all())


@pytest.mark.parametrize("decode", [False, True])
def test_attention_mma_finds_a_far_key_and_ignores_what_lies_beyond_the_length(ops, decode):
    nh, nkv, d = 8, 2, 128
    dtype = torch.bfloat16
    L, far = 650, 13
    ps = PagedSetup([L], nkv, d, dtype, seed=17, key_scale=0.05)
    probe = torch.randn(d)
    probe = probe / probe.norm() * 12.0
    q = probe.repeat(nh).view(1, nh * d)
    page = int(ps.table[ps.slots[0], far // 64])
    ps.k_pages[page, :, far % 64] = (probe * 2.0).to(DEV, dtype)
    # the row after the sequence's last key matches even better and must not be seen (the cache keeps
    # such rows finite, see the append kernel; a huge value shows any leak)
    last_page = int(ps.table[ps.slots[0], L // 64])
    ps.k_pages[last_page, :, L % 64] = (probe * 4.0).to(DEV, dtype)
    ps.v_pages[last_page, :, L % 64] = 1e30
    out = torch.zeros(1, nh * d, device=DEV, dtype=dtype)
    qstart = torch.tensor([0, 1], dtype=torch.int32, device=DEV)
    past_t = torch.tensor([L - 1], dtype=torch.int32, device=DEV)
    scratch = torch.zeros(ops.attention_generic_scratch_floats(1, nh, d, 3), device=DEV)
    ops.attention_mma(decode, q.to(DEV, dtype), out, 1, 1, nh, nkv, d, 1 / math.sqrt(d), 0, qstart, past_t, ps.seq_slot,
                      ps.table, ps.num_pages, ps.k_pages, ps.v_pages, scratch if decode else None,
                      256 if decode else 0, 3 if decode else 0, _status())
    v_far = ps.v_pages[page, :, far % 64].float().cpu()
    got = out.float().cpu().view(nh, d)
    for h in range(nh):
        assert torch.allclose(got[h], v_far[h // 4], atol=2e-2)


@pytest.mark.parametrize("M", [1, 3, 8, 9, 16])
@pytest.mark.parametrize("N,K", [(16, 64), (100, 80), (515, 200), (4096, 4096), (1000, 12288), (48, 8)])
def test_gemm_smallm(ops, M, N, K):
    torch.manual_seed(20)
    x = torch.randn(M, K, device=DEV).to(torch.bfloat16)
    w = (torch.randn(N, K, device=DEV) * 0.5).to(torch.bfloat16)
    want = x.float().cpu() @ w.float().cpu().T
    out32 = torch.full((M, N), float("nan"), device=DEV)
    ops.gemm_smallm(x, w, out32)
    assert rel_err(out32.cpu(), want) < 2e-5
    out16 = torch.zeros(M, N + 8, device=DEV, dtype=torch.bfloat16)[:, :N]      # a row stride larger than N
    ops.gemm_smallm(x, w, out16)
    assert rel_err(out16.float().cpu(), want) < KTOL[torch.bfloat16]
    # x as rows of a wider buffer
    wide = torch.randn(M, K + 24, device=DEV).to(torch.bfloat16)
    ops.gemm_smallm(wide[:, :K], w, out32)
    assert rel_err(out32.cpu(), wide[:, :K].float().cpu() @ w.float().cpu().T) < 2e-5


@pytest.mark.parametrize("M", [1, 8, 13])
@pytest.mark.parametrize("I,K", [(176, 80), (200, 96), (3072, 1024), (24, 4096)])
def test_gemm_smallm_with_the_gate_fused(ops, M, I, K):
    torch.manual_seed(21)
    x = torch.randn(M, K, device=DEV).to(torch.bfloat16)
    w = (torch.randn(2 * I, K, device=DEV) * (2.0 / K ** 0.5)).to(torch.bfloat16)
    gu = x.float().cpu() @ w.float().cpu().T
    g, u = gu[:, :I], gu[:, I:]
    want = g / (1 + torch.exp(-g)) * u
    out = torch.zeros(M, I, device=DEV, dtype=torch.bfloat16)
    ops.gemm_smallm(x, w, out, pair_offset=I)
    assert rel_err(out.float().cpu(), want) < KTOL[torch.bfloat16]
    out32 = torch.zeros(M, I, device=DEV)
    ops.gemm_smallm(x, w, out32, pair_offset=I)
    assert rel_err(out32.cpu(), want) < 2e-5


def test_gemm_smallm_refuses_what_it_does_not_take(pe, ops):
    x = torch.zeros(17, 64, device=DEV, dtype=torch.bfloat16)
    w = torch.zeros(32, 64, device=DEV, dtype=torch.bfloat16)
    assert not ops.gemm_smallm_supported(x, w)
    assert not ops.gemm_smallm_supported(x[:4, :60], w[:, :60].contiguous())
    with pytest.raises(pe.kernels.KernelError):
        ops.gemm_smallm(x, w, torch.zeros(17, 32, device=DEV))


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (1, 16, 8), (300, 515, 200), (2048, 1024, 512), (129, 257, 72),
                                   (640, 4096, 1024), (77, 1000, 4096)])
@pytest.mark.parametrize("kernel", ["gemm_umma", "gemm_umma2"])
def test_gemm_umma(ops, M, N, K, kernel):
    gemm = getattr(ops, kernel)    # one SM per 128 x 256 tile, or a pair of SMs per 256 x 256 tile
    if kernel == "gemm_umma2":
        K = -(-K // 64) * 64       # the pair kernel takes whole k blocks of 64
    torch.manual_seed(30)
    x = torch.randn(M, K, device=DEV).to(torch.bfloat16)
    w = (torch.randn(N, K, device=DEV) * 0.5).to(torch.bfloat16)
    want = x.float().cpu() @ w.float().cpu().T
    st = _status()
    out32 = torch.full((M, N), float("nan"), device=DEV)
    gemm(x, w, out32, st)
    assert st.tolist()[0] == 0
    assert rel_err(out32.cpu(), want) < 2e-5
    out16 = torch.zeros(M, N + 8, device=DEV, dtype=torch.bfloat16)[:, :N]
    gemm(x, w, out16, st)
    assert rel_err(out16.float().cpu(), want) < KTOL[torch.bfloat16]
    wide = torch.randn(M, K + 24, device=DEV).to(torch.bfloat16)
    gemm(wide[:, :K], w, out32, st)
    assert rel_err(out32.cpu(), wide[:, :K].float().cpu() @ w.float().cpu().T) < 2e-5
    assert st.tolist()[0] == 0


def row_errors(y, x, w):
    """The largest error of a row against 64 bits: 2-norm over that of the row (where its sums cancel, over what K independent
    products of such operands sum to)."""
    want, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t() / x.shape[1] ** 0.5
    return float(((y.double() - want).norm(dim=1) / torch.maximum(want.norm(dim=1), size.norm(dim=1))).max())


@pytest.mark.parametrize("M,N,K", [(1, 1, 4), (16, 128, 64), (63, 127, 60), (65, 132, 68), (129, 260, 1000), (200, 1024, 3072),
                                   (600, 4096, 1024), (40, 256, 8192)])
def test_gemm_split32(ops, M, N, K):
    """Float32 products on the tensor cores at the edges of tiles, chunks and ranges of K: no further from 64 bits than float32
    multiply-adds, for rows of any scale and next to numbers that have no bfloat16 parts."""
    torch.manual_seed(32)
    wide = torch.randn(M, K + 8, device=DEV) * torch.logspace(-18, 18, M, device=DEV)[:, None]
    x, w = wide[:, :K], torch.randn(N, K, device=DEV) * 0.5
    assert ops.gemm_split32_supported(x, w)
    out = torch.full((M, -(-N // 4) * 4 + 4), float("nan"), device=DEV)
    st = _status()
    ops.gemm_split32(x, w, out[:, :N], st)
    assert st.tolist()[0] == 0 and bool(out[:, N:].isnan().all())
    # parts: the three products left out are below 2^-25 of theirs; sums: per 64 of K the tensor core adds four times 16 large
    # products, cut to float32 (2^-23 at worst), and a chain of K / 64 roundings of 2^-24 joins them: 2^-21 for every K here.
    # Without one of the second-order products (2^-18 and less of its product) the error is 6 times that bound.
    err, library = (row_errors(y, x, w) for y in (out[:, :N], torch.mm(x, w.t())))
    assert err < 2.0 ** -21 and err < library + 2.0 ** -22
    if M >= 16 and K >= 64:
        x = x.contiguous().clone()
        x[3, 5], x[7, 0], x[9, 9], x[11, 1] = float("inf"), float("nan"), 3.4e38, -float("inf")
        w = w.clone()
        w[N // 2, 2] = float("inf")
        ops.gemm_split32(x, w, out[:, :N], st)
        ref = torch.mm(x, w.t())
        assert torch.equal(out[:, :N].isnan(), ref.isnan()) and torch.equal(out[:, :N].isinf(), ref.isinf())
        fin = ref.isfinite()
        assert rel_err(out[:, :N][fin].cpu() / ref[fin].abs().max().cpu(), ref[fin].cpu() / ref[fin].abs().max().cpu()) < 1e-5


@pytest.mark.parametrize("M,N,K", [(40, 200, 1000), (50, 132, 68), (150, 130, 60), (600, 4100, 68)])   # ranges of K; tiles of 64, of 128 rows
def test_gemm_split32_at_the_ends_of_float32s_range(ops, M, N, K):
    """Operands and results that bfloat16 parts do not hold: as close as a chain of float32 multiply-adds."""
    torch.manual_seed(33)
    near_one = lambda *shape: (torch.rand(*shape, device=DEV) + 0.5) * torch.randn(*shape, device=DEV).sign()
    st = _status()

    def check(x, w):
        x, w = x.contiguous(), w.contiguous()
        out = torch.full((M, -(-N // 4) * 4), float("nan"), device=DEV)[:, :N]
        ops.gemm_split32(x, w, out, st)
        want, size = x.double() @ w.double().t(), (x.double().abs() @ w.double().abs().t())
        # A chain of K multiply-adds has K roundings: up to 2^-24 of a partial sum each (deviation 0.58 of that) or, below 2^-126,
        # half the smallest subnormal.  Partial sums are a random walk of K products, sqrt(K) products = size / sqrt(K) high, in the
        # worst of 2.5 million outputs three times that, with an error of 3.5 deviations: 3.5 * 0.58 * 3 * 2^-24 * size.  (Operands cut
        # to 16 bits give 2^-16 / sqrt(K) of size and more.)  The library's chain has to keep the bound, too.
        bound = 6 * 2.0 ** -24 * size + K * 2.0 ** -150
        ratios = [float(((y.double() - want).abs() / bound).nan_to_num(0.0).max()) for y in (out, torch.mm(x, w.t()))]
        assert bool(out.isfinite().all()) and max(ratios) <= 1.0, ratios

    steps = lambda n, lo, hi: 2.0 ** torch.linspace(lo, hi, n, device=DEV, dtype=torch.float64).round()[:, None]
    check((near_one(M, K) * steps(M, -148, -90)).float(), near_one(N, K))           # small rows of x, of w, of both
    check(near_one(M, K), (near_one(N, K) * steps(N, -148, -90)).float())
    check((near_one(M, K) * steps(M, -80, -50)).float(), (near_one(N, K) * steps(N, -80, -40)).float())
    x, w = near_one(M, K), near_one(N, K)                                          # small values where the weights are large, and
    x[:, ::2] *= 2.0 ** -122                                                        # ordinary ones where there are none
    w[:, ::2] *= 2.0 ** 110
    w[:, 1::2] = 0
    check(x, w)
    check(x * torch.tensor([1.0, 0.0], device=DEV).repeat(K // 2), w)
    x, w = torch.zeros(M, K, device=DEV), torch.zeros(N, K, device=DEV)             # one product a sum, close to the largest number
    x[:, 4], w[:, 4] = 3.4028e38, 0.999
    check(x, w)
    x[:, 4], w[:, 4] = 1.9999 * 2.0 ** 63, 1.9999 * 2.0 ** 63
    check(x, w)
    assert st.tolist()[0] == 0
    bad = near_one(M, K)                                                            # nothing but NaN
    bad[:] = float("nan")
    out = torch.zeros(M, -(-N // 4) * 4, device=DEV)[:, :N]
    ops.gemm_split32(bad, near_one(N, K), out, st)
    assert bool(out.isnan().all()) and st.tolist()[0] == 0


@pytest.mark.parametrize("M,less,K", [(257, 4, 68), (300, 0, 1000), (320, 0, 128)])
def test_gemm_split32_tiles_of_160_rows(ops, M, less, K):
    """Tiles of 160 rows, which save a wave of blocks where two of them a column of tiles are one block an SM: a last tile of 97 rows,
    of 140, and whole ones."""
    N = 128 * (ops.sm_count(torch.device(DEV)) // 2) - less
    test_gemm_split32(ops, M, N, K)
    if K == 68:
        test_gemm_split32_at_the_ends_of_float32s_range(ops, M, N, K)


@pytest.mark.parametrize("M,I,K", [(128, 128, 64), (200, 384, 200), (1000, 1280, 1024), (5, 256, 4096)])
@pytest.mark.parametrize("kernel", ["gemm_umma", "gemm_umma2"])
def test_gemm_umma_with_the_gate_fused(ops, M, I, K, kernel):
    if kernel == "gemm_umma2":
        K = -(-K // 64) * 64
    torch.manual_seed(31)
    x = torch.randn(M, K, device=DEV).to(torch.bfloat16)
    w = (torch.randn(2 * I, K, device=DEV) * (2.0 / K ** 0.5)).to(torch.bfloat16)
    gu = x.float().cpu() @ w.float().cpu().T
    g, u = gu[:, :I], gu[:, I:]
    want = g / (1 + torch.exp(-g)) * u
    out = torch.zeros(M, I, device=DEV, dtype=torch.bfloat16)
    st = _status()
    getattr(ops, kernel)(x, w, out, st, pair_offset=I)
    assert st.tolist()[0] == 0
    assert rel_err(out.float().cpu(), want) < KTOL[torch.bfloat16]


@pytest.mark.parametrize("M,N,K,fused", [(2048, 4096, 12288, False), (1536, 6144, 4096, False), (1024, 4096, 4096, False),
                                         (2048, 12288, 4096, True)])
@pytest.mark.parametrize("kernel", ["gemm_umma", "gemm_umma2"])
def test_gemm_umma_at_the_layer_shapes_of_an_8b_model(ops, M, N, K, fused, kernel):
    """The products of a 2,048-token prompt at width 4,096 / 12,288 (K = 12,288 is 192 k blocks: the 3- and 4-stage
    rings turn over dozens of times).  Every output against the library's true float32 product on the device, and
    a sample of rows against a float64 product on the CPU."""
    torch.manual_seed(33)
    x = torch.randn(M, K, device=DEV).to(torch.bfloat16)
    rows_w = 2 * N if fused else N
    w = (torch.randn(rows_w, K, device=DEV) * (2.0 / K ** 0.5)).to(torch.bfloat16)
    st = _status()
    out = torch.full((M, N), float("nan"), device=DEV, dtype=torch.bfloat16 if fused else torch.float32)
    getattr(ops, kernel)(x, w, out, st, **({"pair_offset": N} if fused else {}))
    assert st.tolist()[0] == 0

    def finish(prod):
        if not fused:
            return prod
        g, u = prod[:, :N], prod[:, N:]
        return g / (1 + torch.exp(-g)) * u

    prev = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = False
    try:
        want = finish(torch.mm(x.float(), w.float().t()))
    finally:
        torch.backends.cuda.matmul.allow_tf32 = prev
    tol = KTOL[torch.bfloat16] if fused else 2e-5
    assert rel_err(out.float().cpu(), want.cpu()) < tol
    pick = torch.randperm(M)[:48].sort().values
    exact = finish(x[pick].double().cpu() @ w.double().cpu().T)
    assert rel_err(out[pick].double().cpu(), exact) < tol


@pytest.mark.parametrize("nh,nkv,K,norm,rotate", [(8, 2, 256, True, True), (3, 1, 320, True, True), (6, 3, 192, False, True),
                                                  (4, 4, 128, True, False)])
def test_qkv_product_with_norm_rotation_and_append_in_its_epilogue(ops, nh, nkv, K, norm, rotate):
    """The q|k|v product with q/k-norm, rotation and cache append in its epilogue against the three kernels it
    stands for (product, then norm + rotation + append): three sequences, one of which starts in this step and one
    ends in the middle of a page; 3 and 5 heads' worth of columns do not fill the last 256-column tile.  Queries as
    the separate kernels leave them, the cache's pages bit for bit except the rounding of the norm's sum."""
    torch.manual_seed(41)
    d, dtype = 128, torch.bfloat16
    lens, q_lens = [300, 130, 200], [230, 130, 136]
    N = sum(q_lens)
    x = torch.randn(N, K, device=DEV).to(dtype)
    w = (torch.randn((nh + 2 * nkv) * d, K, device=DEV) * (1.5 / K ** 0.5)).to(dtype)
    qw = (1 + 0.2 * torch.randn(d, device=DEV)) if norm else None
    kw = (1 + 0.2 * torch.randn(d, device=DEV)) if norm else None
    eps, theta, max_pos = 1e-5, 1e4, 512
    ang = torch.outer(torch.arange(max_pos, dtype=torch.float32), plain.rope_inv_freq(d, theta))
    cos, sin = (torch.cos(ang).to(DEV), torch.sin(ang).to(DEV)) if rotate else (None, None)
    token_seq = torch.tensor(sum(([b] * n for b, n in enumerate(q_lens)), []), dtype=torch.int32, device=DEV)
    pos_list = sum(([lens[b] - q_lens[b] + i for i in range(q_lens[b])] for b in range(3)), [])
    token_pos = torch.tensor(pos_list, dtype=torch.int32, device=DEV)
    qstart = torch.tensor([0, q_lens[0], q_lens[0] + q_lens[1], N], dtype=torch.int32, device=DEV)
    assert ops.gemm_umma2_qkv_rope_supported(x, w, nh, nkv, d, d if rotate else 0)
    results = []
    for fused in (False, True):
        ps = PagedSetup(lens, nkv, d, dtype, seed=41)
        ld = (nh + 2 * nkv) * d
        qkv = torch.zeros(N, ld, device=DEV, dtype=dtype)
        st = _status()
        if fused:
            ops.gemm_umma2_qkv_rope(x, w, qkv, nh, nkv, d, qw, kw, eps, cos, sin, d if rotate else 0, token_seq, token_pos,
                                    ps.seq_slot, qstart, ps.table, ps.num_pages, ps.k_pages, ps.v_pages, True, st)
        else:
            ops.gemm_umma2(x, w, qkv, st)
            ops.qk_norm_rope_append(qkv, N, nh, nkv, d, qw, kw, eps, cos, sin, d if rotate else 0, token_seq, token_pos,
                                    ps.seq_slot, qstart, ps.table, ps.num_pages, ps.k_pages, ps.v_pages, True, st)
        assert st.tolist()[0] == 0
        results.append((qkv[:, : nh * d].float().cpu(), ps.k_pages.float().cpu(), ps.v_pages.float().cpu()))
    (q0, k0, v0), (q1, k1, v1) = results
    assert rel_err(q1, q0) < 4e-3 and rel_err(k1, k0) < 4e-3         # one bfloat16 step where the norm's sum rounds differently
    assert (q1 != q0).float().mean() < 0.02 and (k1 != k0).float().mean() < 0.02
    assert torch.equal(v1, v0)                                        # values are copied: bit for bit, cleared rows included
    # and against the plain formulas
    prod = x.float().cpu() @ w.float().cpu().T
    prod = prod.to(dtype).float()
    q_in = prod[:, : nh * d].view(N, nh, d)
    want = plain.rms_norm(q_in, qw.cpu(), eps) if norm else q_in
    if rotate:
        c, s_ = plain.rope_cos_sin(torch.tensor(pos_list), d, theta)
        want = plain.rope_rotate_neox(want, c, s_, d)
    assert rel_err(q1.view(N, nh, d), want) < KTOL[dtype]
    # a layer that only reads a cache: nothing is appended
    ps = PagedSetup(lens, nkv, d, dtype, seed=41)
    k_before = ps.k_pages.clone()
    qkv = torch.zeros(N, (nh + 2 * nkv) * d, device=DEV, dtype=dtype)
    ops.gemm_umma2_qkv_rope(x, w, qkv, nh, nkv, d, qw, kw, eps, cos, sin, d if rotate else 0, token_seq, token_pos,
                            ps.seq_slot, qstart, ps.table, ps.num_pages, ps.k_pages, ps.v_pages, False, _status())
    assert torch.equal(ps.k_pages, k_before) and torch.equal(qkv[:, : nh * d].float().cpu(), q1)


def test_sampler_greedy_and_ties(ops):
    torch.manual_seed(8)
    logits = torch.randn(6, 1000, device=DEV)
    logits[2, 17] = logits[2, 900] = 50.0                     # a tie: the lower index wins
    logits[3, 999] = 60.0
    req = torch.arange(6, dtype=torch.int32, device=DEV)
    step = torch.zeros(6, dtype=torch.int32, device=DEV)
    out = torch.empty(6, dtype=torch.int32, device=DEV)
    ops.sample(logits, 0.0, 0, 1.0, 0.0, 1, req, step, out)
    want = logits.argmax(-1).tolist()
    want[2] = 17
    assert out.tolist() == want


@pytest.mark.parametrize("filters", [dict(), dict(top_k=5), dict(top_k=40, top_p=0.9, min_p=0.05), dict(top_p=0.6),
                                     dict(min_p=0.2), dict(top_k=1500)])
def test_sampler_matches_the_plain_draw(ops, filters):
    torch.manual_seed(9)
    V, rows = 2000, 24
    logits = torch.randn(rows, V, device=DEV) * 2.5
    req = torch.arange(rows, dtype=torch.int32, device=DEV) % 5
    step = torch.arange(rows, dtype=torch.int32, device=DEV) // 5
    out = torch.empty(rows, dtype=torch.int32, device=DEV)
    kw = dict(top_k=0, top_p=1.0, min_p=0.0)
    kw.update(filters)
    ops.sample(logits, 0.8, kw["top_k"], kw["top_p"], kw["min_p"], 1234, req, step, out)
    got = out.tolist()
    agree = 0
    for r in range(rows):
        want = plain.sample_token(logits[r].cpu(), seed=1234, request=int(req[r]), step=int(step[r]), temperature=0.8, **kw)
        _, probs = plain.filter_logits(logits[r].cpu(), temperature=0.8, **kw)
        assert probs[got[r]] > 0, "the kernel drew a token that the filters exclude"
        agree += got[r] == want
    assert agree >= rows - 1     # float32 vs float64 Gumbel arithmetic may flip one near-tie


@pytest.mark.parametrize("V", [4097, 10000, 151936])
def test_sampler_with_scratch_greedy(ops, V):
    """Rows cut into chunks by a first kernel: the same argmax, ties to the lower index, across chunk borders."""
    torch.manual_seed(11)
    rows = 5
    logits = torch.randn(rows, V, device=DEV)
    logits[1, 4095] = logits[1, 4096] = 40.0                  # a tie across the first chunk border
    logits[2, V - 1] = 41.0                                   # the last entry of the last (short) chunk
    logits[3, 0] = 42.0
    logits[4, 5000 % V] = float("nan")                        # NaN never wins
    req = torch.arange(rows, dtype=torch.int32, device=DEV)
    step = torch.zeros(rows, dtype=torch.int32, device=DEV)
    out = torch.empty(rows, dtype=torch.int32, device=DEV)
    need = ops.sample_scratch_bytes(rows, V, 0.0, 0)
    assert need > 0
    scratch = torch.empty(need, dtype=torch.uint8, device=DEV)
    ops.sample(logits, 0.0, 0, 1.0, 0.0, 1, req, step, out, scratch=scratch)
    want = torch.nan_to_num(logits, nan=-float("inf")).argmax(-1).tolist()
    want[1] = 4095
    assert out.tolist() == want


@pytest.mark.parametrize("filters", [dict(top_k=5), dict(top_k=40, top_p=0.9, min_p=0.05), dict(top_k=40, top_p=0.95, min_p=0.05),
                                     dict(top_k=64, top_p=0.5), dict(top_k=1)])
def test_sampler_with_scratch_matches_the_plain_draw_and_the_single_kernel(ops, filters):
    torch.manual_seed(12)
    V, rows = 20011, 16
    logits = torch.randn(rows, V, device=DEV) * 2.5
    logits[3, 100:140] = 9.0                                  # forty ties at the top of one chunk
    logits[5, :] = 0.25                                       # every entry ties: the chunks overflow, the row is read whole
    req = torch.arange(rows, dtype=torch.int32, device=DEV) % 5
    step = torch.arange(rows, dtype=torch.int32, device=DEV) // 5
    kw = dict(top_k=0, top_p=1.0, min_p=0.0)
    kw.update(filters)
    need = ops.sample_scratch_bytes(rows, V, 0.8, kw["top_k"], kw["top_p"], kw["min_p"])
    assert need > 0
    scratch = torch.empty(need, dtype=torch.uint8, device=DEV)
    out = torch.empty(rows, dtype=torch.int32, device=DEV)
    single = torch.empty(rows, dtype=torch.int32, device=DEV)
    ops.sample(logits, 0.8, kw["top_k"], kw["top_p"], kw["min_p"], 99, req, step, out, scratch=scratch)
    ops.sample(logits, 0.8, kw["top_k"], kw["top_p"], kw["min_p"], 99, req, step, single)
    got = out.tolist()
    assert sum(a != b for a, b in zip(got, single.tolist())) <= 1
    agree = 0
    for r in range(rows):
        want = plain.sample_token(logits[r].cpu(), seed=99, request=int(req[r]), step=int(step[r]), temperature=0.8, **kw)
        _, probs = plain.filter_logits(logits[r].cpu(), temperature=0.8, **kw)
        if r != 5:    # with every entry tied, which k of them a top-k keeps is not defined
            assert probs[got[r]] > 0, "the kernel drew a token that the filters exclude"
            agree += got[r] == want
    assert agree >= rows - 2
    assert ops.sample_scratch_bytes(rows, V, 0.8, 0, 0.9) == 0 and ops.sample_scratch_bytes(rows, 3000, 0.8, 40) == 0


@pytest.mark.parametrize("V,k", [(4097, 50), (16384, 224), (16385, 200), (16387, 225), (50001, 17), (151936, 200)])
def test_sampler_top_k_at_the_edges_of_its_chunks(ops, V, k):
    """A last chunk of one entry or with fewer entries than k, rows without 16-byte alignment, k at the largest that
    the register kernel takes and beyond it, masked rows, ties: the same draws as one kernel over the whole row."""
    torch.manual_seed(14)
    rows = 8
    logits = torch.randn(rows, V, device=DEV) * 2.5
    logits[1, k // 2:] = -float("inf")                        # fewer finite entries than k
    logits[2, ::3] = float("nan")
    logits[3, V - 1] = 30.0
    logits[4, :3 * k] = 8.0                                   # 3 k entries tie at the top: more than a chunk has room for
    logits[5] = -float("inf")
    logits[6, 7] = float("inf")
    req = torch.arange(rows, dtype=torch.int32, device=DEV)
    step = torch.zeros(rows, dtype=torch.int32, device=DEV)
    need = ops.sample_scratch_bytes(rows, V, 0.8, k, 0.95, 0.0)
    assert need > 0
    scratch = torch.empty(need, dtype=torch.uint8, device=DEV)
    for top_p, min_p in ((1.0, 0.0), (0.95, 0.0), (0.7, 0.02)):
        a, b = (torch.empty(rows, dtype=torch.int32, device=DEV) for _ in range(2))
        ops.sample(logits, 0.8, k, top_p, min_p, 3, req, step, a, scratch=scratch)
        ops.sample(logits, 0.8, k, top_p, min_p, 3, req, step, b)
        assert a.tolist() == b.tolist(), (top_p, min_p)
        for r in (0, 1, 2, 3):
            row = logits[r].cpu()
            row[row.isnan()] = -float("inf")                  # where the kernels sort them
            _, probs = plain.filter_logits(row, temperature=0.8, top_k=k, top_p=top_p, min_p=min_p)
            assert probs[a[r]] > 0


@pytest.mark.parametrize("V,k", [(50001, 50), (50001, 200), (151936, 1), (151936, 224)])
def test_sampler_large_entries_side_by_side(ops, V, k):
    """Rows whose largest entries fill a few groups, so that their maxima bound the k-th value from far below, and rows of ties: the
    same draws as one kernel over the whole row, and (but for the ties) in a few times what other rows take."""
    torch.manual_seed(34)
    x = torch.randn(8, V, device=DEV) * 2.5
    rows = torch.arange(V, device=DEV) * -1e-3 + 5e-4 * x     # fall with the id
    rows[1] = x[1].sort(descending=True)[0]
    rows[2] = torch.full_like(x[2], -float("inf"))
    rows[2, 20000:25000] = x[2, 20000:25000]                  # some thousand entries of one range
    rows[3] = x[3].sort()[0]                                  # the last, ragged group holds the largest
    rows[4, ::7] = float("nan")
    rows[5, 1000:1000 + 2 * k] = 6.0                          # ties at the top
    rows[6] = 0.25                                            # nothing but ties
    rows[7] = torch.where(rows[2].isinf(), torch.full_like(x[7], -1e9), x[7])
    req, step = torch.arange(8, dtype=torch.int32, device=DEV), torch.zeros(8, dtype=torch.int32, device=DEV)
    scratch = torch.empty(ops.sample_scratch_bytes(8, V, 0.8, k, 0.95, 0.0), dtype=torch.uint8, device=DEV)
    a, b = (torch.empty(8, dtype=torch.int32, device=DEV) for _ in range(2))
    for top_p, min_p in ((1.0, 0.0), (0.95, 0.0), (0.7, 0.02)):
        ops.sample(rows, 0.8, k, top_p, min_p, 3, req, step, a, scratch=scratch)
        ops.sample(rows, 0.8, k, top_p, min_p, 3, req, step, b)
        assert a.tolist() == b.tolist(), (top_p, min_p)

    def took(logits):
        times = []
        for _ in range(9):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda._sleep(100000)                         # the launches are queued behind this
            start.record()
            ops.sample(logits, 0.8, k, 0.95, 0.0, 3, req, step, a, scratch=scratch)
            end.record()
            torch.cuda.synchronize()
            times.append(start.elapsed_time(end))
        return sorted(times)[4]

    # a search over the whole row takes some fifteen times as long as a draw from other rows
    assert took(rows[:6].repeat(2, 1)[:8]) < 6 * took(x)


def test_sampler_with_scratch_unfiltered_draw_is_the_single_kernels(ops):
    torch.manual_seed(13)
    rows, V = 12, 30000
    logits = torch.randn(rows, V, device=DEV) * 2
    req = torch.arange(rows, dtype=torch.int32, device=DEV)
    step = torch.full((rows,), 3, dtype=torch.int32, device=DEV)
    a, b = (torch.empty(rows, dtype=torch.int32, device=DEV) for _ in range(2))
    scratch = torch.empty(ops.sample_scratch_bytes(rows, V, 0.9, 0), dtype=torch.uint8, device=DEV)
    assert scratch.numel() > 0
    ops.sample(logits, 0.9, 0, 1.0, 0.0, 5, req, step, a, scratch=scratch)
    ops.sample(logits, 0.9, 0, 1.0, 0.0, 5, req, step, b)
    assert a.tolist() == b.tolist()


def test_sampler_is_keyed_by_request_and_step_not_by_row(ops):
    torch.manual_seed(10)
    row = torch.randn(1, 3000, device=DEV)
    logits = row.repeat(4, 1)
    req = torch.tensor([3, 3, 4, 3], dtype=torch.int32, device=DEV)
    step = torch.tensor([0, 1, 0, 0], dtype=torch.int32, device=DEV)
    out = torch.empty(4, dtype=torch.int32, device=DEV)
    ops.sample(logits, 1.0, 0, 1.0, 0.0, 77, req, step, out)
    a = out.tolist()
    assert a[0] == a[3] and len({a[0], a[1], a[2]}) >= 2
    ops.sample(logits, 1.0, 0, 1.0, 0.0, 78, req, step, out)
    assert out.tolist() != a


def test_repetition_penalty(ops):
    logits = torch.tensor([[2.0, -1.0, 0.5, 3.0], [1.0, 1.0, 1.0, 1.0]], device=DEV)
    recent = torch.tensor([[3, 1, 3, 0], [2, 0, 0, 0]], dtype=torch.int32, device=DEV)
    count = torch.tensor([3, 1], dtype=torch.int32, device=DEV)
    ops.repetition_penalty(logits, recent, count, 2.0)
    assert logits.tolist() == [[2.0, -2.0, 0.5, 1.5], [1.0, 1.0, 0.5, 1.0]]


def test_unsupported_sizes_are_refused(pe, ops):
    q = torch.zeros(1, 1024, device=DEV)
    with pytest.raises(pe.kernels.KernelError, match="size"):
        ops.attention_generic(False, q, q.clone(), 1, 1, 1, 1, 1024, 1.0, 0, torch.zeros(2, dtype=torch.int32, device=DEV),
                              torch.zeros(1, dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV),
                              torch.zeros(1, 1, dtype=torch.int32, device=DEV), 1, q, q, None, 0, 0, _status())
    with pytest.raises(pe.kernels.KernelError):
        ops.embed_gather(torch.zeros(4, 4), torch.zeros(1, dtype=torch.int32), torch.zeros(1, 4), torch.zeros(4, dtype=torch.int32))


def test_a_bounded_wait_gives_up_within_seconds(ops):
    """Every wait inside a kernel polls an mbarrier a limited number of times.  A poll that finds the phase incomplete
    takes microseconds (the hardware parks the thread for a while), so the limit in polls is a limit in time: the
    probe kernel polls a barrier on which nothing arrives, a counted number of times, and ends by itself."""
    poll = ops.wait_poll_seconds(DEV, polls=20000)
    assert 1e-7 < poll < 2e-5, f"one failing poll took {poll * 1e6:.2f} us"
    limit = ops.wait_limit_seconds(DEV)
    assert 0.5 < limit < 10.0, f"a wait that nothing ends would last {limit:.1f} s"


def _near(got, want, tol):
    return float((got.double() - want).norm() / want.norm()) < tol


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 5e-6), (torch.bfloat16, 6e-3)])   # float32 chains of 25 tokens; one rounding
@pytest.mark.parametrize("heads,kv_heads,d,dv", [(4, 2, 128, 128), (2, 2, 64, 48), (3, 1, 32, 16), (2, 1, 128, 256)])
@pytest.mark.parametrize("head_decay", [False, True])
def test_delta_rule_walk(ops, dtype, tol, heads, kv_heads, d, dv, head_decay):
    """Sequences that end before, at and behind a stage of eight tokens, from states that are not zero, against 64 bits and
    against the kernel that keeps a head in one block."""
    torch.manual_seed(40)
    lens, slots = [1, 7, 8, 9, 25], [3, 0, 5, 1, 2]
    N, n = sum(lens), len(lens)
    qkv = torch.randn(N, 2 * kv_heads * d + heads * dv, device=DEV).to(dtype)
    a = torch.randn(N, heads if head_decay else heads * d, device=DEV)
    dt = torch.randn(a.shape[1], device=DEV) - 3.0
    A_log, b = torch.randn(heads, device=DEV) * 0.5, torch.randn(N, heads, device=DEV)
    gate, w = torch.randn(N, heads * dv, device=DEV).to(dtype), torch.rand(dv, device=DEV) + 0.5
    S0 = torch.randn(6, heads, d, dv, device=DEV)
    qstart = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    slot = torch.tensor(slots, dtype=torch.int32, device=DEV)
    floats = ops.delta_rule_walk_scratch_floats(N, heads, kv_heads, d, dv)
    assert floats > 0 and ops.delta_rule_walk_scratch_floats(N, heads, kv_heads, 96, dv) == 0 and ops.delta_rule_walk_scratch_floats(N, heads, kv_heads, d, 24) == 0
    S, S1, st = S0.clone(), S0.clone(), _status()
    out, out1 = (torch.zeros(N, heads * dv, device=DEV, dtype=dtype) for _ in range(2))
    args = (qkv, a, dt, A_log, b, gate, w, 1e-5, d ** -0.5)
    form = dict(head_decay=head_decay, gate_silu=head_decay)
    ops.delta_rule_walk(*args, out, S, slot, qstart, n, heads, kv_heads, d, dv, st, torch.full((floats,), float("nan"), device=DEV), **form)
    ops.delta_rule_recurrence(*args, out1, S1, slot, qstart, n, max(lens), heads, kv_heads, d, dv, st, **form)
    assert st.tolist()[0] == 0
    q, k, v = qkv.double().split([kv_heads * d, kv_heads * d, heads * dv], 1)
    q, k = (x.view(N, kv_heads, d).repeat_interleave(heads // kv_heads, 1) for x in (q, k))
    q = q / (q.pow(2).sum(-1, keepdim=True) + 1e-6).sqrt() * d ** -0.5
    k = k / (k.pow(2).sum(-1, keepdim=True) + 1e-6).sqrt()
    z = (a.double() + dt.double()).view(N, heads, -1)
    g = torch.exp(-A_log.double().exp()[None, :, None] * torch.nn.functional.softplus(z)).expand(N, heads, d)
    o, end = torch.empty(N, heads, dv, dtype=torch.float64, device=DEV), S0.double()
    t = 0
    for L, s in zip(lens, slots):
        M = end[s]
        for _ in range(L):
            M = g[t][:, :, None] * M
            u = torch.sigmoid(b[t].double())[:, None] * (v[t].view(heads, dv) - torch.einsum("hij,hi->hj", M, k[t]))
            M = M + k[t][:, :, None] * u[:, None]
            o[t] = torch.einsum("hij,hi->hj", M, q[t])
            t += 1
        end[s] = M
    gd = gate.double().view(N, heads, dv)
    y = o / (o.pow(2).mean(-1, keepdim=True) + 1e-5).sqrt() * w.double() * torch.sigmoid(gd) * (gd if head_decay else 1.0)
    assert _near(out, y.reshape(N, -1), tol) and _near(S, end, 5e-6)
    assert _near(out1, y.reshape(N, -1), tol) and torch.equal(S[4], S0[4])     # the slot that no sequence has


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 6e-3)])   # (a small denominator magnifies its sum's rounding)
@pytest.mark.parametrize("heads,d,dv", [(3, 128, 256), (2, 64, 48), (5, 32, 16)])
def test_mlstm_walk(ops, dtype, tol, heads, d, dv):
    """As above for the matrix memory with exponential gates; one sequence is longer than a tile of its gates."""
    torch.manual_seed(41)
    lens, slots = [1, 8, 9, 23, 1030], [3, 0, 5, 1, 2]
    N, n = sum(lens), len(lens)
    rows = torch.randn(N, 2 * heads * (d + dv), device=DEV).to(dtype)
    q, k, v, g = rows.split([heads * d, heads * d, heads * dv, heads * dv], 1)
    gates, bias = torch.randn(N, 2 * heads, device=DEV), torch.cat([torch.randn(heads), torch.randn(heads) + 4.0]).to(DEV)
    w = torch.rand(heads * dv, device=DEV) + 0.5
    S0, n0, m0 = torch.randn(6, heads, d, dv, device=DEV), torch.randn(6, heads, d, device=DEV), torch.randn(6, heads, device=DEV)
    qstart = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    slot = torch.tensor(slots, dtype=torch.int32, device=DEV)
    floats = ops.mlstm_walk_scratch_floats(N, heads, d, dv)
    assert floats > 0 and ops.mlstm_walk_scratch_floats(N, heads, 96, dv) == 0
    S, nv, m, st = S0.clone(), n0.clone(), m0.clone(), _status()
    out = torch.zeros(N, heads * dv, device=DEV, dtype=dtype)
    ops.mlstm_walk(q, k, v, g, gates, bias, w, 15.0, 1e-5, d ** -0.5, out, S, nv, m, slot, qstart, n, heads, d, dv, st,
                   torch.full((floats,), float("nan"), device=DEV))
    assert st.tolist()[0] == 0
    z = 15.0 * torch.tanh((gates.double() + bias.double()) / 15.0)
    gi, gf = z[:, :heads], torch.nn.functional.logsigmoid(z[:, heads:])
    qd, kd, vd = q.double().view(N, heads, d) * d ** -0.5, k.double().view(N, heads, d), v.double().view(N, heads, dv)
    o, eS, en, em = torch.empty(N, heads, dv, dtype=torch.float64, device=DEV), S0.double(), n0.double(), m0.double()
    t = 0
    for L, s in zip(lens, slots):
        M, nn, mm = eS[s], en[s], em[s]
        for _ in range(L):
            new = torch.maximum(gf[t] + mm, gi[t])
            keep, take = torch.exp(gf[t] + mm - new)[:, None], torch.exp(gi[t] - new)[:, None]
            M = keep[..., None] * M + (take * kd[t])[:, :, None] * vd[t][:, None]
            nn, mm = keep * nn + take * kd[t], new
            den = torch.maximum((nn * qd[t]).sum(-1).abs(), torch.exp(-mm)) + 1e-6
            o[t] = torch.einsum("hij,hi->hj", M, qd[t]) / den[:, None]
            t += 1
        eS[s], en[s], em[s] = M, nn, mm
    y = o / (o.pow(2).mean(-1, keepdim=True) + 1e-5).sqrt() * w.double().view(heads, dv) * torch.sigmoid(g.double().view(N, heads, dv))
    assert _near(out, y.reshape(N, -1), tol) and _near(S, eS, 1e-5) and _near(nv, en, 1e-5) and _near(m, em, 1e-5)
    assert torch.equal(S[4], S0[4])
