"""The recurrent mixers' kernels alone at the sizes where their cuts can go wrong: chunks and tiles with one token or one column
left over, sequences that end inside a block of tokens, launches that carry a state on, rows on and off 16-byte borders (GPU)."""

import pytest
import torch

import helpers
from idempotent_llm_b200.cache import CacheNeed, SequenceCache
from idempotent_llm_b200.engine.batch import context_from_packed, pack_step_host

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    from idempotent_llm_b200.kernels import Kernels
    return Kernels(torch.float32, torch.device("cuda:0"))


def _randn(*shape, seed):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).cuda()


def _ctx(starts, lens):
    slots = list(range(len(lens)))
    packed, n, q_lens = pack_step_host(slots, starts, [[0] * L for L in lens])
    return context_from_packed(packed.cuda(), n, slots, q_lens, starts)


def _pieces(lens, cut):
    """Steps that bring each sequence at most ``cut`` tokens: (starts, counts) until all are through."""
    at = [0] * len(lens)
    while any(a < n for a, n in zip(at, lens)):
        counts = [min(cut, n - a) for a, n in zip(at, lens)]
        yield list(at), counts
        at = [a + c for a, c in zip(at, counts)]


def _step_rows(lens, starts, counts):
    """Rows of the step's tokens among all sequences' rows, one after another; sequences without a token left out."""
    first = [sum(lens[:i]) for i in range(len(lens))]
    keep = [i for i, c in enumerate(counts) if c]
    return keep, [first[i] + starts[i] + j for i in keep for j in range(counts[i])]


# ------------------------------------------------------------------------------------------------ short filters
@pytest.mark.parametrize("taps", [2, 4])
@pytest.mark.parametrize("lens,channels", [([1601], 1500), ([3, 1, 700, 9, 801, 2], 1700), ([8, 8, 1589], 1536)])
def test_short_conv_of_eight_tokens_a_thread(K, taps, lens, channels):
    """A prompt long enough for eight tokens a thread gives a token the bits that single tokens get."""
    n = sum(lens)
    proj = _randn(n, channels + 12, seed=1)
    w, b = _randn(channels, taps, seed=2), _randn(channels, seed=3)
    start = _randn(len(lens), (taps - 1) * channels, seed=4)
    starts = [5 * (i % 3) for i in range(len(lens))]               # (some sequences go on from a state, with fewer tokens than taps too)
    out = K.short_conv(proj, 7, channels, w, b, 1, start.clone(), _ctx(starts, lens))
    want, state = torch.empty_like(out), start.clone()
    for at, counts in _pieces([min(L, 12) for L in lens], 1):
        keep, rows = _step_rows(lens, at, counts)
        slots = keep
        packed, _, q_lens = pack_step_host(slots, [starts[i] + at[i] for i in keep], [[0]] * len(keep))
        ctx = context_from_packed(packed.cuda(), len(keep), slots, q_lens, [starts[i] + at[i] for i in keep])
        want[rows] = K.short_conv(proj[rows].contiguous(), 7, channels, w, b, 1, state, ctx)
    first = [sum(lens[:i]) for i in range(len(lens))]
    rows = [first[i] + j for i, L in enumerate(lens) for j in range(min(L, 12))]
    # (a single token moves its state on; one-token sequences of the long step did so as well)
    assert torch.equal(out[rows], want[rows])
    u = torch.zeros(n, channels, dtype=torch.float64, device="cuda")
    for j in range(taps):
        u[taps - 1:] += w[:, j].double() * proj[j:n - taps + 1 + j, 7:7 + channels].double()
    deep = [first[i] + j for i, L in enumerate(lens) for j in range(taps, L)]
    z = u[deep] + b.double()
    assert helpers.rel_err(out[deep], z * torch.sigmoid(z)) < 1e-5


@pytest.mark.parametrize("maps,dk,half", [(1, 128, 32), (2, 128, 16), (1, 24, 0), (1, 40, 20)])
def test_conv_qkv_of_eight_tokens_a_thread(K, maps, dk, half):
    """Enough tokens for eight a thread (a block of 256 threads for eight tokens and 256 items, 1 184 blocks at least): the bits
    that single tokens get, and the same sums in 64 bits."""
    lens, n_q, n_kv, dv, taps = [1300, 3, 1090], 6, 2, 72, 3
    n_q, n_kv = (n_q, n_kv) if dk == 128 else (20, 10)
    n, channels = sum(lens), (n_q + n_kv) * dk + n_kv * dv
    items = (n_q + n_kv) * (dk - maps * half) + n_kv * dv
    assert n // 8 * -(-items // 256) >= 1184
    proj, w = _randn(n, channels + 4, seed=5), _randn(channels, taps, seed=6)
    cs = _randn(n, half, 2, seed=7) if half else None
    start = _randn(len(lens), (taps - 1) * channels, seed=8)

    def fresh():
        cache = SequenceCache({0: CacheNeed("full", n_kv, dk, k_row=(n_kv, dk), v_row=(n_kv, dv))}, 64 * 48, torch.float32, "cuda:0",
                              max_seqs=3, max_seq_len=2048)
        cache.reserve([(cache.alloc_slot(), L) for L in lens]); cache.flush()
        return cache.view(0)
    kv = fresh()
    q = K.conv_qkv_cache(proj, 4, w, start.clone(), n_q, n_kv, dk, dv, cs, kv, _ctx([0] * 3, lens), maps=maps)
    other, state, one = fresh(), start.clone(), torch.empty_like(q)
    for at, counts in _pieces([min(L, 20) for L in lens], 1):
        keep, rows = _step_rows(lens, at, counts)
        packed, _, q_lens = pack_step_host(keep, [at[i] for i in keep], [[0]] * len(keep))
        ctx = context_from_packed(packed.cuda(), len(keep), keep, q_lens, [at[i] for i in keep])
        one[rows] = K.conv_qkv_cache(proj[rows].contiguous(), 4, w, state, n_q, n_kv, dk, dv, None if cs is None else cs[rows].contiguous(),
                                     other, ctx, maps=maps)
    first = [0, lens[0], lens[0] + lens[1]]
    for i, L in enumerate(lens):
        m = min(L, 20)
        assert torch.equal(q[first[i]:first[i] + m], one[first[i]:first[i] + m])
        page, page2 = int(kv.table[i, 0]), int(other.table[i, 0])
        assert torch.equal(kv.k[page][:, :m], other.k[page2][:, :m]) and torch.equal(kv.v[page][:, :m], other.v[page2][:, :m])
        # all tokens of the sequence: filtered, q and k turned in every part, a q row per part with zeros outside it
        x = proj[first[i]:first[i] + L, 4:].double()
        u = torch.zeros_like(x)
        for j in range(taps):
            back = taps - 1 - j
            u[back:] += w[:, j].double() * x[:max(L - back, 0)]
        turned = u[:, :(n_q + n_kv) * dk].reshape(L, n_q + n_kv, maps, dk // maps).clone()
        if half:
            c, sn = cs[first[i]:first[i] + L].double().permute(2, 0, 1)[:, :, None, None, :]
            a, b = turned[..., :half].clone(), turned[..., half:2 * half].clone()
            turned[..., :half], turned[..., half:2 * half] = a * c - b * sn, b * c + a * sn
        rows = torch.zeros(L, n_q, maps, maps, dk // maps, dtype=torch.float64, device="cuda")
        for z in range(maps):
            rows[:, :, z, z] = turned[:, :n_q, z]
        pages = kv.table[i, :-(-L // 64)].long()
        keys = kv.k[pages].transpose(1, 2).reshape(-1, n_kv, dk)[:L]
        values = kv.v[pages].transpose(1, 2).reshape(-1, n_kv, dv)[:L]
        assert helpers.rel_err(q[first[i]:first[i] + L].reshape(L, -1), rows.reshape(L, -1)) < 1e-6
        assert helpers.rel_err(keys.reshape(L, -1), turned[:, n_q:].reshape(L, -1)) < 1e-6
        assert helpers.rel_err(values.reshape(L, -1), u[:, (n_q + n_kv) * dk:]) < 1e-6


# rows of the turns' table that leave room for three rounds of eight tokens, for one, and for none (a token a block)
@pytest.mark.parametrize("dk,half", [(344, 170), (800, 400), (1284, 641)])
def test_conv_qkv_with_wide_turns(K, dk, half):
    test_conv_qkv_of_eight_tokens_a_thread(K, 1, dk, half)


# ------------------------------------------------------------------------------------------------ delta rule
def _delta_inputs(n, H, Hk, dk, dv, seed, pad=0):
    k = torch.nn.functional.normalize(_randn(n, Hk, dk, seed=seed), dim=-1)
    q = torch.nn.functional.normalize(_randn(n, Hk, dk, seed=seed + 1), dim=-1) * dk ** -0.5
    v = _randn(n, H * dv, seed=seed + 2)
    gap = torch.zeros(n, pad, device="cuda")
    c = torch.cat([gap, q.reshape(n, -1), k.reshape(n, -1), v], dim=1).contiguous()
    g = torch.exp(-3.0 * _randn(n, H * dk, seed=seed + 3).abs() ** 3)     # (some decays underflow within a chunk)
    g[_randn(n, H * dk, seed=seed + 4) > 1.5] = 1.0
    beta = torch.sigmoid(_randn(n, H, seed=seed + 5))
    return c, g.contiguous(), beta, (pad, pad + Hk * dk, pad + 2 * Hk * dk)


def _delta_64(c, cols, g, beta, S, H, Hk, dk, dv):
    """One sequence in 64 bits from S [H, dv, dk]; returns the read-outs and moves S on."""
    out = []
    for t in range(c.shape[0]):
        q, k = (c[t, a:a + Hk * dk].double().view(Hk, dk).repeat_interleave(H // Hk, dim=0) for a in cols[:2])
        v = c[t, cols[2]:].double().view(H, dv)
        S *= g[t].double().view(H, 1, dk)
        u = beta[t].double()[:, None] * (v - (S @ k[:, :, None])[:, :, 0])
        S += u[:, :, None] * k[:, None, :]
        out.append((S @ q[:, :, None])[:, :, 0].reshape(-1))
    return torch.stack(out)


# chunks of 32 with one token left over or missing, a half chunk and one more, keys below and at the kernels' sizes, columns that are no
# whole group of 16; enough sequences that a launch takes one chunk of each and the state carries over
@pytest.mark.parametrize("lens,H,Hk,dk,dv,pad", [
    ([5, 31, 32, 33], 4, 2, 128, 64, 0), ([16, 17, 65, 200], 2, 2, 64, 40, 4), ([100, 7], 3, 1, 20, 24, 0), ([97], 6, 3, 128, 16, 3),
    ([40, 33], 2, 1, 100, 72, 1), ([70] * 24, 64, 16, 128, 64, 0)])
def test_delta_chunks_against_64_bits(K, lens, H, Hk, dk, dv, pad):
    n = sum(lens)
    c, g, beta, cols = _delta_inputs(n, H, Hk, dk, dv, 20, pad)
    state = _randn(len(lens), H * dv * dk, seed=30)
    start = state.clone()
    o = K.delta_scan(c, *cols, g, 0, beta, state, _ctx([0] * len(lens), lens), H, Hk, dk, dv)
    at = 0
    for i, L in enumerate(lens[:4]):
        S = start[i].double().view(H, dv, dk).clone()
        want = _delta_64(c[at:at + L], cols, g[at:at + L], beta[at:at + L], S, H, Hk, dk, dv)
        # 32-bit sums of up to 128 products over a chain of up to 200 tokens whose state does not grow
        assert helpers.rel_err(o[at:at + L], want) < 2e-5 and helpers.rel_err(state[i].view(H, dv, dk), S) < 2e-5, f"sequence {i}"
        at += L
    # a later token that is not a number leaves the ones before it alone
    bad = c.clone()
    bad[lens[0] - 1] = float("nan")
    o2 = K.delta_scan(bad, *cols, g, 0, beta, start.clone(), _ctx([0] * len(lens), lens), H, Hk, dk, dv)
    assert torch.equal(o2[:lens[0] - 1], o[:lens[0] - 1])


# chunks of 32 split from the state (one sequence: 32 blocks) and the chain of chunks of 16 (six of them, 192 blocks): portions of one
# token more than the border between them, with and without a chunk's rest, keys at and below 128, keys that lie close together
@pytest.mark.parametrize("L,dk,dv,pad,close", [(129, 128, 64, 0, 0.0), (160, 100, 64, 1, 0.0), (201, 128, 64, 0, 0.1), (257, 72, 56, 4, 0.3)])
def test_delta_forms_in_64_bits_and_beside_one_another(K, L, dk, dv, pad, close):
    H, Hk, seqs = 8, 4, 6
    c, g, beta, cols = _delta_inputs(L, H, Hk, dk, dv, 60, pad)
    if close:
        k = torch.nn.functional.normalize(_randn(1, Hk, dk, seed=66) + close * _randn(L, Hk, dk, seed=67), dim=-1)
        c[:, cols[1]:cols[2]] = k.reshape(L, -1)
        g.fill_(0.9999); beta.fill_(0.98)
    start = _randn(1, H * dv * dk, seed=68)
    S = start[0].double().view(H, dv, dk).clone()
    want = _delta_64(c, cols, g, beta, S, H, Hk, dk, dv)
    one = start.clone()
    o = K.delta_scan(c, *cols, g, 0, beta, one, _ctx([0], [L]), H, Hk, dk, dv)
    many = start.repeat(seqs, 1)
    o6 = K.delta_scan(c.repeat(seqs, 1), *cols, g.repeat(seqs, 1), 0, beta.repeat(seqs, 1), many, _ctx([0] * seqs, [L] * seqs), H, Hk, dk, dv)
    assert all(torch.equal(o6[i * L:(i + 1) * L], o6[:L]) and torch.equal(many[i], many[0]) for i in range(seqs))
    assert not torch.equal(o, o6[:L])                              # (two orders of the same sums)
    for mine, other, ref in ((o, o6[:L], want), (one[0].view(H, dv, dk), many[0].view(H, dv, dk), S)):
        a, b = helpers.rel_err(mine, ref), helpers.rel_err(other, ref)
        assert a < 2e-5 and b < 2e-5 and a < 1.5 * b + 1e-7, (a, b)    # (simulated in 32 bits: 1.0 to 1.1 times, close keys among them)


# a decay per head: chunks of 32 with one token left over or missing, keys below 128, columns that are no whole group of 16, key heads of one to
# nine heads (a warp weighs a head: four at a time), sequences that share places of 32 tokens, keys that lie close together
@pytest.mark.parametrize("lens,H,Hk,dk,dv,close", [
    ([5, 31, 32, 33, 1, 49], 4, 2, 128, 64, 0.0), ([97, 64], 6, 3, 100, 40, 0.0), ([200], 9, 1, 68, 17, 0.0), ([161, 7], 8, 2, 128, 64, 0.1),
    ([257], 3, 3, 128, 16, 0.3)])
def test_delta_by_heads_against_64_bits(K, lens, H, Hk, dk, dv, close):
    n = sum(lens)
    c, _, beta, cols = _delta_inputs(n, H, Hk, dk, dv, 120)
    g = torch.exp(-3.0 * _randn(n, H, seed=125).abs() ** 3)        # (some underflow within a chunk)
    g[_randn(n, H, seed=126) > 1.5] = 1.0
    if close:
        c[:, cols[1]:cols[2]] = torch.nn.functional.normalize(_randn(1, Hk, dk, seed=127) + close * _randn(n, Hk, dk, seed=128), dim=-1).reshape(n, -1)
        g.fill_(0.9999); beta.fill_(0.98)
    c = torch.cat([c, torch.zeros(n, -c.shape[1] % 4, device="cuda")], dim=1).contiguous()    # (rows of whole pieces)
    wide = g.repeat_interleave(dk, dim=1).contiguous()
    start = _randn(len(lens), H * dv * dk, seed=130)

    def run(c, start, lens, g=g, beta=beta):
        ctx, state = _ctx([0] * len(lens), lens), start.clone()
        want = K.delta_by_heads(c, *cols[:2], ctx, H, Hk, dk, dv)
        assert want > 0
        return K.delta_heads(c, *cols, g.contiguous(), beta.contiguous(), state, ctx, H, Hk, dk, dv, want), state
    o, state = run(c, start, lens)
    other = start.clone()
    o2 = K.delta_scan(c, *cols, wide, 0, beta, other, _ctx([0] * len(lens), lens), H, Hk, dk, dv)
    at = 0
    for i, L in enumerate(lens):
        S, rows = start[i].double().view(H, dv, dk).clone(), slice(at, at + L)
        want = _delta_64(c[rows, :cols[2] + H * dv], cols, wide[rows], beta[rows], S, H, Hk, dk, dv)
        # 32-bit sums of up to 128 products over a chain whose state does not grow; no further off than the chain of decays per channel
        for mine, theirs, ref in ((o[rows], o2[rows], want), (state[i].view(H, dv, dk), other[i].view(H, dv, dk), S)):
            a, b = helpers.rel_err(mine, ref), helpers.rel_err(theirs, ref)
            assert a < 2e-5 and a < 1.5 * b + 1e-7, (i, a, b)
        alone = run(c[rows].contiguous(), start[i:i + 1], [L], g[rows], beta[rows]) if L > 48 else None
        assert alone is None or (torch.equal(alone[0], o[rows]) and torch.equal(alone[1][0], state[i]))
        at += L
    # a later token that is not a number leaves the ones before it alone, in the sequence before it in the step too; a value that is
    # infinite reaches its own column and goes on as a number, as sums of products make it
    bad, last = c.clone(), lens[0] - 1
    bad[last] = float("nan")
    o3, state3 = run(bad, start, lens)
    assert torch.equal(o3[:last], o[:last]) and torch.isnan(o3[last]).all() and torch.isnan(state3[0]).all()
    assert torch.equal(o3[lens[0]:], o[lens[0]:]) and torch.equal(state3[1:], state[1:])
    bad = c.clone()
    bad[last, cols[2]] = float("inf")                               # head 0, column 0 of its last token
    o4, state4 = run(bad, start, lens)
    keep = torch.ones(H * dv, dtype=torch.bool, device="cuda"); keep[0] = False
    assert torch.equal(o4[:last], o[:last]) and helpers.rel_err(o4[:, keep], o[:, keep].double()) < 1e-5
    assert torch.isinf(o4[last, 0]) and torch.isinf(state4[0].view(H, dv, dk)[0, 0]).all()


def test_delta_by_heads_lays_down_whole_groups_of_columns(K):
    """What the walk reads is all written: as many words of the scratch are touched with 17 columns as with 32 (groups of 16), with 40 as with 48."""
    H, Hk, dk, lens = 4, 2, 128, [65, 50]
    left = {}
    for dv in (17, 32, 40, 48):
        n = sum(lens)
        c, g, beta, cols = _delta_inputs(n, H, Hk, dk, dv, 130)
        g = g.view(n, H, dk)[:, :, 0].contiguous()
        state, ctx = torch.zeros(len(lens), H * dv * dk, device="cuda"), _ctx([0] * len(lens), lens)
        want = K.delta_by_heads(c, *cols[:2], ctx, H, Hk, dk, dv)
        scratch = torch.full((want,), 0x7FC12345, dtype=torch.int32, device="cuda")     # (a number that is not one)
        o = torch.empty(n, H * dv, device="cuda")
        rc = K.lib.idm_delta_heads(c.data_ptr(), c.shape[1], *cols, g.data_ptr(), beta.data_ptr(), state.data_ptr(), state.shape[1], o.data_ptr(),
                                   H * dv, ctx.cu_q.data_ptr(), ctx.slots.data_ptr(), ctx.n_seqs, n, H, Hk, dk, dv, max(lens), scratch.data_ptr(),
                                   torch.cuda.current_stream().cuda_stream)
        assert rc == 0 and torch.isfinite(o).all()
        left[dv] = int((scratch == 0x7FC12345).sum())
    assert left[17] == left[32] and left[40] == left[48], left


def test_delta_by_heads_through_a_window(K):
    """More chunks than the scratch holds: the bits that each sequence gets alone, and no more memory for a longer prompt."""
    H, Hk, dk, dv, lens = 64, 8, 128, 64, [700, 33, 900, 1, 50, 400]      # 70 places of 3.1 MB
    n = sum(lens)
    c, _, beta, cols = _delta_inputs(n, H, Hk, dk, dv, 140)
    g = torch.exp(-3.0 * _randn(n, H, seed=145).abs() ** 3)
    start = _randn(len(lens), H * dv * dk, seed=146)

    def run(rows, start, lens):
        ctx, state = _ctx([0] * len(lens), lens), start.clone()
        want = K.delta_by_heads(c, *cols[:2], ctx, H, Hk, dk, dv)
        assert 0 < want <= 32 << 20
        args = c[rows].contiguous(), g[rows].contiguous(), beta[rows].contiguous()
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        o = K.delta_heads(args[0], *cols, args[1], args[2], state, ctx, H, Hk, dk, dv, want)
        assert torch.cuda.max_memory_allocated() - before <= 4 * (o.numel() + (32 << 20)) + (2 << 20)
        return o, state
    o, state = run(slice(0, n), start, lens)
    at = 0
    for i, L in enumerate(lens):
        rows = slice(at, at + L)
        if L > 48:
            alone = run(rows, start[i:i + 1], [L])
            assert torch.equal(alone[0], o[rows]) and torch.equal(alone[1][0], state[i]), i
        if i in (0, 3):
            S = start[i].double().view(H, dv, dk).clone()
            want = _delta_64(c[rows], cols, g[rows].repeat_interleave(dk, dim=1), beta[rows], S, H, Hk, dk, dv)
            assert helpers.rel_err(o[rows], want) < 2e-5 and helpers.rel_err(state[i].view(H, dv, dk), S) < 2e-5, i
        at += L


def test_delta_scratch_is_for_the_tokens_that_are_there(K):
    """One portion among many single tokens, and many sequences of many heads: nothing is sized by the longest portion times all."""
    for lens, H in (([300] + [1] * 63, 32), ([40] * 64, 64)):
        n, Hk, dk, dv = sum(lens), 8, 128, 64
        c, g, beta, cols = _delta_inputs(n, H, Hk, dk, dv, 80)
        state, ctx = torch.zeros(len(lens), H * dv * dk, device="cuda"), _ctx([0] * len(lens), lens)
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        o = K.delta_scan(c, *cols, g, 0, beta, state, ctx, H, Hk, dk, dv)
        # the read-outs, and the chain's numbers: 32 floats a token and head
        assert torch.cuda.max_memory_allocated() - before < 4 * (o.numel() + 32 * n * H) + (2 << 20)


# the forms' border by the tokens of a sequence on average: 16 with 32 heads, 24 with 64
@pytest.mark.parametrize("lens,H,by_heads", [([300] + [1] * 63, 32, False), ([300] + [1] * 63, 64, False), ([2048] + [1] * 60, 32, True), ([2048] + [1] * 60, 64, True),
                                             ([241] + [1] * 15, 32, True), ([240] + [1] * 15, 32, False), ([369] + [1] * 15, 64, True),
                                             ([368] + [1] * 15, 64, False), ([48] * 8, 32, False), ([49] * 8, 64, True)])
def test_delta_form_of_a_portion_among_single_tokens(K, lens, H, by_heads):
    """A portion among many single tokens takes no chunk for each of those, in time or in memory."""
    Hk, dk, dv, n = 8, 128, 64, sum(lens)
    c, _, beta, cols = _delta_inputs(n, H, Hk, dk, dv, 150)
    ctx = _ctx([0] * len(lens), lens)
    assert (K.delta_by_heads(c, *cols[:2], ctx, H, Hk, dk, dv) > 0) == by_heads


@pytest.mark.parametrize("dk,dv,pad", [(128, 64, 0), (64, 40, 4), (24, 9, 0), (100, 64, 0), (30, 16, 0), (128, 64, 1), (160, 16, 0)])
def test_delta_single_tokens_against_64_bits_and_however_cut(K, dk, dv, pad):
    H, Hk, lens = 4, 2, [8, 3, 5]
    n = sum(lens)
    c, g, beta, cols = _delta_inputs(n, H, Hk, dk, dv, 40, pad)
    start = _randn(len(lens), H * dv * dk, seed=50)
    got = {}
    for cut in (1, 3, 4):
        state, o = start.clone(), torch.empty(n, H * dv, device="cuda")
        for at, counts in _pieces(lens, cut):
            keep, rows = _step_rows(lens, at, counts)
            packed, _, q_lens = pack_step_host(keep, [at[i] for i in keep], [[0] * counts[i] for i in keep])
            ctx = context_from_packed(packed.cuda(), len(rows), keep, q_lens, [at[i] for i in keep])
            o[rows] = K.delta_scan(c[rows].contiguous(), *cols, g[rows].contiguous(), 0, beta[rows].contiguous(), state, ctx, H, Hk, dk, dv)
        got[cut] = (o, state)
    for cut in (3, 4):
        assert torch.equal(got[cut][0], got[1][0]) and torch.equal(got[cut][1], got[1][1])
    at = 0
    for i, L in enumerate(lens):
        S = start[i].double().view(H, dv, dk).clone()
        want = _delta_64(c[at:at + L], cols, g[at:at + L], beta[at:at + L], S, H, Hk, dk, dv)
        assert helpers.rel_err(got[1][0][at:at + L], want) < 5e-6 and helpers.rel_err(got[1][1][i].view(H, dv, dk), S) < 5e-6
        at += L


def test_delta_single_tokens_are_the_same_bits_in_any_batch(K):
    """Enough sequences for eight columns a warp, and one alone (two columns)."""
    H, Hk, dk, dv, n = 16, 4, 128, 64, 20
    c, g, beta, cols = _delta_inputs(n, H, Hk, dk, dv, 55)
    start = _randn(n, H * dv * dk, seed=56)
    together = start.clone()
    o = K.delta_scan(c, *cols, g, 0, beta, together, _ctx([3] * n, [1] * n), H, Hk, dk, dv)
    for i in (0, 7, n - 1):
        state = start[i:i + 1].clone()
        one = K.delta_scan(c[i:i + 1].contiguous(), *cols, g[i:i + 1].contiguous(), 0, beta[i:i + 1].contiguous(), state, _ctx([3], [1]), H, Hk, dk, dv)
        assert torch.equal(one[0], o[i]) and torch.equal(state[0], together[i])


@pytest.mark.parametrize("head", [False, True])
def test_delta_prep_and_out_on_and_off_16_byte_borders(K, head):
    """Rows shifted by one column take the element by element kernels: the same numbers up to the order of a norm's sum."""
    n, H, Hk, dk, dv = 37, 6, 3, 64, 40
    qk, a, proj = _randn(n, 2 * Hk * dk, seed=60), _randn(n, H * dk, seed=61), _randn(n, 2 * H + 3, seed=62)
    dt, rate = _randn(H if head else H * dk, seed=63), _randn(H, seed=64)
    o, w, gate = _randn(n, H * dv, seed=65), _randn(dv, seed=66), _randn(n, H * dv, seed=67)
    got = []
    for shift in (0, 1):
        c = torch.cat([torch.zeros(n, 4 * shift + shift, device="cuda"), qk], dim=1).contiguous()
        dec = torch.cat([torch.zeros(n, shift, device="cuda"), a], dim=1).contiguous()
        beta = K.delta_prep(c, 5 * shift, 5 * shift + Hk * dk, dec, shift, proj, 0, dt, rate, H, Hk, dk, head_col=H if head else -1)
        gates = torch.cat([torch.zeros(n, shift, device="cuda"), gate], dim=1).contiguous()
        out = torch.zeros(n, H * dv + 4, device="cuda")
        K.delta_out(o, w, 1e-6, gates, shift, 0.7, out, 4 - shift, H, dv, gate_act=1)
        got.append((c[:, 5 * shift:], dec[:, shift:], beta, out[:, 4 - shift:4 - shift + H * dv]))
    for x, y in zip(*got):
        assert helpers.rel_err(x, y.double()) < 1e-6


# pairs of channels a thread (even columns) and one to four rounds of eight tokens: the bits of the kernels of one token a thread, which steps
# of few tokens take.  Ends of rounds and of sequences everywhere, sequences that go on from a state
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("lens,n_q,dk", [([1601, 7, 40], 20, 64), ([1300, 3, 9, 1, 1090], 12, 128), ([31, 33, 1, 2600], 20, 128)])
def test_filters_in_pairs_and_rounds(K, lens, n_q, dk, shift):
    n_kv, dv, half, taps = n_q // 2, 72, 16, 4
    n, channels, starts = sum(lens), (n_q + n_kv) * dk + n_kv * dv, [6 * (i % 2) for i in range(len(lens))]
    items = (n_q + n_kv) * (dk - half) + n_kv * dv
    assert n // 8 * -(-items // 256) >= 1184
    proj, w = _randn(n, channels + 2 + shift, seed=11), _randn(channels, taps, seed=12)
    cs, start = _randn(n, half, 2, seed=13), _randn(len(lens), (taps - 1) * channels, seed=14)
    got = []
    for cut in (1 << 30, 64):
        cache = SequenceCache({0: CacheNeed("full", n_kv, dk, k_row=(n_kv, dk), v_row=(n_kv, dv))}, 64 * 64, torch.float32, "cuda:0",
                              max_seqs=8, max_seq_len=4096)
        cache.reserve([(cache.alloc_slot(), s + L) for s, L in zip(starts, lens)]); cache.flush()
        kv = cache.view(0)
        kv.k.zero_(); kv.v.zero_()
        state, state2 = start.clone(), start.clone()
        q, y = torch.empty(n, n_q, dk, device="cuda"), torch.empty(n, channels, device="cuda")
        for at, counts in _pieces(lens, cut):
            keep, rows = _step_rows(lens, at, counts)
            packed, tokens, q_lens = pack_step_host(keep, [starts[i] + at[i] for i in keep], [[0] * counts[i] for i in keep])
            ctx = context_from_packed(packed.cuda(), tokens, keep, q_lens, [starts[i] + at[i] for i in keep])
            piece = proj[rows].contiguous()
            q[rows] = K.conv_qkv_cache(piece, 2 + shift, w, state, n_q, n_kv, dk, dv, cs[rows].contiguous(), kv, ctx)
            K.conv_state_update(piece, 2 + shift, channels, taps, state, ctx)
            y[rows] = K.short_conv(piece, 2 + shift, channels, w, None, 0, state2, ctx)
            K.conv_state_update(piece, 2 + shift, channels, taps, state2, ctx)
        table = [kv.table[i, :-(-(starts[i] + L) // 64)].long() for i, L in enumerate(lens)]
        got.append([q, y, state, state2] + [pool[t] for t in table for pool in (kv.k, kv.v)])
    for a, b in zip(*got):
        assert torch.equal(a, b)


# ------------------------------------------------------------------------------------------------ products over chunks
# chunks of 64 with one token left over, columns and dims that are no whole tiles, heads that share keys, blocks with several panels
@pytest.mark.parametrize("lens,heads,groups,P,N,shift", [
    ([129, 200, 3], 4, 2, 64, 128, 0), ([257], 6, 3, 40, 36, 0), ([130, 191], 3, 1, 72, 100, 0), ([193, 64], 2, 2, 20, 7, 1), ([150], 8, 1, 64, 200, 0)])
def test_state_space_chunks_against_the_walk(K, lens, heads, groups, P, N, shift):
    n, inner, gn = sum(lens), heads * P, groups * N
    xbc = torch.cat([torch.zeros(n, shift, device="cuda"), _randn(n, inner + 2 * gn, seed=70)], dim=1).contiguous()
    cols = (shift, shift + inner, shift + inner + gn)
    proj = _randn(n, inner + heads, seed=71)
    dt_bias, a_log, skip = _randn(heads, seed=72) - 2.0, _randn(heads, seed=73), _randn(heads, seed=74)
    start = _randn(len(lens), heads * N * P, seed=75)
    out = []
    for walk in (128, 1 << 30):
        K.SSD_WALK = walk
        state = start.clone()
        out.append((K.ssd_scan(xbc, cols, proj, 0, inner, dt_bias, a_log, skip, state, _ctx([0] * len(lens), lens), heads, groups, P, N), state))
    K.SSD_WALK = type(K).SSD_WALK
    # the same sums of up to N + 64 products per token in another order
    assert helpers.rel_err(out[0][0], out[1][0].double()) < 1e-5 and helpers.rel_err(out[0][1], out[1][1].double()) < 1e-5
    bad = xbc.clone()
    bad[lens[0] - 1] = float("nan")
    y = K.ssd_scan(bad, cols, proj, 0, inner, dt_bias, a_log, skip, start.clone(), _ctx([0] * len(lens), lens), heads, groups, P, N)
    assert torch.equal(y[:lens[0] - 1], out[0][0][:lens[0] - 1])       # (a later token leaves the ones before it alone)


@pytest.mark.parametrize("lens,H,dk,dv,shift", [([65, 128, 9], 2, 128, 256, 0), ([127], 3, 64, 72, 0), ([64, 1, 193], 2, 20, 36, 0), ([130], 1, 200, 40, 1)])
def test_retention_chunks_against_the_walk(K, lens, H, dk, dv, shift):
    n = sum(lens)
    proj = torch.cat([torch.zeros(n, shift, device="cuda"), _randn(n, 2 * H * dk + H * dv, seed=80)], dim=1).contiguous()
    cols = (shift, shift + H * dk, shift + 2 * H * dk)
    decay = torch.tensor([0.96875, 0.5, 0.9995][:H], device="cuda")
    start = _randn(len(lens), H * dk * dv, seed=81)
    out = []
    for walk in (8, 1 << 30):
        K.RETENTION_WALK = walk
        state = start.clone()
        out.append((K.retention(proj.clone(), cols, None, dk ** -0.5, decay, state, _ctx([0] * len(lens), lens), H, dk, dv), state))
    K.RETENTION_WALK = type(K).RETENTION_WALK
    assert helpers.rel_err(out[0][0], out[1][0].double()) < 1e-5 and helpers.rel_err(out[0][1], out[1][1].double()) < 1e-5


# what a chunk adds to the state, as products of parts: a value that has none (infinite, not a number, at the end of the range) moves the state as
# the walk of plain sums moves it, and leaves the other columns' bits alone; dims behind the first 128, columns that are no whole tile
@pytest.mark.parametrize("dk,dv", [(128, 256), (200, 40), (36, 70)])
def test_chunk_states_with_numbers_that_have_no_parts(K, dk, dv):
    H, L = 2, 150
    proj = _randn(L, 2 * H * dk + H * dv, seed=140)
    cols, decay = (0, H * dk, 2 * H * dk), torch.tensor([0.97, 0.5], device="cuda")
    start = _randn(1, H * dk * dv, seed=141)

    def run(proj, walk):
        K.RETENTION_WALK, state = walk, start.clone()
        o = K.retention(proj.clone(), cols, None, dk ** -0.5, decay, state, _ctx([0], [L]), H, dk, dv)
        K.RETENTION_WALK = type(K).RETENTION_WALK
        return o, state.view(H, dk, dv)
    clean = run(proj, 8)[1]
    bad = proj.clone()
    for t, j, x in ((5, 3, float("inf")), (70, 7, float("nan")), (149, dv + 1, -float("inf")), (148, 9, 3.4e38)):
        bad[t, cols[2] + j] = x
    got, want = run(bad, 8)[1], run(bad, 1 << 30)[1]
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
    keep = torch.ones(H, 1, dv, dtype=torch.bool, device="cuda")
    for j in (3, 7, 9): keep[0, 0, j] = False
    keep[1, 0, 1] = False
    assert torch.equal(got[keep.expand_as(got)], clean[keep.expand_as(got)])
    assert helpers.rel_err(got[0, :, 9] / 1e38, want[0, :, 9].double() / 1e38) < 1e-5


# a block of the read-outs takes one panel of 64 columns (in either kernel), two or all four of a group's, by how many chunks and heads a
# step has: a sequence's bits are the same beside any others (148 SMs: at most 296 blocks, at most 355, more)
@pytest.mark.parametrize("kind", ["retention", "state space"])
def test_chunks_give_the_same_bits_however_panels_are_dealt_out(K, kind):
    H, dk, dv, L = 8, 100, 256, 691                                # 11 chunks of 8 heads (groups): 88 x 4 panels
    first = None
    for others in ([], [64], [L], [L] * 2, [L] * 7, [200] * 3):
        lens = [L] + others
        n, ctx = sum(lens), _ctx([0] * len(lens), lens)
        state = torch.cat([_randn(1, H * dk * dv, seed=100), _randn(len(lens), H * dk * dv, seed=101)[1:]]).contiguous()
        if kind == "retention":
            proj = torch.cat([_randn(L, 2 * H * dk + H * dv, seed=102), _randn(n, 2 * H * dk + H * dv, seed=103)[L:]]).contiguous()
            decay = torch.tensor([0.96875, 0.5, 0.9995, 0.9, 0.99, 0.8, 0.999, 0.7], device="cuda")
            o = K.retention(proj, (0, H * dk, 2 * H * dk), None, dk ** -0.5, decay, state, ctx, H, dk, dv)
        else:
            heads, P = 4 * H, 64                                   # four heads a group
            width = heads * P + 2 * H * dk
            xbc = torch.cat([_randn(L, width, seed=104), _randn(n, width, seed=105)[L:]]).contiguous()
            proj = torch.cat([_randn(L, heads * P + heads, seed=106), _randn(n, heads * P + heads, seed=107)[L:]]).contiguous()
            o = K.ssd_scan(xbc, (0, heads * P, heads * P + H * dk), proj, 0, heads * P, _randn(heads, seed=108) - 2.0, _randn(heads, seed=109),
                           _randn(heads, seed=110), state, ctx, heads, H, P, dk)
        if first is None:
            first = (o[:L].clone(), state[0].clone())
        assert torch.equal(o[:L], first[0]) and torch.equal(state[0], first[1]), f"beside {others}"


def test_group_norm_and_gate_scale_on_and_off_16_byte_borders(K):
    n, parts, length = 21, 5, 132
    y, w = _randn(n, parts * length, seed=90), _randn(parts * length, seed=91)
    got = []
    for shift in (0, 1):
        out = torch.zeros(n, parts * length + 4, device="cuda")
        K.ssd_group_norm(y, parts, w, 1e-6, 0.5, out, shift)
        got.append(out[:, shift:shift + parts * length])
    assert helpers.rel_err(got[0], got[1].double()) < 1e-6


def test_a_plan_is_not_made_under_capture(K):
    """The lists of a step of long portions go up from host memory that does not outlive the call: a graph must not read them again."""
    from idempotent_llm_b200.kernels.ops import KernelError
    H, dk, dv, L = 2, 64, 64, 200
    proj, state, ctx = _randn(L, H * (2 * dk + dv), seed=120), torch.zeros(1, H * dk * dv, device="cuda"), _ctx([0], [L])
    decay = torch.tensor([0.5, 0.9], device="cuda")
    torch.cuda.synchronize()
    with pytest.raises(KernelError, match="capture"):
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            K.retention(proj, (0, H * dk, 2 * H * dk), None, dk ** -0.5, decay, state, ctx, H, dk, dv)
    o = K.retention(proj, (0, H * dk, 2 * H * dk), None, dk ** -0.5, decay, state, ctx, H, dk, dv)      # as before, not captured
    assert torch.isfinite(o).all()
