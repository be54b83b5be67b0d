"""Long runs of tokens through recurrent_forward (blocks of 16 tokens, the state in fp32 from the first token to the last)
against the fp32 oracle.  bf16 results are off by their rounding, 2^-9 relative per element at most; the rest are sums of at
most 256 products in fp32, 64 terms of 2^-17 in the worst direction: 2^-9 + 2^-11.  An fp32 state (token by token) has no rounding to bf16:
sums of 256 products rounded to 2^-24 each, added up over the tokens a state remembers, 2^-24 * 256 = 2^-16.
"""
import pytest
import torch

from oracle import gdn_oracle as O
from h100_gdn_cuda_b200 import synthetic

pytestmark = pytest.mark.gpu
REL, REL32 = 2.0 ** -9 + 2.0 ** -11, 2.0 ** -16


@pytest.fixture(scope="module")
def gdn():
    import h100_gdn_cuda_b200 as g
    from h100_gdn_cuda_b200 import build
    build.build()
    return g


def close(x, ref, tol, what):
    x = x.float().cpu()
    assert torch.isfinite(x).all(), what
    assert O.rel_fro(x, ref) <= tol, "%s: rel_fro %.3e" % (what, O.rel_fro(x, ref))


def inputs(B, T, kh, vh, d, norm, seed):
    p = synthetic.prefill_inputs(B, T, kh, vh, d, seed=seed, with_state=True, mild_gate=True, normalize=not norm)
    return p, {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in p.items()}


# around whole blocks, around the turn of the four preparing warps, one CTA and several waves of them
@pytest.mark.parametrize("B,T,kh,vh,d", [(1, 17, 1, 1, 64), (2, 31, 1, 2, 128), (1, 32, 2, 2, 192), (1, 33, 1, 1, 256), (3, 63, 1, 3, 64),
                                         (1, 64, 2, 4, 128), (1, 65, 1, 2, 256), (40, 47, 2, 8, 128), (24, 40, 2, 8, 64)])
@pytest.mark.parametrize("norm,f32,state", [(True, False, True), (False, True, True), (True, True, False)])
def test_padded(gdn, B, T, kh, vh, d, norm, f32, state):
    if f32 and d > 128:
        pytest.skip("fp32 states are built for dk 64 and 128")
    p, c = inputs(B, T, kh, vh, d, norm, 7 * T + d)
    s0 = (c["state"].float() if f32 else c["state"]) if state else None
    if f32 and not state:
        s0 = torch.zeros_like(c["state"], dtype=torch.float32)
    o, s = gdn.recurrent_forward(c["q"], c["k"], c["v"], s0, c["beta"], c["g"], inference_mode=gdn.Decode, is_qk_norm=norm)
    o_ref, s_ref = O.recurrent_ref(p["q"].float(), p["k"].float(), p["v"].float(), p["beta"].float(), p["g"],
                                   p["state"].float() if state else None, is_qk_norm=norm)
    assert s.dtype == (torch.float32 if f32 else torch.bfloat16)
    close(o, o_ref, REL, "O")
    close(s, s_ref, REL32 if f32 else REL, "state")


def test_caps_pool_and_gating(gdn):
    """sequences that end inside a block, before the first token and at the last one, their states in a pool with a padding
    sequence, beta and the gate made inside"""
    B, T, kh, vh, d = 6, 50, 1, 2, 128
    p, c = inputs(B, T, kh, vh, d, True, 3)
    gen = torch.Generator().manual_seed(4)
    A_log, dt_bias = torch.rand(vh, generator=gen).bfloat16(), torch.randn(vh, generator=gen).bfloat16()
    a, b = torch.randn(B, T, vh, generator=gen).bfloat16(), torch.randn(B, T, vh, generator=gen).bfloat16()
    nat = torch.tensor([50, 0, 17, 33, 48, 1], dtype=torch.int32)
    slots = torch.tensor([4, 0, 6, -1, 2, 1], dtype=torch.int32)
    pool = (torch.randn(8, vh, d, d, generator=gen) * 0.02).bfloat16()
    beta, g = O.gating_ref(A_log, dt_bias, a, b)
    got = pool.cuda()
    o, _ = gdn.recurrent_forward(c["q"], c["k"], c["v"], got, None, None, None, nat.cuda(), gdn.Decode, True,
                                 gating=(A_log.cuda(), dt_bias.cuda(), a.cuda(), b.cuda()), state_indices=slots.cuda())
    want = pool.clone()
    for i in range(B):
        n, sl = int(nat[i]), int(slots[i])
        if sl < 0:
            continue
        if n:
            o_ref, s_ref = O.recurrent_ref(p["q"][i:i + 1, :n].float(), p["k"][i:i + 1, :n].float(), p["v"][i:i + 1, :n].float(),
                                           beta[i:i + 1, :n].float(), g[i:i + 1, :n], pool[sl:sl + 1].float(), is_qk_norm=True)
            close(o[i:i + 1, :n], o_ref, REL, "O of sequence %d" % i)
            want[sl] = s_ref[0].bfloat16()
    close(got, want.float(), REL, "pool")
    for sl in (0, 3, 5, 7):
        assert torch.equal(got[sl].cpu(), pool[sl])


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("what", ["v", "k", "state"])
def test_undefined_values_stay_behind_their_token(gdn, what, bad):
    B, T, kh, vh, d, at = 1, 60, 1, 1, 128, 21
    p, c = inputs(B, T, kh, vh, d, False, 5)
    run = lambda: gdn.recurrent_forward(c["q"], c["k"], c["v"], c["state"], c["beta"], c["g"], inference_mode=gdn.Decode)
    o0, s0 = run()
    if what == "state":  # one row of the state: the others are untouched
        c["state"] = c["state"].clone()
        c["state"][0, 0, 5, 7] = bad
        o1, s1 = run()
        rows = [r for r in range(d) if r != 5]
        assert torch.equal(o0[..., rows], o1[..., rows]) and torch.equal(s0[:, :, rows], s1[:, :, rows])
        assert not torch.isfinite(s1[0, 0, 5]).any() and not torch.isfinite(o1[0, :, 0, 5]).any()
    else:
        c[what] = c[what].clone()
        c[what][0, at, 0, 9] = bad
        o1, s1 = run()
        assert torch.equal(o0[:, :at], o1[:, :at])
        if what == "v":
            rows = [r for r in range(d) if r != 9]
            assert torch.equal(o0[..., rows], o1[..., rows]) and torch.equal(s0[:, :, rows], s1[:, :, rows])
            assert not torch.isfinite(o1[0, at:, 0, 9]).any()
        else:
            assert not torch.isfinite(o1[:, at:]).any()


def unit(x):
    return torch.nn.functional.normalize(x, dim=-1).bfloat16()


def flat_inputs(n, kh, vh, d, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    return unit(r(n, kh, d)), unit(r(n, kh, d)), r(n, vh, d).bfloat16(), torch.sigmoid(r(n, vh)).bfloat16(), -torch.nn.functional.softplus(r(n, vh))


# on both sides of the line between the token recurrence and the blocks of every head dim and state type
@pytest.mark.parametrize("d,f32,T", [(64, False, 31), (64, False, 40), (64, False, 41), (64, True, 40), (64, True, 41), (128, False, 17), (128, False, 24),
                                     (128, False, 25), (128, True, 24), (128, True, 25), (192, False, 26), (192, False, 27), (256, False, 22), (256, False, 23)])
def test_bits_do_not_depend_on_company(gdn, d, f32, T):
    """a sequence alone, in a batch that fills the GPU and packed, and a shard of its heads: the same bits"""
    B, kh, vh = 40, 4, 8
    x = [t.view(B, T, *t.shape[1:]) for t in flat_inputs(B * T, kh, vh, d, d + T)]
    s0 = (torch.randn(B, vh, d, d, device="cuda") * 0.02).to(torch.float32 if f32 else torch.bfloat16)
    run = lambda x, s, **kw: gdn.recurrent_forward(*x[:3], s, *x[3:], inference_mode=gdn.Decode, **kw)
    o, s = run(x, s0)
    for i in (0, 39):
        oi, si = run([t[i:i + 1] for t in x], s0[i:i + 1])
        assert torch.equal(oi, o[i:i + 1]) and torch.equal(si, s[i:i + 1])
    heads = [t[:, :, :1] for t in x[:2]] + [t[:, :, :2] for t in x[2:]]
    oh, sh = run(heads, s0[:, :2].contiguous())
    assert torch.equal(oh, o[:, :, :2]) and torch.equal(sh, s[:, :2])
    cu = torch.arange(0, B * T + 1, T, dtype=torch.int32, device="cuda")
    op, sp = run([t.flatten(0, 1) for t in x], s0, cu_seqlens=cu)
    assert torch.equal(op.view_as(o), o) and torch.equal(sp, s)


@pytest.mark.parametrize("chunked", [False, True])
@pytest.mark.parametrize("d", [64, 128, 192, 256])
@pytest.mark.parametrize("lens", [[300] + [1] * 99 + [22, 41, 0, 25, 27, 60, 17], [0] * 70 + [40, 0, 41, 26, 200], [23, 24, 45, 1000, 64, 41],
                                  [45 + i % 4 if i % 5 == 0 or i > 190 else 1 for i in range(200)], [70 + i % 3 for i in range(50)]])
def test_packed_runs_of_unequal_length(gdn, lens, d, chunked):
    """few long sequences among many short ones, among empty ones, none but long ones, more of either than CTAs: the bits each has alone"""
    if chunked and d <= 128:
        pytest.skip("head dims up to 128 have kernels of their own in chunked_forward")
    kh, vh = 2, 4
    x = flat_inputs(sum(lens), kh, vh, d, d)
    s0 = (torch.randn(len(lens), vh, d, d, device="cuda") * 0.02).bfloat16()
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    i32 = lambda t: torch.tensor(t, dtype=torch.int32, device="cuda")
    if chunked:
        run = lambda x, s, *meta: gdn.chunked_forward(*x, None, s, *meta)
        o, s = run(x, s0, i32(cu), i32(synthetic.prepare_chunk_indices(cu)), i32(synthetic.prepare_cu_chunks(cu)))
    else:
        run = lambda x, s, **kw: gdn.recurrent_forward(*x[:3], s, *x[3:], inference_mode=gdn.Decode, **kw)
        o, s = run(x, s0, cu_seqlens=i32(cu))
    for i, n in enumerate(lens):
        if not n:
            assert torch.equal(s[i], s0[i])
        elif n > 8 or i in (1, 50, 99):
            sl = slice(cu[i], cu[i + 1])
            oi, si = run([t[None, sl] for t in x], s0[i:i + 1])
            assert torch.equal(oi[0], o[sl]) and torch.equal(si[0], s[i]), n


# The token recurrence for runs of more than 16 tokens and the blocks, each next to the line between them, on more CTAs than the GPU
# holds at a time
LINES = [(64, False, 17), (64, False, 40), (64, False, 41), (64, True, 40), (64, True, 41), (128, False, 17), (128, False, 24), (128, False, 25),
         (128, True, 22), (128, True, 24), (128, True, 25), (192, False, 20), (192, False, 26), (192, False, 27), (256, False, 20), (256, False, 22), (256, False, 23)]


@pytest.mark.parametrize("d,vh", [(192, 7), (256, 6)])
@pytest.mark.parametrize("lens", [[27, 27], [33, 33], [95, 95], [28, 96], [1200] + [1] * 30 + [27], [33] + [1] * 30, [40] * 20 + [1] * 200])
def test_two_groups_of_rows(gdn, d, vh, lens):
    """Batches with more tiles of 16 rows than SMs whose CTAs own 32 rows (padded, packed, and walked, in the last one several units per CTA): the
    bits of every sequence alone, where they own 16."""
    B, N = len(lens), sum(lens)
    walked = N // {192: 27, 256: 23}[d] < B and len(set(lens)) > 1  # fewer sequences can be long than there are
    tiles = (N // {192: 27, 256: 23}[d] if walked else B) * vh * (d // 16)
    one = 4.3 * (tiles // 296) + (0 if tiles % 296 == 0 else 2.8 if tiles % 296 <= 148 else 4.3)
    assert 4.1 * -(-tiles // 296) < one and walked == (lens[-1] == 1)  # (block_groups)
    p = synthetic.varlen_inputs(lens, 1, vh, d, seed=d + N, mild_gate=True)
    c = {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in p.items()}
    run = lambda sl, state, cu: gdn.recurrent_forward(c["q"][sl], c["k"][sl], c["v"][sl], state, c["beta"][sl], c["g"][sl], cu,
                                                      inference_mode=gdn.Decode, is_qk_norm=True)
    if lens == [lens[0]] * B:
        x = lambda k: c[k].view(B, lens[0], *c[k].shape[1:])
        o, s = gdn.recurrent_forward(x("q"), x("k"), x("v"), c["state"], x("beta"), x("g"), inference_mode=gdn.Decode, is_qk_norm=True)
        o = o.view(N, vh, d)
    else:
        o, s = run(slice(None), c["state"], c["cu_seqlens"])
    at = 0
    for i, n in enumerate(lens):
        if n > 1:
            sl = slice(at, at + n)
            oi, si = run(sl, c["state"][i:i + 1], torch.tensor([0, n], dtype=torch.int32, device="cuda"))
            assert torch.equal(o[sl], oi) and torch.equal(s[i], si[0])
        at += n


@pytest.mark.parametrize("d,vh", [(192, 12), (256, 9)])
def test_two_groups_repeat_bit_for_bit(gdn, d, vh):
    """The groups of a CTA run apart by up to a block, differently each time: what one of them writes may not lie where the other still
    reads."""
    p, c = inputs(2, 600, vh, vh, d, False, d)
    run = lambda: gdn.recurrent_forward(c["q"], c["k"], c["v"], c["state"], c["beta"], c["g"], inference_mode=gdn.Decode, is_qk_norm=False)
    o, s = run()
    for _ in range(40):
        oi, si = run()
        assert torch.equal(o, oi) and torch.equal(s, si)


@pytest.mark.parametrize("d,f32,T", LINES)
def test_either_side_of_the_line(gdn, d, f32, T):
    norm = T % 2 == 0
    p, c = inputs(40, T, 4, 8, d, norm, d + T)
    s0 = p["state"].float() + (1e-4 * torch.randn(p["state"].shape, generator=torch.Generator().manual_seed(1)) if f32 else 0.0)
    o, s = gdn.recurrent_forward(c["q"], c["k"], c["v"], s0.cuda() if f32 else c["state"], c["beta"], c["g"], inference_mode=gdn.Decode,
                                 is_qk_norm=norm)
    o_ref, s_ref = O.recurrent_ref(p["q"].float(), p["k"].float(), p["v"].float(), p["beta"].float(), p["g"], s0, is_qk_norm=norm)
    close(o, o_ref, REL, "O")
    close(s, s_ref, REL32 if f32 else REL, "state")


@pytest.mark.parametrize("d,f32,T", [l for l in LINES if l[2] > 17])
def test_caps_pool_and_gating_either_side(gdn, d, f32, T):
    """accepted-token caps, states in a pool with padding sequences, beta and the gate made inside"""
    B, kh, vh = 24, 2, 4
    gen = torch.Generator().manual_seed(d + T)
    p, c = inputs(B, T, kh, vh, d, True, T)
    A_log, dt_bias = torch.rand(vh, generator=gen).bfloat16(), torch.randn(vh, generator=gen).bfloat16()
    a, b = torch.randn(B, T, vh, generator=gen).bfloat16(), torch.randn(B, T, vh, generator=gen).bfloat16()
    nat = torch.randint(0, T + 1, (B,), generator=gen, dtype=torch.int32)
    nat[0], nat[1], nat[2] = T, 0, 1
    slots = torch.randperm(B + 6, generator=gen)[:B].int()
    slots[5] = slots[17] = -1
    pool = torch.randn(B + 6, vh, d, d, generator=gen) * 0.02
    pool = pool if f32 else pool.bfloat16()
    beta, g = O.gating_ref(A_log, dt_bias, a, b)
    got = pool.cuda()
    o, _ = gdn.recurrent_forward(c["q"], c["k"], c["v"], got, None, None, None, nat.cuda(), gdn.Decode, True,
                                 gating=(A_log.cuda(), dt_bias.cuda(), a.cuda(), b.cuda()), state_indices=slots.cuda())
    live = (slots >= 0).nonzero().flatten()
    at = slots[live].long()
    o_ref, s_ref = O.recurrent_ref(p["q"][live].float(), p["k"][live].float(), p["v"][live].float(), beta[live].float(), g[live], pool[at].float(),
                                   is_qk_norm=True, num_accepted_tokens=nat[live])
    rows = torch.arange(T)[None] < nat[live][:, None]
    close(o.cpu()[live][rows], o_ref[rows], REL, "O")
    # (the fast exponential and logarithm of the gating inside are a few units of 2^-22 off, which T tokens add up)
    close(got[at], s_ref, REL32 + T * 2.0 ** -20 if f32 else REL, "pool")
    rest = [i for i in range(B + 6) if i not in at.tolist()]
    assert torch.equal(got[rest].cpu(), pool[rest])


@pytest.mark.parametrize("d,f32", [(64, False), (64, True), (128, False), (128, True), (192, False), (256, False)])
def test_packed_about_the_line(gdn, d, f32):
    """packed runs of 0 to 44 tokens, 20 on average: sequences of either kernel, in every order"""
    gen = torch.Generator().manual_seed(d)
    lens = torch.randint(0, 45, (60,), generator=gen).tolist() + [16, 17, 22, 23, 24, 25, 26, 27, 40, 41] + [1] * 10
    p = synthetic.varlen_inputs(lens, 2, 4, d, seed=d, mild_gate=True)
    c = {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in p.items()}
    s0 = c["state"].float() if f32 else c["state"]
    o, s = gdn.recurrent_forward(c["q"], c["k"], c["v"], s0, c["beta"], c["g"], cu_seqlens=c["cu_seqlens"], inference_mode=gdn.Decode)
    o_ref, s_ref = O.recurrent_ref(p["q"].float(), p["k"].float(), p["v"].float(), p["beta"].float(), p["g"], p["state"].float(),
                                   cu_seqlens=p["cu_seqlens"])
    close(o, o_ref, REL, "O")
    close(s, s_ref, REL32 if f32 else REL, "states")


@pytest.mark.parametrize("d", [64, 128])
def test_fp32_state_is_the_token_recurrences(gdn, d):
    """The matrix instructions cut their sums off, which an fp32 state would show: it is advanced token by token whatever the run's
    length, with the bits of the last one where a state per token is kept."""
    B, T, kh, vh = 2, 100, 2, 4
    x = [t.view(B, T, *t.shape[1:]) for t in flat_inputs(B * T, kh, vh, d, d)]
    s0 = torch.randn(B, vh, d, d, device="cuda") * 0.02
    o, s = gdn.recurrent_forward(*x[:3], s0, *x[3:], inference_mode=gdn.Decode)
    o1, steps = gdn.recurrent_forward(*x[:3], s0, *x[3:], inference_mode=gdn.SpecVerify)
    assert torch.equal(o, o1) and torch.equal(s, steps[:, -1])
