"""One-token batches: the units of the last round over the CTAs are cut into parts, and states in a pool have instances of their
own whose slots come through a table of 64 units per CTA.  A sequence has the same bits whatever round or part it falls into: batches
at the edges of rounds and parts against batches of one sequence at a time, which the oracle tests hold to the reference.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


def inputs(B, kh, vh, d, f32, slots, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    q, k, v = r(B, 1, kh, d).bfloat16(), r(B, 1, kh, d).bfloat16(), r(B, 1, vh, d).bfloat16()
    a, b = r(B, 1, vh).bfloat16(), r(B, 1, vh).bfloat16()
    par = (r(vh).bfloat16(), (0.1 * r(vh)).bfloat16())
    s = (0.02 * r(slots, vh, d, d)).bfloat16()
    return q, k, v, par, a, b, s.float() if f32 else s


def step(gdn, q, k, v, par, a, b, s, idx=None, inplace=False):
    return gdn.recurrent_forward(q, k, v, s, None, None, inference_mode=gdn.Decode, is_qk_norm=True, gating=(*par, a, b),
                                 inplace_state=inplace, state_indices=idx)


# 592 CTAs at 16-bit states and head dims up to 128 (444 at fp32, d=128): one part per tile, halves, whole, one unit more than a round, a
# round and quarters, halves or more of it, several rounds; head counts that are no power of two; d=192: tiles that halve but do not quarter
@pytest.mark.parametrize("kh,vh,d,f32,batches", [(16, 32, 128, False, (4, 5, 9, 10, 18, 19, 23, 28, 40, 80)), (2, 6, 128, False, (24, 25, 49, 50, 99, 124)),
                                                 (16, 32, 64, False, (9, 10, 19)), (16, 32, 128, True, (3, 4, 6, 7, 14, 17, 21, 28)),
                                                 (2, 6, 192, False, (16, 17, 24, 25, 49, 50))])
@pytest.mark.parametrize("pool", [False, True])
def test_rounds_and_parts(kh, vh, d, f32, batches, pool):
    import h100_gdn_cuda_b200 as gdn
    for B in batches:
        slots = B + 3 if pool else B
        q, k, v, par, a, b, s = inputs(B, kh, vh, d, f32, slots, B)
        idx = torch.randperm(slots, device="cuda", generator=torch.Generator(device="cuda").manual_seed(B))[:B].int() if pool else None
        if pool:
            idx[B // 2] = -1  # a padding sequence: its outputs are not written, no state moves
        o, s1 = step(gdn, q, k, v, par, a, b, s.clone(), idx)  # (a pool is updated where it lies either way)
        o2, s2 = step(gdn, q, k, v, par, a, b, s.clone(), idx, inplace=True)
        for i in sorted({0, 1, B // 2, B - 2, B - 1}):
            at = int(idx[i]) if pool else i
            if at < 0:
                continue
            sl = slice(i, i + 1)
            oi, si = step(gdn, q[sl], k[sl], v[sl], par, a[sl], b[sl], s[at:at + 1])
            assert torch.equal(o[i], oi[0]) and torch.equal(o2[i], oi[0]), (B, i)
            assert torch.equal(s2[at], si[0]) and torch.equal(s1[at], si[0]), (B, i)
        if pool:
            unused = torch.ones(slots, dtype=torch.bool)
            unused[idx[idx >= 0].long().cpu()] = False
            assert torch.equal(s2[unused.cuda()], s[unused.cuda()])


@pytest.mark.parametrize("B", [1184, 1200, 2400])
def test_more_units_than_one_table(B):
    """64 units per CTA and more (592 CTAs, 32 v-heads): the slots of the next 64 are read as the first of them begins"""
    import h100_gdn_cuda_b200 as gdn
    q, k, v, par, a, b, s = inputs(B, 1, 32, 64, False, B + 7, 5)
    idx = torch.randperm(B + 7, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))[:B].int()
    o, s1 = step(gdn, q, k, v, par, a, b, s.clone(), idx, inplace=True)
    o_ref, s_ref = step(gdn, q, k, v, par, a, b, s[idx.long()].contiguous())
    assert torch.equal(o, o_ref) and torch.equal(s1[idx.long()], s_ref)


@pytest.mark.parametrize("dv,vh,f32", [(8192, 1, False), (8224, 1, False), (8224, 2, True), (4096, 2, False)])
def test_more_parts_than_a_byte_counts(dv, vh, f32):
    """One sequence whose v-heads have more than 255 tiles of state rows (the C entry point has no upper limit on dv): every tile by itself, as
    many parts as tiles.  A row of the state needs nothing of the others, so the same rows as heads of 32 each are the reference."""
    import ctypes as C
    import h100_gdn_cuda_b200 as gdn
    from h100_gdn_cuda_b200 import _cabi as cabi, api
    d = 128
    q, k, _, par, a, b, _ = inputs(1, 1, vh, d, f32, 1, dv)
    g = torch.Generator(device="cuda").manual_seed(dv + 1)
    v = torch.randn(1, 1, vh, dv, device="cuda", generator=g).bfloat16()
    s = (0.02 * torch.randn(1, vh, dv, d, device="cuda", generator=g)).bfloat16()
    s = s.float() if f32 else s
    out, s_out = torch.full_like(v, float("nan")), torch.full_like(s, float("nan"))
    r = cabi.RecurrentArgs()
    r.shape = api._shape(1, 1, 1, 1, vh, d, dv)
    r.q, r.k, r.v, r.out = (api._token_tensor(t, False) for t in (q, k, v, out))
    r.gating_a, r.gating_b = api._token_scalar(a, False), api._token_scalar(b, False)
    r.A_log, r.dt_bias = par[0].data_ptr(), par[1].data_ptr()
    r.state_in, r.state_out = api._state_desc(s), api._state_desc(s_out)
    r.state_dtype = cabi.GDN_F32 if f32 else cabi.GDN_BF16
    r.scale, r.is_qk_norm = d ** -0.5, 1
    assert cabi.load().gdn_recurrent_forward(C.byref(r), torch.cuda.current_stream().cuda_stream) == 0, cabi.load().gdn_last_error()
    heads = dv // 32
    rep = lambda t: t.reshape(-1).repeat_interleave(heads)
    o_ref, s_ref = torch.empty(1, 1, vh * heads, 32, device="cuda", dtype=torch.bfloat16), torch.empty(1, vh * heads, 32, d, device="cuda", dtype=s.dtype)
    par2, a2, b2 = [rep(t) for t in par], rep(a).view(1, 1, -1), rep(b).view(1, 1, -1)
    r.shape = api._shape(1, 1, 1, 1, vh * heads, d, 32)
    r.v, r.out = api._token_tensor(v.view(1, 1, vh * heads, 32), False), api._token_tensor(o_ref, False)
    r.gating_a, r.gating_b = api._token_scalar(a2, False), api._token_scalar(b2, False)
    r.A_log, r.dt_bias = par2[0].data_ptr(), par2[1].data_ptr()
    r.state_in, r.state_out = api._state_desc(s.view(1, vh * heads, 32, d)), api._state_desc(s_ref)
    assert cabi.load().gdn_recurrent_forward(C.byref(r), torch.cuda.current_stream().cuda_stream) == 0, cabi.load().gdn_last_error()
    assert torch.isfinite(o_ref.float()).all()
    assert torch.equal(out.view(-1), o_ref.view(-1)) and torch.equal(s_out.view(-1), s_ref.view(-1))
