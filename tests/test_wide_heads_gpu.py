"""chunked_forward for head dims 129 .. 256, which keep the state and every intermediate in fp32.  The error against the
fp32 oracle is that of rounding the results: at most 2^-9 relative per element, hence at most 2^-9 = 1.95e-3 in the
relative Frobenius norm; the tolerance adds 64 terms of 2^-17 in the worst direction (0.5e-3).
"""
import pytest
import torch

from oracle import gdn_oracle as O
from h100_gdn_cuda_b200 import synthetic

pytestmark = pytest.mark.gpu
REL = 2.0 ** -9 + 64 * 2.0 ** -17


@pytest.fixture(scope="module")
def gdn():
    import h100_gdn_cuda_b200 as g
    from h100_gdn_cuda_b200 import build
    build.build()
    return g


def dev(d):
    return {k: (v.cuda() if torch.is_tensor(v) else v) for k, v in d.items()}


def close(x, ref, what):
    x = x.float().cpu()
    assert torch.isfinite(x).all(), what
    assert O.rel_fro(x, ref) <= REL, "%s: rel_fro %.3e" % (what, O.rel_fro(x, ref))


@pytest.mark.parametrize("B,T,kh,vh,d,norm,state", [
    (1, 1, 1, 1, 256, False, True), (1, 64, 1, 2, 256, False, False), (2, 65, 1, 1, 136, False, True),
    (1, 300, 2, 6, 192, True, True), (2, 130, 2, 2, 200, True, False), (1, 128, 1, 3, 250, False, True),
    (1, 1500, 2, 4, 256, False, True),
])
@pytest.mark.parametrize("mild", [False, True])
def test_padded(gdn, B, T, kh, vh, d, norm, state, mild):
    p = synthetic.prefill_inputs(B, T, kh, vh, d, seed=T + d, with_state=state, mild_gate=mild, normalize=not norm)
    o_ref, s_ref = O.recurrent_ref(p["q"].float(), p["k"].float(), p["v"].float(), p["beta"].float(), p["g"],
                                   p["state"].float() if state else None, is_qk_norm=norm)
    pd = dev(p)
    o, s = gdn.chunked_forward(pd["q"], pd["k"], pd["v"], pd["beta"], pd["g"], None, pd["state"], is_qk_norm=norm)
    assert o.shape == p["v"].shape and s.shape == (B, vh, d, d)
    close(o, o_ref, "O")
    close(s, s_ref, "final state")


@pytest.mark.parametrize("lens,kh,vh,d,norm", [([65, 1, 130, 0, 64], 2, 4, 256, False), ([70, 3], 1, 2, 192, True),
                                               ([1 + (37 * i) % 90 for i in range(40)] + [0], 1, 2, 256, False)])
def test_packed(gdn, lens, kh, vh, d, norm):
    """ragged tails next to other sequences, empty sequences, and more CTAs than SMs (longest sequences first)"""
    p = synthetic.varlen_inputs(lens, kh, vh, d, seed=sum(lens), mild_gate=True, normalize=not norm)
    o_ref, s_ref = O.recurrent_ref(p["q"].float(), p["k"].float(), p["v"].float(), p["beta"].float(), p["g"],
                                   p["state"].float(), cu_seqlens=p["cu_seqlens"], is_qk_norm=norm)
    pd = dev(p)
    o, s = gdn.chunked_forward(pd["q"], pd["k"], pd["v"], pd["beta"], pd["g"], None, pd["state"], pd["cu_seqlens"],
                               pd["chunk_indices"], pd["cu_chunks"], p["total_chunks"], is_qk_norm=norm)
    close(o, o_ref, "O")
    close(s, s_ref, "final states")
    for i, n in enumerate(lens):
        if n == 0:
            assert torch.equal(s[i], pd["state"][i])


@pytest.mark.parametrize("B,T,kh,vh,d,norm,gate", [(2, 233, 4, 8, 200, False, True), (1, 1500, 2, 4, 256, True, False),
                                                   (1, 6000, 1, 2, 256, False, False)])
def test_intermediates_keep_32_bits(gdn, B, T, kh, vh, d, norm, gate):
    """Against the recurrence in 64 bits: how many of the bf16 results are not the 64-bit value rounded to bf16.  A result
    with a relative error e before rounding goes to the wrong neighbour with a probability of at most e / 2^-8 (the
    spacing of bf16 numbers is 2^-8 to 2^-7 of their value).  Sums of 256 products in fp32, each rounded to 2^-24, are off
    by some sqrt(256) 2^-24 = 2^-20: at most 2^-12 of the results where a strong gate keeps only the last few tokens.  Without one
    the state adds up the errors of some thousand tokens that overwrite one another: 2^-18 and 2^-10, and twice that for the
    small results, whose relative error is larger.  (Operands of 16 significand bits instead of 24 gave 4e-3 to 6e-3 without
    a gate and 1e-3 with one; fp32 gives 3e-4 to 6e-4 and 5e-5.)"""
    gen = torch.Generator(device="cuda").manual_seed(T + d)
    r = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    q, k = r(B, T, kh, d), r(B, T, kh, d)
    if not norm:
        q, k = (torch.nn.functional.normalize(x, dim=-1) for x in (q, k))
    q, k, v, beta = q.bfloat16(), k.bfloat16(), r(B, T, vh, d).bfloat16(), torch.sigmoid(r(B, T, vh)).bfloat16()
    g = -torch.nn.functional.softplus(r(B, T, vh)) * 8 if gate else torch.zeros(B, T, vh, device="cuda")
    s0 = (r(B, vh, d, d) * 0.02).bfloat16()
    o, s = gdn.chunked_forward(q, k, v, beta, g, None, s0, is_qk_norm=norm)
    q, k = (x.double() * (torch.rsqrt(x.double().square().sum(-1, keepdim=True) + 1e-6) if norm else 1.0) for x in (q, k))
    q, k = (x.repeat_interleave(vh // kh, 2).unsqueeze(-1) for x in (q, k))
    S, a, b, v = s0.double(), g.double().exp()[..., None, None], beta.double()[..., None, None], v.double().unsqueeze(-1)
    wrong = 0
    for t in range(T):
        S = S * a[:, t]
        S = S + b[:, t] * (v[:, t] - S @ k[:, t]) @ k[:, t].mT
        wrong += ((S @ q[:, t])[..., 0] * d ** -0.5).bfloat16().ne(o[:, t]).sum()
    bound = 2.0 ** -12 if gate else 2.0 ** -9
    assert wrong.item() <= bound * o.numel()
    assert S.bfloat16().ne(s).sum().item() <= bound * s.numel()
