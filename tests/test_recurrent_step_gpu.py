"""Short padded runs (2 .. 8 tokens per sequence) of recurrent_forward on bf16 states: the kernel on warp matrix
instructions.  Its products are exact bf16 products accumulated in fp32 and its coefficients keep 24 bits, so against the
fp32 oracle only the rounding of the bf16 results shows: 2^-9 of every element at most, plus 2^-14 for fp32 sums of 128
terms and the fast exponentials.
"""
import pytest
import torch

from oracle import gdn_oracle as O
from h100_gdn_cuda_b200 import synthetic

pytestmark = pytest.mark.gpu
REL = 2.0 ** -9 + 2.0 ** -14


@pytest.fixture(scope="module")
def gdn():
    import h100_gdn_cuda_b200 as g
    from h100_gdn_cuda_b200 import build
    build.build()
    return g


def close(x, ref, what):
    x = x.float().cpu()
    assert torch.isfinite(x).all(), what
    assert O.rel_fro(x, ref) <= REL, "%s: rel_fro %.3e" % (what, O.rel_fro(x, ref))


def problem(B, T, kh, vh, d, seed):
    p = synthetic.decode_inputs(B, T, kh, vh, d, seed=seed)
    beta, g = O.gating_ref(*(p[n].float() for n in ("A_log", "dt_bias", "a", "b")))
    return p, {k: v.cuda() for k, v in p.items()}, beta, g


@pytest.mark.parametrize("B,T,kh,vh,d", [
    (1, 2, 1, 1, 64), (1, 8, 1, 1, 128),      # one unit: most warps have nothing to do
    (3, 7, 2, 6, 128), (2, 3, 3, 3, 64),      # head counts that are no power of two
    (40, 4, 16, 32, 128),                     # one round of whole units and a rest cut across units (1184 warps)
    (37, 5, 16, 32, 64), (75, 2, 8, 32, 128),
])
@pytest.mark.parametrize("norm", [False, True])
def test_against_the_recurrence(gdn, B, T, kh, vh, d, norm):
    p, pd, beta, g = problem(B, T, kh, vh, d, seed=B * 10 + T)
    g[:, T // 2] = -30.0  # a gate that wipes the state out in the middle of the run
    bb = beta.bfloat16()
    q, k = (x if norm else torch.nn.functional.normalize(x.float(), dim=-1).bfloat16() for x in (p["q"], p["k"]))
    ref = dict(is_qk_norm=norm, store_step_state=True)
    o_ref, st_ref = O.recurrent_ref(q.float(), k.float(), p["v"].float(), bb.float(), g, p["state"].float(), **ref)
    args = (q.cuda(), k.cuda(), pd["v"], pd["state"], bb.cuda(), g.cuda())
    o, steps = gdn.recurrent_forward(*args, inference_mode=gdn.SpecVerify, is_qk_norm=norm)
    close(o, o_ref, "o")
    close(steps, st_ref, "step states")
    o1, s1 = gdn.recurrent_forward(*args, inference_mode=gdn.Decode, is_qk_norm=norm)
    assert torch.equal(o1, o) and torch.equal(s1, steps[:, -1])
    s_in = pd["state"].clone()
    o2, s2 = gdn.recurrent_forward(*args[:3], s_in, *args[4:], inference_mode=gdn.Decode, is_qk_norm=norm, inplace_state=True)
    assert s2.data_ptr() == s_in.data_ptr() and torch.equal(s2, s1) and torch.equal(o2, o)


@pytest.mark.parametrize("d", [64, 128])
def test_caps_pool_and_gating(gdn, d):
    """accepted-token caps down to zero, a state pool with a padding sequence, beta and the gate computed inside"""
    B, T, kh, vh = 6, 6, 2, 4
    p, pd, beta, g = problem(B, T, kh, vh, d, seed=d)
    acc = torch.tensor([0, 6, 1, 3, 5, 2], dtype=torch.int32)
    slots = torch.tensor([7, 2, -1, 0, 5, 3], dtype=torch.int32)
    pool = (torch.randn(9, vh, d, d, generator=torch.Generator().manual_seed(1)) * 0.02).bfloat16()
    _, st_ref = O.recurrent_ref(p["q"].float(), p["k"].float(), p["v"].float(), beta, g, pool[slots.clamp(min=0).long()].float(),
                                is_qk_norm=True, store_step_state=True)
    pc = pool.cuda()
    gdn.recurrent_forward(pd["q"], pd["k"], pd["v"], pc, None, None, None, acc.cuda(), gdn.Decode, True,
                          gating=(pd["A_log"], pd["dt_bias"], pd["a"], pd["b"]), state_indices=slots.cuda())
    for s in range(B):
        if slots[s] >= 0 and acc[s] > 0:
            close(pc[slots[s]], st_ref[s, acc[s] - 1], "slot of sequence %d" % s)
    untouched = [i for i in range(9) if i not in slots.tolist()] + [7]  # slot 7: no token accepted
    assert torch.equal(pc[untouched].cpu(), pool[untouched])


def test_no_state_no_gate(gdn):
    p, pd, beta, _ = problem(2, 4, 1, 2, 128, seed=9)
    bb = beta.bfloat16()
    o_ref, s_ref = O.recurrent_ref(p["q"].float(), p["k"].float(), p["v"].float(), bb.float(), torch.zeros(2, 4, 2), None, is_qk_norm=True)
    o, s = gdn.recurrent_forward(pd["q"], pd["k"], pd["v"], None, bb.cuda(), None, is_qk_norm=True)
    close(o, o_ref, "o")
    close(s, s_ref, "state")


@pytest.mark.parametrize("B,T,vh,d", [(14, 2, 32, 128), (15, 2, 32, 128), (18, 4, 32, 128), (37, 3, 16, 128), (38, 2, 16, 128), (16, 5, 32, 128),
                                      (11, 2, 32, 64), (12, 3, 32, 64), (37, 4, 16, 64)])
@pytest.mark.parametrize("steps", [False, True])
def test_one_wave_of_units(gdn, B, T, vh, d, steps):
    """on either side of the band of units (474 to 592 at d=128, 356 to 592 at d=64) where short runs stay with the FMA kernel"""
    p, pd, beta, g = problem(B, T, vh // 2, vh, d, seed=B + T)
    bb = beta.bfloat16()
    o_ref, s_ref = O.recurrent_ref(p["q"].float(), p["k"].float(), p["v"].float(), bb.float(), g, p["state"].float(), is_qk_norm=True, store_step_state=True)
    o, s = gdn.recurrent_forward(pd["q"], pd["k"], pd["v"], pd["state"], bb.cuda(), g.cuda(), inference_mode=gdn.SpecVerify if steps else gdn.Decode, is_qk_norm=True)
    close(o, o_ref, "o")
    close(s, s_ref if steps else s_ref[:, -1], "states")


@pytest.mark.parametrize("B", [1, 4, 5])
def test_one_token_tiles_apart_or_together(gdn, B):
    """one token per sequence: up to 592 tiles of 32 rows (B=4 with 32 v-heads of 128 rows is 512) every tile is a work unit,
    above that the tiles of a head stay together"""
    p, pd, beta, g = problem(B, 1, 16, 32, 128, seed=40 + B)
    bb = beta.bfloat16()
    o_ref, s_ref = O.recurrent_ref(p["q"].float(), p["k"].float(), p["v"].float(), bb.float(), g, p["state"].float(), is_qk_norm=True)
    o, s = gdn.recurrent_forward(pd["q"], pd["k"], pd["v"], pd["state"], bb.cuda(), g.cuda(), inference_mode=gdn.Decode, is_qk_norm=True)
    close(o, o_ref, "o")
    close(s, s_ref, "state")


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("where", ["q", "k", "v", "beta", "gate"])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_undefined_values_stay_behind_their_token(gdn, d, where, bad):
    """An undefined or infinite input of one token reaches no earlier token's output or state, as in the recurrence."""
    B, T, kh, vh, t = 2, 6, 2, 4, 3
    p, pd, beta, g = problem(B, T, kh, vh, d, seed=3 * d)
    x = dict(q=pd["q"], k=pd["k"], v=pd["v"], beta=beta.bfloat16().cuda(), gate=g.cuda())
    call = lambda: gdn.recurrent_forward(x["q"], x["k"], x["v"], pd["state"], x["beta"], x["gate"], inference_mode=gdn.SpecVerify, is_qk_norm=True)
    o_ref, s_ref = call()
    x[where] = x[where].clone()
    x[where][0, t].flatten()[0] = bad  # k-head 0 or v-head 0 of sequence 0
    o, s = call()
    assert torch.equal(o[:, :t], o_ref[:, :t]) and torch.equal(s[:, :t], s_ref[:, :t])
    assert torch.equal(o[1], o_ref[1]) and torch.equal(s[1], s_ref[1]) and torch.equal(o[0, :, 2:], o_ref[0, :, 2:])
    assert not torch.isfinite(o[0, t:, 0]).all()


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("steps", [False, True])
def test_infinite_value_gives_an_infinite_row(gdn, sign, steps):
    """v infinite in one row: that row of the token's state is infinite with the sign of v k, the others are untouched"""
    T, d, t = 2, 128, 1
    p, pd, beta, g = problem(1, T, 1, 1, d, seed=12)
    args = lambda v: (pd["q"], pd["k"], v, pd["state"], beta.bfloat16().cuda(), g.cuda())
    kw = dict(inference_mode=gdn.SpecVerify if steps else gdn.Decode, is_qk_norm=True)
    last = lambda s: s[0, t, 0] if steps else s[0, 0]
    s_ref = last(gdn.recurrent_forward(*args(pd["v"]), **kw)[1])
    v = pd["v"].clone()
    v[0, t, 0, 37] = sign * float("inf")
    s = last(gdn.recurrent_forward(*args(v), **kw)[1])
    rows = [r for r in range(d) if r != 37]
    assert torch.equal(s[rows], s_ref[rows])
    k = pd["k"][0, t, 0].float()
    assert (k != 0).all() and torch.equal(s[37].float(), torch.where(k * sign > 0, float("inf"), float("-inf")))


@pytest.mark.parametrize("T", [2, 8])
def test_no_token_accepted_passes_any_state(gdn, T):
    p, pd, beta, g = problem(2, T, 1, 2, 128, seed=T)
    s0 = pd["state"].clone()
    s0[0, 0, 5, 7], s0[0, 1, 0, 0], s0[1, 1, 127, 127] = float("inf"), float("nan"), float("-inf")
    acc = torch.zeros(2, dtype=torch.int32, device="cuda")
    _, s = gdn.recurrent_forward(pd["q"], pd["k"], pd["v"], s0, beta.bfloat16().cuda(), g.cuda(), None, acc, gdn.Decode, True)
    assert torch.equal(s.nan_to_num(12345.0), s0.nan_to_num(12345.0)) and torch.equal(s.isnan(), s0.isnan())
