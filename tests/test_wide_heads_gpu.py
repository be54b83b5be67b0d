"""chunked_forward for head dims 129 .. 256: the tensor-core kernels on 256 columns whose operands are sums of two bf16
terms.  Nothing is rounded to fewer than 16 significand bits before the bf16 results are, so the error against the fp32
oracle stays that of rounding the results: at most 2^-9 relative per element, hence at most 2^-9 = 1.95e-3 in the
relative Frobenius norm, plus 64 terms of 2^-17 in the worst direction (0.5e-3).
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
