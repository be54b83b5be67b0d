"""causal_conv1d where the launch picks its tokens per thread: just above one block, blocks below and above 32 tokens, a last
block of one token, packed sequences whose ends fall anywhere in a block."""
import pytest
import torch

from oracle import gdn_oracle as O

pytestmark = pytest.mark.gpu

# bf16 output: half a unit in the last place is at most 2^-9 of a value; SiLU's hardware tanh adds 2^-11 on a factor of
# (1 + tanh) / 2: together below 2^-8
TOL = 2.0 ** -8


@pytest.fixture(scope="module")
def gdn():
    import h100_gdn_cuda_b200 as g
    return g


@pytest.mark.parametrize("B,T,C_,W", [(1, 33, 64, 4), (2, 37, 8, 3), (1, 505, 2048, 2), (3, 1000, 1032, 3), (1, 4097, 8192, 4)])
def test_conv_padded_blocks(gdn, B, T, C_, W):
    gen = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(B, T, C_, generator=gen, device="cuda").bfloat16()
    w = (torch.randn(C_, W, generator=gen, device="cuda") * 0.5).bfloat16()
    s0 = torch.randn(B, W - 1, C_, generator=gen, device="cuda").bfloat16()
    y, fin = gdn.api.causal_conv1d(x, w, None, s0, return_final_state=True)
    y_ref, fin_ref = O.causal_conv1d_ref(x.cpu(), w.cpu(), None, s0.cpu())
    assert O.rel_fro(y.cpu(), y_ref) < TOL
    assert torch.equal(fin.float().cpu(), fin_ref)


def test_conv_packed_blocks(gdn):
    lens = [5, 0, 61, 1, 1, 130, 7, 64, 300]
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32)
    gen = torch.Generator().manual_seed(9)
    x = torch.randn(sum(lens), 520, generator=gen).bfloat16()
    w = (torch.randn(520, 4, generator=gen) * 0.5).bfloat16()
    s0 = torch.randn(len(lens), 3, 520, generator=gen).bfloat16()
    y, fin = gdn.api.causal_conv1d(x.cuda(), w.cuda(), None, s0.cuda(), cu_seqlens=cu.cuda(), return_final_state=True)
    y_ref, fin_ref = O.causal_conv1d_ref(x, w, None, s0, cu_seqlens=cu.tolist())
    assert O.rel_fro(y.cpu(), y_ref) < TOL
    assert torch.equal(fin.float().cpu(), fin_ref)


@pytest.mark.parametrize("lens", [[1] * 70, [3, 0, 0, 1, 9, 0, 0, 0] * 8 + [0] * 80, [0, 40, 1, 2] + [0] * 60, [0] * 64 + [64]])
@pytest.mark.parametrize("C_,W", [(8192, 4), (520, 2)])
def test_conv_packed_state_in_place(gdn, lens, C_, W):
    """No more tokens than sequences, but sequences of any length (8192 channels: blocks of 4 tokens, which they span): the
    state updated where it lies, the same bits as into a buffer of its own."""
    assert sum(lens) <= len(lens)
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32).cuda()
    gen = torch.Generator(device="cuda").manual_seed(len(lens))
    x = torch.randn(sum(lens), C_, generator=gen, device="cuda").bfloat16()
    w = (torch.randn(C_, W, generator=gen, device="cuda") * 0.5).bfloat16()
    s0 = torch.randn(len(lens), W - 1, C_, generator=gen, device="cuda").bfloat16()
    y_ref, s_ref = gdn.api.causal_conv1d(x, w, None, s0, cu_seqlens=cu, return_final_state=True)
    y, s = gdn.api.causal_conv1d(x, w, None, s0, cu_seqlens=cu, final_state=s0)
    assert s.data_ptr() == s0.data_ptr()
    assert torch.equal(y, y_ref) and torch.equal(s, s_ref)


@pytest.mark.parametrize("W", [2, 3, 4])
def test_conv_weight_alignment(gdn, W):
    """The taps are read 16 bytes at a time where the weight allows it: a weight at an odd element gives the same bits."""
    gen = torch.Generator(device="cuda").manual_seed(W)
    x = torch.randn(2, 70, 72, generator=gen, device="cuda").bfloat16()
    flat = torch.randn(72 * W + 1, generator=gen, device="cuda").bfloat16()
    w = flat[1:].view(72, W)
    assert torch.equal(gdn.api.causal_conv1d(x, w), gdn.api.causal_conv1d(x, w.clone()))
