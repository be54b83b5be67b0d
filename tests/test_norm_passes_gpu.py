"""gated_rmsnorm at the edges of its dispatch on the row length (lanes per row, passes of 256 elements) and of the rows a
block takes."""
import pytest
import torch

from oracle import gdn_oracle as O

pytestmark = pytest.mark.gpu

# bf16 output: at most 2^-9 of a value; SiLU's hardware tanh adds 2^-11 on a factor of (1 + tanh) / 2: together below 2^-8
TOL = 2.0 ** -8


@pytest.mark.parametrize("dim", [8, 32, 40, 128, 136, 256, 264, 512, 520, 1024])
@pytest.mark.parametrize("rows", [1, 17, 130])
def test_norm_dims(dim, rows):
    import h100_gdn_cuda_b200 as gdn
    gen = torch.Generator().manual_seed(dim + rows)
    x, z = (torch.randn(rows, dim, generator=gen).bfloat16() for _ in range(2))
    w = torch.randn(dim, generator=gen).bfloat16()
    y = gdn.api.gated_rmsnorm(x.cuda(), z.cuda(), w.cuda())
    assert O.rel_fro(y.cpu(), O.gated_rmsnorm_ref(x, z, w)) < TOL
