"""Norm kernel by row length: the edges between one, four and eight warps per row, and the sum left out."""
import pytest
import torch

from oracle import kernl_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("rows, cols", [(3, 8), (1500, 1024), (1500, 1032), (9, 2048), (1100, 3080), (5, 4096), (5, 4104), (1030, 6152), (2, 8192), (3, 16384)])
def test_norm_row_lengths(lib, rows, cols, rms, dtype):
    from kernl_b200.implementations.layer_norm import layer_norm

    g = torch.Generator().manual_seed(cols)
    x = (torch.randn((rows, cols), generator=g) - 20 * (cols % 3)).to(dtype)  # large means too
    r = torch.randn((rows, cols), generator=g).to(dtype)
    w, b = torch.rand((cols,), generator=g).to(dtype) + 0.5, torch.randn((cols,), generator=g).to(dtype)
    bias = None if rms else b
    total = (x.float() + r.float()).to(dtype)
    eps, bound = (1.6e-5, 1e-2) if dtype == torch.float16 else (1e-5, 8e-2)  # fp16 clamps eps; bf16 keeps three bits less
    ref = (lambda t: O.rms_norm(t, w, eps)) if rms else (lambda t: O.layer_norm(t, w, b, eps))
    xc, rc, wc, bc = x.cuda(), r.cuda(), w.cuda(), None if rms else b.cuda()
    O.assert_parity(layer_norm(xc, wc, bc, 1e-5, use_rms_norm=rms), ref(x), max_abs=bound, what="norm")
    y, s = layer_norm(xc, wc, bc, 1e-5, use_rms_norm=rms, residual=rc)
    assert torch.equal(s.cpu(), total)
    O.assert_parity(y, ref(total), max_abs=bound, what="add + norm")
    alone = layer_norm(xc, wc, bc, 1e-5, use_rms_norm=rms, residual=rc, with_sum=False)
    assert torch.equal(alone, y)
