"""Norm kernel by row length: the edges between one, four and eight warps per row, and the sum left out."""
import pytest
import torch

from oracle import kernl_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("rows, cols", [(3, 8), (1500, 1024), (1500, 1032), (9, 2048), (1100, 3080), (5, 4096), (5, 4104), (1030, 6152), (2, 8192), (3, 16384)])
def test_norm_row_lengths(lib, rows, cols, rms):
    from kernl_b200.implementations.layer_norm import layer_norm

    g = torch.Generator().manual_seed(cols)
    x = (torch.randn((rows, cols), generator=g) - 20 * (cols % 3)).half()  # large means too
    r = torch.randn((rows, cols), generator=g).half()
    w, b = torch.rand((cols,), generator=g).half() + 0.5, torch.randn((cols,), generator=g).half()
    bias = None if rms else b
    total = (x.float() + r.float()).half()
    ref = (lambda t: O.rms_norm(t, w, 1.6e-5)) if rms else (lambda t: O.layer_norm(t, w, b, 1.6e-5))
    xc, rc, wc, bc = x.cuda(), r.cuda(), w.cuda(), None if rms else b.cuda()
    O.assert_parity(layer_norm(xc, wc, bc, 1e-5, use_rms_norm=rms), ref(x), what="norm")
    y, s = layer_norm(xc, wc, bc, 1e-5, use_rms_norm=rms, residual=rc)
    assert torch.equal(s.cpu(), total)
    O.assert_parity(y, ref(total), what="add + norm")
    alone = layer_norm(xc, wc, bc, 1e-5, use_rms_norm=rms, residual=rc, with_sum=False)
    assert torch.equal(alone, y)
