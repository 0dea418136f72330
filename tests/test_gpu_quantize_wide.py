"""Row quantisation on 32-byte loads, at the edges of what it takes, against the operator-by-operator path."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# One access; a thread's share and one more; every block size; rows longer than the registers hold; bases and row strides
# that allow 32-byte, 16-byte or single accesses.
@pytest.mark.parametrize("rows,cols", [(1, 16), (3, 1024), (3, 1040), (5, 4096), (600, 4112), (2, 8192), (2, 8208), (2, 16384), (2, 16400), (1, 49168)])
@pytest.mark.parametrize("offset,gap", [(0, 0), (8, 0), (0, 8), (1, 0), (0, 1), (16, 16)])
def test_quantize_rows(rows, cols, offset, gap):
    from torchcomms_b200.ops.tp import quantize_rows

    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    base = torch.randn(offset + rows * (cols + gap), generator=g, device="cuda").to(torch.bfloat16)
    x = base[offset:].view(rows, cols + gap)[:, :cols]
    x[-1, -1] = 9.0  # the maximum at the end of a row, where a remainder would miss it
    scale = x.float().abs().amax(dim=1).clamp_min(1e-8) / 448.0
    want = (x.float() / scale.unsqueeze(1)).to(torch.float8_e4m3fn)
    q, s = quantize_rows(x)
    assert torch.equal(s, scale) and torch.equal(q.view(torch.uint8), want.view(torch.uint8))
