"""One-launch patches, their transpose and the (channel, position) index lists of NormDistConv against PyTorch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,C,H,W,kernel,stride,padding,dilation",
                         [(3, 4, 9, 7, (3, 3), 1, 0, 1), (2, 3, 16, 16, (8, 8), 8, 0, 1), (5, 2, 11, 13, (3, 5), 2, 2, 1),
                          (1, 1, 10, 10, (2, 3), 3, 1, 2), (70, 3, 5, 5, (5, 5), 1, 2, 1)])
def test_unfold_matches_torch(B, C, H, W, kernel, stride, padding, dilation):
    """One-launch patches: values exact; the sum back in kernel order (fp32, as many terms as the kernel has)."""
    from sortnet_b200.layers import _UnfoldF
    x = torch.randn(B, C, H, W, device="cuda", requires_grad=True)
    y = _UnfoldF.apply(x, kernel, stride, padding, dilation)
    want = torch.nn.functional.unfold(x, kernel, dilation, padding, stride)
    assert torch.equal(y, want)
    g = torch.randn_like(y)
    (gx,) = torch.autograd.grad(y, x, g)
    (wx,) = torch.autograd.grad(want, x, g)
    assert torch.allclose(gx, wx, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("S,G,kept,channels,hw", [(3, 1, 5, 8, 1), (2, 3, 4, 12, 4), (1, 2, 6, 12, 9)])
def test_plane_index(S, G, kept, channels, hw):
    from sortnet_b200.layers import _plane_index
    index = torch.stack([torch.stack([torch.randperm(channels // G)[:kept].sort()[0] for _ in range(G)]) for _ in range(S)]).int()
    assert torch.equal(_plane_index(index.cuda(), channels, hw).cpu(), _plane_index(index, channels, hw))
