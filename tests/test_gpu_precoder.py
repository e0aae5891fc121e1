"""The downlink precoder over its cluster split (one to eight CTAs a group, and
the two-pass form past what an eighth of W fits), against torch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _csi(G, M, K, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.complex(torch.randn(G, M, K, generator=g), torch.randn(G, M, K, generator=g))


@pytest.mark.parametrize("M,K", [(1, 1), (31, 3), (32, 64), (33, 7), (64, 16), (129, 33), (200, 64), (256, 300),
                                 (300, 5), (2000, 16), (1000, 255)])
def test_precoder_cluster_split(M, K):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from megastation_b200 import ops
    W = _csi(5, M, K, M + K).cuda()
    P = torch.zeros(5, K, M, dtype=torch.complex64, device="cuda")
    ops.Beamform.beamform_downlink(W, P)
    # |w| as the kernel forms it, then one reciprocal and one product each
    v = torch.view_as_real(W)
    mag = (v[..., 0] * v[..., 0] + v[..., 1] * v[..., 1]).sqrt().amax((1, 2))
    ref = (W.transpose(1, 2) * (1.0 / mag)[:, None, None])
    assert float((P - ref).abs().max()) <= 2.0 ** -22
