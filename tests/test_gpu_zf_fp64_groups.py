"""Mixed-precision zero forcing: the FP64 solve at the edges of its tiles of
antennas and of its paddings of users, and the learned start of 33 to 64 users, in
launches of fewer and of more groups than SMs, against FP64 and one another."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mb():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import megastation_b200 as m
    return m


def _csi(G, M, K):
    g = torch.Generator().manual_seed(1000 * K + M)
    return torch.complex(torch.randn(G, M, K, generator=g), torch.randn(G, M, K, generator=g))


def _solve(C):
    Ch = C.to(torch.complex128).transpose(1, 2)
    return torch.linalg.solve(Ch @ Ch.mH, Ch).transpose(1, 2)


def _twice(mb, C, **kw):
    """W and status of C's groups, and of C repeated past the number of SMs."""
    out = []
    for n in (1, 160 // C.shape[0]):
        d = C.repeat(n, 1, 1).cuda()
        G, M, K = d.shape
        status = torch.full((G,), 9, dtype=torch.int32, device="cuda")
        mb.Beamform(M, K, G, precision=mb._lib.MB_ZF_MIXED, **kw).beamform_uplink(d, G * 16, 16, status=status)
        torch.cuda.synchronize()
        out.append((d.cpu(), status.cpu()))
    (a, sa), (b, sb) = out
    assert b.shape[0] > 148 >= a.shape[0]
    assert torch.equal(a.repeat(b.shape[0] // a.shape[0], 1, 1), b)
    assert torch.equal(sa.repeat(b.shape[0] // a.shape[0]), sb)
    assert mb.ops.device_error() == 0
    return a.to(torch.complex128), sa


# tiles of 31 antennas (up to 16 users: half as many as the CSI's, an odd number)
@pytest.mark.parametrize("M,K", [(2, 2), (31, 5), (62, 16), (63, 7), (257, 16), (31, 17), (93, 32), (94, 31), (64, 33),
                                 (64, 48), (64, 64), (70, 50), (130, 64)])
def test_fp64_groups(mb, M, K):
    C = _csi(5, M, K)
    C[3, :, K - 1] = 0  # no channel: W = 0
    W, status = _twice(mb, C, cond_threshold=0.5)
    assert status.tolist() == [2, 2, 2, 1, 2]
    assert float(W[3].abs().max()) == 0
    keep = [0, 1, 2, 4]
    ref = _solve(C[keep])
    err = (W[keep] - ref).flatten(1).norm(dim=1) / ref.flatten(1).norm(dim=1)
    assert float(err.max()) <= 4 * 2.0 ** -24  # stored in FP32


@pytest.mark.parametrize("M,K", [(128, 33), (200, 48), (256, 63), (256, 64)])
def test_learned_start(mb, M, K):
    """From the best fixed cubic of these groups' own spectra.  The BF16 factors
    allow 2^-8 of the magnitudes |X| |C| each; over 33 and more users their signs
    leave less than a quarter of that in the norm (seen: 0.11)."""
    from megastation_b200 import learned
    C = _csi(8, M, K)
    Ch = C.to(torch.complex128).transpose(1, 2)
    A = Ch @ Ch.mH
    lam = torch.linalg.eigvalsh(A)
    lam = (lam / lam.mean(-1, keepdim=True)).flatten()
    V = torch.stack([lam ** k for k in range(1, 5)], 1)
    coef = torch.linalg.lstsq(V, torch.ones_like(lam)[:, None]).solution[:, 0].numpy().astype(np.float32)
    net = learned.MLP(6, 64, 4, max_batch=256, out_bias=coef)
    W, status = _twice(mb, C, init_net=net)
    assert (status == 3).all(), status
    X = torch.linalg.inv(A)
    bound = 2.0 ** -7 * torch.einsum("guv,gbv->gbu", X.abs(), C.abs().double())
    err = (W - _solve(C)).flatten(1).norm(dim=1) / bound.flatten(1).norm(dim=1)
    assert float(err.max()) <= 0.25
