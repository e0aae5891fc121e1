"""The FP32 / FP64 zero forcing at the edges of its tiles (users past a
power of two, antennas past a column block, a last block of one row, partial
last groups) and its not-positive-definite report, against FP64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _csi(G, M, K, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.complex(torch.randn(G, M, K, generator=g), torch.randn(G, M, K, generator=g))


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("M,K", [(1, 1), (3, 2), (8, 5), (33, 16), (40, 17), (64, 32), (65, 33), (100, 50), (256, 64),
                                 (300, 7), (513, 16), (64, 63), (96, 47), (96, 48), (96, 49)])
def test_zf_edges(prec, M, K):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from megastation_b200 import _lib, ops
    G, sg = 3, 8
    C = _csi(G, M, K, 100 * K + M)
    d = C.cuda()
    status = torch.full((G,), 7, dtype=torch.int32, device="cuda")
    cond = torch.zeros(G, device="cuda")
    z = ops.Beamform(M, K, G, precision=_lib.MB_ZF_FP32 if prec == "fp32" else _lib.MB_ZF_FP64)
    if prec == "fp64" and 16 * K * (M + K + 2) + 1088 > 232448:
        with pytest.raises(_lib.MbError):
            z.beamform_uplink(d, G * sg, sg, status=status, cond=cond)
        return
    z.beamform_uplink(d, G * sg, sg, status=status, cond=cond)
    Ch = C.to(torch.complex128).transpose(1, 2)
    A = Ch @ Ch.mH
    ref = torch.linalg.solve(A, Ch).transpose(1, 2)
    kappa = float(torch.linalg.cond(A).max())
    eps = 2.0 ** -24 if prec == "fp32" else 2.0 ** -24  # FP64 results are stored in FP32
    bound = (K + M) * eps * (kappa if prec == "fp32" else 1.0)
    got = d.cpu().to(torch.complex128)
    err = (got - ref).norm() / ref.norm()
    assert float(err) <= max(bound, 4 * eps)
    if prec == "fp32":
        # The forward bound says little once kappa is large ((64, 63): 1e4, 9%); the residual of A W = C does not
        # grow with it: the Gram's M roundings, the elimination's K and the two products' 2 K, of eps each and of
        # either sign (so their root), relative to |A| |W|.  Seen: 1e-7 at (64, 63), 3.2e-7 at (513, 16).
        X = got.transpose(1, 2)
        res = (A @ X - Ch).flatten(1).norm(dim=1)
        size = torch.linalg.matrix_norm(A, 2) * X.flatten(1).norm(dim=1)
        assert (res <= (M + 3 * K) ** 0.5 * eps * size).all()
    assert (status.cpu() == 0).all()
    # (max / min pivot) of L D L^H is below the condition number
    assert (cond.cpu() <= 1.01 * kappa + 1e-3).all() and (cond.cpu() >= 0.99).all()


def test_zf_not_positive_definite_keeps_other_groups():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from megastation_b200 import _lib, ops
    for K in (5, 20, 40):
        C = _csi(3, 80, K, K)
        C[1, :, K - 1] = 0  # a user without a channel
        d = C.cuda()
        status = torch.zeros(3, dtype=torch.int32, device="cuda")
        ops.Beamform(80, K, 3, precision=_lib.MB_ZF_FP32).beamform_uplink(d, 48, 16, status=status)
        assert status.cpu().tolist() == [0, 1, 0]
        assert float(d[1].abs().max()) == 0 and float(d[0].abs().max()) > 0
