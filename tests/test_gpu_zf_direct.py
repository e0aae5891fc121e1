"""The mixed-precision detector with up to 16 users (direct FP32 inverse):
edges of its tiles, the condition estimate, the FP64 solve of ill-conditioned
groups and the report of rank-deficient ones, against FP64; and the slot with
it against the slot with the tensor-core kernel (cells, path 2)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _csi(G, M, K, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.complex(torch.randn(G, M, K, generator=g), torch.randn(G, M, K, generator=g))


def _solve(C):
    Ch = C.to(torch.complex128).transpose(1, 2)
    A = Ch @ Ch.mH
    return A, torch.linalg.solve(A, Ch).transpose(1, 2)


@pytest.mark.parametrize("M,K", [(1, 1), (5, 2), (12, 3), (32, 16), (33, 15), (64, 8), (65, 9), (127, 16), (129, 4),
                                 (256, 16), (257, 7), (600, 16)])
def test_direct_edges(M, K):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from megastation_b200 import _lib, ops
    G = 5
    C = _csi(G, M, K, 31 * K + M)
    A, ref = _solve(C)
    d = C.cuda()
    status = torch.full((G,), 9, dtype=torch.int32, device="cuda")
    cond = torch.zeros(G, device="cuda")
    ops.Beamform(M, K, G, precision=_lib.MB_ZF_MIXED, cond_threshold=1e6).beamform_uplink(d, G * 16, 16, status=status,
                                                                                       cond=cond)
    assert (status.cpu() == 0).all()
    X = torch.linalg.inv(A)
    k1 = A.abs().sum(1).amax(1) * X.abs().sum(1).amax(1)  # 1-norms
    assert float(((cond.cpu().double() - k1).abs() / k1).max()) <= (K + M) * 2.0 ** -23 * float(k1.max()) + 1e-5
    # W = X C from BF16 X and C: each product off by 2^-8 of its magnitude
    bound = 2.0 ** -7 * torch.einsum("guv,gbv->gbu", X.abs(), C.abs().double()) + 1e-12
    assert ((d.cpu().to(torch.complex128) - ref).abs() <= bound).all()


def test_direct_ill_conditioned_and_deficient():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from megastation_b200 import _lib, ops
    for K in (2, 7, 16):
        M = 40
        C = _csi(4, M, K, K)
        C[1, :, K - 1] = C[1, :, 0] * (1 + 1e-3) + 1e-3 * C[1, :, K - 1]  # nearly parallel: FP64
        C[2, :, K - 1] = 0                                               # no channel: W = 0
        _, ref = _solve(C[[0, 1, 3]])
        d = C.cuda()
        status = torch.zeros(4, dtype=torch.int32, device="cuda")
        ops.Beamform(M, K, 4, precision=_lib.MB_ZF_MIXED, cond_threshold=1e4).beamform_uplink(d, 64, 16, status=status)
        assert status.cpu().tolist() == [0, 2, 1, 0]
        assert float(d[2].abs().max()) == 0
        got = d.cpu().to(torch.complex128)[[0, 1, 3]]
        err = (got - ref).flatten(1).norm(dim=1) / ref.flatten(1).norm(dim=1)
        assert float(err[1]) <= 1e-6 and float(err.max()) <= 2e-2


def test_direct_slot_matches_tensor_core_slot():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from megastation_b200 import cells, datagen
    cfgs = [datagen.CellConfig(M=M, K=K, N=N, S=S, sg=16, Qm=Qm, U=5, snr_db=22.0, seed=M + K)
            for M, K, N, S, Qm in ((32, 8, 1024, 601, 4), (70, 16, 2048, 1199, 6), (64, 3, 4096, 3276, 2))]
    iq = [torch.from_numpy(datagen.make_slot(c)["iq"]).cuda() for c in cfgs]
    cs = cells.Cells(cfgs)
    st = torch.cuda.Stream()
    out = []
    for path in (0, 2):
        t = cs.tuning()
        for c in t:
            c["zf_path"] = path
        cs.set_tuning(t)
        llr, hard = cs(iq, stream=st)
        st.synchronize()
        out.append([(a.float().cpu(), h.cpu().numpy()) for a, h in zip(llr, hard)])
    for c, (a, ha), (b, hb) in zip(cfgs, *out):
        # each path rounds X and C to BF16 (2^-9 an entry, differently scaled):
        # W y is off by 2 * 2^-9 |X| |G| of the symbols, twice for the two paths
        H = datagen.make_slot(c)["H"][:: c.sg]
        G = np.conj(H.transpose(0, 2, 1)) @ H
        amp = (np.abs(np.linalg.inv(G)) @ np.abs(G)).sum(2).max()
        assert float((a - b).norm() / b.norm()) <= 2.0 ** -7 * amp
        assert np.mean(np.unpackbits(ha) != np.unpackbits(hb)) <= 1e-3
