"""Kernels of a chain are set up while the one ahead drains and wait for its
completion on the device.  Chains over buffers that are written again each time, run
back to back and with a synchronisation after every call, must agree bit for
bit: a read before the wait, or of a line cached before it, would show.  So must
the same chains in a caller's graph, where the edges between kernels are
programmatic and those to copies are not."""
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


def twice(chain):
    """chain(sync) -> outputs, back to back and then with sync() after every call"""
    a = chain(lambda: None)
    torch.cuda.synchronize()
    b = chain(torch.cuda.synchronize)
    torch.cuda.synchronize()
    for x, y in zip(a, b, strict=True):
        assert torch.equal(x, y)


@pytest.mark.parametrize("mixed,M,K,N,S", [(False, 64, 16, 2048, 1200), (True, 64, 32, 4096, 3276),
                                           (True, 32, 8, 2048, 1200), (True, 96, 48, 4096, 1204)])
def test_pilots_to_equalizer(mb, mixed, M, K, N, S):
    sg, n_sym, Qm, n = 16, 3, 4, 12
    G, P, start = -(-S // sg), -(-K // sg), (N - S) // 2
    g = torch.Generator(device="cuda").manual_seed(N + K)
    iq = [torch.randn(P, M, N, 2, generator=g, device="cuda").mul(2000).short() for _ in range(3)]
    y = [torch.randn(n_sym, M, S, dtype=torch.complex64, generator=g, device="cuda") for _ in range(3)]
    pilot, scr = mb.PilotFFT(start, N, S, M, K, sg), mb.Scrambler(num_bits=S * Qm)
    zf = mb.Beamform(M, K, G, precision=mb._lib.MB_ZF_MIXED if mixed else mb._lib.MB_ZF_FP32)
    csi = torch.zeros(G, M, K, dtype=torch.complex64, device="cuda")
    pre = [torch.zeros(G, K, M, dtype=torch.complex64, device="cuda") for _ in range(n)]
    llr = [torch.zeros(n_sym, K, S * Qm, dtype=torch.float16, device="cuda") for _ in range(n)]

    def chain(sync):
        csi.zero_()
        for i in range(n):
            (pilot.mixed if mixed else pilot)(iq[i % 3], csi)
            sync()
            zf.beamform_uplink(csi, S, sg)
            sync()
            mb.Beamform.beamform_downlink(csi, pre[i])
            sync()
            eq = mb.Equalize.equalize_tc if mixed else mb.Equalize.equalize
            eq(csi, y[i % 3], llr[i], sg, Qm, S * Qm, 0, scrambler=scr)
            sync()
        return [t.clone() for t in pre + llr + [csi]]

    twice(chain)
    assert mb.ops.device_error() == 0


@pytest.mark.parametrize("mixed", [False, True])
def test_downlink(mb, mixed):
    M, K, sg, D, Qm, n = 128, 16, 16, 6, 6, 12
    N, S = (4096, 3276) if mixed else (2048, 1200)
    g = torch.Generator(device="cuda").manual_seed(1)
    P = torch.randn(-(-S // sg), K, M, dtype=torch.complex64, generator=g, device="cuda")
    bits = [torch.randint(0, 256, (D * K, S * Qm // 8), generator=g, device="cuda").to(torch.uint8) for _ in range(3)]
    sym = torch.zeros(D * K, S, dtype=torch.complex64, device="cuda")
    z = torch.zeros(D, M, N, 2, dtype=torch.float16, device="cuda") if mixed else \
        torch.zeros(D, M, N, dtype=torch.complex64, device="cuda")
    out = [torch.zeros(D, M, N, 2, dtype=torch.float16, device="cuda") for _ in range(n)]
    ifft = mb.DownlinkIFFT((N - S) // 2, N, S, M)

    def chain(sync):
        for i in range(n):
            mb.Modulation.modulate(bits[i % 3], sym, Qm)
            sync()
            (mb.Precode.precode_tc if mixed else mb.Precode.precode)(P, sym.view(D, K, S), z, sg, (N - S) // 2)
            sync()
            (ifft.mixed if mixed else ifft)(z, out[i])
            sync()
        return [t.clone() for t in out]

    twice(chain)


@pytest.mark.parametrize("width,batch", [(128, 100), (256, 4096)])
def test_training(mb, width, batch):
    from megastation_b200 import learned
    g = torch.Generator(device="cuda").manual_seed(width)
    x = torch.rand(batch, 22, generator=g, device="cuda")
    A = torch.eye(4, device="cuda").expand(batch, 4, 4).contiguous()
    b = torch.randn(batch, 4, generator=g, device="cuda")
    c = torch.ones(batch, device="cuda")
    init = 0.05 * np.random.default_rng(0).standard_normal(learned.MLP(22, width, 4, max_batch=batch).params().size)

    def chain(sync):
        net = learned.MLP(22, width, 4, max_batch=batch)
        net.set_params(init.astype(np.float32))
        for _ in range(20):
            net.loss_grad(x, A, b, c)
            sync()
            net.adam_step(1e-3)
            sync()
        return [torch.from_numpy(np.ascontiguousarray(v)) for v in (net.params(), net.grads())]

    twice(chain)


@pytest.mark.parametrize("copies", [False, True])
@pytest.mark.parametrize("mixed,M,K,N,S", [(False, 64, 16, 2048, 1200), (True, 64, 32, 4096, 3276),
                                           (True, 96, 48, 4096, 1204)])
def test_uplink_in_a_callers_graph(mb, copies, mixed, M, K, N, S):
    """Three rounds of pilots, detector, precoder and equalizer in one graph,
    with a copy node between every two launches or with none."""
    sg, n_sym, Qm, n = 16, 3, 4, 3
    G, P, start = -(-S // sg), -(-K // sg), (N - S) // 2
    g = torch.Generator(device="cuda").manual_seed(K + 1)
    src = [torch.randn(n, P, M, N, 2, generator=g, device="cuda").mul(2000).short() for _ in range(3)]
    y = [torch.randn(n_sym, M, S, dtype=torch.complex64, generator=g, device="cuda") for _ in range(n)]
    pilot, scr = mb.PilotFFT(start, N, S, M, K, sg), mb.Scrambler(num_bits=S * Qm)
    zf = mb.Beamform(M, K, G, precision=mb._lib.MB_ZF_MIXED if mixed else mb._lib.MB_ZF_FP32)
    iq, stage = torch.empty_like(src[0]), src[0].clone()
    csi = torch.zeros(G, M, K, dtype=torch.complex64, device="cuda")
    W = torch.zeros_like(csi)
    pre = torch.zeros(n, G, K, M, dtype=torch.complex64, device="cuda")
    llr = torch.zeros(n, n_sym, K, S * Qm, dtype=torch.float16, device="cuda")
    eq = mb.Equalize.equalize_tc if mixed else mb.Equalize.equalize

    def chain():
        iq.copy_(stage)
        for i in range(n):
            (pilot.mixed if mixed else pilot)(iq[i], csi)
            if copies:
                W.copy_(csi)
            w = W if copies else csi
            zf.beamform_uplink(w, S, sg)
            if copies:
                csi.copy_(W)
            mb.Beamform.beamform_downlink(csi, pre[i])
            if copies:
                W.copy_(csi)
            eq(w, y[i], llr[i], sg, Qm, S * Qm, 0, scrambler=scr)

    ref = []
    for s in src:
        stage.copy_(s)
        chain()
        torch.cuda.synchronize()
        ref.append((pre.clone(), llr.clone()))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain()
    for i in (0, 1, 2, 1, 0):
        stage.copy_(src[i])
        pre.zero_(), llr.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(pre, ref[i][0]) and torch.equal(llr, ref[i][1])
    assert mb.ops.device_error() == 0


def test_training_in_a_callers_graph(mb):
    from megastation_b200 import learned
    g = torch.Generator(device="cuda").manual_seed(7)
    x, A = torch.rand(500, 22, generator=g, device="cuda"), torch.eye(4, device="cuda").expand(500, 4, 4).contiguous()
    b, loss = torch.randn(500, 4, generator=g, device="cuda"), torch.zeros(1, device="cuda")
    y = torch.zeros(500, 4, device="cuda")
    net = learned.MLP(22, 128, 4, max_batch=500)
    p0 = (0.05 * np.random.default_rng(0).standard_normal(net.params().size)).astype(np.float32)

    def chain():  # (the optimiser's step count is the handle's, so it stays outside)
        for _ in range(3):
            net.loss_grad(x, A, b, loss=loss)
            net.forward(x, out=y)

    net.set_params(p0)
    chain()
    torch.cuda.synchronize()
    ref = [loss.clone(), y.clone(), torch.from_numpy(net.grads())]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain()
    loss.zero_(), y.zero_()
    graph.replay()
    torch.cuda.synchronize()
    for a, c in zip([loss, y, torch.from_numpy(net.grads())], ref, strict=True):
        assert torch.equal(a, c)
