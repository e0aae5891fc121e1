"""The performance cases: what a base-station program has this library do.

Single operators over the sizes of the repository's workloads (the plain FP32
path and the mixed-precision one, both directions, each sample format), the
LDPC codec, the learned initialiser's inference and training, and two whole
calls (one cell's uplink slot, a set of uneven cells).  Every input is drawn
on the GPU from the seed.  `exact` restates each path in 64-bit torch.
"""
import math
import random

import numpy as np
import torch

from megastation_b200 import _lib, cells, datagen, learned, ops, slot

DEV = "cuda"
IQ_BYTES = {"c64": 8, "int16": 4, "int8": 2, "f16": 4}
IQ_TORCH = {"int16": torch.int16, "int8": torch.int8, "f16": torch.float16}
PRECISION = {"fp32": _lib.MB_ZF_FP32, "mixed": _lib.MB_ZF_MIXED}


def listed():
    return [
        # one antenna panel's symbol of a narrow 20 MHz cell: the smallest
        # call of the FFT operator, where the launch itself counts
        dict(name="fft_1024x32", kind="fft", M=32, N=1024, S=600, n_sym=1, iq="c64", out="c64"),
        # pilots to detector of the 64 x 16 cell with the reference's FP32 arithmetic
        dict(name="zf_fp32_64x16", kind="zf", M=64, K=16, N=2048, S=1200, sg=16, precision="fp32", iq="c64",
             precoder=False),
        # pilots to detector and downlink precoder of the 256 x 64 full-slot cell, mixed precision
        dict(name="zf_mixed_256x64", kind="zf", M=256, K=64, N=4096, S=3276, sg=16, precision="mixed", iq="int16",
             precoder=True),
        # equalize + demap + descramble of the 64 x 16 cell's 13 data symbols in FP32
        dict(name="equalize_fp32_64x16", kind="equalize", M=64, K=16, S=1200, sg=16, n_sym=13, Qm=4,
             precision="fp32"),
        # the same step of the 256 x 32 cell's 12 data symbols on the tensor cores
        dict(name="equalize_mixed_256x32", kind="equalize", M=256, K=32, S=3276, sg=16, n_sym=12, Qm=6,
             precision="mixed"),
        # downlink of a 128 x 16 cell: modulate, precode, inverse FFT to int16 samples
        dict(name="downlink_fp32_128x16", kind="downlink", M=128, K=16, N=2048, S=1200, sg=16, n_sym=6, Qm=6,
             precision="fp32", out="int16"),
        # one slot's 384 code blocks of the 256 x 32 cell at rate 1/3, 8 passes
        dict(name="ldpc_decode_384", kind="ldpc_decode", kb=22, Z=288, rows=46, batch=384, iters=8),
        # the downlink code blocks of a 256 x 64 cell's five symbols
        dict(name="ldpc_encode_320", kind="ldpc_encode", kb=22, Z=352, rows=46, batch=320),
        # per-subcarrier detector of a 128 x 16 cell from the learned blend, two Newton-Schulz steps
        dict(name="lzf_128x16", kind="lzf", M=128, K=16, N=2048, S=1200, sg=16, iters=2, delay_ns=150),
        # eight optimiser steps of the blend network on mini-batches of 4096
        dict(name="train_256", kind="train", n_in=22, width=256, n_out=4, batch=4096, steps=8),
        # the uplink slot of the 256 x 32 cell from int8 samples: pilots to
        # LLRs and hard bits, learned start of the inverse, replayed as a graph
        dict(name="slot_256x32", kind="slot", M=256, K=32, N=4096, S=3276, sg=16, Qm=6, U=12, snr_db=25.0,
             iq="int8", precision="mixed", learned=True, sym_batch=12, graph=True),
        # 32 cells of uneven shape served by one GPU, one call for a slot of each
        dict(name="cells_32", kind="cells", count=32, cell_seed=3, symbols=14),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fft", "zf", "equalize", "downlink", "ldpc_decode", "ldpc_encode", "lzf", "train", "slot",
                       "cells"])
    N = rng.choice([512, 1024, 2048, 4096])
    S = rng.randint(int(0.5 * N), int(0.82 * N))
    if kind == "fft":
        return dict(kind=kind, M=_log_int(rng, 4, 256), N=N, S=S, n_sym=_log_int(rng, 1, 14),
                    iq=rng.choice(["c64", "int16", "int8", "f16"]), out=rng.choice(["c64", "bf16"]))
    if kind in ("zf", "equalize", "downlink", "slot"):
        K = _log_int(rng, 2, 64)
        M = max(K, _log_int(rng, max(2 * K, 8), 256) if K <= 32 else rng.randint(2 * K, 256))
        sg = rng.choice([8, 16, 16, 16, 32])
        precision = rng.choice(["fp32", "mixed"])
        if kind == "zf":
            return dict(kind=kind, M=M, K=K, N=N, S=S, sg=sg, precision=precision,
                        iq=rng.choice(["c64", "int16", "int8", "f16"]), precoder=rng.random() < 0.5)
        if kind == "equalize":
            return dict(kind=kind, M=M, K=K, S=S, sg=sg, n_sym=_log_int(rng, 1, 14), Qm=rng.choice([2, 4, 6, 8]),
                        precision=precision)
        if kind == "downlink":
            return dict(kind=kind, M=M, K=K, N=N, S=S, sg=sg, n_sym=_log_int(rng, 1, 8), Qm=rng.choice([2, 4, 6, 8]),
                        precision=precision if N == 4096 else "fp32", out=rng.choice(["int16", "f16"]))
        U = rng.randint(2, 13)
        return dict(kind=kind, M=M, K=K, N=N, S=S, sg=sg, Qm=rng.choice([2, 4, 6]), U=U, snr_db=rng.uniform(15, 30),
                    iq=rng.choice(["c64", "int16", "int8"]), precision=precision,
                    learned=precision == "mixed" and rng.random() < 0.5, sym_batch=rng.choice([4, U]),
                    graph=rng.random() < 0.5)
    if kind.startswith("ldpc"):
        kb, rows = rng.choice([(22, rng.randint(8, 46)), (10, rng.randint(8, 42))])
        Z = rng.choice([24, 52, 72, 104, 144, 208, 288, 352])
        c = dict(kind=kind, kb=kb, Z=Z, rows=rows, batch=_log_int(rng, 1, 320))
        return dict(c, iters=rng.randint(3, 8)) if kind == "ldpc_decode" else c
    if kind == "lzf":
        K = rng.randint(2, 16)
        return dict(kind=kind, M=_log_int(rng, 2 * K, 128), K=K, N=2048, S=rng.randint(300, 1200),
                    sg=rng.choice([8, 16]), iters=rng.randint(1, 3), delay_ns=rng.randint(50, 300))
    if kind == "train":
        n_in, n_out = rng.choice([(6, 4), (22, 4), (14, 4)])
        return dict(kind=kind, n_in=n_in, width=rng.choice([64, 128, 200, 256]), n_out=n_out,
                    batch=_log_int(rng, 128, 4096), steps=rng.randint(1, 8))
    return dict(kind="cells", count=rng.randint(3, 16), cell_seed=rng.randrange(1 << 16), symbols=rng.randint(6, 14))


# ------------------------------------------------------------- inputs ----
def _gen(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(1000003 * int(seed) + salt)
    return g


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV)


def _cn(g, *shape):
    return torch.complex(_randn(g, *shape), _randn(g, *shape)) * math.sqrt(0.5)


def _qam(g, Qm, *shape):
    """Uniform symbols of the square 2^Qm constellation at unit power."""
    n = 1 << (Qm // 2)
    a, b = (2 * torch.randint(0, n, shape, generator=g, device=DEV) - (n - 1) for _ in range(2))
    return torch.complex(a.float(), b.float()) / math.sqrt(2 * (n * n - 1) / 3)


def _bins(N, S):
    """FFT bin of each data subcarrier."""
    return (torch.arange(S, device=DEV) + (N - S) // 2 + N // 2) % N


def _pilots(S):
    """The comb pilot of each subcarrier: a Zadoff-Chu sequence of the largest
    prime length up to min(S, 2039), turned by pi/4 a subcarrier; phases
    rounded to float, as a transmitter in single precision forms them."""
    L = min(S, 2039)
    while any(L % d == 0 for d in range(2, int(math.isqrt(L)) + 1)):
        L -= 1
    i = np.arange(S)
    m = (i % L).astype(np.float64)
    turn = (-np.pi * np.floor(L * 2.0 / 31.0 + 0.5) * m * (m + 1) / L).astype(np.float32).astype(np.float64)
    spin = (np.float32(np.pi / 4) * i.astype(np.float32)).astype(np.float64)
    return torch.from_numpy(np.exp(1j * (turn + spin)).astype(np.complex64)).to(DEV)


def _tdl(g, c, taps=8, rho=0.5, decay=2.0, delay_ns=None):
    """Frequency response [S][M][K] of a tapped-delay-line channel with
    exponential power-delay profile and exponential antenna correlation;
    delay_ns spreads the taps over three such delay spreads (30 kHz spacing)."""
    M, K, N, S = c["M"], c["K"], c["N"], c["S"]
    if delay_ns:
        ds = delay_ns * 1e-9 * N * 30e3
        tau = torch.arange(taps, device=DEV, dtype=torch.float64) * (3 * ds / (taps - 1))
        pdp = torch.exp(-tau / ds)
    else:
        tau = torch.arange(taps, device=DEV, dtype=torch.float64)
        pdp = torch.exp(-tau / decay)
    w = _cn(g, taps, M, K) * torch.sqrt(pdp / pdp.sum()).float()[:, None, None]
    if rho:
        i = torch.arange(M, device=DEV)
        w = torch.linalg.cholesky(rho ** (i[:, None] - i[None, :]).abs().double()).to(w.dtype) @ w
    f = (_bins(N, S) + N // 2) % N - N // 2
    turn = torch.exp(-2j * math.pi * f.double()[:, None] * tau / N).to(torch.complex64)
    return (turn @ w.reshape(taps, M * K)).reshape(S, M, K)


def _iid(g, c):
    """Frequency response [S][M][K], i.i.d. Rayleigh per subcarrier group."""
    G = -(-c["S"] // c["sg"])
    return _cn(g, G, c["M"], c["K"])[torch.arange(c["S"], device=DEV) // c["sg"]]


def _to_samples(c, Y, iq):
    """Time-domain samples [sym][M][N] (pairs for the integer and FP16 formats) of the
    subcarrier values Y [sym][M][S]; integer formats at a quarter of full scale."""
    row = torch.zeros(*Y.shape[:-1], c["N"], dtype=torch.complex64, device=DEV)
    row[..., _bins(c["N"], c["S"])] = Y
    x = torch.fft.ifft(row)
    if iq == "c64":
        return x
    v = torch.view_as_real(x)
    if iq == "f16":
        return (v * math.sqrt(c["N"])).half()
    top = 32768 if iq == "int16" else 128
    v = v * (0.25 / v.square().sum(-1).mean().sqrt())
    return torch.clamp(torch.round(v * top), -top, top - 1).to(IQ_TORCH[iq])


def _received(c, g, H, snr_db, U, Qm):
    """Subcarrier values [P + U][M][S]: comb pilots (user p sg + s mod sg on
    subcarrier s of pilot symbol p), then U symbols of QAM data, plus noise."""
    M, K, S, sg = c["M"], c["K"], c["S"], c["sg"]
    P = -(-K // sg)
    s = torch.arange(S, device=DEV)
    pil = _pilots(S)
    Y = torch.zeros(P + U, M, S, dtype=torch.complex64, device=DEV)
    for p in range(P):
        u = p * sg + s % sg
        Y[p] = (H[s, :, u.clamp(max=K - 1)] * (pil * (u < K))[:, None]).T
    if U:
        Y[P:] = (H @ _qam(g, Qm, S, K, U)).permute(2, 1, 0)
    return Y + _cn(g, P + U, M, S) * 10 ** (-snr_db / 20)


def _cell_config(c, **kw):
    return datagen.CellConfig(M=c["M"], K=c["K"], N=c["N"], S=c["S"], sg=c["sg"], Qm=c["Qm"], U=c["U"],
                              iq_dtype=c["iq"], **kw)


def _start_net(H, sg, width=64):
    """Network of the learned Newton-Schulz start, its coefficients those of
    the best fixed cubic for this cell's Gram spectra (what training finds for
    one shape), with small weights on the features."""
    C = H[::sg][:32].to(torch.complex128)
    lam = torch.linalg.eigvalsh(C.mH @ C)
    lam = (lam / lam.mean(-1, keepdim=True)).flatten()
    A = torch.stack([lam ** k for k in range(1, 5)], 1)
    coef = torch.linalg.lstsq(A, torch.ones_like(lam)[:, None]).solution[:, 0].cpu().numpy()
    net = learned.MLP(6, width, 4, max_batch=256, out_bias=coef)
    p = net.params()
    p[-4 - 4 * width:-4] = 1e-3 * np.random.default_rng(0).standard_normal(4 * width)
    net.set_params(p)
    return net


def _blend_net(sg, width=256):
    """Network of the per-subcarrier blend: linear interpolation between the
    neighbouring groups' inverses by the subcarrier's offset (the one-hot
    inputs), with small weights elsewhere."""
    r = np.random.default_rng(1)
    n_in = sg + 6
    W1, W2 = (0.01 * r.standard_normal((n, width)) for n in (n_in, width))
    W3 = 0.01 * r.standard_normal((width, 4))
    t = (np.arange(sg) - sg // 2) / sg
    for o in range(sg):
        W1[o, :], W2[o, :] = 0, 0
        W1[o, o], W2[o, o] = 1, 1
        W3[o] = [max(0, -t[o]), 1 - abs(t[o]), max(0, t[o]), 0]
    z = np.zeros(width)
    net = learned.MLP(n_in, width, 4, max_batch=8192)
    net.set_params(np.concatenate([a.ravel() for a in (W1, z, W2, z, W3, np.zeros(4))]))
    return net


def _graph(c):
    """Base graph entries (row, column, shift) with the NR block structure:
    four core rows with a dual-diagonal core parity block, then extension rows
    of falling degree over the information and core parity columns."""
    r = random.Random(c["kb"])
    kb, Z, e = c["kb"], c["Z"], []
    for i in range(c["rows"]):
        if i < 4:
            cols = sorted(r.sample(range(2, kb), int(0.7 * kb))) + [0, 1][:2 if kb > 12 else 1 + i % 2]
        else:
            deg = max(2, (9 if kb > 12 else 5) - i // 6)
            cols = [i % 2] + r.sample(range(2, kb + (4 if i < 16 else 0)), deg)
        e += [(i, j, r.randrange(384) % Z) for j in cols]
        if i < 4:  # columns kb .. kb + 3: the first three times (shift 1, 0, 1), then the diagonal pair
            e += [(i, kb, {0: 1, 1: 0, 3: 1}[i])] if i != 2 else []
            e += [(i, kb + 1 + j, 0) for j in (i - 1, i) if 0 <= j < 3]
        else:
            e += [(i, kb + i, 0)]
    return e


def _encode(c, info):
    """Codewords [B][kb + rows][Z] (bits) of info [B][kb][Z] by the parity equations."""
    kb, e = c["kb"], _graph(c)
    B, Z = info.shape[0], c["Z"]
    x = torch.zeros(B, kb + c["rows"], Z, dtype=torch.uint8, device=DEV)
    x[:, :kb] = info

    def part(i, lo, hi):
        acc = torch.zeros(B, Z, dtype=torch.uint8, device=DEV)
        for r, j, s in e:
            if r == i and lo <= j < hi:
                acc ^= torch.roll(x[:, j], -(s % Z), -1)
        return acc

    lam = [part(i, 0, kb) for i in range(4)]
    x[:, kb] = lam[0] ^ lam[1] ^ lam[2] ^ lam[3]  # the diagonal and the shift-1 pair cancel in the sum
    first = [torch.roll(x[:, kb], -(1 % Z), -1), x[:, kb], None, None]
    x[:, kb + 1] = lam[0] ^ first[0]
    x[:, kb + 2] = lam[1] ^ first[1] ^ x[:, kb + 1]
    x[:, kb + 3] = lam[2] ^ x[:, kb + 2]
    for i in range(4, c["rows"]):
        x[:, kb + i] = part(i, 0, kb + 4)
    return x


def _pack(bits):
    pad = -bits.shape[-1] % 8
    b = torch.nn.functional.pad(bits, (0, pad)).reshape(*bits.shape[:-1], -1, 8)
    return (b * torch.tensor([128, 64, 32, 16, 8, 4, 2, 1], device=DEV, dtype=torch.uint8)).sum(-1).to(torch.uint8)


def _cells(c):
    """The cells of a batched case: antennas, users, carriers and modulations
    of the uneven-cells workload, drawn from the case's own cell_seed."""
    r = random.Random(c["cell_seed"])
    out = []
    for _ in range(c["count"]):
        M, S = r.choice([32, 64, 128]), r.choice([600, 1200, 3276])
        K = min(r.choice([4, 8, 16, 32]), M // 2)
        sg = 16
        out.append(dict(M=M, K=K, N={600: 1024, 1200: 2048, 3276: 4096}[S], S=S, sg=sg,
                        Qm=r.choice([2, 4, 6]), U=c["symbols"] - -(-K // sg), iq="c64",
                        snr_db=r.uniform(15.0, 25.0)))
    return out


def _equalize_inputs(c, seed):
    g = _gen(seed)
    M, K, S, sg = c["M"], c["K"], c["S"], c["sg"]
    G = -(-S // sg)
    H = _cn(g, G, M, K)
    W = torch.linalg.solve(H.mH @ H, H.mH).transpose(1, 2).contiguous()  # [G][M][K]
    x = _qam(g, c["Qm"], G, K, c["n_sym"] * sg)
    y = (H @ x).reshape(G, M, c["n_sym"], sg).permute(2, 1, 0, 3).reshape(c["n_sym"], M, G * sg)[..., :S]
    return W, (y + 0.05 * _cn(g, c["n_sym"], M, S)).contiguous()


def _downlink_inputs(c, seed):
    g = _gen(seed)
    P = _cn(g, -(-c["S"] // c["sg"]), c["K"], c["M"])
    rows, row = c["n_sym"] * c["K"], (c["S"] * c["Qm"] + 7) // 8
    bits = torch.randint(0, 256, (rows, row), generator=g, device=DEV).to(torch.uint8)
    return P / P.abs().amax((1, 2), keepdim=True), bits


def _slot_inputs(c, seed, salt=0):
    g = _gen(seed, salt)
    H = _tdl(g, c) if c["kind"] == "slot" else _iid(g, c)
    return H, _to_samples(c, _received(c, g, H, c["snr_db"], c["U"], c["Qm"]), c["iq"])


def _zf_inputs(c, seed):
    g = _gen(seed)
    return _to_samples(c, _received(c, g, _tdl(g, c), 25.0, 0, 2), c["iq"])


def _lzf_inputs(c, seed):
    g = _gen(seed)
    M, K, S, sg = c["M"], c["K"], c["S"], c["sg"]
    G = -(-S // sg)
    H = _tdl(g, c, rho=0.0, delay_ns=c["delay_ns"])
    s = (torch.arange(G, device=DEV)[:, None] * sg + torch.arange(K, device=DEV) % sg).clamp(max=S - 1)
    csi = H[s, :, torch.arange(K, device=DEV)].transpose(1, 2).conj()
    return (csi + 0.03 * _cn(g, G, M, K)).contiguous()


def _train_inputs(c, seed):
    g = _gen(seed)
    B, O = c["steps"] * c["batch"], c["n_out"]
    x = torch.rand(B, c["n_in"], generator=g, device=DEV)
    Y = _randn(g, B, O, 6)
    w = torch.eye(O, device=DEV)[1] + 0.3 * torch.tanh(x[:, :O] - 0.5)
    A = Y @ Y.mT / 6 + 0.1 * torch.eye(O, device=DEV)
    b = (A @ w[..., None])[..., 0]
    one = (b * w).sum(-1) + 0.01
    cut = [t.split(c["batch"]) for t in (x, A.contiguous(), b.contiguous(), one)]
    n = c["n_in"], c["width"], O
    r = np.random.default_rng(seed)
    p = [r.standard_normal((n[0], n[1])) * math.sqrt(2 / n[0]), np.zeros(n[1]),
         r.standard_normal((n[1], n[1])) * math.sqrt(2 / n[1]), np.zeros(n[1]),
         r.standard_normal((n[1], O)) * math.sqrt(0.1 / n[1]), np.eye(O)[1]]
    return list(zip(*cut)), [a.astype(np.float32) for a in p]


def _ldpc_inputs(c, seed):
    g = _gen(seed)
    info = torch.randint(0, 2, (c["batch"], c["kb"], c["Z"]), generator=g, device=DEV, dtype=torch.uint8)
    if c["kind"] == "ldpc_encode":
        return _pack(info.flatten(1))
    x = _encode(c, info).flatten(1)
    sigma = 0.9
    llr = 2 / sigma ** 2 * (1 - 2.0 * x + sigma * _randn(g, *x.shape))
    llr[:, :2 * c["Z"]] = 0
    return llr.half()


def prepare(case, seed):
    c, k = case, case["kind"]
    if k == "fft":
        g = _gen(seed)
        st = dict(c=c, iq=_to_samples(c, _cn(g, c["n_sym"], c["M"], c["S"]) * 4, c["iq"]),
                  op=ops.UplinkFFT((c["N"] - c["S"]) // 2, c["N"], c["S"], c["M"]))
        if c["out"] == "bf16":
            st["out"] = torch.zeros(c["n_sym"], 2, c["M"], -(-c["S"] // 8) * 8, dtype=torch.bfloat16, device=DEV)
        else:
            st["out"] = torch.zeros(c["n_sym"], c["M"], c["S"], dtype=torch.complex64, device=DEV)
        return st
    if k == "zf":
        G = -(-c["S"] // c["sg"])
        return dict(c=c, iq=_zf_inputs(c, seed), csi=torch.zeros(G, c["M"], c["K"], dtype=torch.complex64, device=DEV),
                    P=torch.zeros(G, c["K"], c["M"], dtype=torch.complex64, device=DEV) if c["precoder"] else None,
                    status=torch.zeros(G, dtype=torch.int32, device=DEV),
                    pilot=ops.PilotFFT((c["N"] - c["S"]) // 2, c["N"], c["S"], c["M"], c["K"], c["sg"]),
                    zf=ops.Beamform(c["M"], c["K"], G, precision=PRECISION[c["precision"]]))
    if k == "equalize":
        W, y = _equalize_inputs(c, seed)
        n = c["S"] * c["Qm"]
        return dict(c=c, W=W, y=y, scr=ops.Scrambler(num_bits=n),
                    llr=torch.zeros(c["n_sym"], c["K"], n, dtype=torch.float16, device=DEV),
                    hard=torch.zeros(c["n_sym"], c["K"], (n + 7) // 8, dtype=torch.uint8, device=DEV))
    if k == "downlink":
        M, K, N, S, D = c["M"], c["K"], c["N"], c["S"], c["n_sym"]
        P, bits = _downlink_inputs(c, seed)
        st = dict(c=c, P=P, bits=bits, sym=torch.zeros(D * K, S, dtype=torch.complex64, device=DEV),
                  ifft=ops.DownlinkIFFT((N - S) // 2, N, S, M),
                  out=torch.zeros(D, M, N, 2, dtype=IQ_TORCH[c["out"]], device=DEV))
        if c["precision"] == "mixed":
            st["z"] = torch.zeros(D, M, N, 2, dtype=torch.float16, device=DEV)
            n = _lib.U64()
            _lib.check(_lib.LIB.mb_precode_tc_scratch(M, K, S, c["sg"], n), "mb_precode_tc_scratch")
            st["scratch"] = torch.empty(n.value, dtype=torch.uint8, device=DEV)
        else:
            st["z"] = torch.zeros(D, M, N, dtype=torch.complex64, device=DEV)
        return st
    if k.startswith("ldpc"):
        code = ops.Ldpc(_graph(c), c["kb"], c["Z"], c["rows"], max_batch=c["batch"])
        cols = code.info_bytes if k == "ldpc_decode" else (code.cw_bits + 7) // 8
        return dict(c=c, code=code, inp=_ldpc_inputs(c, seed),
                    out=torch.zeros(c["batch"], cols, dtype=torch.uint8, device=DEV))
    if k == "lzf":
        return dict(c=c, csi=_lzf_inputs(c, seed), lzf=learned.LearnedZF(c["M"], c["K"], c["S"], c["sg"]),
                    net=_blend_net(c["sg"]),
                    W=torch.zeros(c["S"], c["M"], c["K"], dtype=torch.complex64, device=DEV))
    if k == "train":
        data, p = _train_inputs(c, seed)
        net = learned.MLP(c["n_in"], c["width"], c["n_out"], max_batch=c["batch"])
        net.set_params(np.concatenate([a.ravel() for a in p]))
        return dict(c=c, data=data, net=net, loss=torch.zeros(1, device=DEV))
    if k == "slot":
        H, iq = _slot_inputs(c, seed)
        run_ = slot.UplinkSlot(_cell_config(c), precision=c["precision"], sym_batch=c["sym_batch"],
                               use_graph=c["graph"])
        if c["learned"]:
            run_.set_zf_init(_start_net(H, c["sg"]))
        return dict(c=c, slot=run_, iq=iq, stream=torch.cuda.Stream())
    cs = _cells(c)
    return dict(c=c, cells=cells.Cells([_cell_config(d) for d in cs]), stream=torch.cuda.Stream(),
                iq=[_slot_inputs(dict(d, kind="cells"), seed, 7919 * (i + 1))[1] for i, d in enumerate(cs)])


# ---------------------------------------------------------------- run ----
def run(state):
    st, c = state, state["c"]
    k = c["kind"]
    if k == "fft":
        if c["out"] == "c64":
            st["op"](st["iq"], st["out"])
            return st["out"]
        st["op"].uplink_bf16(st["iq"], st["out"], st["out"].shape[-1])
        return st["out"][..., :c["S"]]  # the columns past S are padding
    if k == "zf":
        (st["pilot"] if c["precision"] == "fp32" else st["pilot"].mixed)(st["iq"], st["csi"])
        st["zf"].beamform_uplink(st["csi"], c["S"], c["sg"], status=st["status"])
        if c["precoder"]:
            ops.Beamform.beamform_downlink(st["csi"], st["P"])
        return {"W": st["csi"], "P": st["P"], "status": st["status"]}
    if k == "equalize":
        f = ops.Equalize.equalize if c["precision"] == "fp32" else ops.Equalize.equalize_tc
        f(st["W"], st["y"], st["llr"], c["sg"], c["Qm"], c["S"] * c["Qm"], 0, hard=st["hard"], scrambler=st["scr"])
        return {"llr": st["llr"], "hard": st["hard"]}
    if k == "downlink":
        M, K, N, S, D = c["M"], c["K"], c["N"], c["S"], c["n_sym"]
        ops.Modulation.modulate(st["bits"], st["sym"], c["Qm"])
        sym = st["sym"].view(D, K, S)
        if c["precision"] == "mixed":
            ops.Precode.precode_tc(st["P"], sym, st["z"], c["sg"], (N - S) // 2, scratch=st["scratch"])
            st["ifft"].mixed(st["z"], st["out"])
        else:
            ops.Precode.precode(st["P"], sym, st["z"], c["sg"], (N - S) // 2)
            st["ifft"](st["z"], st["out"])
        return {"spectra": st["z"], "samples": st["out"]}
    if k == "ldpc_encode":
        return st["code"].encode(st["inp"], out=st["out"])
    if k == "ldpc_decode":
        return st["code"].decode(st["inp"], max_iter=c["iters"], out=st["out"])
    if k == "lzf":
        return st["lzf"].run(st["csi"], learned.LEARNED, c["iters"], mlp=st["net"], W=st["W"])
    if k == "train":
        for x, A, b, one in st["data"]:
            st["net"].loss_grad(x, A, b, one, loss=st["loss"])
            st["net"].adam_step(1e-3)
        return {"loss": st["loss"], "grads": st["net"].grads(), "params": st["net"].params()}
    if k == "slot":
        llr, hard = st["slot"](st["iq"], stream=st["stream"])
        return {"llr": llr, "hard": hard}
    llr, hard = st["cells"](st["iq"], stream=st["stream"])
    return {"llr": llr, "hard": hard}


# ------------------------------------------------- work and tolerances ----
def _slot_work(c):
    M, K, N, S, sg, Qm, U = (c[n] for n in ("M", "K", "N", "S", "sg", "Qm", "U"))
    P, G = -(-K // sg), -(-S // sg)
    cb, _, stride = _cell_config(c).ldpc()
    n = min(S * Qm, cb)
    byt = (P + U) * M * N * IQ_BYTES[c["iq"]] + U * K * (2 * n + n / 8)
    return byt, (P + U) * M * 5 * N * math.log2(N) + G * _zf_flops(M, K) + U * S * 8 * M * K


def _zf_flops(M, K):
    """Hermitian Gram, Cholesky factor, two triangular solves of M columns."""
    return 4 * K * K * M + 4 / 3 * K ** 3 + 8 * K * K * M


def work(case):
    c, k = case, case["kind"]
    if k == "fft":
        rows = c["n_sym"] * c["M"]
        return dict(bytes=rows * (c["N"] * IQ_BYTES[c["iq"]] + c["S"] * (8 if c["out"] == "c64" else 4)),
                    flops=rows * 5 * c["N"] * math.log2(c["N"]))
    if k == "zf":
        M, K = c["M"], c["K"]
        P, G = -(-K // c["sg"]), -(-c["S"] // c["sg"])
        return dict(bytes=P * M * c["N"] * IQ_BYTES[c["iq"]] + G * M * K * 8 * (1 + c["precoder"]),
                    flops=P * M * 5 * c["N"] * math.log2(c["N"]) + G * _zf_flops(M, K))
    if k == "equalize":
        M, K, S, L = c["M"], c["K"], c["S"], c["n_sym"]
        return dict(bytes=8 * (-(-S // c["sg"]) * M * K + L * M * S) + L * K * S * c["Qm"] * (2 + 1 / 8),
                    flops=8 * M * K * S * L)
    if k == "downlink":
        M, K, N, S, D = c["M"], c["K"], c["N"], c["S"], c["n_sym"]
        z = 4 if c["precision"] == "mixed" else 8
        return dict(bytes=D * K * S * c["Qm"] / 8 + 8 * -(-S // c["sg"]) * M * K + D * M * N * (z + 4),
                    flops=8 * M * K * S * D + D * M * 5 * N * math.log2(N))
    if k == "ldpc_decode":
        e = len(_graph(c))
        return dict(bytes=c["batch"] * c["Z"] * (2 * (c["kb"] + c["rows"]) + c["kb"] / 8),
                    flops=6.0 * e * c["Z"] * c["batch"] * c["iters"])
    if k == "ldpc_encode":
        return dict(bytes=c["batch"] * c["Z"] * (2 * c["kb"] - 2 + c["rows"]) / 8,
                    flops=len(_graph(c)) * c["Z"] * c["batch"] / 32)
    if k == "lzf":
        M, K, S = c["M"], c["K"], c["S"]
        return dict(bytes=8 * M * K * (-(-S // c["sg"]) + S),
                    flops=S * (4 * K * K * M + c["iters"] * 16 * K ** 3 + 8 * K * K * M + 8 * M * K))
    if k == "train":
        n = c["n_in"] * c["width"] + c["width"] ** 2 + c["width"] * c["n_out"]
        return dict(bytes=c["steps"] * (4 * c["batch"] * (c["n_in"] + c["n_out"] ** 2 + c["n_out"] + 1) + 28 * n),
                    flops=c["steps"] * c["batch"] * 6 * n)
    w = [_slot_work(d) for d in (_cells(c) if k == "cells" else [c])]
    return dict(bytes=sum(a for a, _ in w), flops=sum(b for _, b in w))


def tolerance(case):
    """About four times what two correct forms differ by: measured against
    64 bits, FP32 paths are 1e-7 to 4e-7 off, FP16 LLRs 3e-4 (their own
    rounding), BF16 operands 1.4e-3 in one product and 3e-3 to 7e-3 through
    FFT, inverse and product, the network's gradients 1e-2 to 4e-2 (BF16
    operands and eight updates on the way)."""
    c, k = case, case["kind"]
    if k.startswith("ldpc"):
        return "exact"
    if k == "fft":
        return {"rel": 1e-6} if c["out"] == "c64" else {"rel": 8e-3, "max": 0.05}
    if k == "zf":  # the inverse's condition on top
        return {"rel": 2e-5, "max": 2e-3} if c["precision"] == "fp32" else {"rel": 2e-2, "max": 0.5}
    if k == "equalize":  # hard bits differ where an LLR is next to zero
        return {"rel": 1e-3, "max": 0.02, "differ": 1e-3} if c["precision"] == "fp32" else \
            {"rel": 6e-3, "max": 0.1, "differ": 1e-2}
    if k == "downlink":  # int16 samples differ where a value is next to a half
        if c["precision"] == "mixed":
            return {"rel": 1e-2, "max": 0.1, "differ": 1e-2}
        return {"rel": 1e-6 if c["out"] == "int16" else 1e-3, "max": 0.02, "differ": 5e-3}
    if k == "lzf":
        return {"rel": 6e-5, "max": 6e-3}
    if k == "train":
        return {"rel": 2e-2, "max": 0.5}
    mixed = k == "cells" or c["precision"] == "mixed"
    return {"rel": 2e-2, "max": 0.5, "differ": 1e-2} if mixed else {"rel": 1e-3, "max": 0.05, "differ": 2e-3}


# --------------------------------------------------------------- exact ----
def _as_c128(iq):
    if iq.is_complex():
        return iq.to(torch.complex128)
    full = {torch.int16: 32768.0, torch.int8: 128.0, torch.float16: 1.0}[iq.dtype]
    return torch.view_as_complex(iq.double() / full)


def _fft64(c, iq):
    return torch.fft.fft(_as_c128(iq))[..., _bins(c["N"], c["S"])]


def _detector64(c, X):
    """W [G][M][K] from the pilot symbols' subcarriers X [P][M][S]."""
    M, K, S, sg = c["M"], c["K"], c["S"], c["sg"]
    G = -(-S // sg)
    pil = _pilots(S).to(torch.complex128)
    est = X.conj() * (pil / pil.abs().square())
    est = torch.nn.functional.pad(est, (0, G * sg - S)).reshape(-1, M, G, sg)  # [P][M][G][sg]
    csi = est.permute(2, 1, 0, 3).reshape(G, M, -1)[..., :K].clone()
    if S % sg and G > 1:
        gone = torch.arange(K, device=DEV) % sg >= S % sg
        csi[-1][:, gone] = csi[-2][:, gone]
    C = csi.transpose(1, 2)
    return torch.linalg.solve(C @ C.mH, C).transpose(1, 2)


def _equalize64(c, W, y):
    """x [sym][K][S] = sum over antennas of W[group] y."""
    G, M, K = W.shape
    L, S, sg = y.shape[0], c["S"], c["sg"]
    Y = torch.nn.functional.pad(y, (0, G * sg - S)).reshape(L, M, G, sg).permute(2, 1, 0, 3).reshape(G, M, L * sg)
    x = (W.transpose(1, 2) @ Y).reshape(G, K, L, sg)
    return x.permute(2, 1, 0, 3).reshape(L, K, G * sg)[..., :S]


def _demap64(x, Qm):
    """Max-log LLRs [sym][K][S Qm] of the library's scale (100 a unit of amplitude)."""
    v = torch.view_as_real(x)
    if Qm == 2:
        return (-20 * math.sqrt(2) * v).flatten(-2)
    levels, unit = [100 * v], 100 / math.sqrt({4: 10, 6: 42, 8: 170}[Qm])
    for i in range(Qm // 2 - 1, 0, -1):
        levels.append(2 ** i * unit - levels[-1].abs())
    return torch.stack(levels, -2).reshape(*x.shape[:-1], -1)


def _slot64(c, iq):
    X = _fft64(c, iq)
    P = -(-c["K"] // c["sg"])
    llr = _demap64(_equalize64(c, _detector64(c, X[:P]), X[P:]), c["Qm"])
    cb, zeros, stride = _cell_config(c).ldpc()
    n = min(c["S"] * c["Qm"], cb)
    return torch.nn.functional.pad(llr[..., :n], (zeros, stride - zeros - n))


def _map64(bits, S, Qm):
    """QAM symbols [rows][S] of packed rows, bit t of a row bit t % 8 of byte
    t / 8 and the first of a symbol's bits its index's most significant."""
    b = ((bits[..., None].long() >> torch.arange(8, device=DEV)) & 1).flatten(-2)[..., :S * Qm].reshape(-1, S, Qm)
    v = {2: [-1, 1], 4: [1, 3, -1, -3], 6: [3, 1, 5, 7, -3, -1, -5, -7],
         8: [-15, -13, -9, -11, -1, -3, -7, -5, 15, 13, 9, 11, 1, 3, 7, 5]}[Qm]
    v = torch.tensor(v, device=DEV, dtype=torch.float64) / math.sqrt({2: 2, 4: 10, 6: 42, 8: 170}[Qm])
    w = 2 ** torch.arange(Qm // 2 - 1, -1, -1, device=DEV)
    return torch.complex(v[(b[..., 0::2] * w).sum(-1)], v[(b[..., 1::2] * w).sum(-1)])


def _train64(c, seed):
    data, p = _train_inputs(c, seed)
    p = [torch.from_numpy(a).to(DEV).double().requires_grad_() for a in p]
    m, v = ([torch.zeros_like(a) for a in p] for _ in range(2))
    for t, (x, A, b, one) in enumerate(data, 1):
        x, A, b, one = x.double(), A.double(), b.double(), one.double()
        y = torch.relu(torch.relu(x @ p[0] + p[1]) @ p[2] + p[3]) @ p[4] + p[5]
        loss = ((y * (A @ y[..., None])[..., 0]).sum(-1) - 2 * (b * y).sum(-1) + one).mean()
        g = torch.autograd.grad(loss, p)
        with torch.no_grad():
            for i in range(6):
                m[i] = 0.9 * m[i] + 0.1 * g[i]
                v[i] = 0.999 * v[i] + 0.001 * g[i] ** 2
                p[i] -= 1e-3 * (m[i] / (1 - 0.9 ** t)) / ((v[i] / (1 - 0.999 ** t)).sqrt() + 1e-8)
    flat = [torch.cat([a.detach().flatten() for a in q]).cpu().numpy() for q in (g, p)]
    return {"loss": loss.detach().reshape(1), "grads": flat[0], "params": flat[1]}


def _lzf64(c, seed):
    csi = _lzf_inputs(c, seed).to(torch.complex128)
    G, M, K = csi.shape
    S, sg = c["S"], c["sg"]
    at = (torch.arange(S, device=DEV).double()[:, None] - torch.arange(K, device=DEV) % sg) / sg  # [S][K]
    g0 = at.floor().clamp(0, max(G - 2, 0)).long()
    t = (at - g0).clamp(0, 1)[:, None] if G > 1 else torch.zeros(1, device=DEV)
    u = torch.arange(K, device=DEV)
    a, b = (csi[i, :, u].transpose(1, 2) for i in (g0, (g0 + 1).clamp(max=G - 1)))
    C = ((1 - t) * a + t * b).transpose(1, 2)
    return torch.linalg.solve(C @ C.mH, C).transpose(1, 2)


def exact(case, seed):
    c, k = case, case["kind"]
    if k.startswith("ldpc"):
        return None
    if k == "fft":
        g = _gen(seed)
        X = _fft64(c, _to_samples(c, _cn(g, c["n_sym"], c["M"], c["S"]) * 4, c["iq"]))
        return X if c["out"] == "c64" else torch.stack([X.real, X.imag], 1)
    if k == "zf":
        W = _detector64(c, _fft64(c, _zf_inputs(c, seed)))
        P = W.transpose(1, 2) / W.abs().amax((1, 2))[:, None, None] if c["precoder"] else None
        return {"W": W, "P": P, "status": None}
    if k == "equalize":
        W, y = _equalize_inputs(c, seed)
        return {"llr": _demap64(_equalize64(c, W.to(torch.complex128), y.to(torch.complex128)), c["Qm"]),
                "hard": None}
    if k == "downlink":
        P, bits = _downlink_inputs(c, seed)
        D, K, N = c["n_sym"], c["K"], c["N"]
        s = _map64(bits, c["S"], c["Qm"]).reshape(D, K, c["S"])
        z = torch.zeros(D, c["M"], N, dtype=torch.complex128, device=DEV)
        # precoding is the equalizer's contraction with users in place of antennas
        z[..., _bins(N, c["S"])] = _equalize64(dict(c, M=K), P.to(torch.complex128), s)
        out = torch.view_as_real(torch.fft.ifft(z)) if c["out"] == "f16" else None
        return {"spectra": torch.view_as_real(z) if c["precision"] == "mixed" else z, "samples": out}
    if k == "lzf":
        return _lzf64(c, seed)
    if k == "train":
        return _train64(c, seed)
    if k == "slot":
        return {"llr": _slot64(c, _slot_inputs(c, seed)[1]), "hard": None}
    cs = _cells(c)
    return {"llr": [_slot64(d, _slot_inputs(dict(d, kind="cells"), seed, 7919 * (i + 1))[1])
                    for i, d in enumerate(cs)], "hard": [None] * len(cs)}
