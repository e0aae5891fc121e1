"""Tensor-core FFT of 1- to 4-byte samples, whose CTA runs two pipelines that
take its units of two rows in turn: row counts that leave a pipeline one unit,
fewer units than its neighbour, none, or half a unit, against a 64-bit FFT.
Tolerance per output as in test_gpu_fft_tc.py: BF16 rounding (2^-8 of the
value) plus 2e-3 of the row's RMS for the FP16 operands; the inverse writes
FP16 samples (2^-11 of the value) and takes the same 2e-3."""
import pytest
import torch

pytestmark = pytest.mark.gpu
N, S = 4096, 3276


@pytest.fixture(scope="module")
def mb():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import megastation_b200 as m
    return m


# units per CTA on 148 SMs: 1 (the last half a unit), 2 (the last CTA 1), 3, 7 (odd row count)
@pytest.mark.parametrize("M,n_sym", [(5, 1), (33, 9), (199, 3), (211, 9)])
@pytest.mark.parametrize("dtype", [torch.int8, torch.int16, torch.float16])
def test_uplink_rows(mb, dtype, M, n_sym):
    g = torch.Generator(device="cuda").manual_seed(M)
    if dtype == torch.float16:
        gain = 2.0 ** torch.randint(-6, 7, (n_sym, M, 1, 1), generator=g, device="cuda")
        iq = (torch.randn(n_sym, M, N, 2, generator=g, device="cuda") * gain).to(dtype)
        full = 1.0
    else:
        full = 128.0 if dtype == torch.int8 else 32768.0
        iq = torch.randint(-int(full), int(full), (n_sym, M, N, 2), generator=g, device="cuda").to(dtype)
    start, pitch = (N - S) // 2, (S + 7) // 8 * 8
    out = torch.full((n_sym, 2, M, pitch), 7.0, dtype=torch.bfloat16, device="cuda")
    mb.UplinkFFT(start, N, S, M).uplink_bf16(iq, out, pitch)
    torch.cuda.synchronize()
    assert mb.ops.device_error() == 0
    bins = (torch.arange(S, device="cuda") + start + N // 2) % N
    ref = torch.fft.fft(torch.view_as_complex(iq.double() / full))[..., bins]
    o = out.double()
    got = torch.complex(o[:, 0, :, :S], o[:, 1, :, :S])
    rms = ref.abs().square().mean(-1, keepdim=True).sqrt()
    assert ((got - ref).abs() <= 2.0 ** -8 * ref.abs() + 2e-3 * rms).all()


@pytest.mark.parametrize("M,D", [(1, 1), (33, 9), (199, 3)])
def test_inverse_rows(mb, M, D):
    g = torch.Generator(device="cuda").manual_seed(M)
    gain = 2.0 ** torch.randint(-3, 4, (D, M, 1, 1), generator=g, device="cuda")
    z = (torch.randn(D, M, N, 2, generator=g, device="cuda") * gain).half()
    out = torch.zeros(D, M, N, 2, dtype=torch.float16, device="cuda")
    mb.DownlinkIFFT((N - S) // 2, N, S, M).mixed(z, out)
    torch.cuda.synchronize()
    assert mb.ops.device_error() == 0
    ref = torch.fft.ifft(torch.view_as_complex(z.double()))
    got = torch.view_as_complex(out.double())
    rms = ref.abs().square().mean(-1, keepdim=True).sqrt()
    assert ((got - ref).abs() <= 2.0 ** -10 * ref.abs() + 2e-3 * rms).all()


# one unit a CTA and three of 4-byte samples take one pipeline, the others two
@pytest.mark.parametrize("M,P", [(5, 1), (37, 8), (33, 9), (199, 3), (211, 5)])
@pytest.mark.parametrize("dtype", [torch.int8, torch.int16, torch.float16])
def test_pilot_rows(mb, dtype, M, P):
    """The LS estimates against the FP32 operator's: 2e-3 of the rows' RMS
    (FP16 operands; the pilots have unit modulus, the rows one power)."""
    sg, g = 16, torch.Generator(device="cuda").manual_seed(M + P)
    full = {torch.int8: 128, torch.int16: 32768}.get(dtype)
    iq = torch.randint(-full, full, (P, M, N, 2), generator=g, device="cuda").to(dtype) if full else \
        torch.randn(P, M, N, 2, generator=g, device="cuda").to(dtype)
    op = mb.PilotFFT((N - S) // 2, N, S, M, sg * P, sg)
    ref, got = (torch.zeros(-(-S // sg), M, sg * P, dtype=torch.complex64, device="cuda") for _ in range(2))
    op(iq, ref)
    op.mixed(iq, got)
    torch.cuda.synchronize()
    assert mb.ops.device_error() == 0
    rms = ref.abs().square().mean().sqrt()  # within 10% of each row's
    assert float(rms) > 0 and float((got - ref).abs().max()) <= 2e-3 * float(rms) * 1.1
