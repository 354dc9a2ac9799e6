"""GPU parity tests of the FP64 path: bit-identical (0 ulp) to the reference's
double transform d_sr24_cp_fft (lab/serial/double/serial_d_fft6.c:93-429)."""
import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def M():
    import mpfft_b200

    return mpfft_b200


def _bits_equal(a, b):
    return np.array_equal(np.asarray(a).view(np.uint64), np.asarray(b).view(np.uint64))


@pytest.mark.parametrize("n", [1, 2, 4, 8, 16, 32, 64, 128, 1024, 4096, 1 << 16, 1 << 20])
def test_d_bitexact_vs_reference_restatement(M, orc, n):
    O = orc
    xr, xi = O.d_uniform(n, 100 + n)
    er, ei = O.DFFT(n)(xr, xi)
    yr, yi = np.zeros(n), np.zeros(n)
    assert M.d_sr24_cp_fft(n, 1, 0, xr, xi, yr, yi) == M.OK, M.last_error()
    assert _bits_equal(yr, er) and _bits_equal(yi, ei)


@pytest.mark.parametrize("g", load_golden("d_"), ids=lambda g: g["name"])
def test_d_bitexact_vs_reference_golden(M, g):
    xr = np.array([float.fromhex(v) for v in g["inr"]])
    xi = np.array([float.fromhex(v) for v in g["ini"]])
    er = np.array([float.fromhex(v) for v in g["outr"]])
    ei = np.array([float.fromhex(v) for v in g["outi"]])
    n = g["N"]
    yr, yi = np.zeros(n), np.zeros(n)
    assert M.d_sr24_cp_fft(n, 1, 0, xr, xi, yr, yi) == M.OK
    assert _bits_equal(yr, er) and _bits_equal(yi, ei)
    vr, vi = np.zeros(n), np.zeros(n)
    assert M.d_sr24_cp_fft_v2(n, 0, 1, 0, xr, xi, vr, vi) == M.OK
    assert _bits_equal(vr, er) and _bits_equal(vi, ei)


def test_d_scaled_and_strided(M, orc):
    O = orc
    n, s = 2048, 2
    xr, xi = O.d_uniform(n * s, 3)
    yr, yi = np.zeros(n), np.zeros(n)
    assert M.d_sr24_cp_fft(n, s, 0, xr, xi, yr, yi) == M.OK
    er, ei = O.DFFT(n)(np.ascontiguousarray(xr[::s]), np.ascontiguousarray(xi[::s]))
    assert _bits_equal(yr, er) and _bits_equal(yi, ei)
    sr, si = np.zeros(n), np.zeros(n)
    assert M.d_sr24_cp_fft_scaled(n, s, 0, xr, xi, sr, si) == M.OK
    assert _bits_equal(sr, er / n) and _bits_equal(si, ei / n)


def test_d_batched_device_api(M, orc):
    import torch

    O = orc
    n, batch = 4096, 33
    xr = np.zeros((batch, n))
    xi = np.zeros((batch, n))
    for b in range(batch):
        xr[b], xi[b] = O.d_uniform(n, 500 + b)
    plan = M.DPlan(n)
    yr, yi = np.zeros_like(xr), np.zeros_like(xi)
    plan.execute(batch, xr, xi, yr, yi)
    f = O.DFFT(n)
    for b in range(batch):
        er, ei = f(xr[b], xi[b])
        assert _bits_equal(yr[b], er) and _bits_equal(yi[b], ei)
    # device layout [c][b][p]
    d_in = torch.from_numpy(np.stack([xr, xi]).copy()).cuda()
    d_out = torch.empty_like(d_in)
    plan.execute_device(batch, d_in.data_ptr(), d_out.data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    out = d_out.cpu().numpy()
    assert _bits_equal(out[0], yr) and _bits_equal(out[1], yi)


@pytest.mark.parametrize("n", [1, 16, 1024, 65536])
def test_d_inverse_bitexact_vs_reference_procedure(M, orc, n):
    """d_sr24_cp_ifft is bit-identical to the reference's test() inverse:
    swap re/im, forward transform, swap back, divide by N
    (lab/serial/double/serial_d_fft6.c:511-524)."""
    O = orc
    xr, xi = O.d_uniform(n, 900 + n)
    fr, fi = O.DFFT(n)(xi, xr)           # forward of the swapped input
    er, ei = fi / n, fr / n              # swap back, divide by N
    yr, yi = np.zeros(n), np.zeros(n)
    assert M.d_sr24_cp_ifft(n, 1, 0, xr, xi, yr, yi) == M.OK
    assert _bits_equal(yr, er) and _bits_equal(yi, ei)
    plan = M.DPlan(n)
    zr, zi = np.zeros(n), np.zeros(n)
    plan.execute(1, xr, xi, zr, zi, scaled=True, inverse=True)
    assert _bits_equal(zr, er) and _bits_equal(zi, ei)


@pytest.mark.parametrize("n,batch", [(8, 700), (16, 129), (32, 333), (64, 65), (128, 33), (256, 301), (512, 9),
                                     (1024, 5), (2048, 3), (4096, 2), (8192, 3), (16384, 2), (32768, 1), (131072, 1),
                                     (1 << 19, 1)])
@pytest.mark.parametrize("inverse", [False, True])
def test_d_register_passes_bitexact(M, orc, n, batch, inverse):
    """Every chain of base cases and register passes (up to three levels each,
    in shared memory and above), CTAs of several signals with a partly filled
    last one, planes exchanged and scaled outputs: the same bits as the
    reference's transform (inverse: its swap procedure, lab/serial/double/
    serial_d_fft6.c:511-524)."""
    import torch

    rng = np.random.default_rng(n + batch)
    x = rng.uniform(-1, 1, (2, batch, n))
    d_in = torch.from_numpy(x).cuda()
    d_out = torch.full_like(d_in, float("nan"))
    plan = M.DPlan(n)
    plan.execute_device(batch, d_in.data_ptr(), d_out.data_ptr(), scaled=inverse, inverse=inverse,
                        stream=torch.cuda.current_stream().cuda_stream)
    y = d_out.cpu().numpy()
    f = orc.DFFT(n)
    for b in sorted({0, batch // 2, batch - 1}):
        if inverse:
            ei, er = f(x[1, b].copy(), x[0, b].copy())
            er, ei = er / n, ei / n
        else:
            er, ei = f(x[0, b].copy(), x[1, b].copy())
        assert _bits_equal(y[0, b], er) and _bits_equal(y[1, b], ei), b


@pytest.mark.parametrize("n,batch", [(1, 5000), (2, 3001), (4, 2049), (16, 331), (32, 4801), (64, 1201), (128, 2371),
                                     (256, 601), (512, 2401), (1024, 1187), (2048, 601), (8192, 75), (65536, 10),
                                     (131072, 11)])
@pytest.mark.parametrize("inverse", [False, True])
def test_d_several_signals_or_chunks_per_cta(M, orc, n, batch, inverse):
    """Batches in which a CTA takes several signals (the last CTA partly filled) or
    several chunks of one signal: every signal has the bits of its single call
    (one per CTA), and three of them those of the reference's transform."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(n + batch)
    x = 2 * torch.rand((2, batch, n), dtype=torch.float64, device="cuda", generator=gen) - 1
    y, ref = torch.full_like(x, float("nan")), torch.empty_like(x)
    plan = M.DPlan(n)
    s = torch.cuda.current_stream().cuda_stream
    plan.execute_device(batch, x.data_ptr(), y.data_ptr(), scaled=inverse, inverse=inverse, stream=s)
    for b in range(batch):
        one = x[:, b].contiguous()
        out = torch.empty_like(one)
        plan.execute_device(1, one.data_ptr(), out.data_ptr(), scaled=inverse, inverse=inverse, stream=s)
        ref[:, b] = out
    assert torch.equal(y.view(torch.int64), ref.view(torch.int64))
    h, f = x.cpu().numpy(), orc.DFFT(n)
    for b in (0, batch // 2, batch - 1):
        r, i = h[0, b].copy(), h[1, b].copy()
        if inverse:
            ei, er = f(i, r)
            er, ei = er / n, ei / n
        else:
            er, ei = f(r, i)
        assert _bits_equal(y[0, b].cpu().numpy(), er) and _bits_equal(y[1, b].cpu().numpy(), ei), b


@pytest.mark.parametrize("form,n,bytes_per_point", [("fp64", 1 << 22, 8), ("dd", 1 << 20, 16), ("qd", 1 << 19, 32),
                                                    ("ff", 1 << 21, 8)])
def test_plan_holds_its_twiddles_once(M, form, n, bytes_per_point):
    """Device memory of a plan: the twiddles of all levels (N/2 complex values of the
    form's words) and tables that do not grow with them; freed with the plan."""
    import torch

    torch.cuda.synchronize()
    make = (lambda k: M.DPlan(k)) if form == "fp64" else (lambda k: M.MultiwordPlan(k, form))
    make(64).close()
    free = torch.cuda.mem_get_info()[0]
    plan = make(n)
    held = free - torch.cuda.mem_get_info()[0]
    assert bytes_per_point * n <= held + (2 << 20) and held <= bytes_per_point * n + (6 << 20), held
    plan.close()
    assert free - torch.cuda.mem_get_info()[0] <= 2 << 20
