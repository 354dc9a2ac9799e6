"""GPU tests of the tensor-core (tcgen05 kind::i8) twiddle products used at
large precision (35..260 limbs, P from about 1050 to 8200 bits at N = 1024).

The product is checked bit for bit against its integer definition (byte
columns >= J0 of |x|*w, rounded at bit 32L-1), and the transforms that use it
against the 2P-bit MPFR DFT and against the integer-pipe streaming kernels.
"""
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MPFR_T = 32


@pytest.fixture(scope="module")
def M():
    import mpfft_b200

    return mpfft_b200


def _tc_expected(x: int, w: int, L: int) -> int:
    """sign(x) * floor((S + 2^(32L-2)) / 2^(32L-1)), S = the byte columns
    j >= J0 = (4L-8) rounded down to 16 of |x|*w."""
    j0 = (4 * L - 8) & ~15
    a = abs(x)
    full = a * w
    low = 0
    for i in range(j0):  # partial products x_i * w_c with i + c < j0
        xi = (a >> (8 * i)) & 0xFF
        if xi:
            low += (xi * (w & ((1 << (8 * (j0 - i))) - 1))) << (8 * i)
    r = (full - low + (1 << (32 * L - 2))) >> (32 * L - 1)
    return -r if x < 0 else r


def _to_planes(vals, L):
    B = len(vals)
    out = np.zeros((L, B), dtype=np.uint32)
    for b, v in enumerate(vals):
        u = v % (1 << (32 * L))
        for i in range(L):
            out[i, b] = (u >> (32 * i)) & 0xFFFFFFFF
    return out


def _from_planes(planes):
    L, B = planes.shape
    vals = []
    for b in range(B):
        u = 0
        for i in range(L):
            u |= int(planes[i, b]) << (32 * i)
        if u >> (32 * L - 1):
            u -= 1 << (32 * L)
        vals.append(u)
    return vals


@pytest.mark.parametrize("L,B", [(35, 128), (41, 77), (64, 128), (65, 1), (65, 300), (100, 129), (129, 256), (257, 130), (260, 64)])
def test_tc_product_bit_exact(M, L, B):
    import torch

    rng = random.Random(1000 * L + B)
    xs = [rng.randrange(-(1 << (32 * L - 2)) + 1, 1 << (32 * L - 2)) for _ in range(B)]
    xs[0] = (1 << (32 * L - 2)) - 1  # largest magnitude
    if B > 2:
        xs[1], xs[2] = 0, -((1 << (32 * L - 2)) - 1)
    w = rng.randrange(0, 1 << (32 * L))
    wl = np.array([(w >> (32 * i)) & 0xFFFFFFFF for i in range(L)], dtype=np.uint32)
    d_x = torch.from_numpy(_to_planes(xs, L).view(np.int32)).cuda()
    d_w = torch.from_numpy(wl.view(np.int32)).cuda()
    d_o = torch.full((L, B), 7, dtype=torch.int32, device="cuda")
    M.tc_mul(L, B, d_x.data_ptr(), d_w.data_ptr(), d_o.data_ptr())
    torch.cuda.synchronize()
    M.tc_error()
    got = _from_planes(d_o.cpu().numpy().view(np.uint32))
    for b in range(B):
        assert got[b] == _tc_expected(xs[b], w, L), b
        # within one unit of the correctly rounded full product
        full = (abs(xs[b]) * w + (1 << (32 * L - 2))) >> (32 * L - 1)
        assert abs(abs(got[b]) - full) <= 1


@pytest.mark.parametrize("n,p,batch", [(128, 1200, 40), (256, 2048, 1), (64, 2048, 130), (32, 4096, 3), (16, 8192, 2)])
def test_tc_transform_matches_oracle_and_integer_path(M, orc, n, p, batch):
    O = orc
    L = O.lib()
    tc = M.MpPlan(n, p)
    assert 35 <= tc.limbs <= 260
    xr, xi = O.mp_pair(n * batch, p)
    O.fill_uniform(xr, xi, 31 + p)
    yr, yi = O.mp_pair(n * batch, p)
    tc.execute(batch, xr.ptr, xi.ptr, yr.ptr, yi.ptr)
    zr, zi = O.mp_pair(n * batch, p)
    M.MpPlan(n, p, tensor=False).execute(batch, xr.ptr, xi.ptr, zr.ptr, zi.ptr)
    bound = O.mp_bound_log2(n, p)
    for b in sorted({0, batch - 1}):
        sl = lambda a, pr=p: _slice(O, a, b * n, n, pr)
        sr, si = sl(xr), sl(xi)
        dr, di = O.mp_pair(n, 2 * p)
        O.mp_dft(sr, si, dr, di)
        e_tc = O.mp_errors(sl(yr), sl(yi), dr, di)["log2_rel"]
        e_int = O.mp_errors(sl(zr), sl(zi), dr, di)["log2_rel"]
        rr, ri = O.mp_pair(n, p)
        O.MpFFT(n, p)(sr, si, rr, ri)
        e_ref = O.mp_errors(rr, ri, dr, di)["log2_rel"]
        assert e_tc <= bound and e_tc <= e_ref + 0.5, (e_tc, e_ref, bound)
        assert abs(e_tc - e_int) <= 1.0, (e_tc, e_int)


def _slice(O, a, start, count, prec):
    out = O.MpArray(count, prec)
    O.lib().orc_mp_copy(out.ptr, a.ptr + start * MPFR_T, count)
    return out


@pytest.mark.parametrize("n,p,B", [(8, 1100, 1), (16, 1300, 130), (64, 1070, 257), (128, 2100, 3), (256, 4200, 129),
                                   (1024, 1600, 2), (512, 8100, 1)])
def test_tc_items_match_one_launch_per_level(M, n, p, B):
    """The persistent launch, whose items wait for the three items they need,
    against one launch per level (the timed call): the same bits, for one and
    several signal groups and every level order from one level up."""
    import torch

    from mpfft_b200.mparray import synthetic_planes

    plan = M.MpPlan(n, p)
    host = synthetic_planes(n, plan.limbs, plan.frac_bits, B, seed=n + B)
    s = torch.cuda.current_stream().cuda_stream
    d_in = torch.from_numpy(host.view(np.int32)).cuda()
    a, b = torch.full_like(d_in, -1), torch.full_like(d_in, -1)
    for _ in range(3):
        plan.execute_device(B, d_in.data_ptr(), a.data_ptr(), s)
        plan.execute_device_timed(B, d_in.data_ptr(), b.data_ptr(), s)
        assert torch.equal(a, b)
    M.tc_error()


def test_tc_segment_carries(M):
    """Operands whose carries and signs run through whole segments: zeros,
    powers of two, all ones, one limb of ones between zeros."""
    import torch

    for L in (35, 36, 41, 64, 129, 257):
        full = (1 << (32 * L - 2)) - 1
        xs = [0, 1, -1, full, -full, 1 << (16 * L), -(1 << (16 * L)), (1 << (16 * L)) - 1, -((1 << (16 * L)) - 1),
              0xFFFFFFFF << 64, -(0xFFFFFFFF << 64), full ^ 0xFFFFFFFF, -(full ^ ((1 << (32 * (L // 2))) - 1))]
        for w in ((1 << (32 * L)) - 1, 1 << (32 * L - 1), (1 << (32 * L - 1)) - 1):
            x = torch.from_numpy(_to_planes(xs, L).view(np.int32)).cuda()
            d_w = torch.from_numpy(_to_planes([w], L).view(np.int32)).cuda()
            y = torch.zeros_like(x)
            M.tc_mul(L, len(xs), x.data_ptr(), d_w.data_ptr(), y.data_ptr(),
                     torch.cuda.current_stream().cuda_stream)
            got = _from_planes(y.cpu().numpy().view(np.uint32))
            for v, g in zip(xs, got):
                assert g == _tc_expected(v, w, L), (L, hex(v)[:20], hex(w)[:20])


@pytest.mark.parametrize("L", [8, 9, 13, 14, 17, 21, 25, 28, 29, 30, 31, 34])
@pytest.mark.parametrize("n,B", [(8, 3), (64, 1), (64, 130)])
def test_tc_forced_below_its_default_range(M, L, n, B):
    """Plans forced onto the tensor cores (one tile of byte columns up to 28 limbs
    and at 30, two at 29 and from 31) against the integer pipe: both round each
    product to within a unit of the last place.  A difference e of a level's inputs
    becomes at most (2e + 1) + (sqrt 2 e + 1) in a twiddled value, twice that in
    their sum, plus e: 8e + 4.  Signals cut from the batch have the batch's bits."""
    import torch

    from mpfft_b200.mparray import synthetic_planes

    lg = n.bit_length() - 1
    plan = M.MpPlan(n, 32 * L - 7 - 2 * lg, tensor="force")
    ref = M.MpPlan(n, 32 * L - 7 - 2 * lg, tensor=False)
    assert plan.limbs == ref.limbs == L and plan.form() != ref.form()
    host = synthetic_planes(n, L, plan.frac_bits, B, seed=n + L).reshape(2, L, n, B)
    s = torch.cuda.current_stream().cuda_stream
    d_in = torch.from_numpy(np.ascontiguousarray(host).view(np.int32)).cuda()
    a, b = torch.full_like(d_in, -1), torch.full_like(d_in, -1)
    plan.execute_device(B, d_in.data_ptr(), a.data_ptr(), s)
    ref.execute_device(B, d_in.data_ptr(), b.data_ptr(), s)
    for i in {0, B - 1}:
        one = d_in[..., i].contiguous()
        out = torch.empty_like(one)
        plan.execute_device(1, one.data_ptr(), out.data_ptr(), s)
        assert torch.equal(out, a[..., i].contiguous()), i
    M.tc_error()
    bound = 0
    for _ in range(lg - 2):  # levels n = 8 ..
        bound = 8 * bound + 4
    ints = lambda t: np.ascontiguousarray(t.cpu().numpy().view(np.uint32).transpose(0, 2, 3, 1)).reshape(-1, L)
    top = 1 << (32 * L)
    for x, y in zip(ints(a), ints(b)):
        d = (int.from_bytes(x.tobytes(), "little") - int.from_bytes(y.tobytes(), "little")) % top
        assert min(d, top - d) <= bound, (hex(d), bound)
