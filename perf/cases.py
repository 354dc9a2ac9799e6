"""The transforms that users of mpfft_b200 run, as performance cases.

A case is a dict of plain values; `kind` names the entry point:

* ``dropin``   one signal in host mpfr_t arrays through ``mp_sr24_cp_fft``
* ``host``     a batch in host mpfr_t arrays through ``MpPlan.execute``
* ``mp``       a batch of device limb planes through ``MpPlan.execute_device``
* ``fp64``     a batch of device double planes through ``DPlan.execute_device``
* ``tier``     the same for a compensated tier through ``MultiwordPlan``
* ``adjoint``  double-double forward and backward pass through ``autograd.dd_fft``
* ``uneven``   signals of many lengths and precisions through ``BatchPlan``

``listed()`` holds the named cases, ``draw(rng)`` one more of the same ranges.
``prepare`` makes what a program holds before the call, ``run`` is one pass,
``work`` the bytes and operations the pass cannot do without, and ``exact`` the
result in 64-bit arithmetic where the outputs are floating-point numbers (limb
planes and mpfr_t fields are whole numbers).
"""
import math

import numpy as np
import torch

import mpfft_b200 as M
from mpfft_b200 import autograd as AG

TIERS = {"ff": (2, torch.float32), "dd": (2, torch.float64), "qd": (4, torch.float64)}


def listed():
    return [
        # the reference's calling pattern: one signal per call, host mpfr_t arrays in and out
        {"name": "dropin_1024_256b", "kind": "dropin", "n": 1024, "prec": 256, "batch": 1},
        # the same arrays in a batch, converted, transformed and rounded back in one call
        {"name": "host_1024_1024b_x256", "kind": "host", "n": 1024, "prec": 1024, "batch": 256},
        # one signal that stays on the device: launches and latency
        {"name": "mp_1024_1024b_x1", "kind": "mp", "n": 1024, "prec": 1024, "batch": 1},
        # the precision sweep's batch at a moderate precision
        {"name": "mp_1024_256b_x256", "kind": "mp", "n": 1024, "prec": 256, "batch": 256},
        # throughput: the batch of the benchmark
        {"name": "mp_1024_1024b_x2048", "kind": "mp", "n": 1024, "prec": 1024, "batch": 2048},
        # a ragged batch of longer signals at a precision between the usual ones
        {"name": "mp_4096_600b_x37", "kind": "mp", "n": 4096, "prec": 600, "batch": 37},
        # large precision: twiddle products on the tensor cores
        {"name": "mp_1024_4096b_x256", "kind": "mp", "n": 1024, "prec": 4096, "batch": 256},
        # FP64 batch, one shared-memory sub-transform per signal
        {"name": "fp64_4096_x4096", "kind": "fp64", "n": 4096, "batch": 4096, "inverse": False, "scaled": False},
        # one long FP64 signal, normalised inverse: levels above the sub-transforms
        {"name": "fp64_1m_x1_inverse", "kind": "fp64", "n": 1 << 20, "batch": 1, "inverse": True, "scaled": True},
        # training through the double-double transform: forward and adjoint
        {"name": "dd_adjoint_65536_x64", "kind": "adjoint", "n": 65536, "batch": 64},
        # quad-double batch
        {"name": "qd_4096_x512", "kind": "tier", "tier": "qd", "n": 4096, "batch": 512, "inverse": False,
         "scaled": False},
        # signals of every length and precision class in one launch
        {"name": "uneven_2000", "kind": "uneven", "count": 2000, "lg_max": 16},
    ]


def _log_int(rng, lo, hi):
    """Log-uniform integer in [lo, hi]."""
    return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(["dropin", "host", "mp", "mp", "mp", "mp", "large", "large", "fp64", "fp64", "tier", "tier",
                       "adjoint", "uneven"])
    if kind == "dropin":
        return {"kind": kind, "n": 1 << rng.randint(4, 12), "prec": _log_int(rng, 53, 1024), "batch": 1}
    if kind == "host":
        n, prec = 1 << rng.randint(6, 12), _log_int(rng, 53, 1024)
        return {"kind": kind, "n": n, "prec": prec, "batch": _log_int(rng, 2, max(2, 256 * 1024 // n))}
    if kind == "mp":
        n, prec = 1 << rng.randint(5, 14), _log_int(rng, 53, 1024)
        return {"kind": kind, "n": n, "prec": prec, "batch": _log_int(rng, 1, max(1, 2048 * 1024 // n // 2))}
    if kind == "large":
        n, prec = 1 << rng.randint(6, 11), _log_int(rng, 1100, 8100)
        most = max(1, int(256 * (1024 / n) * min(1.0, 4096 / prec) ** 2))
        return {"kind": "mp", "n": n, "prec": prec, "batch": _log_int(rng, 1, min(512, most))}
    if kind == "fp64":
        n = 1 << rng.randint(6, 20)
        return {"kind": kind, "n": n, "batch": _log_int(rng, 1, max(1, (1 << 24) // n)), "inverse": rng.random() < 0.5,
                "scaled": rng.random() < 0.5}
    if kind == "tier":
        tier, n = rng.choice(["ff", "dd", "qd"]), 1 << rng.randint(6, 17)
        return {"kind": kind, "tier": tier, "n": n, "batch": _log_int(rng, 1, max(1, (1 << 22) // n)),
                "inverse": rng.random() < 0.5, "scaled": rng.random() < 0.5}
    if kind == "adjoint":
        n = 1 << rng.randint(8, 18)
        return {"kind": kind, "n": n, "batch": _log_int(rng, 1, max(1, (1 << 22) // n))}
    return {"kind": "uneven", "count": _log_int(rng, 50, 1500), "lg_max": rng.randint(10, 16)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

class MpfrFields:
    """n consecutive mpfr_t of precision prec whose significands are spaced as
    malloc spaces those of mpfr_init2 (an 8-byte size field in front, chunks of
    a multiple of 16 bytes).  Values: uniform in [-1, 1) at full precision, or
    zero without a generator."""

    HEAD = np.dtype([("prec", "<i8"), ("sign", "<i4"), ("pad", "<i4"), ("exp", "<i8"), ("d", "<u8")])

    def __init__(self, n, prec, rng=None):
        nl = (prec + 63) // 64
        step = (8 * nl + 8 + 8 + 15) // 16 * 2  # 64-bit words from one significand to the next
        self.words = np.zeros(n * step + 4, dtype=np.int64)
        first = 1 + (self.words.ctypes.data % 16) // 8  # significands 8 bytes off 16-byte alignment
        self.mant = np.lib.stride_tricks.as_strided(self.words[first:], (n, nl), (8 * step, 8))
        self.head = np.zeros(n, dtype=self.HEAD)
        self.head["prec"], self.head["sign"] = prec, 1
        self.head["d"] = np.uint64(self.words.ctypes.data + 8 * first) + np.arange(n, dtype=np.uint64) * np.uint64(8 * step)
        if rng is None:
            self.head["exp"] = -(1 << 63) + 1  # MPFR's exponent of zero
        else:
            self.mant[:] = rng.integers(-(1 << 63), 1 << 63, (n, nl), dtype=np.int64)
            self.mant[:, 0] &= -1 << (64 * nl - prec)
            self.mant[:, nl - 1] |= np.int64(-(1 << 63))
            self.head["exp"] = 1 - np.minimum(rng.geometric(0.5, n), 60)
            self.head["sign"] = 1 - 2 * rng.integers(0, 2, n)
        self.ptr = self.head.ctypes.data

    def fields(self):
        return [self.mant, self.head["exp"], self.head["sign"]]


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _fill_planes(planes, frac_bits, g):
    """planes: int32 (2, L, ...) limb planes; values uniform in (-1, 1) times 2^frac_bits."""
    limbs = planes.shape[1]
    planes.copy_(torch.randint(-(1 << 31), 1 << 31, planes.shape, dtype=torch.int32, device="cuda", generator=g))
    top = frac_bits - 32 * (limbs - 1)
    planes[:, limbs - 1] = torch.randint(-(1 << top), 1 << top, planes[:, limbs - 1].shape, dtype=torch.int32,
                                         device="cuda", generator=g)


def _fill_words(x, g):
    """x: (2, K, ...) tier words; leading words uniform in [-1, 1), each further word below half an ulp of the last."""
    eps = torch.finfo(x.dtype).eps
    x[:, 0] = 2 * torch.rand(x[:, 0].shape, dtype=x.dtype, device="cuda", generator=g) - 1
    for h in range(1, x.shape[1]):
        r = torch.rand(x[:, h].shape, dtype=x.dtype, device="cuda", generator=g) - 0.5
        x[:, h] = x[:, h - 1] * (0.4 * eps) * r


def _float_inputs(case, g):
    """The input (and for the adjoint the cotangent) of a floating-point case."""
    n, batch = case["n"], case["batch"]
    if case["kind"] == "fp64":
        return [2 * torch.rand((2, batch, n), dtype=torch.float64, device="cuda", generator=g) - 1]
    words, dtype = TIERS[case.get("tier", "dd")]
    xs = [torch.empty((2, words, batch, n), dtype=dtype, device="cuda")
          for _ in range(2 if case["kind"] == "adjoint" else 1)]
    for x in xs:
        _fill_words(x, g)
    return xs


class _Span:
    """An arena of a batch plan, for torch.as_tensor: the tensor keeps this
    object, and with it the plan that owns the memory, alive."""

    def __init__(self, plan, ptr, nbytes):
        self.plan = plan
        self.__cuda_array_interface__ = {"shape": (nbytes,), "typestr": "|u1", "data": (ptr, False), "version": 3}


def _uneven_signals(case):
    """Lengths log-uniform over 2^4 .. 2^lg_max, precisions from six classes; one fixed mix per size."""
    r = np.random.default_rng(1000 * case["count"] + case["lg_max"])
    ns = [1 << int(v) for v in r.integers(4, case["lg_max"] + 1, case["count"])]
    precs = sorted(int(v) for v in r.choice([24, 53, 106, 212, 512, 1024], case["count"]))
    return ns, precs


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("dropin", "host"):
        n, prec, total = case["n"], case["prec"], case["n"] * case["batch"]
        rng = np.random.default_rng(seed)
        x = [MpfrFields(total, prec, rng) for _ in range(2)]
        y = [MpfrFields(total, prec) for _ in range(2)]
        return {"case": case, "plan": M.MpPlan(n, prec) if kind == "host" else None, "x": x, "y": y}
    g = _gen(seed)
    if kind == "uneven":
        ns, precs = _uneven_signals(case)
        plan = M.BatchPlan(ns, precs, float_tiers="native")
        a, b, nbytes = plan.arenas()
        ain, aout = (torch.as_tensor(_Span(plan, p, nbytes), device="cuda") for p in (a, b))
        ain.zero_()
        aout.zero_()
        where = [plan.signal_format(i) for i in range(case["count"])]
        parts = {}  # form: (first byte, last byte); the signals of one floating form lie together
        for i, (form, words, off, size) in enumerate(where):
            if form == M.FORM_LIMBS:
                t = ain[off:off + size].view(torch.int32).view(2, words, ns[i])
                _fill_planes(t, 32 * words - 1 - (ns[i].bit_length() - 1 + 2), g)
            else:
                dtype = torch.float32 if form == M.FORM_FLOAT_FLOAT else torch.float64
                _fill_words(ain[off:off + size].view(dtype).view(2, -1, ns[i]), g)
            lo, hi = parts.get(form, (off, off + size))
            parts[form] = (min(lo, off), max(hi, off + size))
        out = []
        for form in sorted(parts):
            lo, hi = parts[form]
            dtype = {M.FORM_LIMBS: torch.int32, M.FORM_FLOAT_FLOAT: torch.float32}.get(form, torch.float64)
            out.append(aout[lo:hi].view(dtype))
        return {"case": case, "plan": plan, "in": ain, "out": out, "where": where, "parts": parts}
    n, batch = case["n"], case["batch"]
    if kind == "mp":
        plan = M.MpPlan(n, case["prec"])
        x = torch.empty((2, plan.limbs, n, batch), dtype=torch.int32, device="cuda")
        _fill_planes(x, plan.frac_bits, g)
        return {"case": case, "plan": plan, "x": x, "y": torch.empty_like(x)}
    if kind == "adjoint":  # the autograd function keeps its plans
        x, grad = _float_inputs(case, g)
        return {"case": case, "x": x.requires_grad_(), "grad": grad}
    plan = M.DPlan(n) if kind == "fp64" else M.MultiwordPlan(n, case["tier"])
    (x,) = _float_inputs(case, g)
    return {"case": case, "plan": plan, "x": x, "y": torch.empty_like(x)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "adjoint":
        y = AG.dd_fft(state["x"])
        (gx,) = torch.autograd.grad(y, state["x"], state["grad"])
        y = y.detach()
        return [y[:, 0], y[:, 1], gx[:, 0], gx[:, 1]]
    if kind == "dropin":
        (xr, xi), (yr, yi) = state["x"], state["y"]
        if M.mp_sr24_cp_fft(case["n"], 1, 0, xr.ptr, xi.ptr, yr.ptr, yi.ptr) != M.OK:
            raise RuntimeError(M.last_error()[1])
        return yr.fields() + yi.fields()
    if kind == "host":
        (xr, xi), (yr, yi) = state["x"], state["y"]
        state["plan"].execute(case["batch"], xr.ptr, xi.ptr, yr.ptr, yi.ptr)
        return yr.fields() + yi.fields()
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "uneven":
        state["plan"].execute_device(stream)
        return state["out"]
    plan, x, y = state["plan"], state["x"], state["y"]
    if kind == "mp":
        plan.execute_device(case["batch"], x.data_ptr(), y.data_ptr(), stream)
        return y
    plan.execute_device(case["batch"], x.data_ptr(), y.data_ptr(), scaled=case["scaled"], stream=stream,
                        inverse=case["inverse"])
    return y if kind == "fp64" else [y[:, 0], y[:, 1:]]


# ---------------------------------------------------------------------------
# work and exact results
# ---------------------------------------------------------------------------

def _mults(n):
    """Real multiplications of one split-radix transform with three per general twiddle product."""
    m = [0] * 64
    lg = n.bit_length() - 1
    for k in range(3, lg + 1):
        m[k] = m[k - 1] + 2 * m[k - 2] + 4 + 6 * ((1 << k) // 4 - 2)
    return m[lg]


def _limbs(n, prec):
    return max(2, -(-(prec + 2 * (n.bit_length() - 1) + 7) // 32))


def _mp_ops(n, prec):
    """Integer operations of one transform: a multiply and an add per partial product, half of them dropped."""
    return _mults(n) * _limbs(n, prec) ** 2


def work(case):
    kind = case["kind"]
    if kind == "uneven":
        nbytes = flops = 0
        for n, p in zip(*_uneven_signals(case)):
            if p > 212:
                nbytes += 16 * n * _limbs(n, p)
                flops += _mp_ops(n, p)
            else:
                per = {24: (8, 12), 53: (8, 4), 106: (16, 60), 212: (32, 330)}[p]
                nbytes += 4 * n * per[0]
                flops += per[1] * n * (n.bit_length() - 1)
        return {"bytes": nbytes, "flops": flops}
    n, batch = case["n"], case["batch"]
    lg = n.bit_length() - 1
    if kind in ("dropin", "host"):
        nl = (case["prec"] + 63) // 64
        return {"bytes": 4 * n * batch * (8 * nl + 32), "flops": batch * _mp_ops(n, case["prec"])}
    if kind == "mp":
        return {"bytes": 16 * n * batch * _limbs(n, case["prec"]), "flops": batch * _mp_ops(n, case["prec"])}
    if kind == "fp64":
        return {"bytes": 32 * n * batch, "flops": 4 * n * lg * batch}
    if kind == "adjoint":
        return {"bytes": 128 * n * batch, "flops": 2 * 60 * n * lg * batch}
    words, dtype = TIERS[case["tier"]]
    per = {"ff": 12, "dd": 60, "qd": 330}[case["tier"]]  # operations per point and level
    return {"bytes": 4 * words * torch.finfo(dtype).bits // 8 * n * batch, "flops": per * n * lg * batch}


def _dft(planes, inverse, scaled):
    """(2, B, n) real and imaginary planes -> the same of the transform, in float64."""
    z = planes[0] + 1j * planes[1]
    n = z.shape[-1]
    y = np.fft.ifft(z) * n if inverse else np.fft.fft(z)
    return np.stack((y.real, y.imag)) / (n if scaled else 1)


def _uneven_exact(state):
    """Leading words of the floating signals in 64 bits (further words zero), laid out as the output arena."""
    ain, out = state["in"].cpu(), []
    for form, (lo, hi) in sorted(state["parts"].items()):
        if form == M.FORM_LIMBS:
            out.append(None)
            continue
        dtype = torch.float32 if form == M.FORM_FLOAT_FLOAT else torch.float64
        part = np.zeros((hi - lo) // dtype.itemsize)
        for f, words, off, size in state["where"]:
            if f == form:
                x = ain[off:off + size].view(dtype).double().numpy()
                at = slice((off - lo) // dtype.itemsize, (off - lo + size) // dtype.itemsize)
                part[at].reshape(2, words, -1)[:, 0] = _dft(x.reshape(2, words, -1).sum(axis=1)[:, None], False, False)[:, 0]
        out.append(part)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "uneven":
        return _uneven_exact(prepare(case, seed))
    if kind not in ("fp64", "tier", "adjoint"):
        return None
    x, *grad = [t.double().cpu().numpy() for t in _float_inputs(case, _gen(seed))]
    if kind == "fp64":
        return _dft(x, case["inverse"], case["scaled"])
    if kind == "tier":
        return [_dft(x.sum(axis=1), case["inverse"], case["scaled"]), None]
    return [_dft(x.sum(axis=1), False, False), None, _dft(grad[0].sum(axis=1), True, False), None]
