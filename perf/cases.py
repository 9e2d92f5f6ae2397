"""The work a user has the solver do, as cases that can be timed and compared.

Kinds of call (``case["kind"]``):

* ``solve``    -- ``Context.solve_device``: CSR, b and x in device memory, one
  complete solve (factorization, spikes, reduced system, FP64 refinement);
* ``host``     -- the reference's drop-in entry points ``?spike_core_host`` on
  page-locked host arrays (``dtype`` d, z, s or c);
* ``factored`` -- ``spike_dsolve_factored_device``: a factorization the program
  keeps, new right-hand sides on every pass;
* ``batch``    -- ``Batch.run``: many uneven systems in one launch.

Every system is a band of ``kl`` sub- and ``ku`` super-diagonals with entries
U[-1, 1) (real and imaginary parts for complex data), of which a share ``fill``
is stored, and a diagonal of ``dom`` times the row's off-diagonal magnitude with
a random sign or phase; x is U[-1, 1) and b = A x.
"""
from __future__ import annotations

import ctypes
import math
import random

import numpy as np
import torch

import hspike_gb300 as hs
from hspike_gb300 import workloads

DEV = "cuda"


def _solve(name, n, k, nrhs, precision="mixed", cplx=False, partitions=0, dom=1.5, ku=None, fill=1.0):
    c = dict(kind="solve", n=n, kl=k, ku=k if ku is None else ku, nrhs=nrhs, precision=precision, complex=cplx,
             partitions=partitions, dom=dom, fill=fill)
    return dict(c, name=name) if name else c


def _host(name, n, k, nrhs, dtype="d", dom=1.5, ku=None, fill=1.0):
    c = dict(kind="host", n=n, kl=k, ku=k if ku is None else ku, nrhs=nrhs, dtype=dtype, dom=dom, fill=fill)
    return dict(c, name=name) if name else c


def _factored(name, n, k, nrhs, precision="mixed", dom=1.5, ku=None, fill=1.0):
    c = dict(kind="factored", n=n, kl=k, ku=k if ku is None else ku, nrhs=nrhs, precision=precision, dom=dom, fill=fill)
    return dict(c, name=name) if name else c


def _batch(name, count, layout, precision="mixed"):
    c = dict(kind="batch", count=count, layout=layout, precision=precision)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: a short pentadiagonal system, where launches and waits are everything
        _solve("penta_1k", 1_000, 2, 1),
        # the reference's own configuration: pentadiagonal, plain FP64, its fixed four partitions
        _solve("penta_100k_fp64_p4", 100_000, 2, 1, precision="fp64", partitions=4, dom=2.0),
        # an ordinary narrow band with every choice left to the library, odd size
        _solve("band8_300k", 300_007, 8, 1),
        # a median request of the serving stream through the drop-in entry point (weak dominance, many columns)
        _host("request_20k_k48", 20_011, 48, 16, dom=1.05),
        # a wide-band request of that stream (128-row tiles)
        _solve("request_33k_k100", 33_000, 100, 8, dom=1.05),
        # repeated right-hand sides against a factorization the program keeps (time stepping)
        _factored("factored_150k_k24", 150_001, 24, 4),
        # the large-band configuration: one and sixteen right-hand sides, and plain FP64
        _solve("large_band_r1", 2_000_000, 64, 1, partitions=256),
        _solve("large_band_r16", 2_000_000, 64, 16, partitions=256),
        _solve("large_band_fp64", 2_000_000, 64, 1, precision="fp64", partitions=256),
        # the complex heptadiagonal configuration
        _solve("complex_hepta_4m", 4_000_000, 3, 4, cplx=True, partitions=512, dom=1.2),
        # a large system whose arrays are in host memory (drop-in entry point, end to end)
        _host("host_band_400k_k64", 400_000, 64, 1),
        # many uneven independent systems, the batched configuration's distribution
        _batch("batch_512", 512, 4),
    ]


# A drawn case stays below the largest listed one by this estimate of its work.
_COST_CAP = 2_000_000 * 64 * 64 * 8.0


def _cost(n, k, nrhs, heavy):
    """tile work of the factorization plus the sweeps and the residual, FP64 / complex scaled up"""
    kb = next(s for s in (2, 4, 8, 16, 32, 64, 128) if s >= k)
    return n * (kb * kb + 12.0 * kb * nrhs) * heavy


def draw(rng: random.Random):
    def logu(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    dom = round(rng.uniform(1.05, 2.0), 3)
    fill = rng.choice((1.0, 1.0, 1.0, 0.3))
    kind = rng.choice(("solve", "solve", "solve", "host", "factored", "batch"))
    if kind == "batch":
        return _batch(None, logu(16, 512), rng.randrange(1, 10_000), rng.choice(("mixed", "mixed", "fp64")))
    if kind == "solve":
        precision = rng.choice(("mixed", "mixed", "mixed", "fp64"))
        cplx = rng.random() < 0.25
        k = logu(1, 64 if cplx or precision == "fp64" else 128)
        heavy = (4.0 if cplx else 1.0) * (8.0 if precision == "fp64" else 1.0)
        nrhs = logu(1, 32)
        n = max(4 * k, min(logu(500, 4_000_000), int(_COST_CAP / _cost(1, k, nrhs, heavy)), 150_000_000 // (2 * k + 1)))
        # a count the caller chose, down to the reference's 25,000 rows per partition
        part = rng.choice((0, 0, 0, max(logu(4, 512), -(-n // 25_000))))
        return _solve(None, n, k, nrhs, precision, cplx, part, max(dom, 1.2) if cplx else dom,
                      max(1, int(k * rng.choice((1.0, 1.0, 0.5)))), fill)
    if kind == "host":
        dtype = rng.choice("dddzsc")
        k = logu(1, 64 if dtype in "zc" else 128)
        n = max(4 * k, min(logu(500, 500_000), 40_000_000 // (2 * k + 1)))
        if dtype in "sc":  # single-precision data: ordinary sizes
            k, n, dom = min(k, 8), min(n, 60_000), max(dom, 1.5)
        return _host(None, max(n, 4 * k), k, logu(1, 32), dtype, max(dom, 1.2) if dtype == "z" else dom,
                     max(1, int(k * rng.choice((1.0, 1.0, 0.5)))), fill)
    precision = rng.choice(("mixed", "mixed", "fp64"))
    k = logu(1, 64 if precision == "fp64" else 128)
    n = max(4 * k, min(logu(500, 1_000_000), 60_000_000 // (2 * k + 1)))
    return _factored(None, n, k, logu(1, 32), precision, dom, max(1, int(k * rng.choice((1.0, 1.0, 0.5)))), fill)


# ---------------------------------------------------------------- inputs
def _system(n, ku, kl, dom, nrhs, cplx, fill, g):
    """The band as an n x (kl + ku + 1) array with a mask of what is stored,
    and x, all on the device; columns of row r start at r - kl."""
    w = kl + ku + 1
    dt = torch.complex128 if cplx else torch.float64

    def uniform(*shape):
        if cplx:
            return torch.view_as_complex(torch.rand(*shape, 2, dtype=torch.float64, device=DEV, generator=g) * 2 - 1)
        return torch.rand(*shape, dtype=torch.float64, device=DEV, generator=g).mul_(2).sub_(1)

    col = torch.arange(n, device=DEV, dtype=torch.int32)[:, None] + torch.arange(-kl, ku + 1, device=DEV,
                                                                                 dtype=torch.int32)
    stored = (col >= 0) & (col < n)
    if fill < 1.0:
        stored &= torch.rand(n, w, device=DEV, generator=g) < fill
    stored[:, kl] = True
    band = uniform(n, w)
    band.mul_(stored)
    band[:, kl] = 0
    weight = torch.zeros(n, dtype=torch.float64, device=DEV)
    for j in range(w):
        weight += band[:, j].abs()
    weight = torch.where(weight > 0, weight, torch.ones_like(weight)) * dom
    phase = torch.rand(n, dtype=torch.float64, device=DEV, generator=g)
    band[:, kl] = torch.polar(weight, phase * (2 * math.pi)) if cplx else torch.where(phase < 0.5, -weight, weight)
    x = uniform(nrhs, n).to(dt)
    return band, col, stored, x


def _times(band, kl, x):
    """A x in 64 bits, x and the result nrhs x n"""
    n, w = band.shape
    pad = torch.zeros(n + w, x.shape[0], dtype=band.dtype, device=DEV)
    pad[kl:kl + n] = x.T
    y = torch.zeros(n, x.shape[0], dtype=band.dtype, device=DEV)
    for j in range(w):
        y.addcmul_(band[:, j:j + 1], pad[j:j + n])
    return y.T.contiguous()


def _csr(band, col, stored):
    rowptr = torch.zeros(band.shape[0] + 1, dtype=torch.int32, device=DEV)
    rowptr[1:] = stored.sum(1).cumsum(0)
    return rowptr, col[stored], band[stored]


def _inputs(n, ku, kl, dom, nrhs, cplx, fill, g):
    """rowptr, colind, values, b (nrhs x n, so column-major n x nrhs), x"""
    band, col, stored, x = _system(n, ku, kl, dom, nrhs, cplx, fill, g)
    b = _times(band, kl, x)
    return (*_csr(band, col, stored), b, x)


def _generator(case, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _layout(case):
    return workloads.batch_draws(case["count"], seed=case["layout"])


_DTYPE = {"d": (torch.float64, torch.float64), "z": (torch.complex128, torch.complex128),
          "s": (torch.float32, torch.float64), "c": (torch.complex64, torch.complex128)}


def _precision(case):
    return hs.SPIKE_PRECISION_FP64 if case["precision"] == "fp64" else hs.SPIKE_PRECISION_MIXED


def prepare(case, seed):
    g = _generator(case, seed)
    kind = case["kind"]
    if kind == "batch":
        arrays, descr = [], []
        for n, k, nrhs, dom in _layout(case):
            rp, ci, a, b, _ = _inputs(n, k, k, dom, nrhs, False, 1.0, g)
            x = torch.zeros_like(b)
            arrays.append((rp, ci, a, b, x))
            descr.append((n, ci.numel(), nrhs, ci.data_ptr(), rp.data_ptr(), a.data_ptr(), x.data_ptr(), b.data_ptr()))
        ctx = hs.Context()
        ctx.set_option(hs.SPIKE_OPT_PRECISION, _precision(case))
        torch.cuda.synchronize()
        # the schedule by rule: the same on every run, where the autotuner picks by timing
        return dict(kind=kind, ctx=ctx, arrays=arrays, batch=hs.Batch(descr, ctx, autotune=False))
    n, nrhs = case["n"], case["nrhs"]
    if kind == "host":
        dt, high = _DTYPE[case["dtype"]]
        rp, ci, a, b, x = _inputs(n, case["ku"], case["kl"], case["dom"], nrhs, high.is_complex, case["fill"], g)
        arrays = []
        for t in (ci, rp, a.to(dt), torch.zeros_like(b, dtype=dt), b.to(dt)):
            h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
            h.copy_(t)
            arrays.append(h)
        torch.cuda.synchronize()
        views = [h.numpy() for h in arrays]
        views[3], views[4] = views[3].T, views[4].T  # n x nrhs, column-major
        return dict(kind=kind, arrays=arrays, args=(n, ci.numel(), nrhs, *views),
                    call=getattr(hs, case["dtype"] + "spike_core_host"))
    cplx = bool(case.get("complex", False))
    rp, ci, a, b, _ = _inputs(n, case["ku"], case["kl"], case["dom"], nrhs, cplx, case["fill"], g)
    x = torch.zeros_like(b)
    ctx = hs.Context()
    ctx.set_option(hs.SPIKE_OPT_PRECISION, _precision(case))
    torch.cuda.synchronize()
    state = dict(kind=kind, ctx=ctx, arrays=(rp, ci, a, b, x))
    if kind == "factored":
        f = ctypes.c_void_p()
        rc = hs.load().spike_dfactor_device(ctx.handle, n, ci.numel(), ci.data_ptr(), rp.data_ptr(), a.data_ptr(),
                                            ctypes.byref(f))
        if rc != hs.SPIKE_SUCCESS:
            raise RuntimeError(hs.last_error())
        return dict(state, factor=_Handle(f), nrhs=nrhs, x=x, b=b)
    ctx.set_option(hs.SPIKE_OPT_PARTITIONS, case["partitions"])
    return dict(state, x=x, complex_=cplx,
                args=(n, ci.numel(), nrhs, ci.data_ptr(), rp.data_ptr(), a.data_ptr(), x.data_ptr(), b.data_ptr()))


class _Handle:
    """A factor handle, released with the state that holds it."""

    def __init__(self, handle):
        self.handle = handle

    def __del__(self):
        hs.load().spike_factor_release(self.handle)


# ---------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "solve":
        state["ctx"].solve_device(*state["args"], complex_=state["complex_"])
        return state["x"]
    if kind == "host":
        if state["call"](*state["args"]) != hs.SPIKE_SUCCESS:
            raise RuntimeError(hs.last_error())
        return state["arrays"][3]
    if kind == "factored":
        rc = hs.load().spike_dsolve_factored_device(state["factor"].handle, state["nrhs"], state["x"].data_ptr(),
                                                    state["b"].data_ptr())
        if rc != hs.SPIKE_SUCCESS:
            raise RuntimeError(hs.last_error())
        return state["x"]
    state["batch"].run()
    # 64 outputs at most: the systems' solutions end to end
    return torch.cat([s[4].reshape(-1) for s in state["arrays"]])


# ---------------------------------------------------------------- what a pass cannot do without
def _work(n, ku, kl, nrhs, cplx, fill, esize, factor=True):
    """CSR and b read once, x written once; a banded LU, its two triangular
    solves and one residual (complex multiply-adds count four real ones)"""
    nnz = n * (1 + fill * (ku + kl))
    m = 4.0 if cplx else 1.0
    size = nnz * (4 + esize) + 4 * (n + 1) + 2 * n * nrhs * esize
    flops = (2.0 * n * kl * ku if factor else 0.0) + n * nrhs * (2.0 * kl + 2.0 * (kl + ku)) + 2.0 * nnz * nrhs
    return size, flops * m


def work(case):
    if case["kind"] == "batch":
        per = [_work(n, k, k, nrhs, False, 1.0, 8) for n, k, nrhs, _ in _layout(case)]
        return {"bytes": float(sum(p[0] for p in per)), "flops": float(sum(p[1] for p in per))}
    dt = _DTYPE[case["dtype"]][0] if case["kind"] == "host" else torch.complex128 if case.get("complex") else torch.float64
    size, flops = _work(case["n"], case["ku"], case["kl"], case["nrhs"], dt.is_complex, case["fill"], dt.itemsize,
                        case["kind"] != "factored")
    return {"bytes": float(size), "flops": float(flops)}


# ---------------------------------------------------------------- the exact outputs
def exact(case, seed):
    """b was formed as A x in 64 bits, so x solves the system as far as 64
    bits tell; for single-precision data A and b are rounded after that, and
    the correction this makes is found by Jacobi sweeps in 64 bits."""
    g = _generator(case, seed)
    if case["kind"] == "batch":
        return torch.cat([_inputs(n, k, k, dom, nrhs, False, 1.0, g)[4].reshape(-1)
                          for n, k, nrhs, dom in _layout(case)])
    n, kl = case["n"], case["kl"]
    dt, high = _DTYPE[case["dtype"]] if case["kind"] == "host" else (None, None)
    cplx = high.is_complex if high else bool(case.get("complex", False))
    band, _, _, x = _system(n, case["ku"], kl, case["dom"], case["nrhs"], cplx, case["fill"], g)
    if dt is None or dt == high:
        return x
    b = _times(band, kl, x).to(dt).to(high)
    band = band.to(dt).to(high)
    diag = band[:, kl].clone()
    for _ in range(100):  # dominance 1.5 or more: each sweep takes a third off the error
        x = x + (b - _times(band, kl, x)) / diag
    return x
