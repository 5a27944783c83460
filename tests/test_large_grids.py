"""Kernels whose launch shape depends on the grid, on every size up to 1024^3,
through the library's own launchers on device memory.

The FP64 row sweeps (from the coefficient planes and from the face sums: 8, 16
or 32 rows per CTA, with and without a cluster) and the face-sum residual run on
a 32^3 problem repeated along the axes, whose solution is the repeated 32^3 one:
bit for bit the oracle's.  The spectral lines run on a few modes of any
frequency, whose derivatives are known."""
import ctypes as C
import math

import numpy as np
import pytest

from conftest import smooth_field

pytestmark = pytest.mark.gpu


class Face64(C.Structure):
    _fields_ = [(f, C.c_void_p) for f in ("bx", "by", "bz", "f2", "f3", "f5", "d", "y")]


@pytest.fixture
def dev(mmh):
    """The library and torch on the legacy default stream; device memory given
    back afterwards."""
    import torch
    yield mmh.lib(), torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()


def call(lib, symbol, *args, restype=None):
    f = getattr(lib, symbol)
    f.restype = restype
    f.argtypes = [{int: C.c_int, float: C.c_double, bool: C.c_bool}.get(type(a), C.c_void_p) for a in args]
    return f(*[C.c_void_p(a.data_ptr()) if hasattr(a, "data_ptr") else C.byref(a) if isinstance(a, Face64) else a
               for a in args])


def metric(lib, d, rho, n, dx, coef):
    call(lib, "_ZN3mmh13launch_metricIdEEvPKT_S3_iS1_PS1_P11CUstream_stbS4_", d, rho, n, dx, coef, None, False, None)


def sweeps(lib, phi, rhs, op, n, dx, count, scratch):
    """The swept field: phi or scratch."""
    if isinstance(op, Face64):
        at = call(lib, "_ZN3mmh18launch_gs64_sweepsEPdPKdRKNS_6Face64EidiS0_P11CUstream_st", phi, rhs, op, n, dx,
                  count, scratch, None, restype=C.c_void_p)
    else:
        at = call(lib, "_ZN3mmh18launch_gs64_sweepsEPdPKdS2_idiS0_P11CUstream_sti", phi, rhs, op, n, dx, count,
                  scratch, None, 16, restype=C.c_void_p)
    return {phi.data_ptr(): phi, scratch.data_ptr(): scratch}[at]


@pytest.mark.parametrize("n", [32, 64, 128, 256, 512, 1024])
def test_row_sweeps(dev, oracle, fields, n):
    lib, torch = dev
    m, dx, count = 32, 2.0, 3
    _, u = fields.initial_state(m, sigma=0.8, seed=17)
    rho, d = np.asfortranarray(u[0]), smooth_field(m, 0.05, 18)
    rng = np.random.default_rng(19)
    rhs, phi = (np.asfortranarray(rng.standard_normal((m, m, m))) for _ in range(2))
    coef0 = oracle.metric(d, rho, dx)
    want = phi.copy(order="F")
    oracle.relax(want, rhs, coef0, dx, count, 18, colour8=True)
    r0 = oracle.residual(want, rhs, coef0, dx)

    def base(a):
        return torch.from_numpy(np.ascontiguousarray(a.transpose(2, 1, 0))).cuda()

    def tiled(a):
        return base(a).repeat(n // m, n // m, n // m)

    def same(t, a):
        t = t.view(torch.int64).view(n // m, m, n // m, m, n // m, m)
        return bool((t == base(a).view(torch.int64)[None, :, None, :, None, :]).all())

    coef = torch.empty((6, n, n, n), device="cuda", dtype=torch.float64)
    metric(lib, tiled(d), tiled(rho), n, dx, coef)
    rhs_t, scratch = tiled(rhs), torch.empty((n, n, n), device="cuda", dtype=torch.float64)
    got = sweeps(lib, tiled(phi), rhs_t, coef, n, dx, count, scratch)
    torch.cuda.synchronize()
    assert same(got, want)
    del got
    # from here on the coefficient planes hold face sums
    planes = torch.empty((2, n, n, n), device="cuda", dtype=torch.float64)
    n3 = 8 * n ** 3
    make = lib._ZN3mmh14launch_faces64EPdiS0_S0_P11CUstream_st
    make.restype, make.argtypes = Face64, [C.c_void_p, C.c_int, C.c_void_p, C.c_void_p, C.c_void_p]
    face = make(coef.data_ptr(), n, planes[0].data_ptr(), planes[1].data_ptr(), None)
    assert face.by == coef.data_ptr() and face.d == coef.data_ptr() + 5 * n3
    got = sweeps(lib, tiled(phi), rhs_t, face, n, dx, count, scratch)
    torch.cuda.synchronize()
    assert same(got, want)
    res = scratch if got is not scratch else torch.empty_like(scratch)
    call(lib, "_ZN3mmh17launch_residual64EPKdS1_RKNS_6Face64EidPdPyP11CUstream_st", got, rhs_t, face, n, dx, res, None,
         None)
    torch.cuda.synchronize()
    assert same(res, r0)


@pytest.mark.parametrize("n", [512, 1024])
def test_spectral_modes(dev, n):
    lib, torch = dev
    rng = np.random.default_rng(n)
    modes = [(1, -2, 3), (n // 2 - 1, 1 - n // 2, n // 2 - 1)]
    modes += [tuple(int(k) for k in rng.integers(1 - n // 2, n // 2, 3)) for _ in range(4)]
    line = torch.arange(n, device="cuda")

    def add(out, table, k):
        i = (k[0] * line % n)[None, None, :] + (k[1] * line % n)[None, :, None]
        out += table[(i + (k[2] * line % n)[:, None, None]) % n]

    src = torch.zeros((n, n, n), device="cuda", dtype=torch.float64)
    want = torch.zeros((4, n, n, n), device="cuda", dtype=torch.float64)
    angle = 2 * math.pi * np.arange(n) / n
    for q, k in enumerate(modes):
        c, s = np.cos(angle + q), np.sin(angle + q)
        kap = [2 * math.pi * a / n for a in k]
        add(src, torch.from_numpy(c).cuda(), k)
        for a in range(3):  # minus the gradient
            add(want[a], torch.from_numpy(kap[a] * s).cuda(), k)
        add(want[3], torch.from_numpy(sum(a * a for a in kap) * c).cuda(), k)
    got = torch.empty_like(want)
    tab = torch.empty(4 * n + 2 * n * n + 1, device="cuda", dtype=torch.float64)
    sums = tab[4 * n:]
    call(lib, "_ZN3mmh17launch_fft_tablesEPdiP11CUstream_st", tab, n, None)
    call(lib, "_ZN3mmh21launch_spectral_linesEPKdiPdS2_S1_S2_PjP11CUstream_st", src, n, got, got[3], tab, sums,
         sums[2 * n * n:], None)
    torch.cuda.synchronize()
    # 2^-53 for each of the ~3 log2(n) roundings on the way to a value and as
    # many in the expected one, of values as large as the largest factor (pi,
    # 3 pi^2) makes them
    tol = 6 * math.log2(n) * 2.0 ** -53 * float(src.norm())
    got -= want
    for a in range(3):
        assert float(got[a].norm()) <= tol * math.pi
    assert float(got[3].norm()) <= tol * 3 * math.pi ** 2
