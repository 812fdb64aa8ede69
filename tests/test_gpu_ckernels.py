"""GPU C-ABI kernels (include/vibe_c_kernels.h) against the reference's own
known-answer tests (tests/unit/test_common.cpp:163-266,
tests/unit/test_time.cpp:53-100, tests/unit/test_gpu_precision.cpp) and
against the oracle on seeded inputs."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# ---- known answers from the reference's tests --------------------------------
def test_thomas_residual_diag_1_m4_1(vg):
    """test_common.cpp:163-175: diag(1,-4,1), d = 1, residual <= 1e-10 (the
    reference's own c_kernels.c fails this with 9e-2)."""
    n = 24
    a = np.ones(n - 1)
    c = np.ones(n - 1)
    b = np.full(n, -4.0)
    d = np.ones(n)
    rc, x = vg.tridiagonal_solve(a, b, c, d)
    assert rc == 0
    lhs = -4.0 * x
    lhs[1:] += x[:-1]
    lhs[:-1] += x[1:]
    assert np.abs(lhs - 1.0).max() <= 1e-10


def test_thomas_singular_and_bad_args(vg):
    """test_common.cpp:177-186."""
    lib = vg.lib
    b = np.zeros(2)
    d = np.ones(2)
    x = np.zeros(2)
    ws = np.zeros(2)
    assert lib.vibe_tridiagonal_solve_f64(None, b.ctypes.data, None, d.ctypes.data, 2, x.ctypes.data,
                                          ws.ctypes.data) == 1
    assert lib.vibe_tridiagonal_solve_f64(None, None, None, None, 2, x.ctypes.data, ws.ctypes.data) == 2
    assert lib.vibe_tridiagonal_solve_f64(None, b.ctypes.data, None, d.ctypes.data, 0, x.ctypes.data,
                                          ws.ctypes.data) == 2


def test_thomas_mms_and_variable_coefficients(vg, oc):
    """test_time.cpp:53-88 pattern; variable coefficients vs the oracle."""
    n = 24
    j = np.arange(n)
    b = 4.0 + 0.1 * j
    d = np.sin(0.3 * j)
    a = np.full(n - 1, -1.0)
    c = np.full(n - 1, -1.2)
    rc, x = vg.tridiagonal_solve(a, b, c, d)
    assert rc == 0
    xo = np.zeros(n)
    ws = np.zeros(n)
    L = oc.port_lib()
    assert L.vo_tridiagonal_solve(a.ctypes.data, b.ctypes.data, c.ctypes.data, d.ctypes.data, n, xo.ctypes.data,
                                  ws.ctypes.data) == 0
    assert np.abs(x - xo).max() <= 1e-12 * np.abs(xo).max()


def test_thomas_batched_matches_oracle(vg, oc):
    rng = np.random.default_rng(7)
    n_sys, n = 1000, 60
    b = 4.0 + rng.random((n_sys, n))
    a = -rng.random((n_sys, n - 1))
    c = -rng.random((n_sys, n - 1))
    d = rng.standard_normal((n_sys, n))
    rc, x = vg.tridiagonal_solve_batched(a, b, c, d)
    assert rc == 0
    L = oc.port_lib()
    for s in (0, 17, 999):
        xo = np.zeros(n)
        ws = np.zeros(n)
        aa, bb, cc, dd = (np.ascontiguousarray(v[s]) for v in (a, b, c, d))
        L.vo_tridiagonal_solve(aa.ctypes.data, bb.ctypes.data, cc.ctypes.data, dd.ctypes.data, n, xo.ctypes.data,
                               ws.ctypes.data)
        assert np.abs(x[s] - xo).max() <= 1e-12 * np.abs(xo).max()


@pytest.mark.parametrize("n,n_sys", [(129, 1), (200, 5), (225, 4), (1000, 37), (4097, 3)])
def test_thomas_tall_systems_warp_cooperative(vg, oc, n, n_sys):
    """n > 128: one warp per system (chunked Thomas per lane + the 2x2
    block-tridiagonal interface system). Agrees with the oracle's sequential
    sweep to rounding (1e-12 of the solution's scale) on diagonally dominant
    systems, including a one-row last chunk (n = 225: 28 chunks of 8 rows and
    one of 1)."""
    rng = np.random.default_rng(n)
    b = 4.0 + rng.random((n_sys, n))
    a = -rng.random((n_sys, n - 1))
    c = -rng.random((n_sys, n - 1))
    d = rng.standard_normal((n_sys, n))
    rc, x = vg.tridiagonal_solve_batched(a, b, c, d)
    assert rc == 0
    L = oc.port_lib()
    for s in range(n_sys):
        xo = np.zeros(n)
        ws = np.zeros(n)
        aa, bb, cc, dd = (np.ascontiguousarray(v[s]) for v in (a, b, c, d))
        L.vo_tridiagonal_solve(aa.ctypes.data, bb.ctypes.data, cc.ctypes.data, dd.ctypes.data, n, xo.ctypes.data,
                               ws.ctypes.data)
        assert np.abs(x[s] - xo).max() <= 1e-12 * np.abs(xo).max()
    # the single-system entry point takes the same path; NULL a / c read as 0
    rc1, x1 = vg.tridiagonal_solve(None, b[0], c[0], d[0])
    assert rc1 == 0
    A = np.diag(b[0]) + np.diag(c[0], 1)
    assert np.abs(x1 - np.linalg.solve(A, d[0])).max() <= 1e-12 * np.abs(x1).max()
    # an exact zero pivot is reported
    bz = b.copy()
    bz[0, 0] = 0.0
    az = a.copy()
    az[0, :] = 0.0
    rcz, _ = vg.tridiagonal_solve_batched(az, bz, c, d)
    assert rcz == 1


def _residual(a, b, c, d, x):
    """max |Ax - d| / max(|A||x| + |d|) of one tridiagonal system."""
    r = b * x - d
    r[1:] += a * x[:-1]
    r[:-1] += c * x[1:]
    scale = np.abs(b * x) + np.abs(d)
    scale[1:] += np.abs(a * x[:-1])
    scale[:-1] += np.abs(c * x[1:])
    return float(np.abs(r).max() / scale.max())


def _oracle_solve(oc, a, b, c, d):
    n = b.size
    xo, ws = np.zeros(n), np.zeros(n)
    aa, bb, cc, dd = (np.ascontiguousarray(v) for v in (a, b, c, d))
    rc = oc.port_lib().vo_tridiagonal_solve(aa.ctypes.data, bb.ctypes.data, cc.ctypes.data, dd.ctypes.data, n,
                                            xo.ctypes.data, ws.ctypes.data)
    return rc, xo


@pytest.mark.parametrize("n", [300, 1000])
def test_thomas_tall_zero_chunk_pivot_falls_back_to_the_sweep(vg, oc, n):
    """A nonsingular system whose diagonal is 0 at the first row of a warp
    chunk (rows per chunk m = ceil(n/32)): the chunked elimination has a zero
    pivot there, the single sweep does not. The reference's contract
    (c_kernels.c:26,34,40) reports singular only on a zero sweep pivot, so
    the solver must solve it, as the oracle's sweep does."""
    m = (n + 31) // 32
    rng = np.random.default_rng(n + 5)
    n_sys = 6
    b = 4.0 + rng.random((n_sys, n))
    a = -rng.random((n_sys, n - 1))
    c = -rng.random((n_sys, n - 1))
    d = rng.standard_normal((n_sys, n))
    for s in range(n_sys):  # a zero at the start of chunk s+1 (every system a different chunk)
        b[s, (s + 1) * m] = 0.0
    rc, x = vg.tridiagonal_solve_batched(a, b, c, d)
    assert rc == 0
    for s in range(n_sys):
        rco, xo = _oracle_solve(oc, a[s], b[s], c[s], d[s])
        assert rco == 0
        assert np.abs(x[s] - xo).max() <= 1e-12 * np.abs(xo).max()
        assert _residual(a[s], b[s], c[s], d[s], x[s]) <= 1e-13


def test_thomas_tall_non_dominant_diagonals(vg, oc):
    """Diagonals of either sign and no dominance (|b| ~ |a| + |c|): every
    system is solved to the sweep's accuracy (residual 1e-10 of the row
    scale, the sweep's own residual within a factor 100), and the return code
    is the sweep's."""
    rng = np.random.default_rng(11)
    n, n_sys = 513, 40
    b = rng.uniform(-2.0, 2.0, (n_sys, n))
    a = rng.uniform(-1.0, 1.0, (n_sys, n - 1))
    c = rng.uniform(-1.0, 1.0, (n_sys, n - 1))
    d = rng.standard_normal((n_sys, n))
    _, x = vg.tridiagonal_solve_batched(a, b, c, d)
    for s in range(n_sys):
        rco, xo = _oracle_solve(oc, a[s], b[s], c[s], d[s])
        assert rco == 0
        r_gpu, r_seq = _residual(a[s], b[s], c[s], d[s], x[s]), _residual(a[s], b[s], c[s], d[s], xo)
        assert r_gpu <= max(1e-10, 100.0 * r_seq), (s, r_gpu, r_seq)
        rc1, x1 = vg.tridiagonal_solve(a[s], b[s], c[s], d[s])
        assert rc1 == rco


def test_host_entry_points_reentrant_and_allocation_free(vg, oc):
    """c_kernels.h:17-18: reentrant, OpenMP-thread-safe, no allocation per
    call. Eight host threads call vibe_tridiagonal_solve_f64 and
    vibe_neumaier_sum_f64 concurrently on their own inputs (ctypes releases
    the interpreter lock during the call); every result matches the oracle.
    After each thread's first calls, further calls of the same sizes make no
    allocation (vibe_c_allocations() stays put). Prints the latency of one
    n = 80 solve."""
    import threading
    import time
    lib = vg.lib
    lib.vibe_c_allocations.restype = ctypes.c_ulonglong
    lib.vibe_neumaier_sum_f64.restype = ctypes.c_double
    lib.vibe_neumaier_sum_f64.argtypes = [ctypes.c_void_p, ctypes.c_size_t]
    L = oc.port_lib()
    nthreads, calls, n = 8, 40, 80
    cases = []
    for t in range(nthreads):
        rng = np.random.default_rng(100 + t)
        sys_ = []
        for q in range(calls):
            b = 4.0 + rng.random(n)
            a, c = -rng.random(n - 1), -rng.random(n - 1)
            d = rng.standard_normal(n)
            xs = rng.standard_normal(5000) * 10.0 ** rng.integers(-8, 8, 5000)
            _, xo = _oracle_solve(oc, a, b, c, d)
            so = L.vo_neumaier_sum(xs.ctypes.data, xs.size)
            sys_.append((a, b, c, d, xo, xs, so))
        cases.append(sys_)
    errors = []
    warm, go, done = threading.Barrier(nthreads + 1), threading.Barrier(nthreads + 1), threading.Barrier(nthreads + 1)

    def worker(t):
        try:
            x, ws = np.zeros(n), np.zeros(n)

            def run_all():
                for a, b, c, d, xo, xs, so in cases[t]:
                    rc = lib.vibe_tridiagonal_solve_f64(a.ctypes.data, b.ctypes.data, c.ctypes.data, d.ctypes.data,
                                                        n, x.ctypes.data, ws.ctypes.data)
                    if rc != 0 or np.abs(x - xo).max() > 1e-12 * np.abs(xo).max():
                        errors.append(("thomas", t, rc))
                    sv = lib.vibe_neumaier_sum_f64(xs.ctypes.data, xs.size)
                    if abs(sv - so) > 1e-13 * np.abs(xs).sum():
                        errors.append(("neumaier", t, sv, so))
            run_all()
            warm.wait()
            go.wait()
            run_all()
            done.wait()
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(("exception", t, repr(e)))
            for bar in (warm, go, done):
                bar.abort()

    threads = [threading.Thread(target=worker, args=(t,)) for t in range(nthreads)]
    for th in threads:
        th.start()
    warm.wait()
    before = lib.vibe_c_allocations()
    go.wait()
    done.wait()
    after = lib.vibe_c_allocations()
    for th in threads:
        th.join()
    assert not errors, errors[:5]
    assert after == before, (before, after)
    a, b, c, d, xo, _, _ = cases[0][0]
    x, ws = np.zeros(n), np.zeros(n)
    for _ in range(20):
        lib.vibe_tridiagonal_solve_f64(a.ctypes.data, b.ctypes.data, c.ctypes.data, d.ctypes.data, n, x.ctypes.data,
                                       ws.ctypes.data)
    t0 = time.perf_counter()
    for _ in range(500):
        lib.vibe_tridiagonal_solve_f64(a.ctypes.data, b.ctypes.data, c.ctypes.data, d.ctypes.data, n, x.ctypes.data,
                                       ws.ctypes.data)
    print("host vibe_tridiagonal_solve_f64, n = 80: %.1f us per call" % ((time.perf_counter() - t0) / 500 * 1e6))


def test_dev_entry_points_share_no_scratch_across_streams(vg, oc):
    """The _dev forms take their scratch from the calling thread's buffer and
    order a call on one stream after the previous call on another: solves
    queued back to back on two streams, the second needing a larger scratch
    than the first (the buffer is replaced only after its last user), with a
    Neumaier sum after each, all come out right."""
    torch = pytest.importorskip("torch")
    dev = torch.device("cuda", 0)
    vp, i = ctypes.c_void_p, ctypes.c_int
    f = vg.lib.vibe_tridiagonal_solve_batched_f64_dev
    f.restype, f.argtypes = i, [vp, vp, vp, vp, i, i, vp, vp, vp]
    g = vg.lib.vibe_neumaier_sum_f64_dev
    g.restype, g.argtypes = i, [vp, ctypes.c_size_t, vp, vp]
    s1, s2 = torch.cuda.Stream(dev), torch.cuda.Stream(dev)
    outs = []
    for q, (n, n_sys, st) in enumerate(((60, 2000, s1), (300, 2000, s2), (60, 20000, s1))):
        rng = np.random.default_rng(q)
        arrs = [4.0 + rng.random((n_sys, n)), -rng.random((n_sys, n - 1)), -rng.random((n_sys, n - 1)),
                rng.standard_normal((n_sys, n))]
        b, a, c, d = (torch.tensor(v, device=dev) for v in arrs)
        x = torch.zeros((n_sys, n), dtype=torch.float64, device=dev)
        assert f(a.data_ptr(), b.data_ptr(), c.data_ptr(), d.data_ptr(), n, n_sys, x.data_ptr(), None,
                 st.cuda_stream) == 0
        xs = torch.tensor(rng.standard_normal(100000), device=dev)
        out = torch.zeros(1, dtype=torch.float64, device=dev)
        assert g(xs.data_ptr(), xs.numel(), out.data_ptr(), s1.cuda_stream) == 0
        outs.append((arrs, x, xs, out))
    torch.cuda.synchronize(dev)
    for arrs, x, xs, out in outs:
        b, a, c, d = arrs
        xg = x.cpu().numpy()
        for s in (0, b.shape[0] - 1):
            _, xo = _oracle_solve(oc, a[s], b[s], c[s], d[s])
            assert np.abs(xg[s] - xo).max() <= 1e-12 * np.abs(xo).max()
        assert abs(float(out.item()) - float(np.sum(xs.cpu().numpy()))) <= 1e-10 * float(xs.abs().sum())


def test_weno5_known_answers(vg, oc):
    """test_common.cpp:188-205: exact on constants, bounded on monotone data."""
    ql, qr = vg.weno5_reconstruct(3.5, 3.5, 3.5, 3.5, 3.5)
    assert abs(ql - 3.5) <= 1e-12 and abs(qr - 3.5) <= 1e-12
    ql, qr = vg.weno5_reconstruct(0.2, -0.4, 1.1, 0.9, 2.3)
    assert -0.4 <= ql <= 2.3 and -0.4 <= qr <= 2.3
    L = oc.port_lib()
    a, b = ctypes.c_double(), ctypes.c_double()
    L.vo_weno5_reconstruct(0.2, -0.4, 1.1, 0.9, 2.3, ctypes.byref(a), ctypes.byref(b))
    assert abs(ql - a.value) <= 1e-14 and abs(qr - b.value) <= 1e-14


def test_bilinear_known_answers(vg):
    """test_common.cpp:207-226."""
    halo, nx, ny, nz = 2, 5, 4, 2
    nsx, nsy = nx + 2 * halo, ny + 2 * halo
    f = np.zeros((nz + 2 * halo, nsy, nsx))
    for k in range(nz):
        for j in range(ny):
            for i in range(nx):
                f[k + halo, j + halo, i + halo] = 10.0 * i + j + 100.0 * k
    assert abs(vg.bilinear(f, halo, nsx, nsy, nz, 2.0, 1.0, 1) - 121.0) <= 1e-12
    assert abs(vg.bilinear(f, halo, nsx, nsy, nz, 1.5, 1.0, 0) - 16.0) <= 1e-12
    assert abs(vg.bilinear(f, halo, nsx, nsy, nz, -50.0, -50.0, 0) - 0.0) <= 1e-12


def test_cfl_scan_known_answers(vg):
    """test_common.cpp:228-242: linear in dt, hand value 0.02, min dz 1000."""
    nx, ny, nz = 4, 3, 3
    u = np.full(nx * ny * nz, 20.0)
    v = np.zeros_like(u)
    w = np.zeros_like(u)
    dzeta = np.array([0.05, 0.10, 0.20])
    c1, mw, mdz = vg.cfl_scan(u, v, w, dzeta, None, nx, ny, nz, 1000.0, 1000.0, 20000.0, 1.0)
    c2, _, _ = vg.cfl_scan(u, v, w, dzeta, None, nx, ny, nz, 1000.0, 1000.0, 20000.0, 2.0)
    assert abs(c2 - 2.0 * c1) <= 1e-12
    assert abs(mw - 20.0) <= 1e-12
    assert abs(mdz - 0.05 * 20000.0) <= 1e-9
    assert abs(c1 - 20.0 / 1000.0) <= 1e-12


def test_cfl_scan_matches_oracle_with_terrain(vg, oc):
    rng = np.random.default_rng(3)
    nx, ny, nz = 37, 23, 19
    n = nx * ny * nz
    u, v, w = (rng.standard_normal(n) * s for s in (15.0, 10.0, 2.0))
    dzeta = rng.random(nz) * 0.1 + 1e-3
    zs = rng.random(nx * ny) * 500.0
    r, mw, mdz = vg.cfl_scan(u, v, w, dzeta, zs, nx, ny, nz, 1000.0, 800.0, 20000.0, 6.0)
    L = oc.port_lib()
    a, b = ctypes.c_double(), ctypes.c_double()
    ro = L.vo_cfl_scan(u.ctypes.data, v.ctypes.data, w.ctypes.data, dzeta.ctypes.data, zs.ctypes.data, nx, ny, nz,
                       1000.0, 800.0, 20000.0, 6.0, ctypes.byref(a), ctypes.byref(b))
    assert r == ro and mw == a.value and mdz == b.value  # max/min are exact


def test_neumaier_cancellation(vg):
    """test_common.cpp:244-254: [1e16, 1 x 9998, -1e16] sums to 9998."""
    n = 10000
    x = np.ones(n)
    x[0] = 1e16
    x[-1] = -1e16
    assert abs(vg.neumaier_sum(x) - (n - 2)) <= 1e-6
    assert abs(vg.neumaier_sum(np.ones(1_000_000)) - 1e6) <= 1e-3  # test_gpu_precision.cpp reduce on 1e6 ones


def test_neumaier_matches_oracle(vg, oc):
    rng = np.random.default_rng(11)
    x = rng.standard_normal(3_000_017) * 10.0 ** rng.integers(-8, 8, 3_000_017)
    L = oc.port_lib()
    ref = L.vo_neumaier_sum(x.ctypes.data, x.size)
    got = vg.neumaier_sum(x)
    assert abs(got - ref) <= 1e-12 * np.abs(x).sum()
    assert vg.neumaier_sum(np.zeros(0)) == 0.0


def test_flux_advection_constant_is_zero(vg):
    """test_common.cpp:256-266."""
    nx, ny, nz = 6, 5, 4
    n = nx * ny * nz
    q, rho, u, v, w = (np.full(n, val) for val in (3.0, 1.2, 7.0, -3.0, 0.5))
    dzeta = np.array([0.05, 0.08, 0.12, 0.2])
    dq = vg.advect_scalar_flux(q, rho, u, v, w, dzeta, None, nx, ny, nz, 1000.0, 1000.0, 20000.0)
    assert np.abs(dq).max() <= 1e-10


def test_flux_advection_matches_oracle(vg, oc):
    rng = np.random.default_rng(5)
    nx, ny, nz = 33, 17, 9
    n = nx * ny * nz
    q = rng.random(n)
    rho = 1.0 + 0.1 * rng.random(n)
    u, v, w = (rng.standard_normal(n) for _ in range(3))
    dzeta = rng.random(nz) * 0.1 + 0.01
    zs = rng.random(nx * ny) * 300.0
    dq = vg.advect_scalar_flux(q, rho, u, v, w, dzeta, zs, nx, ny, nz, 900.0, 1100.0, 15000.0)
    out = np.zeros(n)
    oc.port_lib().vo_advect_scalar_flux(q.ctypes.data, rho.ctypes.data, u.ctypes.data, v.ctypes.data, w.ctypes.data,
                                        dzeta.ctypes.data, zs.ctypes.data, nx, ny, nz, 900.0, 1100.0, 15000.0,
                                        out.ctypes.data)
    assert np.abs(dq - out).max() <= 1e-12 * np.abs(out).max()


# ---- FP32 twins (the *_f32 names of c_kernels.h:15-16) -----------------------
_F = ctypes.c_float
_fp = ctypes.POINTER(ctypes.c_float)


def f32(a):
    return np.ascontiguousarray(a, dtype=np.float32)


def _sig(vg, name, res, args):
    fn = getattr(vg.lib, name)
    fn.restype = res
    fn.argtypes = args
    return fn


def test_f32_thomas(vg):
    """diag(1,-4,1) known answer and variable coefficients at float precision;
    singular and bad-argument codes as the FP64 form."""
    fn = _sig(vg, "vibe_tridiagonal_solve_f32", ctypes.c_int, [ctypes.c_void_p] * 4 + [ctypes.c_int] +
              [ctypes.c_void_p] * 2)
    n = 24
    j = np.arange(n)
    for a, b, c, d in ((np.ones(n - 1), np.full(n, -4.0), np.ones(n - 1), np.ones(n)),
                       (np.full(n - 1, -1.0), 4.0 + 0.1 * j, np.full(n - 1, -1.2), np.sin(0.3 * j))):
        a32, b32, c32, d32 = f32(a), f32(b), f32(c), f32(d)
        x, ws = np.zeros(n, np.float32), np.zeros(n, np.float32)
        assert fn(a32.ctypes.data, b32.ctypes.data, c32.ctypes.data, d32.ctypes.data, n, x.ctypes.data,
                  ws.ctypes.data) == 0
        A = np.diag(b) + np.diag(a, -1) + np.diag(c, 1)
        ref = np.linalg.solve(A, d)
        assert np.abs(x - ref).max() <= 1e-5 * np.abs(ref).max()
    z, one, x, ws = np.zeros(2, np.float32), np.ones(2, np.float32), np.zeros(2, np.float32), np.zeros(2, np.float32)
    assert fn(None, z.ctypes.data, None, one.ctypes.data, 2, x.ctypes.data, ws.ctypes.data) == 1
    assert fn(None, None, None, None, 2, x.ctypes.data, ws.ctypes.data) == 2


def test_f32_weno_bilinear_cfl_neumaier_flux(vg, oc):
    """Each twin against the FP64 entry point on the same (float-representable)
    inputs: relative differences at float rounding."""
    weno = _sig(vg, "vibe_weno5_reconstruct_f32", None, [_F] * 5 + [_fp, _fp])
    rng = np.random.default_rng(9)
    for _ in range(20):
        q = f32(rng.standard_normal(5)).astype(np.float64)
        l32, r32 = _F(), _F()
        weno(*[float(v) for v in q], ctypes.byref(l32), ctypes.byref(r32))
        l64, r64 = vg.weno5_reconstruct(*q)
        assert abs(l32.value - l64) <= 2e-5 * max(1.0, abs(l64)) and abs(r32.value - r64) <= 2e-5 * max(1.0, abs(r64))

    bil = _sig(vg, "vibe_bilinear_f32", _F, [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_int,
                                               ctypes.c_int, _F, _F, ctypes.c_int])
    halo, nx, ny, nz = 2, 7, 5, 3
    nsx, nsy = nx + 2 * halo, ny + 2 * halo
    f = f32(rng.standard_normal(nsx * nsy * (nz + 2 * halo)))
    for xi, yj, k in ((2.25, 1.5, 1), (-3.0, 9.0, 0), (5.75, 3.125, 2)):
        got = bil(f.ctypes.data, halo, nsx, nsy, nz, xi, yj, k)
        ref = vg.bilinear(f.astype(np.float64), halo, nsx, nsy, nz, xi, yj, k)
        assert abs(got - ref) <= 1e-5 * max(1.0, abs(ref))

    cfl = _sig(vg, "vibe_cfl_scan_f32", _F, [ctypes.c_void_p] * 5 + [ctypes.c_int] * 3 + [_F] * 4 + [_fp, _fp])
    nx, ny, nz = 37, 23, 19
    n = nx * ny * nz
    u, v, w = (f32(rng.standard_normal(n) * s) for s in (15.0, 10.0, 2.0))
    dzeta, zs = f32(rng.random(nz) * 0.1 + 1e-3), f32(rng.random(nx * ny) * 500.0)
    mw, mdz = _F(), _F()
    got = cfl(u.ctypes.data, v.ctypes.data, w.ctypes.data, dzeta.ctypes.data, zs.ctypes.data, nx, ny, nz, 1000.0,
              800.0, 20000.0, 6.0, ctypes.byref(mw), ctypes.byref(mdz))
    r, m64, d64 = vg.cfl_scan(*(a.astype(np.float64) for a in (u, v, w, dzeta, zs)), nx, ny, nz, 1000.0, 800.0,
                              20000.0, 6.0)
    assert abs(got - r) <= 1e-5 * r and abs(mw.value - m64) <= 1e-5 * m64 and abs(mdz.value - d64) <= 1e-5 * d64

    neu = _sig(vg, "vibe_neumaier_sum_f32", _F, [ctypes.c_void_p, ctypes.c_size_t])
    x = np.ones(10000, np.float32)
    x[0], x[-1] = 1e8, -1e8
    assert neu(x.ctypes.data, x.size) == 9998.0  # compensation recovers what a plain float sum loses
    y = f32(rng.standard_normal(1_000_003))
    assert abs(neu(y.ctypes.data, y.size) - y.astype(np.float64).sum()) <= 1e-6 * np.abs(y).sum()

    flux = _sig(vg, "vibe_advect_scalar_flux_f32", None, [ctypes.c_void_p] * 7 + [ctypes.c_int] * 3 + [_F] * 3 +
                [ctypes.c_void_p])
    nx, ny, nz = 33, 17, 9
    n = nx * ny * nz
    q, rho = f32(rng.random(n)), f32(1.0 + 0.1 * rng.random(n))
    u, v, w = (f32(rng.standard_normal(n)) for _ in range(3))
    dzeta, zs = f32(rng.random(nz) * 0.1 + 0.01), f32(rng.random(nx * ny) * 300.0)
    out = np.zeros(n, np.float32)
    flux(*(a.ctypes.data for a in (q, rho, u, v, w, dzeta, zs)), nx, ny, nz, 900.0, 1100.0, 15000.0, out.ctypes.data)
    ref = vg.advect_scalar_flux(*(a.astype(np.float64) for a in (q, rho, u, v, w, dzeta, zs)), nx, ny, nz, 900.0,
                                1100.0, 15000.0)
    assert np.abs(out - ref).max() <= 1e-4 * np.abs(ref).max()


# ---- TL / AD of the flux advection ------------------------------------------
def _adv_case(seed, nx=23, ny=17, nz=9, dtype=np.float64):
    rng = np.random.default_rng(seed)
    n = nx * ny * nz
    x = {"q": 0.5 + rng.random(n), "rho": 1.0 + 0.1 * rng.random(n), "u": rng.standard_normal(n),
         "v": rng.standard_normal(n), "w": 0.3 * rng.standard_normal(n)}
    d = {k: rng.standard_normal(n) * (0.1 if k == "rho" else 1.0) for k in x}
    dzeta = rng.random(nz) * 0.1 + 0.01
    zs = rng.random(nx * ny) * 300.0
    cast = lambda a: np.ascontiguousarray(a, dtype=dtype)
    return ({k: cast(a) for k, a in x.items()}, {k: cast(a) for k, a in d.items()}, cast(dzeta), cast(zs),
            (nx, ny, nz))


ADV = ("q", "rho", "u", "v", "w")
GEO = (900.0, 1100.0, 15000.0)


def _tl(vg, x, d, dzeta, zs, dims, f32=False):
    nx, ny, nz = dims
    out = np.zeros(nx * ny * nz, dtype=np.float32 if f32 else np.float64)
    fn = vg.lib.vibe_advect_scalar_flux_tl_f32 if f32 else vg.lib.vibe_advect_scalar_flux_tl_f64
    fn.restype = ctypes.c_int
    F = ctypes.c_float if f32 else ctypes.c_double
    fn.argtypes = [ctypes.c_void_p] * 12 + [ctypes.c_int] * 3 + [F] * 3 + [ctypes.c_void_p]
    rc = fn(*[x[k].ctypes.data for k in ADV], *[d[k].ctypes.data for k in ADV], dzeta.ctypes.data, zs.ctypes.data,
            nx, ny, nz, *GEO, out.ctypes.data)
    assert rc == 0
    return out


def _ad(vg, x, bd, dzeta, zs, dims, acc=None, f32=False):
    nx, ny, nz = dims
    n = nx * ny * nz
    dt = np.float32 if f32 else np.float64
    outs = {k: (acc[k].copy() if acc else np.zeros(n, dtype=dt)) for k in ADV}
    fn = vg.lib.vibe_advect_scalar_flux_ad_f32 if f32 else vg.lib.vibe_advect_scalar_flux_ad_f64
    fn.restype = ctypes.c_int
    F = ctypes.c_float if f32 else ctypes.c_double
    fn.argtypes = [ctypes.c_void_p] * 8 + [ctypes.c_int] * 3 + [F] * 3 + [ctypes.c_void_p] * 5
    rc = fn(*[x[k].ctypes.data for k in ADV], bd.ctypes.data, dzeta.ctypes.data, zs.ctypes.data, nx, ny, nz, *GEO,
            *[outs[k].ctypes.data for k in ADV])
    assert rc == 0
    return outs


def test_flux_advection_tl_matches_finite_differences(vg):
    """Central differences of the FP64 forward kernel (which matches the
    oracle) converge to the TL: error O(eps^2) down to rounding."""
    x, d, dzeta, zs, dims = _adv_case(1)
    nx, ny, nz = dims
    fwd = lambda xx: vg.advect_scalar_flux(*[xx[k] for k in ADV], dzeta, zs, nx, ny, nz, *GEO)
    tl = _tl(vg, x, d, dzeta, zs, dims)
    errs = []
    for eps in (1e-2, 1e-3, 1e-4):
        xp = {k: x[k] + eps * d[k] for k in ADV}
        xm = {k: x[k] - eps * d[k] for k in ADV}
        fd = (fwd(xp) - fwd(xm)) / (2 * eps)
        errs.append(np.abs(fd - tl).max() / np.abs(tl).max())
    # second order (x100 per decade of eps) until rounding takes over
    assert errs[1] <= 0.02 * errs[0] or errs[1] < 1e-9, errs
    assert min(errs) < 1e-7, errs


@pytest.mark.parametrize("dims", [(23, 17, 9), (1, 5, 4), (2, 1, 3)])
def test_flux_advection_adjoint_dot_product(vg, dims):
    """<TL dx, y> = <dx, AD y> over all five inputs (1e-12 in FP64), on
    regular, one-column-wide and two-wide periodic grids; AD accumulates."""
    x, d, dzeta, zs, dims = _adv_case(2, *dims)
    rng = np.random.default_rng(3)
    y = rng.standard_normal(x["q"].size)
    lhs = float(np.dot(_tl(vg, x, d, dzeta, zs, dims), y))
    bar = _ad(vg, x, y, dzeta, zs, dims)
    rhs = float(sum(np.dot(d[k], bar[k]) for k in ADV))
    assert abs(lhs - rhs) <= 1e-12 * max(abs(lhs), abs(rhs)), (lhs, rhs)
    twice = _ad(vg, x, y, dzeta, zs, dims, acc=bar)
    for k in ADV:
        assert np.allclose(twice[k], 2 * bar[k], rtol=1e-14, atol=0)


def test_flux_advection_adjoint_dot_product_f32(vg):
    x, d, dzeta, zs, dims = _adv_case(4, dtype=np.float32)
    y = np.random.default_rng(5).standard_normal(x["q"].size).astype(np.float32)
    lhs = float(np.dot(_tl(vg, x, d, dzeta, zs, dims, f32=True).astype(np.float64), y))
    bar = _ad(vg, x, y, dzeta, zs, dims, f32=True)
    rhs = float(sum(np.dot(d[k].astype(np.float64), bar[k]) for k in ADV))
    assert abs(lhs - rhs) <= 1e-5 * max(abs(lhs), abs(rhs)), (lhs, rhs)


def _dev(vg, name, args):
    import ctypes
    f = getattr(ctypes.CDLL(vg.lib._name), name)
    f.restype, f.argtypes = ctypes.c_int, args
    return f


@pytest.mark.parametrize("bits", [64, 32])
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 16, 17, 80, 128, 129, 200, 363, 364])
@pytest.mark.parametrize("n_sys", [1, 33, 300])
def test_thomas_staged_sweep_edges(vg, oc, bits, n, n_sys):
    """The on-chip sweep at the edges of its stages (8 and 16 levels), its
    32-system blocks and its limits in n and n_sys: against the oracle at the
    bounds of the tests above (1e-12; FP32 1e-5), NULL off-diagonals, and a
    singular system, whose x stays as it was while its neighbours solve."""
    import ctypes
    import torch
    dt = torch.float64 if bits == 64 else torch.float32
    vp, i32 = ctypes.c_void_p, ctypes.c_int
    f = _dev(vg, "vibe_tridiagonal_solve_batched_f%d_dev" % bits, [vp] * 4 + [i32, i32, vp, vp, vp])
    rng = np.random.default_rng(n * 1000 + n_sys)
    a, c = -rng.random((n_sys, max(n - 1, 1))), -rng.random((n_sys, max(n - 1, 1)))
    b, d = 2.5 + rng.random((n_sys, n)), rng.random((n_sys, n))
    bad = n_sys // 2
    if n_sys > 1:
        b[bad, 0] = 0.0  # a zero first pivot
    t = [torch.tensor(v, dtype=dt, device="cuda") for v in (a[:, :n - 1], b, c[:, :n - 1], d)]
    x = torch.full((n_sys, n), 7.0, dtype=dt, device="cuda")
    st = torch.full((n_sys,), -1, dtype=torch.int32, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    p = lambda v: v.data_ptr() if v.numel() else None  # noqa: E731
    assert f(p(t[0]), p(t[1]), p(t[2]), p(t[3]), n, n_sys, x.data_ptr(), st.data_ptr(), stream) == 0
    torch.cuda.synchronize()
    host = [v.double().cpu().numpy() for v in t]
    got, status = x.double().cpu().numpy(), st.cpu().numpy()
    tol = 1e-12 if bits == 64 else 1e-5
    for s in range(n_sys):
        xo, ws = np.zeros(n), np.zeros(n)
        rows = [np.ascontiguousarray(h[s]) for h in host]
        rc = oc.port_lib().vo_tridiagonal_solve(rows[0].ctypes.data, rows[1].ctypes.data, rows[2].ctypes.data,
                                                 rows[3].ctypes.data, n, xo.ctypes.data, ws.ctypes.data)
        assert status[s] == rc == (1 if n_sys > 1 and s == bad else 0)
        if rc:
            if n <= 128:
                assert (got[s] == 7.0).all()
        else:
            assert np.abs(got[s] - xo).max() <= tol * np.abs(xo).max()
    assert f(None, p(t[1]), None, p(t[3]), n, n_sys, x.data_ptr(), None, stream) == 0
    ok = np.arange(n_sys) != (bad if n_sys > 1 else -1)
    q = (host[3] / np.where(host[1] == 0.0, 1.0, host[1]))[ok]
    assert np.abs(x.double().cpu().numpy()[ok] - q).max() <= tol * np.abs(q).max()


@pytest.mark.parametrize("bits", [64, 32])
@pytest.mark.parametrize("dims", [(1, 1, 1), (1, 5, 2), (5, 3, 3), (31, 8, 4), (32, 9, 5), (62, 7, 9), (63, 17, 13)])
def test_flux_advection_tile_edges(vg, oc, bits, dims):
    """Tiles of 31 x 8 columns and chunks of levels, wrapped rows and columns on
    small periodic grids: against the oracle at the bounds above (1e-12; FP32
    1e-4)."""
    import ctypes
    import torch
    nx, ny, nz = dims
    dt = torch.float64 if bits == 64 else torch.float32
    vp, i32 = ctypes.c_void_p, ctypes.c_int
    real = ctypes.c_double if bits == 64 else ctypes.c_float
    f = _dev(vg, "vibe_advect_scalar_flux_f%d_dev" % bits, [vp] * 7 + [i32] * 3 + [real] * 3 + [vp, vp])
    rng = np.random.default_rng(nx * 100 + ny)
    n = nx * ny * nz
    fields = [rng.random(n), 0.5 + rng.random(n), 20 * rng.random(n) - 10, 20 * rng.random(n) - 10,
              rng.random(n) - 0.5, 0.01 + 0.01 * rng.random(nz), 500.0 * rng.random(nx * ny)]
    t = [torch.tensor(v, dtype=dt, device="cuda") for v in fields]
    host = [np.ascontiguousarray(v.double().cpu().numpy()) for v in t]
    for zs in (True, False):
        out = torch.full((n,), float("nan"), dtype=dt, device="cuda")
        args = [v.data_ptr() for v in t[:6]] + [t[6].data_ptr() if zs else None]
        assert f(*args, nx, ny, nz, 900.0, 1100.0, 20000.0, out.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        ref = np.full(n, np.nan)
        oc.port_lib().vo_advect_scalar_flux(*[h.ctypes.data for h in host[:6]], host[6].ctypes.data if zs else None,
                                             nx, ny, nz, 900.0, 1100.0, 20000.0, ref.ctypes.data)
        tol = 1e-12 if bits == 64 else 1e-4
        assert np.abs(out.double().cpu().numpy() - ref).max() <= tol * np.abs(ref).max() or np.abs(ref).max() == 0.0


@pytest.mark.parametrize("kind", ["plain", "calm", "tiny", "huge", "nonfinite", "odd_metric"])
@pytest.mark.parametrize("dims", [(1, 1, 1), (7, 5, 3), (129, 3, 17), (64, 40, 8)])
def test_cfl_scan_bounds_change_no_bit(vg, oc, kind, dims):
    """The FP32 bounds skip cells, never a maximum: the scan equals the oracle's
    bit for bit on ordinary, resting, subnormal, overflowing and non-finite
    winds and on a metric with negative and huge entries."""
    nx, ny, nz = dims
    n = nx * ny * nz
    rng = np.random.default_rng(n)
    u, v, w = (20.0 * rng.standard_normal(n) for _ in range(3))
    dz, zs, dt = 0.01 + 0.02 * rng.random(nz), 500.0 * rng.random(nx * ny), 6.0
    if kind == "calm":
        u, v, w = np.zeros(n), np.zeros(n), np.zeros(n)
    elif kind == "tiny":
        u, v, w = (1e-40 * a for a in (u, v, w))
        u[n // 2] = 1e-310
    elif kind == "huge":
        u, v, w = (10.0 ** rng.uniform(20, 150, n) * np.sign(a) for a in (u, v, w))
    elif kind == "nonfinite":
        u[n // 3], v[n // 2], w[n - 1] = np.nan, -np.inf, np.nan
    elif kind == "odd_metric":
        dz, zs = rng.standard_normal(nz) * 10.0 ** rng.uniform(-3, 3, nz), 40000.0 * rng.random(nx * ny)
    with np.errstate(all="ignore"):
        for step in (dt, -dt, 1e-40):
            r, mw, mdz = vg.cfl_scan(u, v, w, dz, zs, nx, ny, nz, 900.0, 1100.0, 20000.0, step)
            a, b = ctypes.c_double(), ctypes.c_double()
            ro = oc.port_lib().vo_cfl_scan(u.ctypes.data, v.ctypes.data, w.ctypes.data, dz.ctypes.data, zs.ctypes.data,
                                            nx, ny, nz, 900.0, 1100.0, 20000.0, step, ctypes.byref(a), ctypes.byref(b))
            assert (r, mdz) == (ro, b.value), (step, r, ro, mdz, b.value)
            assert mw == a.value or abs(mw - a.value) <= 2.3e-16 * a.value, (mw, a.value)  # the sum's FMA contraction


@pytest.mark.parametrize("kind", ["narrow", "wide", "cancel", "subnormal", "rising"])
@pytest.mark.parametrize("n", [1, 255, 4097, 300000])
def test_neumaier_integer_sum(vg, kind, n):
    """Sums whose exponents stay in, leave and move the integer accumulator's
    window, against math.fsum: one rounding of the result plus the compensated
    sum's second-order bound, 4 eps |s| + 4 n eps^2 sum|x|."""
    import math
    rng = np.random.default_rng(n)
    x = rng.standard_normal(n)
    if kind == "wide":
        x = x * 10.0 ** rng.uniform(-150, 150, n)
    elif kind == "cancel":
        x = x * 10.0 ** rng.uniform(0, 30, n)
        x[n // 2:2 * (n // 2)] = -x[:n // 2]
    elif kind == "subnormal":
        x = x * 1e-310
    elif kind == "rising":
        x = np.sort(np.abs(x) * 10.0 ** rng.uniform(-300, 300, n))
    got, ref = vg.neumaier_sum(x), math.fsum(x)
    eps = 2.0 ** -52
    assert abs(got - ref) <= 4 * eps * abs(ref) + 4 * n * eps * eps * np.abs(x).sum() + 5e-324, (got, ref)
    x[n // 2] = np.inf  # the compensation of an infinite sum is inf - inf, as in the reference
    assert np.isnan(vg.neumaier_sum(x))


@pytest.mark.parametrize("big", [7.0e305, 1e306, 1.7e308, 1e300, 1.0])
@pytest.mark.parametrize("odd", [(np.inf, -np.inf), (np.nan,), (-np.nan,), (np.nan, -np.nan), (np.inf,), (-np.inf,)])
@pytest.mark.parametrize("n", [8, 5000])
def test_neumaier_nonfinite_beside_the_largest(vg, big, odd, n):
    """Infinities and NaN make the compensated sum NaN, as in the reference,
    also beside finite elements up to the largest double."""
    x = np.zeros(n)
    x[0] = big
    x[1:1 + len(odd)] = odd
    x[1 + len(odd)] = -big
    assert np.isnan(vg.neumaier_sum(x))
    x[1:1 + len(odd)] = 0.0
    assert vg.neumaier_sum(x) == 0.0


@pytest.mark.parametrize("case", ["winds", "depth", "dzeta"])
@pytest.mark.parametrize("dims", [(3, 1, 2), (300, 16, 18), (300, 77, 21)])
def test_cfl_scan_bounds_beyond_single_precision(vg, oc, case, dims):
    """Winds under 2^-126 beside tiny spacings, and dzeta and depths that single
    precision cuts to zero while their product is an ordinary thickness: the
    scan equals the oracle's bit for bit."""
    nx, ny, nz = dims
    n = nx * ny * nz
    u, v, w = np.zeros(n), np.zeros(n), np.zeros(n)
    dz, zs, z_top, dx = np.full(nz, 0.01), np.zeros(nx * ny), 20000.0, 1e-9
    if case == "winds":  # both winds of the first cell count as 2^-126, together above the second's
        u[0], v[0], v[1] = 1e-300, 1e-300, 2e-38
    else:  # w = 5 m/s where dz is 3.63 m has the larger bound and the smaller number than 2 m/s where it is 1.32 m
        dx = 1000.0
        w[0], w[nx * ny + 1] = 5.0, 2.0
        if case == "depth":
            dz[:], z_top = 1.1e-38, 3.3e38
            dz[1] = 4e-39
        else:
            dz[:], z_top = 2e38, 1e-38
            dz[1] = 3e38
            w[0], w[nx * ny + 1] = 5.0, 6.0  # dz = 2 m and 3 m: equal bounds per wind, 2.5 /s and 2 /s
    a, b = ctypes.c_double(), ctypes.c_double()
    ro = oc.port_lib().vo_cfl_scan(u.ctypes.data, v.ctypes.data, w.ctypes.data, dz.ctypes.data, zs.ctypes.data, nx, ny,
                                    nz, dx, dx, z_top, 6.0, ctypes.byref(a), ctypes.byref(b))
    r, mw, mdz = vg.cfl_scan(u, v, w, dz, zs, nx, ny, nz, dx, dx, z_top, 6.0)
    assert (r, mdz) == (ro, b.value), (r, ro, mdz, b.value)
    assert mw == a.value or abs(mw - a.value) <= 2.3e-16 * a.value


@pytest.mark.parametrize("dims", [(34, 10, 6), (62, 24, 45)])  # a thread per cell, tiles
@pytest.mark.parametrize("where", ["zs", "dzeta", "rho", "q", "w"])
@pytest.mark.parametrize("nan", [np.nan, -np.nan])
def test_flux_advection_nan_reaches_the_result(vg, oc, where, nan, dims):
    """A NaN in the metric or a field makes the cells that use it NaN, as in
    the oracle, and no others."""
    nx, ny, nz = dims
    rng = np.random.default_rng(1)
    n = nx * ny * nz
    f = dict(q=rng.random(n), rho=0.5 + rng.random(n), u=rng.random(n) - 0.5, v=rng.random(n) - 0.5,
             w=rng.random(n) - 0.5, dzeta=0.01 + 0.01 * rng.random(nz), zs=500.0 * rng.random(nx * ny))
    f[where][f[where].size // 2] = nan
    got = vg.advect_scalar_flux(f["q"], f["rho"], f["u"], f["v"], f["w"], f["dzeta"], f["zs"], nx, ny, nz, 900.0,
                                1100.0, 20000.0)
    ref = np.zeros(n)
    oc.port_lib().vo_advect_scalar_flux(*[f[k].ctypes.data for k in ("q", "rho", "u", "v", "w", "dzeta", "zs")], nx, ny,
                                         nz, 900.0, 1100.0, 20000.0, ref.ctypes.data)
    assert np.isnan(ref).any() and np.array_equal(np.isnan(got), np.isnan(ref))


@pytest.mark.parametrize("n", [1, 2, 7, 80, 129])
def test_thomas_sweep_error_against_64_bits(vg, n):
    """The batched sweep is no further from the extended-precision solution than
    a sweep that divides twice a row (the oracle's arithmetic with fused
    multiply-adds): 2-norms over 2000 diagonally dominant systems, to 2 %."""
    rng = np.random.default_rng(n)
    a, c = -3.0 * rng.random((2000, max(n - 1, 1))), -3.0 * rng.random((2000, max(n - 1, 1)))
    a, c = a[:, :n - 1], c[:, :n - 1]
    b, d = 1.0 + 0.5 * rng.random((2000, n)), rng.random((2000, n)) - 0.5
    b[:, 1:] -= a
    b[:, :-1] -= c
    rc, got = vg.tridiagonal_solve_batched(a, b, c, d)
    assert not np.any(rc)

    def sweep(t):  # t(x): a rounded value; products are exact in the wider type before they are
        w = np.longdouble
        x, cp = np.zeros((2000, n), w), np.zeros((2000, n), w)
        for k in range(n):
            l = a[:, k - 1].astype(w) if k else 0
            den = t(b[:, k] - l * (cp[:, k - 1] if k else 0))
            x[:, k] = t(t(d[:, k] - l * (x[:, k - 1] if k else 0)) / den)
            cp[:, k] = t(c[:, k].astype(w) / den) if k + 1 < n else 0
        for k in range(n - 2, -1, -1):
            x[:, k] = t(x[:, k] - cp[:, k] * x[:, k + 1])
        return x

    exact = sweep(lambda v: v)
    twice = sweep(lambda v: np.asarray(v, np.float64).astype(np.longdouble))
    err = lambda v: float(np.sqrt(((v - exact) ** 2).sum()))  # noqa: E731
    if np.finfo(np.longdouble).nmant <= 52:
        pytest.skip("no wider type on this host")
    assert err(got.reshape(2000, n)) <= 1.02 * err(twice)


@pytest.mark.parametrize("bits,n", [(64, 3), (64, 4), (64, 5), (64, 128), (64, 129), (64, 380), (64, 381), (32, 7),
                                    (32, 8), (32, 9), (32, 128), (32, 129), (32, 764), (32, 765)])
@pytest.mark.parametrize("n_sys", [1, 32, 255, 257, 2999])
def test_thomas_sweep_and_solver_limits(vg, oc, bits, n, n_sys):
    """At the edges of the on-chip sweep's stages (4 and 8 levels), at the tallest
    columns it holds and just above, for few systems and many, whichever kernel
    the batched call takes: against the oracle at the bounds above (1e-12; FP32
    1e-5), with a singular system between others."""
    import torch
    dt = torch.float64 if bits == 64 else torch.float32
    vp, i32 = ctypes.c_void_p, ctypes.c_int
    f = _dev(vg, "vibe_tridiagonal_solve_batched_f%d_dev" % bits, [vp] * 4 + [i32, i32, vp, vp, vp])
    rng = np.random.default_rng(n * 10000 + n_sys)
    a, c = (-rng.random((n_sys, n - 1)) for _ in range(2))
    b, d = 2.5 + rng.random((n_sys, n)), rng.random((n_sys, n)) - 0.5
    bad = n_sys // 3 if n_sys > 1 else -1
    if bad >= 0:
        b[bad, 0] = 0.0
    t = [torch.tensor(v, dtype=dt, device="cuda") for v in (a, b, c, d)]
    x = torch.full((n_sys, n), 7.0, dtype=dt, device="cuda")
    st = torch.full((n_sys,), -1, dtype=torch.int32, device="cuda")
    assert f(*[v.data_ptr() for v in t], n, n_sys, x.data_ptr(), st.data_ptr(),
             torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    host = [np.ascontiguousarray(v.double().cpu().numpy()) for v in t]
    got, status = x.double().cpu().numpy(), st.cpu().numpy()
    tol = 1e-12 if bits == 64 else 1e-5
    xo, ws = np.zeros(n), np.zeros(n)
    for s in range(n_sys):
        rc = oc.port_lib().vo_tridiagonal_solve(*[h[s].ctypes.data for h in host], n, xo.ctypes.data, ws.ctypes.data)
        assert status[s] == rc == (1 if s == bad else 0)
        if rc == 0:
            assert np.abs(got[s] - xo).max() <= tol * np.abs(xo).max()


@pytest.mark.parametrize("bits", [64, 32])
@pytest.mark.parametrize("thin", [False, True])
def test_flux_advection_error_against_wider_type(vg, bits, thin):
    """The tiled kernel is no further from the result in a wider type than the
    formula with its two divisions a cell, rounded at every operation: 2-norms
    over 62 x 40 x 40 cells, to 1 %; thin: layers under 1 m count as 1 m."""
    import torch
    dt, np_t = (torch.float64, np.float64) if bits == 64 else (torch.float32, np.float32)
    if bits == 64 and np.finfo(np.longdouble).nmant <= 52:
        pytest.skip("no wider type on this host")
    nx, ny, nz = 62, 40, 40
    rng = np.random.default_rng(bits)
    u, v, w = ((a * rng.random((nz, ny, nx)) - 0.5 * a).astype(np_t) for a in (40.0, 30.0, 4.0))
    q, rho = (300.0 + 5.0 * rng.random((nz, ny, nx))).astype(np_t), (0.2 + rng.random((nz, ny, nx))).astype(np_t)
    dz = ((2e-5 if thin else 0.01) * (1.0 + rng.random(nz))).astype(np_t)
    zs = (800.0 * rng.random((ny, nx))).astype(np_t)
    f = _dev(vg, "vibe_advect_scalar_flux_f%d_dev" % bits, [ctypes.c_void_p] * 7 + [ctypes.c_int] * 3 +
             [ctypes.c_double if bits == 64 else ctypes.c_float] * 3 + [ctypes.c_void_p] * 2)
    t = [torch.tensor(a, dtype=dt, device="cuda") for a in (q, rho, u, v, w, dz, zs)]
    out = torch.empty((nz, ny, nx), dtype=dt, device="cuda")
    assert f(*[a.data_ptr() for a in t], nx, ny, nz, 900.0, 1100.0, 20000.0, out.data_ptr(),
             torch.cuda.current_stream().cuda_stream) == 0

    def formula(wide, r):  # r rounds to the kernel's type (or not at all)
        U, V, W, Q, R, D, S = (a.astype(wide) for a in (u, v, w, q, rho, dz, zs))
        thick = np.maximum(r(D[:, None, None] * r(wide(20000.0) - S)), 1)

        def diff(vel, ax):  # of the fluxes through a cell's two faces
            f = r(r(vel * r(R + np.roll(R, 1, ax))) * r(Q + np.roll(Q, 1, ax)))
            return r(np.roll(f, -1, ax) - f) / 4

        h = r(r(diff(U, 2) * r(wide(1) / wide(900.0))) + r(diff(V, 1) * r(wide(1) / wide(1100.0))))
        z = diff(W, 0)
        z[0], z[-1] = 0, 0
        return -r(r(h + r(z / thick)) / R)

    wide = np.longdouble if bits == 64 else np.float64
    exact = formula(wide, lambda a: a)
    twice = formula(wide, lambda a: np.asarray(a, np_t).astype(wide))
    err = lambda a: float(np.sqrt(((a - exact) ** 2).sum()))  # noqa: E731
    assert err(out.cpu().numpy().astype(wide)) <= 1.01 * err(twice)


@pytest.mark.parametrize("bits", [64, 32])
@pytest.mark.parametrize("dims", [(63, 17, 120), (94, 25, 61), (31, 8, 400), (62, 9, 200), (124, 48, 11), (186, 16, 25),
                                  (5, 700, 30), (4000, 1, 20), (16, 512, 9), (33, 33, 33)])
def test_flux_advection_tiles_and_cells(vg, oc, bits, dims):
    """Grids large enough for the tiled kernel, with ragged last tiles and level
    chunks, and grids that fill its tiles badly and take a thread per cell:
    against the oracle at the bounds above (1e-12; FP32 1e-4)."""
    import torch
    nx, ny, nz = dims
    dt = torch.float64 if bits == 64 else torch.float32
    f = _dev(vg, "vibe_advect_scalar_flux_f%d_dev" % bits, [ctypes.c_void_p] * 7 + [ctypes.c_int] * 3 +
             [ctypes.c_double if bits == 64 else ctypes.c_float] * 3 + [ctypes.c_void_p] * 2)
    rng = np.random.default_rng(nx + ny)
    n = nx * ny * nz
    fields = [rng.random(n), 0.5 + rng.random(n), 20 * rng.random(n) - 10, 20 * rng.random(n) - 10, rng.random(n) - 0.5,
              0.01 + 0.01 * rng.random(nz), 500.0 * rng.random(nx * ny)]
    t = [torch.tensor(v, dtype=dt, device="cuda") for v in fields]
    host = [np.ascontiguousarray(v.double().cpu().numpy()) for v in t]
    for zs in (True, False):
        out = torch.full((n,), float("nan"), dtype=dt, device="cuda")
        assert f(*[v.data_ptr() for v in t[:6]], t[6].data_ptr() if zs else None, nx, ny, nz, 900.0, 1100.0, 20000.0,
                 out.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        ref = np.full(n, np.nan)
        oc.port_lib().vo_advect_scalar_flux(*[h.ctypes.data for h in host[:6]], host[6].ctypes.data if zs else None,
                                             nx, ny, nz, 900.0, 1100.0, 20000.0, ref.ctypes.data)
        tol = 1e-12 if bits == 64 else 1e-4
        assert np.abs(out.double().cpu().numpy() - ref).max() <= tol * np.abs(ref).max()


@pytest.mark.parametrize("kind", ["white", "uniform", "near", "calm", "tiny", "huge", "nonfinite", "odd_metric", "steps"])
@pytest.mark.parametrize("dims", [(260, 16, 17), (97, 65, 33), (300, 77, 21), (511, 257, 6)])
def test_cfl_scan_tiles_change_no_bit(vg, oc, kind, dims):
    """The tiled scan (two and four levels a tile) equals the oracle's bit for bit:
    also where most cells lie at the best (a uniform wind, one that differs in its
    last bits, one that grows from cell to cell)."""
    nx, ny, nz = dims
    n = nx * ny * nz
    rng = np.random.default_rng(n)
    u, v, w = (20.0 * rng.standard_normal(n) for _ in range(3))
    dz, zs, dt = 0.01 + 0.02 * rng.random(nz), 500.0 * rng.random(nx * ny), 6.0
    if kind == "uniform":
        u[:], v[:], w[:] = -10.0, 5.0, 0.0
    elif kind == "near":
        u, v, w = 10.0 + 1e-14 * rng.standard_normal(n), 1e-6 * v, 1e-7 * w
    elif kind == "calm":
        u, v, w = np.zeros(n), np.zeros(n), np.zeros(n)
    elif kind == "tiny":
        u, v, w = (1e-40 * a for a in (u, v, w))
        u[n // 2] = 1e-310
    elif kind == "huge":
        u, v, w = (10.0 ** rng.uniform(20, 150, n) * np.sign(a) for a in (u, v, w))
    elif kind == "nonfinite":
        u[n // 3], v[n // 2], w[n - 1], zs[0] = np.nan, -np.inf, np.nan, np.nan
    elif kind == "odd_metric":
        dz, zs = rng.standard_normal(nz) * 10.0 ** rng.uniform(-3, 3, nz), 40000.0 * rng.random(nx * ny)
    elif kind == "steps":
        u, v, w = 10.0 + 1e-9 * np.arange(n), -3.0 - 1e-9 * np.arange(n)[::-1], np.full(n, 0.5)
    with np.errstate(all="ignore"):
        for step in (dt, -dt, 1e-40):
            r, mw, mdz = vg.cfl_scan(u, v, w, dz, zs, nx, ny, nz, 900.0, 1100.0, 20000.0, step)
            a, b = ctypes.c_double(), ctypes.c_double()
            ro = oc.port_lib().vo_cfl_scan(u.ctypes.data, v.ctypes.data, w.ctypes.data, dz.ctypes.data, zs.ctypes.data,
                                            nx, ny, nz, 900.0, 1100.0, 20000.0, step, ctypes.byref(a), ctypes.byref(b))
            assert (r, mdz) == (ro, b.value), (step, r, ro, mdz, b.value)
            assert mw == a.value or abs(mw - a.value) <= 2.3e-16 * a.value, (mw, a.value)  # the sum's FMA contraction


@pytest.mark.parametrize("kind", ["white", "uniform", "near", "calm", "nonfinite"])
@pytest.mark.parametrize("dims", [(512, 257, 65), (255, 130, 40)])
def test_cfl_scan_f32_against_torch(vg, kind, dims):
    """FP32, tiled (8.6 M cells) and cell by cell, against the same formula in
    torch's FP32: bit for bit but for the speed, whose sum may be contracted."""
    import torch
    nx, ny, nz = dims
    g = torch.Generator(device="cuda").manual_seed(nx)
    u, v, w = (20.0 * torch.randn(nz, ny, nx, device="cuda", generator=g) for _ in range(3))
    dz = 0.01 + 0.02 * torch.rand(nz, device="cuda", generator=g)
    zs = 500.0 * torch.rand(ny, nx, device="cuda", generator=g)
    if kind == "uniform":
        u, v, w = torch.full_like(u, 10.0), torch.full_like(u, -5.0), torch.zeros_like(u)
    elif kind == "near":
        u, v, w = 10.0 + 1e-6 * u, 1e-4 * v, 1e-5 * w
    elif kind == "calm":
        u, v, w = (torch.zeros_like(u) for _ in range(3))
    elif kind == "nonfinite":
        u.view(-1)[5], v.view(-1)[u.numel() // 2], w.view(-1)[-1] = float("nan"), float("nan"), float("nan")
    f = _dev(vg, "vibe_cfl_scan_f32_dev", [ctypes.c_void_p] * 5 + [ctypes.c_int] * 3 + [ctypes.c_float] * 4 +
             [ctypes.c_void_p] * 2)
    out = torch.empty(3, device="cuda")
    for step in (6.0, -6.0):
        assert f(u.data_ptr(), v.data_ptr(), w.data_ptr(), dz.data_ptr(), zs.data_ptr(), nx, ny, nz, 900.0, 1100.0,
                 20000.0, step, out.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        thick = (dz[:, None, None] * (20000.0 - zs)).clamp(min=1.0)
        dx, dy = torch.full_like(u, 900.0), torch.full_like(u, 1100.0)  # (torch multiplies by a number's reciprocal)
        c = step * (u.abs() / dx + v.abs() / dy + w.abs() / thick)
        s = (u * u + v * v + w * w).sqrt()
        got = out.tolist()
        assert got[0] == max(0.0, float(c.nan_to_num(nan=0.0).max()))
        assert abs(got[1] - float(s.nan_to_num(nan=0.0).max())) <= 2.4e-7 * got[1]
        assert got[2] == float(thick.min())
