"""Failure visibility of the Stokes solve, through the C ABI: a Patera iteration that runs out of
iterations is reported as M3SPH_ERR_NOT_CONVERGED (with the last iterate still delivered), and a
learned smoother that stops contracting is switched off by the outer FP64 CG without changing the
converged answer."""
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def dm_plates(built_lib, tiny_plates):
    from m3tet_sph_gb300 import stokes
    w = tiny_plates
    dm = stokes.DeviceMesh(w['levels'])
    yield w, dm
    dm.close()


def test_itmax_pat_exhausted_is_not_converged(dm_plates):
    from m3tet_sph_gb300 import _lib as L
    w, dm = dm_plates
    dm.setup(w['visc'], w['dens'], w['ifix'], w['vfix'], w['phys'], precision=0)
    kw = dict(rtol_Pat=1e-12, rtol_U=1e-3, itmax_Pat=2, itmin_Pat=1, itmax_U=20)
    with pytest.raises(L.M3SphError) as ei:
        dm.solve(**kw)
    assert ei.value.code == L.ERR_NOT_CONVERGED
    assert 'not converged' in str(ei.value)
    U, P, info = ei.value.result
    assert info['status'] == L.ERR_NOT_CONVERGED and info['itPat'] == 2
    assert np.isfinite(U).all() and np.isfinite(P).all() and np.linalg.norm(U) > 0
    # the same call with the status accepted returns the same iterate
    U2, P2, info2 = dm.solve(allow_not_converged=True, **kw)
    assert info2['status'] == L.ERR_NOT_CONVERGED
    assert np.array_equal(U, U2) and np.array_equal(P, P2)
    # the device-resident step reports it too
    with pytest.raises(L.M3SphError) as ei:
        dm.step_device(**kw)
    assert ei.value.code == L.ERR_NOT_CONVERGED


def test_unreachable_target_is_not_converged(dm_plates):
    from m3tet_sph_gb300 import _lib as L
    w, dm = dm_plates
    dm.setup(w['visc'], w['dens'], w['ifix'], w['vfix'], w['phys'], precision=1)
    U, P, info = dm.solve(rtol_Pat=1e-6, itmax_Pat=6, target_rel_residual=1e-30, allow_not_converged=True)
    assert info['status'] == L.ERR_NOT_CONVERGED and info['rel_residual'] > 1e-30
    # a reachable target converges with status 0
    U, P, info = dm.solve(rtol_Pat=1e-6, itmax_Pat=200, target_rel_residual=1e-8)
    assert info['status'] == 0 and info['rel_residual'] <= 1e-8


def test_learned_smoother_fallback_is_forced_and_harmless(dm_plates):
    """A smoother that amplifies the error (the trained network's correction negated and scaled by
    3) makes the MG-PCG residual grow; the rate check must switch it off (smoother_fallbacks >= 1)
    and the solve must reach the same answer as the Jacobi-smoothed one."""
    from m3tet_sph_gb300 import learned
    w, dm = dm_plates
    dm.setup(w['visc'], w['dens'], w['ifix'], w['vfix'], w['phys'], precision=1)
    p = np.load(Path(learned.__file__).with_name('smoother_c1.npy')).astype(np.float32)
    bad = p.copy()
    bad[8320:] *= -1.0                      # W2 and b2 negated: the correction points the wrong way
    learned.set_params(dm, bad, trained=True)
    dm.set_option("ml_omega_pct", 300)
    kw = dict(rtol_Pat=1e-8, rtol_U=5e-3, itmax_Pat=200, itmax_U=40, target_rel_residual=1e-8)
    try:
        U0, P0, i0 = dm.solve(smoother=0, **kw)
        U1, P1, i1 = dm.solve(smoother=1, **kw)
    finally:
        dm.set_option("ml_omega_pct", 100)
        learned.set_params(dm, p, trained=True)
    assert i1['smoother_fallbacks'] >= 1, i1
    assert i0['smoother_fallbacks'] == 0
    assert i1['rel_residual'] <= 1e-8 and i0['rel_residual'] <= 1e-8
    assert np.linalg.norm(U1 - U0) < 1e-6 * np.linalg.norm(U0)
    Pc0, Pc1 = P0 - P0.mean(), P1 - P1.mean()
    assert np.linalg.norm(Pc1 - Pc0) < 1e-6 * np.linalg.norm(Pc0)


def test_calculate_dt_matches_oracle(dm_plates):
    """Device max-reduction CFL step (calculate_dt.m:40-52) on the resident velocity: bit-identical
    to the oracle's on the same velocity (a max is exact; one division and one multiply)."""
    from oracle import stokes_oracle as O
    w, dm = dm_plates
    dm.setup(w['visc'], w['dens'], w['ifix'], w['vfix'], w['phys'], precision=1)
    dm.solve(rtol_Pat=1e-6, itmax_Pat=200)
    U, _ = dm.solution()
    X = w['levels'][0]['GCOORD']
    for limit, dtmax in ((0.005, 0.1), (0.005, 1e-30), (1.0, 1e30)):
        dt, adv = dm.calculate_dt(limit, dtmax)
        dt_r, adv_r = O.calculate_dt(X, U[0::3], U[1::3], U[2::3], limit, dtmax)
        assert dt == dt_r and adv == adv_r, (limit, dtmax, dt, dt_r)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("is_abs_tol", [False, True])
def test_nan_right_hand_side_leaves_the_iterate(dm_plates, precision, is_abs_tol):
    """A NaN right-hand side is an error with either kind of tolerance, and the resident velocity is
    the initial guess afterwards, bit for bit."""
    from m3tet_sph_gb300 import _lib as L
    w, dm = dm_plates
    dm.setup(w['visc'], w['dens'], w['ifix'], w['vfix'], w['phys'], precision=precision)
    rng = np.random.default_rng(12)
    x0, b = rng.standard_normal(dm.ndof), rng.standard_normal(dm.ndof)
    dm.mgpcg(b, x0, 1e-3, is_abs_tol, itmax=0)          # x0 is the resident velocity now
    U0, _ = dm.solution()
    free = np.setdiff1d(np.arange(dm.ndof), w['ifix'])
    b[free[len(free) // 2]] = np.nan
    with pytest.raises(L.M3SphError, match='RHS vector contains NaNs') as ei:
        dm.mgpcg(b, x0, 1e-3, is_abs_tol, itmax=7)
    assert ei.value.code == 3
    assert np.array_equal(dm.solution()[0], U0)


@pytest.mark.parametrize("word", [1, 2, 3])
@pytest.mark.parametrize("graphs", [0, 1])
def test_a_wait_that_gave_up_is_reported(dm_plates, graphs, word):
    """With the error word of a bounded wait set (as a kernel sets it whose wait gives up, so that its
    products are wrong), the V-cycle, the velocity CG and the solve fail instead of returning a result,
    the CG ends with the iteration that saw it, and the call after is clean."""
    import ctypes as C
    from m3tet_sph_gb300 import _lib as L, learned
    w, dm = dm_plates
    dm.setup(w['visc'], w['dens'], w['ifix'], w['vfix'], w['phys'], precision=1)
    learned.set_params(dm, np.load(Path(learned.__file__).with_name('smoother_c1.npy')), trained=True)

    def launches():
        n = C.c_ulonglong()
        L.check(L.lib().m3sph_launch_count(C.byref(n)))
        return n.value

    rng = np.random.default_rng(9)
    b, x0 = rng.standard_normal(dm.ndof), np.zeros(dm.ndof)
    calls = (lambda: dm.vcycle(b), lambda: dm.mgpcg(b, x0, 0.0, True, 60)[0],
             lambda: dm.mgpcg(b, x0, 0.0, True, 0)[0], lambda: dm.solve(rtol_Pat=1e-4, allow_not_converged=True)[0])
    try:
        dm.set_option("graphs", graphs)
        dm.mgpcg(b, x0, 0.0, True, 1)                    # captures the loop
        n0 = launches()
        dm.mgpcg(b, x0, 0.0, True, 1)
        n1 = launches()
        for k, call in enumerate(calls):
            want = call()
            dm.set_option("wait_error", word)
            n2 = launches()
            with pytest.raises(L.M3SphError, match='bounded wait') as ei:
                call()
            assert ei.value.code == L.ERR_CUDA
            if k == 1:
                assert launches() - n2 == n1 - n0
            assert np.array_equal(call(), want)
    finally:
        dm.set_option("graphs", 1)


@pytest.mark.parametrize("precision,itmax", [(0, 1), (0, 2), (0, 255), (0, 256), (0, 257), (0, 513),
                                             (1, 1), (1, 255), (1, 256), (1, 257)])
def test_captured_loop_and_host_loop_agree(dm_plates, precision, itmax):
    """The captured CG loop runs 256 iterations before the host looks at it; without graphs the host
    runs every iteration. Both launch the same kernels in the same order: exactly itmax iterations for a
    tolerance that is never met, and the same bits. Viscosities over 8 decades and a large right-hand side
    keep the residual of so many iterations above the smallest FP32 (FP64) numbers, where every form breaks
    down."""
    w, dm = dm_plates
    visc = 10.0 ** np.random.default_rng(2).uniform(-4, 4, len(w['visc']))
    dm.setup(visc, w['dens'], w['ifix'], w['vfix'], w['phys'], precision=precision)
    rng = np.random.default_rng(14)
    b, x0 = rng.standard_normal(dm.ndof) * (1e30 if precision else 1e60), rng.standard_normal(dm.ndof)
    out = []
    try:
        for graphs in (1, 0):
            dm.set_option("graphs", graphs)
            # the second ends at the same iteration for both, in between
            out.append(dm.mgpcg(b, x0, 0.0, True, itmax) + dm.mgpcg(b, x0, 1e-3, False, itmax))
    finally:
        dm.set_option("graphs", 1)
    g, h = out
    assert g[1] == h[1] == itmax and g[4] == h[4] <= itmax
    for k in (0, 2, 3, 5):
        assert np.array_equal(g[k], h[k])


@pytest.mark.parametrize("graphs", [0, 1])
def test_solve_with_either_loop(dm_plates, graphs):
    """The learned solve, whose CG may switch the smoother off, with the captured and the host loop."""
    from m3tet_sph_gb300 import learned
    w, dm = dm_plates
    dm.setup(w['visc'], w['dens'], w['ifix'], w['vfix'], w['phys'], precision=1)
    learned.set_params(dm, np.load(Path(learned.__file__).with_name('smoother_c1.npy')), trained=True)
    kw = dict(rtol_Pat=1e-8, rtol_U=5e-3, itmax_Pat=200, itmax_U=40, target_rel_residual=1e-8, smoother=1)
    ref = dm.solve(**kw)
    try:
        dm.set_option("graphs", graphs)
        got = dm.solve(**kw)
    finally:
        dm.set_option("graphs", 1)
    assert got[2]['itPat'] == ref[2]['itPat'] and got[2]['nvcycle'] == ref[2]['nvcycle']
    assert got[2]['smoother_fallbacks'] == ref[2]['smoother_fallbacks']
    assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])


def test_operator_calls_report_a_wait_that_gave_up(dm_plates):
    """The finest-level products and the training pairs made from them do too."""
    from m3tet_sph_gb300 import _lib as L
    w, dm = dm_plates
    dm.setup(w['visc'], w['dens'], w['ifix'], w['vfix'], w['phys'], precision=1)
    x = np.random.default_rng(10).standard_normal(dm.ndof)
    L.check(L.lib().m3sph_ml_reserve(dm.h, 1 << 16))

    def collect():
        L.check(L.lib().m3sph_ml_collect(dm.h, 1, 1, 8, None))

    for call in (lambda: dm.apply(x), lambda: dm.level_apply(0, x), lambda: dm.level_apply32(0, x), collect):
        dm.set_option("wait_error", 1)
        with pytest.raises(L.M3SphError, match='bounded wait'):
            call()
        call()


def test_a_failed_allocation_is_reported_once(built_lib, tiny_plates):
    """An allocation that does not fit fails its call and not the one after it."""
    from m3tet_sph_gb300 import _lib as L, stokes
    w = tiny_plates
    dm = stokes.DeviceMesh(w['levels'])
    try:
        dm.setup(w['visc'], w['dens'], w['ifix'], w['vfix'], w['phys'], precision=1)
        x = np.random.default_rng(11).standard_normal(dm.ndof)
        y = dm.apply(x)
        assert L.lib().m3sph_ml_reserve(dm.h, 10 ** 13) == L.ERR_CUDA
        assert np.array_equal(dm.apply(x), y)
    finally:
        dm.close()
