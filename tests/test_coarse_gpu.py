"""The coarsest-level solve (stands in for cholesky_factorization / cholesky_solve): the blocked
Gauss-Jordan inverse, and on the plain FP64 path for large coarsest levels the FP32 inverse refined
against the FP64 coarsest operator. Through the C ABI."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _vcycles(w, dm, r, f64_direct_max):
    dm.set_option("coarse_f64_direct_max", f64_direct_max)
    try:
        dm.setup(w['visc'], w['dens'], w['ifix'], w['vfix'], w['phys'], precision=0)
        return dm.vcycle(r)
    finally:
        dm.set_option("coarse_f64_direct_max", 6000)


def test_refined_fp64_coarse_solve_equals_the_fp64_inverse(built_lib, tiny_plates):
    """The refined coarse solve (FP32 inverse + 3 refinement steps against the FP64 operator) gives
    the V-cycle of the FP64 inverse to FP64 rounding."""
    from m3tet_sph_gb300 import stokes
    w = tiny_plates
    dm = stokes.DeviceMesh(w['levels'])
    try:
        rng = np.random.default_rng(3)
        r = rng.standard_normal(dm.ndof)
        d_direct = _vcycles(w, dm, r, 6000)
        d_ref = _vcycles(w, dm, r, 0)
        assert np.linalg.norm(d_ref - d_direct) < 1e-12 * np.linalg.norm(d_direct)
    finally:
        dm.close()


def test_17k_coarsest_level(built_lib):
    """The 130,662-DOF shell on 2 levels puts 17,334 dofs on the coarsest level (the size of the
    4-level 8M-DOF and the 5-level 64M-DOF hierarchies). On that problem the plain FP64 path with the
    refined coarse solve and the FP32 V-cycle path (FP32 inverse) both reach the solution of the
    plain FP64 path with the FP64 inverse of the coarsest level."""
    from m3tet_sph_gb300 import stokes, workloads
    kw = dict(rtol_Pat=1e-9, rtol_U=5e-3, itmax_Pat=400, itmax_U=40, target_rel_residual=1e-11)
    w = workloads.make_workload('c1', nmg=2)
    assert 3 * w['levels'][1]['nnod'] == 17334
    sols, its = {}, {}
    dm = stokes.DeviceMesh(w['levels'])
    try:
        for name, prec, direct_max in (("fp64 inverse", 0, 20000), ("fp64 refined", 0, 6000), ("fp32", 1, 6000)):
            dm.set_option("coarse_f64_direct_max", direct_max)
            dm.setup(w['visc'], w['dens'], w['ifix'], w['vfix'], w['phys'], precision=prec)
            U, P, info = dm.solve(**kw)
            assert info['rel_residual'] <= 1e-11, (name, info)
            its[name] = info['nitU'] + info['nitZ']
            print(f"{name}: {its[name]} MG-PCG iterations, set-up {info['t_setup_ms']:.1f} ms")
            sols[name] = (U, P - P.mean())
    finally:
        dm.set_option("coarse_f64_direct_max", 6000)
        dm.close()
    U0, P0 = sols["fp64 inverse"]
    for name in ("fp64 refined", "fp32"):
        U, P = sols[name]
        assert np.linalg.norm(U - U0) < 1e-8 * np.linalg.norm(U0), name
        assert np.linalg.norm(P - P0) < 1e-8 * np.linalg.norm(P0), name
    assert abs(its["fp64 refined"] - its["fp64 inverse"]) <= 2


@pytest.mark.parametrize("precision,direct_max", [(0, 6000), (0, 0), (1, 6000)])
def test_coarsest_level_without_free_dofs(built_lib, tiny_plates, precision, direct_max):
    """Every velocity dof prescribed: the set-up succeeds, the force vector is the one of a set-up with
    free dofs (it does not depend on them) and a V-cycle gives zero."""
    from m3tet_sph_gb300 import stokes
    w = tiny_plates
    dm = stokes.DeviceMesh(w['levels'])
    try:
        dm.setup(w['visc'], w['dens'], w['ifix'], w['vfix'], w['phys'], precision=precision)
        f = dm.force()
        rng = np.random.default_rng(8)
        dm.set_option("coarse_f64_direct_max", direct_max)
        dm.setup(w['visc'], w['dens'], np.arange(dm.ndof), rng.standard_normal(dm.ndof), w['phys'],
                 precision=precision)
        assert np.array_equal(dm.force(), f)
        assert not dm.element_matrices()[0].any()
        assert not dm.vcycle(rng.standard_normal(dm.ndof)).any()
        # the next set-up has free dofs again
        dm.setup(w['visc'], w['dens'], w['ifix'], w['vfix'], w['phys'], precision=precision)
        assert dm.vcycle(rng.standard_normal(dm.ndof)).any()
    finally:
        dm.set_option("coarse_f64_direct_max", 6000)
        dm.close()


# mean relative error of a V-cycle with the unrefined FP32 inverse, when the inverse was formed by FP32
# multiply-adds throughout: (surface level, layers, free dofs of the coarsest level, seeds of the dofs
# fixed for that): over 3 x 8 vectors (None: every free dof, 8 vectors)
FP32_INVERSE = [(2, 2, 100, 1, 3.99e-9), (2, 2, 129, 3, 8.65e-9), (2, 2, 250, 3, 1.81e-8), (2, 2, 500, 3, 5.07e-8),
                (2, 2, None, 1, 1.94e-7), (2, 4, None, 1, 9.58e-8), (3, 2, None, 1, 3.96e-7), (3, 4, 5996, 1, 9.12e-8),
                (3, 4, 6094, 1, 1.01e-7)]


@pytest.mark.parametrize("level,layers,nfree,seeds,bound", FP32_INVERSE)
def test_fp32_inverse_is_as_accurate_as_fp32_multiply_adds(built_lib, level, layers, nfree, seeds, bound):
    """The FP32 inverse by itself (no refinement) against the FP64 inverse, 1 to 48 panels of 128, the last
    ones partial, either side of the size from which the next diagonal block runs ahead: the error of a
    V-cycle is that of an inverse formed with FP32 multiply-adds (the figures above), which may differ by
    20 % with the matrix on small ones. (Without the correction for truncation the errors are 1.1 to 1.3
    times the figures from 7 panels on.)"""
    from m3tet_sph_gb300 import stokes, workloads
    w = workloads.make_workload('c2', level=level, nlayer=layers, nmg=2)
    nc = 3 * w['levels'][-1]['nnod']
    rhs_seeds = range(6) if nfree in (100, 5996, 6094) else range(8)
    d = stokes.DeviceMesh(w['levels'])
    err = []
    try:
        for seed in range(seeds):
            ifix, vfix = w['ifix'], w['vfix']
            if nfree is not None:
                free = np.setdiff1d(np.arange(nc), ifix)
                seed = 7 if seeds == 1 else seed
                more = np.random.default_rng(seed).permutation(free)[:len(free) - nfree]
                ifix, vfix = np.concatenate([ifix, more]), np.concatenate([vfix, np.zeros(len(more))])
            out = []
            for direct_max, sweeps in ((20000, 3), (0, 0)):
                d.set_option("coarse_f64_direct_max", direct_max)
                d.set_option("coarse_refine_sweeps", sweeps)
                d.setup(w['visc'], w['dens'], ifix, vfix, w['phys'], precision=0)
                out.append([d.vcycle(np.random.default_rng(s).standard_normal(d.ndof)) for s in rhs_seeds])
            err += [np.linalg.norm(b - a) / np.linalg.norm(a) for a, b in zip(*out)]
    finally:
        d.set_option("coarse_f64_direct_max", 6000)
        d.set_option("coarse_refine_sweeps", 3)
        d.close()
    assert np.mean(err) <= 1.2 * bound
