"""Finest-level element passes on meshes whose element count is not a multiple of their tiles and blocks
(64 and 128 elements): partially assembled FP32 apply, gradient, divergence and inverse diagonal against
the FP64 element matrices summed on the host."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (surface level, layers, MG levels): 60, 240, 480, 720 and 3,840 elements
SIZES = [(0, 1, 1), (1, 1, 1), (1, 2, 2), (1, 3, 1), (2, 4, 2)]


@pytest.fixture(params=SIZES, ids=lambda p: f"L{p[0]}x{p[1]}")
def dm(request, built_lib):
    from m3tet_sph_gb300 import stokes, workloads
    level, layers, nmg = request.param
    w = workloads.make_workload('c2', level=level, nlayer=layers, nmg=nmg)
    d = stokes.DeviceMesh(w['levels'])
    d.setup(w['visc'], w['dens'], w['ifix'], w['vfix'], w['phys'], precision=1)
    yield w, d
    d.close()


def test_element_passes(dm):
    w, d = dm
    f = w['levels'][0]
    EL, n, nv = f['EL2NOD'], 3 * f['nnod'], d.nvnod
    K, G, _ = d.element_matrices()
    dof = (3 * EL[:, :, None] + np.arange(3)).reshape(len(EL), 30)
    rng = np.random.default_rng(5)
    x, q = rng.standard_normal(n), rng.standard_normal(nv)
    free = np.ones(n, bool)
    free[w['ifix']] = False
    # K is masked: fixed rows and columns are zero
    y = np.bincount(dof.ravel(), np.einsum('eij,ej->ei', K, x[dof]).ravel(), n)
    y32 = d.level_apply32(0, x.astype(np.float32))
    # FP32 rounding (6e-8) over sums of a few hundred terms of either sign
    assert np.linalg.norm(y32 - y) <= 1e-5 * np.linalg.norm(y)
    assert np.all(y32[~free] == 0)
    # FP64 sums of at most a few hundred terms
    g = np.bincount(dof.ravel(), np.einsum('eip,ep->ei', G, q[EL[:, :4]]).ravel(), n)
    assert np.linalg.norm(d.grad(q) - g) <= 1e-13 * np.linalg.norm(g)
    s = np.bincount(EL[:, :4].ravel(), np.einsum('eip,ei->ep', G, x[dof]).ravel(), nv)
    assert np.linalg.norm(d.div(x) - s) <= 1e-13 * np.linalg.norm(s)
    D = np.bincount(dof.ravel(), np.einsum('eii->ei', K).ravel(), n)
    Di = np.where(free & (D != 0), 1.0 / np.where(D != 0, D, 1.0), 0.0)
    assert np.allclose(d.level_inverse_diag32(0), Di, rtol=1e-6, atol=0)


@pytest.mark.parametrize("level,layers", [(1, 2), (1, 4), (2, 2)])
def test_coarse_inverse_panel_edges(level, layers, built_lib):
    """Coarsest levels whose free dofs do not fill the last panel (378, 630 and 1,458 dofs in all): the
    FP64 inverse and the FP32 inverse refined against the FP64 operator give the same V-cycle. Three
    refinements leave (FP32 rounding x condition)^4, far below FP64 rounding; 1e-11 covers the
    conditioning of the levels above."""
    from m3tet_sph_gb300 import stokes, workloads
    w = workloads.make_workload('c2', level=level, nlayer=layers, nmg=2)
    d = stokes.DeviceMesh(w['levels'])
    try:
        r = np.random.default_rng(3).standard_normal(d.ndof)
        out = []
        for direct_max in (6000, 0):
            d.set_option("coarse_f64_direct_max", direct_max)
            d.setup(w['visc'], w['dens'], w['ifix'], w['vfix'], w['phys'], precision=0)
            out.append(d.vcycle(r))
        assert np.linalg.norm(out[1] - out[0]) < 1e-11 * np.linalg.norm(out[0])
    finally:
        d.set_option("coarse_f64_direct_max", 6000)
        d.close()


def test_coarse_inverse_diagonal_block_ahead(built_lib):
    """A coarsest level of 9,630 dofs, whose FP32 inverse updates and inverts each diagonal block beside the
    other tiles, against the FP64 inverse, as above."""
    from m3tet_sph_gb300 import stokes, workloads
    w = workloads.make_workload('c2', level=3, nlayer=4, nmg=2)
    d = stokes.DeviceMesh(w['levels'])
    try:
        r = np.random.default_rng(4).standard_normal(d.ndof)
        out = []
        for direct_max in (20000, 0):
            d.set_option("coarse_f64_direct_max", direct_max)
            d.setup(w['visc'], w['dens'], w['ifix'], w['vfix'], w['phys'], precision=0)
            out.append(d.vcycle(r))
        assert np.linalg.norm(out[1] - out[0]) < 1e-11 * np.linalg.norm(out[0])
    finally:
        d.set_option("coarse_f64_direct_max", 6000)
        d.close()


@pytest.mark.parametrize("split", [0, 1])
def test_products_without_streaming(dm, split):
    """The finest-level products with stream_apply and stream_outer off, either form: FP64, double-float
    and FP32 against the FP64 element matrices summed on the host; one launch for the elements and one for
    the nodes. Tolerances as above: rounding (6e-8, 1e-14 of double-float, 1e-16) over sums of a few
    hundred terms."""
    import ctypes as C
    from m3tet_sph_gb300 import _lib as L

    def launches():
        n = C.c_ulonglong()
        L.check(L.lib().m3sph_launch_count(C.byref(n)))
        return n.value

    w, d = dm
    EL, n = w['levels'][0]['EL2NOD'], 3 * w['levels'][0]['nnod']
    K, _, _ = d.element_matrices()
    dof = (3 * EL[:, :, None] + np.arange(3)).reshape(len(EL), 30)
    x = np.random.default_rng(6).standard_normal(n).astype(np.float32).astype(np.float64)
    y = np.bincount(dof.ravel(), np.einsum('eij,ej->ei', K, x[dof]).ravel(), n)
    opts = dict(stream_apply=0, stream_outer=0, fp32_operator=0, split_apply=split)
    try:
        for k, v in opts.items():
            d.set_option(k, v)
        for fn, tol in ((lambda: d.level_apply(0, x), 1e-13), (lambda: d.apply(x), 1e-11),
                        (lambda: d.level_apply32(0, x.astype(np.float32)), 1e-5)):
            n0 = launches()
            got = fn()
            assert launches() - n0 == 2
            assert np.linalg.norm(got - y) <= tol * np.linalg.norm(y)
            assert np.array_equal(fn(), got)
    finally:
        for k in opts:
            d.set_option(k, 1)
