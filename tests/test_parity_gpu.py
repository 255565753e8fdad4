"""Parity of the CUDA kernels with the oracle (the reference's algorithm
restated in C, pinned to the reference's own kernels) and with the golden
vectors of the reference itself.

Tolerances (largest |out - ref| over the largest |ref|, the reference's
rel_maxdiff, include/bk_harness.h:74-83):
  FP64 engines (DFMA, float-float)     1e-12  (the target of the work)
  FP32 storage (FP32, MIXED)           1e-5   (the reference's fail_mark)
"""
import numpy as np
import pytest
import torch

import oracle
from gpu_util import dev, gpu_apply, host, oracle_apply, random_case, sizes

pytestmark = pytest.mark.gpu

TOL64 = 1e-12
TOL32 = 1e-5
P_ALL = list(range(1, 9))


@pytest.fixture(scope="module", autouse=True)
def _cuda(bklib):
    assert torch.cuda.is_available(), "the GPU tests need CUDA: the product has no CPU path"
    bklib.device_status(reset=True)
    yield
    assert bklib.device_status(reset=True) == bklib.BK_OK


@pytest.mark.parametrize("bk", [1, 3, 5])
@pytest.mark.parametrize("p", P_ALL)
@pytest.mark.parametrize("engine", ["dfma", "ff"])
def test_fp64_random(bklib, bk, p, engine):
    E = 13
    nq, basis, dbasis, g, u = random_case(bk, p, E)
    eng = bklib.ENGINE_DFMA if engine == "dfma" else bklib.ENGINE_FF
    out = gpu_apply(bklib, bk, p, E, basis, dbasis, g, u, bklib.PREC_FP64, engine=eng)
    ref = oracle_apply(bk, nq, E, basis, dbasis, g, u)
    assert np.all(np.isfinite(out))
    assert oracle.rel_maxdiff(out, ref) < TOL64


@pytest.mark.parametrize("bk", [1, 3, 5])
@pytest.mark.parametrize("p", P_ALL)
@pytest.mark.parametrize("prec", ["fp32", "mixed"])
def test_fp32_random(bklib, bk, p, prec):
    E = 13
    nq, basis, dbasis, g, u = random_case(bk, p, E)
    pr = bklib.PREC_FP32 if prec == "fp32" else bklib.PREC_MIXED
    out = gpu_apply(bklib, bk, p, E, basis, dbasis, g, u, pr)
    # the FP32 kernels read the inputs rounded to float
    ref = oracle_apply(bk, nq, E, basis, dbasis, g.astype(np.float32), u.astype(np.float32))
    assert np.all(np.isfinite(out))
    assert oracle.rel_maxdiff(out, ref) < TOL32


@pytest.mark.parametrize("bk", [1, 3, 5])
@pytest.mark.parametrize("p", P_ALL)
def test_golden_vectors(bklib, golden, bk, p):
    """Against the reference's own SumFactorization<double, nq> outputs."""
    arr, meta = golden
    E = meta["E_rand"]
    nq, basis, dbasis, g, u = random_case(bk, p, E, meta["seed"])
    out = gpu_apply(bklib, bk, p, E, basis, dbasis, g, u, bklib.PREC_FP64)
    assert oracle.rel_maxdiff(out, arr[f"bk{bk}_p{p}_rand_f64"]) < TOL64


@pytest.mark.parametrize("bk", [1, 3, 5])
@pytest.mark.parametrize("p", P_ALL)
@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_constant_data_norm(bklib, golden, bk, p, prec):
    """The drivers' known answer: "norm =" on constant data (in = 3, JxW = 1,
    G = 2, cos basis) as printed by the reference's BK1/BK3/BK5."""
    arr, meta = golden
    E = meta["E_const"]
    nq, nm, ngeo = sizes(bk, p)
    dt = np.float32 if prec == "f32" else np.float64
    u = np.full(E * nm ** 3, 3.0)
    g = np.full(E * ngeo, 1.0 if bk == 1 else 2.0)
    basis = oracle.test_basis(nm, nq, dt).astype(np.float64) if bk != 5 else None
    dbasis = oracle.test_basis(nq, nq, dt).astype(np.float64) if bk != 1 else None
    pr = bklib.PREC_FP32 if prec == "f32" else bklib.PREC_FP64
    out = gpu_apply(bklib, bk, p, E, basis, dbasis, g, u, pr)
    ref = meta["norms"][f"bk{bk}_p{p}_const_{prec}"]
    nrm = float(np.sqrt(np.sum(out * out)))
    assert abs(nrm - ref) <= (2e-5 if prec == "f32" else 1e-12) * abs(ref)
    e0 = arr[f"bk{bk}_p{p}_const_{prec}_e0"]
    assert oracle.rel_maxdiff(out[: e0.size], e0) < (TOL32 if prec == "f32" else TOL64)


@pytest.mark.parametrize("E", [1, 2, 3, 5, 16, 33, 100])
@pytest.mark.parametrize("bk,p", [(1, 3), (3, 6), (5, 7), (5, 8), (3, 8)])
def test_element_counts(bklib, bk, p, E):
    """Any element count: partial last batches, batches whose slices start off
    a 16-byte boundary (the TMA head/tail path)."""
    nq, basis, dbasis, g, u = random_case(bk, p, E, seed=E)
    for prec, tol in ((bklib.PREC_FP64, TOL64), (bklib.PREC_FP32, TOL32)):
        out = gpu_apply(bklib, bk, p, E, basis, dbasis, g, u, prec)
        if prec == bklib.PREC_FP32:
            ref = oracle_apply(bk, nq, E, basis, dbasis, g.astype(np.float32), u.astype(np.float32))
        else:
            ref = oracle_apply(bk, nq, E, basis, dbasis, g, u)
        assert oracle.rel_maxdiff(out, ref) < tol


@pytest.mark.parametrize("p", [1, 4, 7, 8])
@pytest.mark.parametrize("nfactors", [6, 9])
@pytest.mark.parametrize("layout", [0, 1, 2])
@pytest.mark.parametrize("engine", ["dfma", "ff", "fp32"])
@pytest.mark.parametrize("kernel", ["sweep", "column"])
def test_bk5_layouts(bklib, p, nfactors, layout, engine, kernel):
    """BK5 with G in every layout and factor count of make_bk5_G
    (include/bk_harness.h:217-244), with both kernel shapes."""
    E = 7
    nq, _, dbasis, g6i, u = random_case(5, p, E)
    G = oracle.make_bk5_G(g6i, E, nq, nfactors, layout)
    kern = bklib.KERNEL_SWEEP if kernel == "sweep" else bklib.KERNEL_COLUMN
    if engine == "fp32":
        dt, prec, eng, tol = "f32", bklib.PREC_FP32, 0, TOL32
        f = lambda a: a.astype(np.float32).astype(np.float64)
        ref = oracle.bk5(nq, E, dbasis, f(g6i), f(u))
    else:
        dt, prec, tol = "f64", bklib.PREC_FP64, TOL64
        eng = bklib.ENGINE_DFMA if engine == "dfma" else bklib.ENGINE_FF
        ref = oracle.bk5(nq, E, dbasis, g6i, u)
    gu, gg = dev(u, dt), dev(G, dt)
    out = torch.full_like(gu, float("nan"))
    bklib.bk5_apply(p, E, dbasis, gg, gu, out, prec=prec, engine=eng, layout=layout, nfactors=nfactors, kernel=kern)
    torch.cuda.synchronize()
    assert oracle.rel_maxdiff(host(out), ref) < tol


@pytest.mark.parametrize("p", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_bk5_kernel_shapes_agree(bklib, p, prec):
    """The sweep and column kernels give the same operator."""
    E = 37
    nq, _, dbasis, g, u = random_case(5, p, E, seed=99)
    pr = bklib.PREC_FP64 if prec == "fp64" else bklib.PREC_MIXED
    dt = "f64" if prec == "fp64" else "f32"
    gu, gg = dev(u, dt), dev(g, dt)
    outs = []
    for kern in (bklib.KERNEL_SWEEP, bklib.KERNEL_COLUMN):
        out = torch.full_like(gu, float("nan"))
        bklib.bk5_apply(p, E, dbasis, gg, gu, out, prec=pr, kernel=kern)
        outs.append(host(out))
    torch.cuda.synchronize()
    assert oracle.rel_maxdiff(outs[1], outs[0]) < (TOL64 if prec == "fp64" else TOL32)


@pytest.mark.parametrize("p", [2, 5, 8])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_bk5_helmholtz_mass(bklib, p, prec):
    E = 9
    nq, _, dbasis, g, u = random_case(5, p, E)
    mass = np.random.default_rng(p).uniform(0.5, 1.5, E * nq ** 3)
    pr = bklib.PREC_FP64 if prec == "fp64" else bklib.PREC_MIXED
    out = gpu_apply(bklib, 5, p, E, None, dbasis, g, u, pr, mass=mass, lam=1.0)
    if pr == bklib.PREC_FP64:
        ref = oracle.bk5(nq, E, dbasis, g, u, mass=mass, lam=1.0)
        tol = TOL64
    else:
        f = lambda a: a.astype(np.float32).astype(np.float64)
        ref = oracle.bk5(nq, E, dbasis, f(g), f(u), mass=f(mass), lam=1.0)
        tol = TOL32
    assert oracle.rel_maxdiff(out, ref) < tol


@pytest.mark.parametrize("p", [1, 4, 6, 8])
@pytest.mark.parametrize("engine", ["dfma", "ff"])
def test_bk3_coefficient(bklib, p, engine):
    E = 5
    nq, basis, dbasis, g, u = random_case(3, p, E)
    k = np.exp(np.random.default_rng(p).normal(0, 0.5, E * nq ** 3))
    eng = bklib.ENGINE_DFMA if engine == "dfma" else bklib.ENGINE_FF
    out = gpu_apply(bklib, 3, p, E, basis, dbasis, g, u, bklib.PREC_FP64, engine=eng, k=k)
    ref = oracle.bk3(nq, E, basis, dbasis, g, u, k=k)
    assert oracle.rel_maxdiff(out, ref) < TOL64


def test_offset_views(bklib):
    """Arrays that start inside an allocation (16-byte aligned views)."""
    p, E = 7, 6
    nq, _, dbasis, g, u = random_case(5, p, E)
    big_u = dev(np.concatenate([np.zeros(2), u]), "f64")[2:]
    big_g = dev(np.concatenate([np.zeros(2), g]), "f64")[2:]
    out = torch.full((E * nq ** 3 + 2,), float("nan"), dtype=torch.float64, device="cuda")[2:]
    bklib.bk5_apply(p, E, dbasis, big_g, big_u, out)
    torch.cuda.synchronize()
    assert oracle.rel_maxdiff(host(out), oracle.bk5(nq, E, dbasis, g, u)) < TOL64
    # a view one double in is not 16-byte aligned: rejected before any launch
    with pytest.raises(bklib.BKError, match="misaligned"):
        bklib.bk5_apply(p, E - 1, dbasis, big_g, big_u[1:], out)


def test_bounded_wait_timeout(bklib):
    """A device-side wait that nothing completes gives up within its limit,
    records BK_ERR_TIMEOUT, and the context stays usable."""
    L = bklib.lib()
    assert bklib.device_status(reset=True) == bklib.BK_OK
    assert L.bk_set_wait_limit(20000) == 0
    try:
        s = torch.cuda.current_stream().cuda_stream
        assert L.bk_test_wait_timeout(s) == 0
        torch.cuda.synchronize()
        assert bklib.device_status(reset=True) == bklib.BK_ERR_TIMEOUT
    finally:
        assert L.bk_set_wait_limit(0) == 0
    # the next apply runs normally
    p, E = 3, 4
    nq, _, dbasis, g, u = random_case(5, p, E)
    out = gpu_apply(bklib, 5, p, E, None, dbasis, g, u, bklib.PREC_FP64)
    assert oracle.rel_maxdiff(out, oracle.bk5(nq, E, dbasis, g, u)) < TOL64
    assert bklib.device_status(reset=True) == bklib.BK_OK


@pytest.mark.parametrize("p", P_ALL)
@pytest.mark.parametrize("engine", ["dfma", "ff", "fp32", "mixed"])
def test_bk5_gll_even_odd(bklib, p, engine):
    """With the GLL derivative matrix (centro-antisymmetric) BK5 takes the
    even-odd contractions; same operator as the oracle's plain sums."""
    E = 11
    nq = p + 1
    D, _, _ = bklib.bk5_matrices(p)
    rng = np.random.default_rng(100 + p)
    u = rng.uniform(-1, 1, E * nq ** 3)
    g = rng.uniform(0.5, 1.5, E * 6 * nq ** 3)
    if engine in ("dfma", "ff"):
        eng = bklib.ENGINE_DFMA if engine == "dfma" else bklib.ENGINE_FF
        out = gpu_apply(bklib, 5, p, E, None, D, g, u, bklib.PREC_FP64, engine=eng)
        ref = oracle.bk5(nq, E, D, g, u)
        tol = TOL64
    else:
        pr = bklib.PREC_FP32 if engine == "fp32" else bklib.PREC_MIXED
        out = gpu_apply(bklib, 5, p, E, None, D, g, u, pr)
        f = lambda a: a.astype(np.float32).astype(np.float64)
        ref = oracle.bk5(nq, E, D, f(g), f(u))
        tol = TOL32
    assert oracle.rel_maxdiff(out, ref) < tol


@pytest.mark.parametrize("p", P_ALL)
@pytest.mark.parametrize("engine", ["dfma", "ff", "fp32", "mixed"])
@pytest.mark.parametrize("coef", [False, True])
def test_bk3_gll_gauss_even_odd(bklib, p, engine, coef):
    """With GLL nodes and Gauss points (B centro-symmetric, D
    centro-antisymmetric) BK3 takes the even-odd contractions, rectangular
    for the interpolation; same operator as the oracle's plain sums."""
    E = 9
    B, D, _, _, _ = bklib.bk1_bk3_matrices(p)
    nq = p + 2
    rng = np.random.default_rng(200 + p)
    u = rng.uniform(-1, 1, E * (nq - 1) ** 3)
    g = rng.uniform(0.5, 1.5, E * 6 * nq ** 3)
    k = np.exp(rng.normal(0, 0.5, E * nq ** 3)) if coef else None
    if engine in ("dfma", "ff"):
        eng = bklib.ENGINE_DFMA if engine == "dfma" else bklib.ENGINE_FF
        out = gpu_apply(bklib, 3, p, E, B, D, g, u, bklib.PREC_FP64, engine=eng, k=k)
        ref = oracle.bk3(nq, E, B, D, g, u, k=k)
        tol = TOL64
    else:
        pr = bklib.PREC_FP32 if engine == "fp32" else bklib.PREC_MIXED
        out = gpu_apply(bklib, 3, p, E, B, D, g, u, pr, k=k)
        f = lambda a: None if a is None else a.astype(np.float32).astype(np.float64)
        ref = oracle.bk3(nq, E, B, D, f(g), f(u), k=f(k))
        tol = TOL32
    assert np.all(np.isfinite(out))
    assert oracle.rel_maxdiff(out, ref) < tol


@pytest.mark.parametrize("p", P_ALL)
@pytest.mark.parametrize("engine", ["dfma", "ff", "fp32", "mixed"])
def test_bk1_gll_gauss_even_odd(bklib, p, engine):
    """With GLL nodes and Gauss points (B centro-symmetric) BK1 takes the
    even-odd interpolation sweeps; same operator as the oracle's sums."""
    E = 10
    B, _, _, _, _ = bklib.bk1_bk3_matrices(p)
    nq = p + 2
    rng = np.random.default_rng(300 + p)
    u = rng.uniform(-1, 1, E * (nq - 1) ** 3)
    jxw = rng.uniform(0.5, 1.5, E * nq ** 3)
    if engine in ("dfma", "ff"):
        eng = bklib.ENGINE_DFMA if engine == "dfma" else bklib.ENGINE_FF
        out = gpu_apply(bklib, 1, p, E, B, None, jxw, u, bklib.PREC_FP64, engine=eng)
        ref = oracle.bk1(nq, E, B, jxw, u)
        tol = TOL64
    else:
        pr = bklib.PREC_FP32 if engine == "fp32" else bklib.PREC_MIXED
        out = gpu_apply(bklib, 1, p, E, B, None, jxw, u, pr)
        f = lambda a: a.astype(np.float32).astype(np.float64)
        ref = oracle.bk1(nq, E, B, f(jxw), f(u))
        tol = TOL32
    assert np.all(np.isfinite(out))
    assert oracle.rel_maxdiff(out, ref) < tol


@pytest.mark.parametrize("p", P_ALL)
@pytest.mark.parametrize("layout", [0, 1, 2])
@pytest.mark.parametrize("with_mass", [False, True])
def test_bk5_split_g_is_bitwise(bklib, p, layout, with_mass):
    """G split once into float-float pairs (bk_g_to_ff) gives bitwise the
    apply on the doubles: the pairs are the engine's own split of each value.
    The conversion also runs in place."""
    E = 13
    nq = p + 1
    D, _, _ = bklib.bk5_matrices(p)
    rng = np.random.default_rng(300 + p)
    u = dev(rng.uniform(-1, 1, E * nq ** 3), "f64")
    g = dev(rng.uniform(0.5, 1.5, E * 6 * nq ** 3) * (1 + 1e-9 * rng.standard_normal(E * 6 * nq ** 3)), "f64")
    mass = dev(rng.uniform(0.5, 1.5, E * nq ** 3), "f64") if with_mass else None
    v0 = torch.empty_like(u)
    v1 = torch.full_like(u, float("nan"))
    bklib.bk5_apply(p, E, D, g, u, v0, layout=layout, mass=mass, lam=0.7 if with_mass else 0.0)
    gff = bklib.g_to_ff(g)
    bklib.bk5_apply(p, E, D, gff, u, v1, layout=layout, mass=mass, lam=0.7 if with_mass else 0.0,
                    gform=bklib.G_FF)
    g_in_place = g.clone()
    bklib.g_to_ff(g_in_place, out=g_in_place)
    torch.cuda.synchronize()
    assert torch.equal(v0, v1)
    assert torch.equal(g_in_place, gff)
    # hi + lo is the double to 2^-48
    pairs = gff.view(torch.float32).view(-1, 2).double()
    assert torch.max(torch.abs(pairs[:, 0] + pairs[:, 1] - g) / torch.abs(g)).item() < 2.0 ** -47


def test_bk5_split_g_unsupported(bklib):
    """The split G form is for the float-float engine's even-odd sweep kernel
    only: every other combination is rejected, none computes."""
    p, E = 4, 3
    nq = p + 1
    D, _, _ = bklib.bk5_matrices(p)
    g = torch.ones(E * 6 * nq ** 3, dtype=torch.float64, device="cuda")
    u = torch.ones(E * nq ** 3, dtype=torch.float64, device="cuda")
    v = torch.empty_like(u)
    for kw in (dict(engine=bklib.ENGINE_DFMA), dict(prec=bklib.PREC_MIXED), dict(nfactors=9),
               dict(kernel=bklib.KERNEL_COLUMN)):
        with pytest.raises(bklib.BKError, match="precision"):
            bklib.bk5_apply(p, E, D, g, u, v, gform=bklib.G_FF, **kw)
    # a D that is not centro-antisymmetric has no even-odd form
    Dn = np.random.default_rng(1).uniform(-1, 1, (nq, nq))
    with pytest.raises(bklib.BKError, match="precision"):
        bklib.bk5_apply(p, E, Dn, g, u, v, gform=bklib.G_FF)


@pytest.mark.parametrize("p", P_ALL)
@pytest.mark.parametrize("coef", [False, True])
def test_bk3_split_g_is_bitwise(bklib, p, coef):
    """BK3 on G split once into float-float pairs gives bitwise the apply on
    the doubles (GLL nodes, Gauss points: the even-odd path)."""
    E = 7
    B, D, _, _, _ = bklib.bk1_bk3_matrices(p)
    nq = p + 2
    rng = np.random.default_rng(400 + p)
    u = dev(rng.uniform(-1, 1, E * (nq - 1) ** 3), "f64")
    g = dev(rng.uniform(0.5, 1.5, E * 6 * nq ** 3) * (1 + 1e-9 * rng.standard_normal(E * 6 * nq ** 3)), "f64")
    k = dev(np.exp(rng.normal(0, 0.5, E * nq ** 3)), "f64") if coef else None
    v0 = torch.empty_like(u)
    v1 = torch.full_like(u, float("nan"))
    bklib.bk3_apply(p, E, B, D, g, u, v0, k=k)
    bklib.bk3_apply(p, E, B, D, bklib.g_to_ff(g), u, v1, k=k, gform=bklib.G_FF)
    torch.cuda.synchronize()
    assert torch.equal(v0, v1)
    with pytest.raises(bklib.BKError, match="precision"):
        bklib.bk3_apply(p, E, B, D, g, u, v1, prec=bklib.PREC_MIXED, gform=bklib.G_FF)


@pytest.mark.parametrize("p", [1, 3, 6, 7, 8])
@pytest.mark.parametrize("nfactors", [6, 9])
@pytest.mark.parametrize("layout", [0, 1, 2])
@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_bk5_make_g_matches_oracle(bklib, p, nfactors, layout, prec):
    """The device make_bk5_G is a permutation (and, for 9 factors, a
    duplication) of G6i: bitwise the oracle's restatement of
    include/bk_harness.h:220-244."""
    E = 5
    q = p + 1
    g6i = np.random.default_rng(500 + p).uniform(-1, 1, E * 6 * q ** 3)
    ref = oracle.make_bk5_G(g6i, E, q, nfactors, layout)
    src = dev(g6i, prec)
    out = bklib.bk5_make_g(p, E, src, nfactors=nfactors, layout=layout)
    torch.cuda.synchronize()
    want = ref if prec == "f64" else ref.astype(np.float32).astype(np.float64)
    assert np.array_equal(host(out), want)


def test_bk5_make_g_feeds_the_apply(bklib):
    """G6i relaid on the device to each layout, 6 and 9 factors: the BK5
    apply agrees with the oracle on the interleaved G6."""
    p, E = 7, 6
    q = p + 1
    D, _, _ = bklib.bk5_matrices(p)
    rng = np.random.default_rng(9)
    u = rng.uniform(-1, 1, E * q ** 3)
    g6i = rng.uniform(0.5, 1.5, E * 6 * q ** 3)
    ref = oracle.bk5(q, E, D, g6i, u)
    for nf in (6, 9):
        for layout in (0, 1, 2):
            G = bklib.bk5_make_g(p, E, dev(g6i, "f64"), nfactors=nf, layout=layout)
            v = torch.empty(E * q ** 3, dtype=torch.float64, device="cuda")
            bklib.bk5_apply(p, E, D, G, dev(u, "f64"), v, layout=layout, nfactors=nf)
            torch.cuda.synchronize()
            assert oracle.rel_maxdiff(host(v), ref) < TOL64, (nf, layout)


@pytest.mark.parametrize("p", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_bk1_transpose_jxw_matches_oracle(bklib, p, prec):
    """The device transpose_jxw is bitwise the oracle's restatement of
    include/bk_harness.h:89-102 (JxW(e,p,q,r) -> JxW_t(e,r,q,p))."""
    E = 7
    q = p + 2
    jxw = np.random.default_rng(700 + p).uniform(0.5, 1.5, E * q ** 3)
    if prec == "f32":
        jxw = jxw.astype(np.float32).astype(np.float64)
    out = bklib.bk1_transpose_jxw(p, E, dev(jxw, prec))
    torch.cuda.synchronize()
    assert np.array_equal(host(out), oracle.transpose_jxw(jxw, E, q))


@pytest.mark.parametrize("p", [1, 3, 4, 6, 8])
@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("basis", ["gll", "test"])
def test_bk1_transposed_jxw_apply(bklib, p, prec, basis):
    """BK1 on JxW_t(e,r,q,p) (jxw_layout RQP, the layout of the SYCL BK1
    variants, sycl/bk1_sycl.cpp:74-98) gives bitwise the apply on JxW(e,p,q,r)
    for every engine, on the even-odd (GLL/Gauss) and the plain (test basis)
    paths, and agrees with the oracle."""
    E = 37
    q, P = p + 2, p + 1
    if basis == "gll":
        B = bklib.bk1_bk3_matrices(p)[0]
    else:
        B = oracle.test_basis(P, q)
    rng = np.random.default_rng(40 + p)
    u = rng.uniform(-1, 1, E * P ** 3)
    jxw = rng.uniform(0.5, 1.5, E * q ** 3)
    dt = "f64" if prec == bklib.PREC_FP64 else "f32"
    du, dj = dev(u, dt), dev(jxw, dt)
    djt = bklib.bk1_transpose_jxw(p, E, dj)
    v0 = torch.full_like(du, float("nan"))
    v1 = torch.full_like(du, float("nan"))
    bklib.bk1_apply(p, E, B, dj, du, v0, prec=prec)
    bklib.bk1_apply(p, E, B, djt, du, v1, prec=prec, jxw_layout=bklib.JXW_RQP)
    torch.cuda.synchronize()
    assert torch.equal(v0, v1)
    tol = TOL64 if prec == bklib.PREC_FP64 else 1e-5
    assert oracle.rel_maxdiff(host(v1), oracle.bk1(q, E, B, jxw, u)) < tol


@pytest.mark.parametrize("p", [4, 7])
@pytest.mark.parametrize("h", [1.0 / 64, 1.0 / 16])
def test_bk5_fp64_smooth_field(bklib, p, h):
    """The FP64 forms on a smooth field, u = sin(pi x) sin(pi y) sin(pi z)
    at the nodes of the jittered trilinear mesh: the operator's image
    cancels (v is a second difference, |v| ~ h^2 |u| ... h |u|), which
    amplifies the float-float engine's 2^-48 rounding of the terms; measured
    3e-13 to 4e-13 at p = 7 (DFMA 1e-14), still inside the 1e-12 bound."""
    import math
    Q, E, n = p + 1, 1024, 256
    D, x, w = bklib.bk5_matrices(p)
    G = torch.empty(E * 6 * Q ** 3, dtype=torch.float64, device="cuda")
    X = torch.empty(E * Q ** 3 * 3, dtype=torch.float64, device="cuda")
    bklib.geom_trilinear(Q, E, 16, 16, x, w, 2, h, 0.15, G=G, layout=bklib.LAYOUT_COLUMN, coords=X)
    xyz = X.view(-1, 3)
    u = (torch.sin(math.pi * xyz[:, 0]) * torch.sin(math.pi * xyz[:, 1]) * torch.sin(math.pi * xyz[:, 2])).contiguous()
    g = host(G[: n * 6 * Q ** 3]).reshape(n, 6, Q, Q, Q).transpose(0, 3, 4, 1, 2).copy().ravel()
    ref = oracle.bk5(Q, n, np.asarray(D), g, host(u[: n * Q ** 3]))
    for eng in (bklib.ENGINE_FF, bklib.ENGINE_DFMA):
        v = torch.full_like(u, float("nan"))
        bklib.bk5_apply(p, E, D, G, u, v, prec=bklib.PREC_FP64, engine=eng, layout=bklib.LAYOUT_COLUMN)
        torch.cuda.synchronize()
        assert oracle.rel_maxdiff(host(v[: n * Q ** 3]), ref) < TOL64, (eng, p, h)


@pytest.mark.parametrize("bk", [3, 5])
@pytest.mark.parametrize("p", P_ALL)
def test_fp64_factor_ranges(bklib, bk, p):
    """The float-float engine splits a point's six factors behind one range
    test: zeros of both signs and values below the fast range (2^-74) beside
    ordinary ones take the careful path for the point, at batch remainders of
    every order's elements per block.  The bound is the FP64 target (the
    small factors contribute nothing to it: they are below 1e-25)."""
    E = 29
    Q, P = (p + 1, p + 1) if bk == 5 else (p + 2, p + 1)
    rng = np.random.default_rng(100 * bk + p)
    u = rng.uniform(-1, 1, E * P ** 3)
    G = rng.uniform(0.1, 1, (E, 6, Q, Q, Q))
    kind = rng.integers(0, 6, G.shape)
    G = np.where(kind == 0, 0.0, np.where(kind == 1, -0.0, np.where(kind == 2, G * 1e-26, G)))
    if bk == 5:
        D = np.asarray(bklib.bk5_matrices(p)[0])
        ref = oracle.bk5(Q, E, D, G.transpose(0, 2, 3, 1, 4).copy().ravel(), u)
        gd, ud = dev(G.transpose(0, 1, 4, 2, 3).copy().ravel(), "f64"), dev(u, "f64")
        v = torch.full_like(ud, float("nan"))
        bklib.bk5_apply(p, E, D, gd, ud, v, layout=bklib.LAYOUT_COLUMN)
    else:
        B, D = (np.asarray(m) for m in bklib.bk1_bk3_matrices(p)[:2])
        ref = oracle.bk3(Q, E, B, D, G.ravel(), u)
        gd, ud = dev(G.ravel(), "f64"), dev(u, "f64")
        v = torch.full_like(ud, float("nan"))
        bklib.bk3_apply(p, E, B, D, gd, ud, v)
    torch.cuda.synchronize()
    assert oracle.rel_maxdiff(host(v), ref) < TOL64


def test_apply_runs_on_the_current_stream(bklib):
    """Without a stream argument an apply is ordered with torch's work on the
    current stream (here a side stream behind a long chain of fills)."""
    p, E = 3, 3000
    B, _, _, _, _ = bklib.bk1_bk3_matrices(p)
    rng = np.random.default_rng(3)
    u, q = rng.uniform(-1, 1, E * 64), rng.uniform(0.1, 1, E * 125)
    ref = oracle.bk1(p + 2, E, np.asarray(B), q, u)
    gq, src = dev(q, "f64"), dev(u, "f64")
    gu, v = torch.zeros_like(src), torch.zeros_like(src)
    big = torch.empty(1 << 27, device="cuda")
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        for k in range(8):
            big.fill_(k)
        gu.copy_(src)
        bklib.bk1_apply(p, E, B, gq, gu, v)
    s.synchronize()
    assert oracle.rel_maxdiff(host(v), ref) < TOL64


@pytest.mark.parametrize("bk", [1, 3, 5])
@pytest.mark.parametrize("p", P_ALL)
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_every_batch_is_taken_once(bklib, bk, p, prec):
    """The blocks of a launch take over the batches of blocks not launched yet:
    a launch of many waves equals the same elements in launches of one wave
    or less, to the bit (the last batch partial, the outputs poisoned)."""
    Q, P = (p + 1, p + 1) if bk == 5 else (p + 2, p + 1)
    E = 40000 * 8 // Q ** 3 * 5 + 11
    pr, dt = (bklib.PREC_FP64, torch.float64) if prec == "fp64" else (bklib.PREC_MIXED, torch.float32)
    gen = torch.Generator(device="cuda").manual_seed(10 * bk + p)
    u = torch.rand(E, P ** 3, generator=gen, device="cuda", dtype=torch.float64).sub_(0.5).to(dt)
    g = torch.rand(E, (1 if bk == 1 else 6) * Q ** 3, generator=gen, device="cuda", dtype=torch.float64).to(dt)
    D5 = bklib.bk5_matrices(p)[0]
    B, D = bklib.bk1_bk3_matrices(p)[:2]

    def apply(e0, e1):
        gg, uu = g[e0:e1].clone(), u[e0:e1].clone()   # (an allocation of its own is aligned)
        v = torch.full_like(uu, float("nan"))
        if bk == 1:
            bklib.bk1_apply(p, e1 - e0, B, gg, uu, v, prec=pr)
        elif bk == 3:
            bklib.bk3_apply(p, e1 - e0, B, D, gg, uu, v, prec=pr)
        else:
            bklib.bk5_apply(p, e1 - e0, D5, gg, uu, v, prec=pr)
        return v

    whole = apply(0, E)
    step = max(1, min(E, 600))
    for e0 in range(0, E, step * 7):   # a seventh of the pieces, and the last
        assert torch.equal(whole[e0:min(E, e0 + step)], apply(e0, min(E, e0 + step)))
    assert torch.equal(whole[max(0, E - step):], apply(max(0, E - step), E))
    assert not torch.isnan(whole).any()


@pytest.mark.parametrize("p", P_ALL)
@pytest.mark.parametrize("nfactors", [6, 9])
@pytest.mark.parametrize("many", [False, True])
def test_bk5_column_vectors(bklib, p, nfactors, many):
    """The column kernel with G in the column layout and FP32 storage, where
    whole columns of v and the mass move as vectors: one element, and several
    batches per block with the last one partial, against the oracle."""
    nq = p + 1
    E = 320000 // nq ** 2 + 3 if many else 1
    nq, _, dbasis, g6i, u = random_case(5, p, E)
    G = oracle.make_bk5_G(g6i, E, nq, nfactors, bklib.LAYOUT_COLUMN)
    mass = np.random.default_rng(p).uniform(0.5, 1.5, E * nq ** 3)
    f = lambda a: a.astype(np.float32).astype(np.float64)
    ref = oracle.bk5(nq, E, dbasis, f(g6i), f(u), mass=f(mass), lam=0.75)
    gu, gg, gm = dev(u, "f32"), dev(G, "f32"), dev(mass, "f32")
    out = torch.full_like(gu, float("nan"))
    bklib.bk5_apply(p, E, dbasis, gg, gu, out, prec=bklib.PREC_MIXED, layout=bklib.LAYOUT_COLUMN, nfactors=nfactors,
                    kernel=bklib.KERNEL_COLUMN, mass=gm, lam=0.75)
    torch.cuda.synchronize()
    assert oracle.rel_maxdiff(host(out), ref) < TOL32


def test_stalled_launch_ends_after_one_limit(bklib):
    """A launch with a block per batch whose copies never come ends after the
    waits of its first resident blocks: the others are cancelled.  The status
    that it leaves stops no later launch, nor a replay of a captured one, before
    the host clears it."""
    L = bklib.lib()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    nbatch = 64 * 4 * sms   # 64 rounds of the resident blocks, four to an SM
    few = 8 * sms           # those, and the ones launched while the first give up
    counts = torch.zeros(2, dtype=torch.int32, device="cuda")

    def walk(stall):
        counts.zero_()
        assert L.bk_test_walk(nbatch, stall, counts.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        return counts.tolist()

    assert bklib.device_status(reset=True) == bklib.BK_OK
    started, done = walk(0)
    assert done == nbatch and started < nbatch
    assert L.bk_set_wait_limit(200000) == 0
    try:
        started, done = walk(1)
        assert 1 <= started <= few and done == 0
        assert bklib.device_status(reset=False) == bklib.BK_ERR_TIMEOUT
        assert walk(0)[1] == nbatch
        assert bklib.device_status(reset=True) == bklib.BK_ERR_TIMEOUT   # the first error stays
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            assert L.bk_test_walk(nbatch, 1, counts.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        for _ in range(2):
            counts.zero_()
            g.replay()
            torch.cuda.synchronize()
            assert 1 <= counts[0].item() <= few and counts[1].item() == 0
    finally:
        assert L.bk_set_wait_limit(0) == 0
        bklib.device_status(reset=True)
    p, E = 3, 4
    nq, _, dbasis, g, u = random_case(5, p, E)
    out = gpu_apply(bklib, 5, p, E, None, dbasis, g, u, bklib.PREC_FP64)
    assert oracle.rel_maxdiff(out, oracle.bk5(nq, E, dbasis, g, u)) < TOL64


def test_joins_agree(bklib):
    """A float-float pair becomes the nearest double of hi + lo by both routes of
    the stores, whichever part is the larger: loose pairs after a cancellation,
    normalised ones, powers of two with a part below, zeros."""
    rng = np.random.default_rng(11)
    n = 1 << 20
    hi = (rng.uniform(1, 2, n) * 2.0 ** rng.integers(-30, 30, n) * rng.choice([-1, 1], n)).astype(np.float32)
    lo = (rng.uniform(1, 2, n) * np.abs(hi) * 2.0 ** rng.integers(-50, 30, n) * rng.choice([-1, 1], n)).astype(np.float32)
    hi[::7] = np.exp2(np.floor(np.log2(np.abs(hi[::7]))))
    hi[::1001], lo[::1003] = 0, 0
    hi[5], lo[5] = 2.0 ** -24, 1 + 2.0 ** -23
    pairs = torch.from_numpy(np.stack([hi, lo], axis=1)).cuda()
    out = torch.empty(2, n, dtype=torch.float64, device="cuda")
    assert bklib.lib().bk_test_join(n, pairs.data_ptr(), out.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    want = hi.astype(np.float64) + lo.astype(np.float64)
    got = out.cpu().numpy()
    assert np.array_equal(got[1], want) and np.array_equal(got[0], want)


@pytest.mark.parametrize("p", P_ALL)
@pytest.mark.parametrize("layout", [0, 1, 2])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_bk5_column_elements_per_block(bklib, prec, layout, p):
    """The column kernel's elems_per_block: 0, the documented default and about
    128 columns are taken and give the same result (elements are independent of
    the block they are in), every other number is refused."""
    nq, E = p + 1, 37
    _, _, dbasis, g6i, u = random_case(5, p, E)
    G = oracle.make_bk5_G(g6i, E, nq, 6, layout)
    t = "f64" if prec == "fp64" else "f32"
    gu, gg = dev(u, t), dev(G, t)
    pr = bklib.PREC_FP64 if prec == "fp64" else bklib.PREC_MIXED
    allowed = {0, (32, 15, 8, 6, 4, 3, 2, 2)[p - 1] if prec == "mixed" or p < 7 else 1}
    if prec == "mixed" and layout == bklib.LAYOUT_COLUMN:
        allowed.add((32, 7, 4, 5, 3, 1, 1, 1)[p - 1])
    ref = None
    for eb in range(65):
        out = torch.full_like(gu, float("nan"))

        def run():
            bklib.bk5_apply(p, E, dbasis, gg, gu, out, prec=pr, layout=layout, kernel=bklib.KERNEL_COLUMN,
                            elems_per_block=eb)

        if eb not in allowed:
            with pytest.raises(bklib.BKError, match="invalid argument"):
                run()
            continue
        run()
        torch.cuda.synchronize()
        ref = out if ref is None else ref
        assert torch.equal(out, ref)
    tol = TOL64 if prec == "fp64" else TOL32
    f = (lambda a: a) if prec == "fp64" else (lambda a: a.astype(np.float32).astype(np.float64))
    assert oracle.rel_maxdiff(host(ref), oracle.bk5(nq, E, dbasis, f(g6i), f(u))) < tol


WALKS = [("bk1", "fp64", "pqr"), ("bk1", "fp64", "rqp"), ("bk1", "mixed", "pqr"), ("bk1", "fp32", "rqp"),
         ("bk3", "fp64", ""), ("bk3", "fp64", "k"), ("bk3", "fp64", "split"), ("bk3", "fp64", "split k"),
         ("bk3", "mixed", "k"), ("bk3", "fp32", ""), ("bk5", "fp64", "column"), ("bk5", "fp64", "factor mass"),
         ("bk5", "fp64", "column mass"), ("bk5", "fp64", "column split mass"), ("bk5", "mixed", "column mass"),
         ("bk5", "mixed", "factor"), ("adjoint", "fp64", ""), ("adjoint", "fp64", "split"), ("adjoint", "mixed", "")]


@pytest.mark.parametrize("p", P_ALL)
@pytest.mark.parametrize("op,prec,form", WALKS)
def test_launch_sizes_agree(bklib, op, prec, form, p):
    """The same 840 elements over and over (840 is a multiple of every number of
    elements a block takes), in launches of all kinds: 840 elements, at most 840
    batches, fewer than eight per SM, are dealt to the blocks; a few thousand take
    the shapes for launches of a few waves and those of many; and with 40000
    batches and more (no SM holds more than 32 blocks) the blocks take over one
    another's.  Every repetition to the bit, the last one partial."""
    q = p + 1 if op == "bk5" else p + 2
    nb, nu, nq = 840, (p + 1) ** 3, q ** 3
    dt = torch.float64 if prec == "fp64" else torch.float32
    pr = {"fp64": bklib.PREC_FP64, "fp32": bklib.PREC_FP32, "mixed": bklib.PREC_MIXED}[prec]
    gen = torch.Generator(device="cuda").manual_seed(7 * p + WALKS.index((op, prec, form)))
    rnd = lambda n, lo: (torch.rand(nb, n, generator=gen, device="cuda", dtype=torch.float64) + lo).to(dt)
    u, res, w, G = rnd(nu, -0.5), rnd(nu, -0.5), rnd(nq, 0.5), rnd(6 * nq, 0.1)
    B, D = bklib.bk1_bk3_matrices(p)[:2]
    D5 = bklib.bk5_matrices(p)[0]
    split = bklib.G_FF if "split" in form else bklib.G_STORAGE
    lay = bklib.LAYOUT_FACTOR if "factor" in form else bklib.LAYOUT_COLUMN

    def run(E):
        many = lambda x: x.expand(-(-E // nb), *x.shape).reshape(-1, x.shape[1])[:E].contiguous()
        eu = many(u)
        v = torch.full_like(eu, float("nan"))
        if op == "bk1":
            bklib.bk1_apply(p, E, B, many(w), eu, v, prec=pr,
                            jxw_layout=bklib.JXW_RQP if form == "rqp" else bklib.JXW_PQR)
            return [v]
        g = many(G)
        if "split" in form:
            g = bklib.g_to_ff(g.reshape(-1))
        if op == "bk3":
            bklib.bk3_apply(p, E, B, D, g, eu, v, k=many(w) if "k" in form else None, prec=pr, gform=split)
            return [v]
        if op == "bk5":
            bklib.bk5_apply(p, E, D5, g, eu, v, prec=pr, layout=lay, kernel=bklib.KERNEL_SWEEP,
                            mass=many(w) if "mass" in form else None, lam=0.75, gform=split)
            return [v]
        dk, dG = (torch.full((E, n), float("nan"), dtype=dt, device="cuda") for n in (nq, 6 * nq))
        bklib.bk3_adjoint(p, E, B, D, g, many(w), eu, many(res), dk, dG, prec=pr, gform=split)
        return [dk, dG]

    base = run(nb)
    torch.cuda.synchronize()
    assert not any(torch.isnan(b).any() for b in base)
    eb = min(16, max(1, 256 // q ** 2))   # at least a block's elements
    for E in (nb + 1, 2 * nb + 17, 5 * nb + 3, 12 * nb + 1, 40000 * eb + 11):
        for out, b in zip(run(E), base):
            n = E // nb
            assert torch.equal(out[:n * nb].reshape(n, nb, -1), b.expand(n, *b.shape))
            assert torch.equal(out[n * nb:], b[:E - n * nb])
            del out
