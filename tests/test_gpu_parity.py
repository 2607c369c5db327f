"""Parity of the CUDA path (called through the C ABI) with the oracle and with the reference.

Bars (the reference's own): bit-exact CSR patterns, colourings and AMG hierarchies (aggregates,
P, R, Galerkin operators, omega, coarse inverse); assembled values within 1e-12 per row; ILU
factors within 1e-12; solutions to the solver tolerance (tol 1e-10: 1e-8 relative); mixed
precision solves reach the same 1e-10 residual and match the FP64 solution to 1e-7.
"""
import numpy as np
import pytest

import fixtures as F
from oracle import oracle as O
from tests.conftest import MeshFromGolden, golden
from tests.test_oracle import rows_rel_err

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

import cfa_b200 as cfa  # noqa: E402

MESHES = {}


def mesh(name):
    if name not in MESHES:
        if name == "113k":   # level 0 beyond the ring tiles (512 rows per SM)
            import batch as B
            MESHES[name] = B.batch_system(3, 77_001, 77_001).mesh
            assert MESHES[name].n > 512 * torch.cuda.get_device_properties(0).multi_processor_count
        else:
            MESHES[name] = F.make_mesh(name)
    return MESHES[name]


@pytest.fixture(scope="module")
def ctx():
    return cfa.default_context()


def dev(a, dtype=torch.float64):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda", dtype)


def host(t):
    torch.cuda.synchronize()
    return t.cpu().numpy()


def fields(m):
    return (F.fourier_field(m.x, m.y, 1), F.fourier_field(m.x, m.y, 2), 0.3 * F.fourier_field(m.x, m.y, 3))


# ------------------------------------------------------------------------------------------------
# a1: CSR pattern
# ------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("name", ["tiny", "small", "medium"])
def test_csr_build_bit_exact(ctx, name):
    m = mesh(name)
    rp, ci = cfa.csr_build(ctx, m.n, dev(m.elem_v, torch.int32))
    orp, oci = O.csr_build(m.n, m.elem_v)
    assert np.array_equal(host(rp), orp) and np.array_equal(host(ci), oci)


def test_csr_build_matches_reference_golden(ctx):
    g = golden("ref_host_small.npz")
    m = MeshFromGolden(g)
    rp, ci = cfa.csr_build(ctx, m.n, dev(m.elem_v, torch.int32))
    assert np.array_equal(host(rp), g["rp"]) and np.array_equal(host(ci), g["ci"])


# ------------------------------------------------------------------------------------------------
# a3-a9: assembly
# ------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("name", ["small", "medium"])
def test_assembly_matches_oracle(ctx, name):
    m = mesh(name)
    dm = cfa.DeviceMesh(ctx, m)
    rp, ci = dm.host_pattern()
    n, ne, nnz = m.n, m.ne, dm.nnz
    u, v, p = fields(m)
    prm_o, prm = O.bdf2_params(), cfa.bdf2_params()
    # momentum + BCs
    A, ru, rv, mass = O.assemble_momentum(m, rp, ci, u, v, u, v, p, prm_o)
    uu, vv = u.copy(), v.copy()
    O.apply_bc_momentum(m, rp, ci, A, ru, rv, uu, vv)
    dA, dru, drv, dmass = (torch.zeros(k, dtype=torch.float64, device="cuda") for k in (nnz, n, n, n))
    du, dv = dev(u), dev(v)
    du_old, dv_old, dp_old = dev(u), dev(v), dev(p)
    cfa.assemble_momentum(ctx, dm, du_old, dv_old, du_old, dv_old, dp_old, prm, dA, dru, drv, dmass, du, dv,
                          u_max=1.5, H=1.0)
    assert rows_rel_err(host(dA), A, rp) < 1e-12
    for got, want in ((dru, ru), (drv, rv), (dmass, mass), (du, uu), (dv, vv)):
        assert np.abs(host(got) - want).max() <= 1e-12 * max(np.abs(want).max(), 1e-300)
    # lumped mass kernel (|det|/6 form)
    dm2 = torch.zeros(n, dtype=torch.float64, device="cuda")
    cfa.lumped_mass(ctx, dm, dm2)
    assert np.abs(host(dm2) - O.lumped_mass(m)).max() <= 1e-12 * mass.max()
    # PPE + OSS with BCs, the driver's Step B
    dt_proj = 2e-3 / 3
    s = O.oss_weights(m, uu, vv, dt_proj, 1.0, 1e-3, 0.3)
    ds = torch.zeros(ne, dtype=torch.float64, device="cuda")
    cfa.oss_weights(ctx, dm, du, dv, dt_proj, 1.0, 1e-3, 0.3, ds)
    assert np.abs(host(ds) - s).max() <= 1e-12 * np.abs(s).max()
    gx, gy = O.scalar_gradient(m, p, s)
    dgx, dgy = torch.zeros(n, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda")
    cfa.scalar_gradient(ctx, dm, dp_old, ds, dgx, dgy)
    assert np.abs(host(dgx) - gx).max() <= 1e-12 * np.abs(gx).max()
    assert np.abs(host(dgy) - gy).max() <= 1e-12 * np.abs(gy).max()
    Kp, rhs, div = O.assemble_ppe(m, rp, ci, uu, vv, p, gx, gy, mass, s, dt_proj, 1.0, 0.3)
    dp0 = np.ones(n)
    O.apply_bc_pressure(m, rp, ci, Kp, rhs, dp0, mass)
    oss, inv_m = O.assemble_oss(m, rp, ci, s, mass)
    dKp, drhs, ddiv = torch.zeros(nnz, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda")
    ddp = torch.ones(n, dtype=torch.float64, device="cuda")
    doss, dinv = torch.zeros(4 * nnz, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda")
    cfa.assemble_pressure_system(ctx, dm, du, dv, dp_old, dgx, dgy, dmass, ds, dt_proj, 1.0, 0.3, dKp, drhs, ddiv, ddp,
                                 doss, dinv)
    assert rows_rel_err(host(dKp), Kp, rp) < 1e-12
    assert np.abs(host(drhs) - rhs).max() <= 1e-12 * np.abs(rhs).max()
    assert np.abs(host(ddiv) - div).max() <= 1e-12 * np.abs(div).max()
    assert np.array_equal(host(ddp), dp0)
    hoss = host(doss)
    for q in range(4):
        assert rows_rel_err(hoss[q * nnz:(q + 1) * nnz], oss[q * nnz:(q + 1) * nnz], rp) < 1e-11
    assert np.abs(host(dinv) - inv_m).max() <= 1e-12 * inv_m.max()
    # the separate drop-in entry points give the same pressure system
    dKp2, drhs2, ddiv2 = torch.zeros_like(dKp), torch.zeros_like(drhs), torch.zeros_like(ddiv)
    ddp2 = torch.ones(n, dtype=torch.float64, device="cuda")
    cfa.assemble_ppe(ctx, dm, du, dv, dp_old, dgx, dgy, dmass, ds, dt_proj, 1.0, 0.3, dKp2, drhs2, ddiv2, ddp2)
    doss2, dinv2 = torch.zeros_like(doss), torch.zeros_like(dinv)
    cfa.assemble_oss(ctx, dm, ds, dmass, doss2, dinv2)
    assert torch.equal(dKp2, dKp) and torch.equal(drhs2, drhs) and torch.equal(doss2, doss)
    # OSS apply (a8) against the oracle
    xin = np.random.default_rng(3).uniform(-0.5, 0.5, n)
    out = np.zeros(n)
    O.oss_apply(m, rp, ci, oss, inv_m, xin, out)
    dout = torch.zeros(n, dtype=torch.float64, device="cuda")
    cfa.oss_apply(ctx, dm, doss, dinv, dev(xin), dout)
    assert np.abs(host(dout) - out).max() <= 1e-12 * np.abs(out).max()


def test_assembly_deterministic(ctx):
    m = mesh("medium")
    dm = cfa.DeviceMesh(ctx, m)
    u, v, p = fields(m)
    outs = []
    for _ in range(2):
        dA = torch.zeros(dm.nnz, dtype=torch.float64, device="cuda")
        bufs = [torch.zeros(m.n, dtype=torch.float64, device="cuda") for _ in range(3)]
        cfa.assemble_momentum(ctx, dm, dev(u), dev(v), dev(u), dev(v), dev(p), cfa.bdf2_params(), dA, *bufs,
                              dev(u), dev(v), u_max=1.5)
        outs.append(host(dA))
    assert np.array_equal(outs[0], outs[1])


def test_assembly_matches_reference_golden(ctx):
    """The reference's GPU assembly of one step (FP64 atomics) against ours: 1e-12 per row."""
    g = golden("ref_gpu_small.npz")
    h = golden("ref_host_small.npz")
    m = MeshFromGolden(h)
    dm = cfa.DeviceMesh(ctx, m, dev(h["rp"], torch.int32), dev(h["ci"], torch.int32))
    rp = h["rp"]
    n, nnz = m.n, rp[-1]
    u, v, p = h["u"], h["v"], h["p"]
    dA, dru, drv, dmass = (torch.zeros(k, dtype=torch.float64, device="cuda") for k in (nnz, n, n, n))
    cfa.assemble_momentum(ctx, dm, dev(u), dev(v), dev(u), dev(v), dev(p), cfa.bdf2_params(), dA, dru, drv, dmass,
                          dev(u), dev(v), u_max=1.5)
    assert rows_rel_err(host(dA), g["step_A_val"], rp) < 1e-12
    assert np.abs(host(dru) - g["step_rhs_u"]).max() <= 1e-12 * np.abs(g["step_rhs_u"]).max()
    us, vs = dev(g["step_u"]), dev(g["step_v"])
    dt_proj = 2e-3 / 3
    ds = torch.zeros(m.ne, dtype=torch.float64, device="cuda")
    cfa.oss_weights(ctx, dm, us, vs, dt_proj, 1.0, 1e-3, 0.3, ds)
    dgx, dgy = torch.zeros(n, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda")
    cfa.scalar_gradient(ctx, dm, dev(p), ds, dgx, dgy)
    dKp, drhs, ddiv, ddp = (torch.zeros(k, dtype=torch.float64, device="cuda") for k in (nnz, n, n, n))
    doss, dinv = torch.zeros(4 * nnz, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda")
    cfa.assemble_pressure_system(ctx, dm, us, vs, dev(p), dgx, dgy, dmass, ds, dt_proj, 1.0, 0.3, dKp, drhs, ddiv, ddp,
                                 doss, dinv)
    assert rows_rel_err(host(dKp), g["step_Kp_val"], rp) < 1e-12
    assert np.abs(host(drhs) - g["step_rhs_p"]).max() <= 1e-12 * np.abs(g["step_rhs_p"]).max()
    hoss = host(doss)
    for q in range(4):
        assert rows_rel_err(hoss[q * nnz:(q + 1) * nnz], g["step_oss_val"][q * nnz:(q + 1) * nnz], rp) < 1e-11


# ------------------------------------------------------------------------------------------------
# a15-a17: multicolour ILU(0)
# ------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("precision", [cfa.FP64, cfa.MIXED])
def test_ilu_colouring_factor_apply(ctx, precision):
    from tests.golden.make_golden import momentum_ilu_matrix
    m = mesh("small")
    rp, ci = O.csr_build(m.n, m.elem_v)
    n = m.n
    a, b = momentum_ilu_matrix(rp, ci)
    oi = O.Ilu(rp, ci)
    lu, _, _, _ = oi.factor(a)
    drp, dci = dev(rp, torch.int32), dev(ci, torch.int32)
    ilu = cfa.MulticolourIlu0(ctx, precision)
    ilu.set_pattern(n, rp, ci, drp, dci)
    assert ilu.n_colours == oi.nc and np.array_equal(ilu.colour_start, oi.colour_start)
    ilu.factor(dev(a))
    col, rows, dlu = ilu.device_arrays(ci.size)
    assert np.array_equal(host(col), oi.colour) and np.array_equal(host(rows), oi.rows)
    assert rows_rel_err(host(dlu), lu, rp) < 1e-12
    z = torch.zeros(2 * n, dtype=torch.float64, device="cuda")
    ilu.apply(dev(b), z, nrhs=2)
    zo = oi.apply(b, nrhs=2)
    tol = 1e-12 if precision == cfa.FP64 else 1e-5
    assert np.abs(host(z) - zo).max() <= tol * np.abs(zo).max()
    # the momentum solve's sweeps: both right-hand sides interleaved per row (FP64: the same
    # operations as the stacked sweeps; mixed: FP32 arithmetic on an FP32 work vector)
    zi = torch.zeros(2 * n, dtype=torch.float64, device="cuda")
    ilu.apply_interleaved(dev(np.stack([b[:n], b[n:]], 1).ravel()), zi)
    got = host(zi).reshape(n, 2).T.ravel()
    if precision == cfa.FP64:
        assert np.array_equal(got, host(z))
    assert np.abs(got - zo).max() <= tol * np.abs(zo).max()


@pytest.mark.parametrize("precision", [cfa.FP64, cfa.MIXED])
def test_ilu_sweep_orders_agree(ctx, precision, monkeypatch):
    """The interleaved-pair ILU apply in its two sweep forms: rows in the reference's natural order
    (CFA_ILU_PERM=0) and the work vector in colour order between a first and a last pass over all
    rows (the default): the same terms per row, so the results agree to rounding."""
    from tests.golden.make_golden import momentum_ilu_matrix
    m = mesh("c0")
    rp, ci = O.csr_build(m.n, m.elem_v)
    n = m.n
    a, b = momentum_ilu_matrix(rp, ci)
    ilu = cfa.MulticolourIlu0(ctx, precision)
    ilu.set_pattern(n, rp, ci, dev(rp, torch.int32), dev(ci, torch.int32))
    assert ilu.n_colours >= 3
    ilu.factor(dev(a))
    r = dev(np.stack([b[:n], b[n:]], 1).ravel())
    out = {}
    for order in ("0", "1"):
        monkeypatch.setenv("CFA_ILU_PERM", order)
        z = torch.full((2 * n,), np.nan, dtype=torch.float64, device="cuda")
        ilu.apply_interleaved(r, z)
        out[order] = host(z)
    assert np.isfinite(out["1"]).all()
    tol = 1e-13 if precision == cfa.FP64 else 1e-6
    assert np.abs(out["0"] - out["1"]).max() <= tol * np.abs(out["0"]).max()


@pytest.mark.parametrize("precision", [cfa.FP64, cfa.MIXED])
def test_ilu_set_pattern_reuses_the_handle(ctx, precision):
    """set_pattern on a handle that held another (larger) pattern gives the same colouring, factor
    and sweeps as a fresh handle, and the transposed factor follows the new pattern."""
    from tests.golden.make_golden import momentum_ilu_matrix
    big, m = mesh("medium"), mesh("small")
    rpb, cib = O.csr_build(big.n, big.elem_v)
    rp, ci = O.csr_build(m.n, m.elem_v)
    a, b = momentum_ilu_matrix(rp, ci)
    drp, dci = dev(rp, torch.int32), dev(ci, torch.int32)
    drpb, dcib = dev(rpb, torch.int32), dev(cib, torch.int32)   # device patterns outlive their use
    reused = cfa.MulticolourIlu0(ctx, precision)
    reused.set_pattern(big.n, rpb, cib, drpb, dcib)
    ab, _ = momentum_ilu_matrix(rpb, cib)
    reused.factor_transposed(dev(ab))
    reused.set_pattern(m.n, rp, ci, drp, dci)
    fresh = cfa.MulticolourIlu0(ctx, precision)
    fresh.set_pattern(m.n, rp, ci, drp, dci)
    assert reused.n_colours == fresh.n_colours and np.array_equal(reused.colour_start, fresh.colour_start)
    out = []
    for ilu in (reused, fresh):
        ilu.factor(dev(a))
        z = torch.zeros(2 * m.n, dtype=torch.float64, device="cuda")
        ilu.apply(dev(b), z, nrhs=2)
        ilu.factor_transposed(dev(a))
        zt = torch.zeros(2 * m.n, dtype=torch.float64, device="cuda")
        ilu.apply(dev(b), zt, nrhs=2)
        out.append((host(z), host(zt)))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


def test_ilu_row_too_long_is_an_error(ctx):
    n = 40
    rp = np.array([0, n] + list(range(n + 1, 2 * n)), np.int32)   # row 0 full, others diagonal
    ci = np.array(list(range(n)) + list(range(1, n)), np.int32)
    ilu = cfa.MulticolourIlu0(ctx)
    with pytest.raises(cfa.CfaError) as e:
        ilu.set_pattern(n, rp, ci, dev(rp, torch.int32), dev(ci, torch.int32))
    assert e.value.status == cfa.CFA_ROW_TOO_LONG


# ------------------------------------------------------------------------------------------------
# a18-a21: two-component BiCGSTAB
# ------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("precision", [cfa.FP64, cfa.MIXED])
def test_bicgstab2_matches_oracle(ctx, precision):
    from tests.golden.make_golden import momentum_ilu_matrix
    m = mesh("small")
    rp, ci = O.csr_build(m.n, m.elem_v)
    n = m.n
    a, b = momentum_ilu_matrix(rp, ci)
    oi = O.Ilu(rp, ci)
    oi.factor(a)
    xu, xv, reps = O.bicgstab2(rp, ci, a, b[:n], b[n:], np.zeros(n), np.zeros(n), oi, 200, 1e-10)
    drp, dci = dev(rp, torch.int32), dev(ci, torch.int32)
    ilu = cfa.MulticolourIlu0(ctx, precision)
    ilu.set_pattern(n, rp, ci, drp, dci)
    da = dev(a)
    ilu.factor(da)
    s = cfa.GpuBicgstab2(ctx)
    du, dv = torch.zeros(n, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda")
    db = dev(b)
    s.solve(n, drp, dci, da, db[:n], db[n:], du, dv, 200, 1e-10, ilu)
    assert s.converged == [True, True]
    x = np.concatenate([host(du), host(dv)])
    xo = np.concatenate([xu, xv])
    assert np.abs(x - xo).max() < 1e-8 * np.abs(xo).max()
    if precision == cfa.FP64:
        assert abs(s.iters[0] - reps[0].iterations) <= 1 and abs(s.iters[1] - reps[1].iterations) <= 1
    # true residual of each component
    for comp, xx, bb in ((0, host(du), b[:n]), (1, host(dv), b[n:])):
        r = bb - O.spmv(rp, ci, a, xx)
        assert np.linalg.norm(r) <= 1.5e-10 * np.linalg.norm(bb) or np.linalg.norm(r) < 1e-11


@pytest.mark.parametrize("precision", [cfa.FP64, cfa.MIXED])
def test_bicgstab2_staged_ilu_input_gives_the_same_bits(ctx, precision, monkeypatch):
    """BiCGSTAB2 with its p and s updates writing the ILU apply's colour-order work vector as they
    form p and s (the default) against the apply's own first pass (CFA_ILU_STAGED=0): the same
    values reach the sweeps, so iterations and solutions are bit for bit the same."""
    from tests.golden.make_golden import momentum_ilu_matrix
    m = mesh("c0")
    rp, ci = O.csr_build(m.n, m.elem_v)
    n = m.n
    a, b = momentum_ilu_matrix(rp, ci)
    drp, dci = dev(rp, torch.int32), dev(ci, torch.int32)
    ilu = cfa.MulticolourIlu0(ctx, precision)
    ilu.set_pattern(n, rp, ci, drp, dci)
    da, db = dev(a), dev(b)
    ilu.factor(da)
    out = {}
    for staged in ("1", "0"):
        monkeypatch.setenv("CFA_ILU_STAGED", staged)
        s = cfa.GpuBicgstab2(ctx)
        du, dv = torch.zeros(n, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda")
        s.solve(n, drp, dci, da, db[:n], db[n:], du, dv, 200, 1e-10, ilu)
        assert s.converged == [True, True]
        out[staged] = (list(s.iters), np.concatenate([host(du), host(dv)]))
    assert out["1"][0] == out["0"][0]
    assert np.array_equal(out["1"][1], out["0"][1])


def test_bicgstab2_not_converged_status(ctx):
    from tests.golden.make_golden import momentum_ilu_matrix
    m = mesh("small")
    rp, ci = O.csr_build(m.n, m.elem_v)
    n = m.n
    a, b = momentum_ilu_matrix(rp, ci)
    drp, dci, da, db = dev(rp, torch.int32), dev(ci, torch.int32), dev(a), dev(b)
    ilu = cfa.MulticolourIlu0(ctx)
    ilu.set_pattern(n, rp, ci, drp, dci)
    ilu.factor(da)
    s = cfa.GpuBicgstab2(ctx)
    du, dv = torch.zeros(n, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda")
    s.solve(n, drp, dci, da, db[:n], db[n:], du, dv, 2, 1e-14, ilu)
    assert s.converged == [False, False] and s.iters == [2, 2]


def test_bicgstab_jacobi_matches_oracle(ctx):
    from tests.golden.make_golden import momentum_ilu_matrix
    m = mesh("small")
    rp, ci = O.csr_build(m.n, m.elem_v)
    n = m.n
    a, b = momentum_ilu_matrix(rp, ci)
    xo, rep = O.bicgstab(rp, ci, a, b[:n], np.zeros(n), 400, 1e-10)
    s = cfa.GpuLinearSolver(ctx)
    dx = torch.zeros(n, dtype=torch.float64, device="cuda")
    it = s.solve_bicgstab(n, dev(rp, torch.int32), dev(ci, torch.int32), dev(a), dev(b[:n]), dx, 400, 1e-10)
    assert s.converged and abs(it - rep.iterations) <= 1
    assert np.abs(host(dx) - xo).max() < 1e-8 * np.abs(xo).max()


# ------------------------------------------------------------------------------------------------
# a22-a25: SA-AMG
# ------------------------------------------------------------------------------------------------
def laplacian(rp, ci):
    from tests.golden.make_golden import shifted_laplacian
    return shifted_laplacian(rp, ci)


def check_hierarchy(amg, oa):
    assert amg.num_levels() == oa.nlev + 1
    assert amg.coarse_n == oa.coarse_n
    for l in range(oa.nlev):
        L, OL = amg.level(l), oa.level(l)
        assert L["omega"] == OL["omega"]
        assert np.array_equal(host(L["agg"]), OL["agg"])
        for name in ("A", "P", "R"):
            rp_, ci_, v_ = (host(t) for t in L[name])
            _, _, orp, oci, ov = OL[name]
            assert np.array_equal(rp_, orp), (l, name)
            assert np.array_equal(ci_, oci), (l, name)
            assert np.array_equal(v_, ov), (l, name)
    _, inv = oa.coarse()
    assert np.array_equal(host(amg.coarse_inverse()), inv)


@pytest.mark.parametrize("agg", ["device", "host"])
@pytest.mark.parametrize("name,which", [("small", "lap"), ("medium", "lap"), ("medium", "ppe"), ("c0", "ppe"),
                                        ("c1", "ppe")])
def test_amg_setup_bit_exact(ctx, name, which, agg, monkeypatch):
    """The device setup (strength, the aggregation -- the dataflow kernels on the device, or the
    sequential host loop --, smoothing, transpose, Galerkin SpGEMM, coarse inverse) against the
    oracle's sequential host setup, bit for bit, up to the ~400k-node adaptive mesh."""
    monkeypatch.setenv("CFA_AGG_HOST", "0" if agg == "device" else "1")
    m = mesh(name)
    rp, ci = O.csr_build(m.n, m.elem_v)
    if which == "lap":
        a = laplacian(rp, ci)
    else:
        from tests.golden.make_golden import oracle_pressure_matrix
        u, v, p = fields(m)
        a = oracle_pressure_matrix(m, rp, ci, u, v, p)
    oa = O.Amg(rp, ci, a)
    amg = cfa.AmgPreconditioner(ctx)
    amg.setup(m.n, ci.size, dev(rp, torch.int32), dev(ci, torch.int32), dev(a))
    check_hierarchy(amg, oa)
    # V-cycle against the oracle's
    r = np.sin(0.37 * np.arange(m.n)) + 0.2
    z = torch.zeros(m.n, dtype=torch.float64, device="cuda")
    amg.apply(dev(r), z)
    zo = oa.apply(r)
    assert np.abs(host(z) - zo).max() <= 1e-12 * np.abs(zo).max()
    # mixed precision V-cycle: same hierarchy in FP32
    amg32 = cfa.AmgPreconditioner(ctx, cfa.MIXED)
    amg32.setup(m.n, ci.size, dev(rp, torch.int32), dev(ci, torch.int32), dev(a))
    z32 = torch.zeros(m.n, dtype=torch.float64, device="cuda")
    amg32.apply(dev(r), z32)
    assert np.abs(host(z32) - zo).max() <= 1e-4 * np.abs(zo).max()


@pytest.mark.parametrize("name", ["medium", "c1"])
def test_vcycle_composite_and_fused_transfers_match_level_chain(ctx, name, monkeypatch):
    """The V-cycle's two reformulations against the plain chain of level kernels: the composite
    coarse operator (the V-cycle below the first level of at most 2048 rows formed once as a dense
    matrix) and the fused transfers (the restricted residual R b - (R A) x in one pass, the
    prolongation folded into the first post-smoothing sweep through [A | A P] and [I | P]): the
    default (restriction fused on the levels >= 1, prolongation on those of at most 16384 rows)
    and both fused on every level. Each sums the same terms in another order: the
    V-cycles agree to 1e-13 relative in FP64 and 1e-5 in mixed precision, and PCG to 1e-10 takes
    the same number of iterations within 1."""
    from tests.golden.make_golden import oracle_pressure_matrix
    m = mesh(name)
    rp, ci = O.csr_build(m.n, m.elem_v)
    a = dev(oracle_pressure_matrix(m, rp, ci, *fields(m)))
    drp, dci = dev(rp, torch.int32), dev(ci, torch.int32)
    r = dev(np.sin(0.37 * np.arange(m.n)) + 0.2)
    out = {}
    # (composite rows, fused levels, largest level with the prolongation folded)
    configs = {"chain": ("0", "0", "0"), "default": ("2048", "1", "16384"), "fused_all": ("0", "2", "1000000000")}
    for cfg, (comp, fuse, addjac) in configs.items():
        monkeypatch.setenv("CFA_COMPOSITE_ROWS", comp)
        monkeypatch.setenv("CFA_VC_FUSE", fuse)
        monkeypatch.setenv("CFA_VC_ADDJAC_ROWS", addjac)
        for prec in (cfa.FP64, cfa.MIXED):
            amg = cfa.AmgPreconditioner(ctx, prec)
            amg.setup(m.n, ci.size, drp, dci, a)
            lv, rows = amg.composite()
            if comp == "0":
                assert lv == -1
            else:
                assert lv >= 1 and 0 < rows <= 2048
                assert amg.level(lv)["rows"] == rows
            z = torch.zeros(m.n, dtype=torch.float64, device="cuda")
            amg.apply(r, z)
            s = cfa.GpuLinearSolver(ctx)
            x = torch.zeros(m.n, dtype=torch.float64, device="cuda")
            it = s.solve_pcg(m.n, drp, dci, a, r, x, 4000, 1e-10, None, amg)
            assert s.converged
            out[cfg, prec] = (host(z), it, host(x))
    # the per-handle setter (0, 0, 0) gives the chain bit for bit, whatever the environment says
    for prec in (cfa.FP64, cfa.MIXED):
        amg = cfa.AmgPreconditioner(ctx, prec)
        amg.set_vcycle(0, 0, 0)
        amg.setup(m.n, ci.size, drp, dci, a)
        assert amg.composite()[0] == -1
        z = torch.zeros(m.n, dtype=torch.float64, device="cuda")
        amg.apply(r, z)
        assert np.array_equal(host(z), out["chain", prec][0])
    for cfg in ("default", "fused_all"):
        for prec, tol in ((cfa.FP64, 1e-13), (cfa.MIXED, 1e-5)):
            (z1, it1, x1), (z0, it0, x0) = out[cfg, prec], out["chain", prec]
            assert np.abs(z1 - z0).max() <= tol * np.abs(z0).max(), (cfg, prec)
            assert abs(it1 - it0) <= 1, (cfg, prec, it1, it0)
            assert np.abs(x1 - x0).max() <= 1e-8 * np.abs(x0).max(), (cfg, prec)


@pytest.mark.parametrize("prec", [cfa.FP64, cfa.MIXED])
def test_autotuned_tiles_give_the_same_vcycle_bits(ctx, prec):
    """The tile-height autotuner changes which CTA streams which rows, never a row's own sum: the
    V-cycle through a tuned hierarchy equals the default one bit for bit. Its choices are logged
    per pattern class, and a second setup of the same matrix takes them from the cache."""
    from tests.golden.make_golden import oracle_pressure_matrix
    m = mesh("c0")
    rp, ci = O.csr_build(m.n, m.elem_v)
    a = dev(oracle_pressure_matrix(m, rp, ci, *fields(m)))
    drp, dci = dev(rp, torch.int32), dev(ci, torch.int32)
    r = dev(np.sin(0.37 * np.arange(m.n)) + 0.2)
    zs = []
    try:
        for tune in (False, True, True):
            cfa.autotune(tune)
            n_log = len(cfa.autotune_log())
            amg = cfa.AmgPreconditioner(ctx, prec)
            amg.setup(m.n, ci.size, drp, dci, a)
            z = torch.zeros(m.n, dtype=torch.float64, device="cuda")
            amg.apply(r, z)
            zs.append(host(z))
            if tune:
                log = cfa.autotune_log()
                if len(zs) == 2:
                    assert len(log) > n_log
                    for rec in log[n_log:]:
                        assert rec["row_shift"] in (-2, -1, 0, 1) and str(rec["row_shift"]) in rec["us"]
                else:
                    assert len(log) == n_log   # every class cached
    finally:
        cfa.autotune(False)
    assert np.array_equal(zs[0], zs[1]) and np.array_equal(zs[0], zs[2])


def test_amg_matches_reference_golden(ctx):
    for name in ("tiny", "small"):
        g = golden(f"ref_host_{name}.npz")
        rp, ci = g["rp"], g["ci"]
        for which in ("ppe", "lap"):
            amg = cfa.AmgPreconditioner(ctx)
            amg.setup(rp.size - 1, ci.size, dev(rp, torch.int32), dev(ci, torch.int32), dev(g[f"{which}_val"]))
            assert amg.num_levels() == int(g[f"{which}_levels"][0]) + 1
            for l in range(int(g[f"{which}_levels"][0])):
                L = amg.level(l)
                assert L["omega"] == g[f"{which}_L{l}_omega"][0]
                for nm in ("A", "P", "R"):
                    for part, t in zip(("rp", "ci", "v"), L[nm]):
                        assert np.array_equal(host(t), g[f"{which}_L{l}_{nm}_{part}"]), (name, which, l, nm, part)
            assert np.array_equal(host(amg.coarse_inverse()).ravel(), g[f"{which}_coarse_inv"])


def test_amg_vcycle_matches_reference_gpu_golden(ctx):
    g = golden("ref_gpu_small.npz")
    h = golden("ref_host_small.npz")
    rp, ci = h["rp"], h["ci"]
    n = rp.size - 1
    amg = cfa.AmgPreconditioner(ctx)
    amg.setup(n, ci.size, dev(rp, torch.int32), dev(ci, torch.int32), dev(h["lap_val"]))
    z = torch.zeros(n, dtype=torch.float64, device="cuda")
    amg.apply(dev(np.sin(0.37 * np.arange(n)) + 0.2), z)
    # bit-identical hierarchy; the V-cycle's row sums are ordered differently (tile kernels)
    assert np.abs(host(z) - g["lap_vcycle_z"]).max() <= 1e-12 * np.abs(g["lap_vcycle_z"]).max()


@pytest.mark.parametrize("precision", [cfa.FP64, cfa.MIXED])
def test_amg_cluster_tail_matches_level_kernels(ctx, precision, monkeypatch):
    """The opt-in coarse tail (one thread-block cluster for the levels below CFA_TAIL_ROWS rows)
    gives the V-cycle of the per-level kernels."""
    m = mesh("medium")
    rp, ci = O.csr_build(m.n, m.elem_v)
    val = laplacian(rp, ci)
    r = dev(np.cos(0.11 * np.arange(m.n)))
    out = []
    for tail in (None, "7000"):   # tail from level 1 (6.4k rows) down
        if tail is None:
            monkeypatch.delenv("CFA_TAIL_ROWS", raising=False)
        else:
            monkeypatch.setenv("CFA_TAIL_ROWS", tail)
        amg = cfa.AmgPreconditioner(ctx, precision=precision)
        amg.setup(m.n, ci.size, dev(rp, torch.int32), dev(ci, torch.int32), dev(val))
        assert amg.num_levels() >= 3
        z = torch.zeros(m.n, dtype=torch.float64, device="cuda")
        amg.apply(r, z)
        out.append(host(z))
    assert np.abs(out[1] - out[0]).max() <= 1e-12 * np.abs(out[0]).max()


@pytest.mark.parametrize("precision", [cfa.FP64, cfa.MIXED])
def test_amg_remap_matches_oracle(ctx, precision):
    """remap (a24) against the oracle's restatement: the level-0 prolongator and restriction
    bit-exact, the V-cycle within 1e-12 (FP64) / 1e-6 (FP32 hierarchy); an unchanged mesh gives the
    setup's V-cycle; the remapped hierarchy after a local refinement solves to 1e-10 within the
    reference's iteration bound."""
    from tests.golden.make_golden import shifted_laplacian
    m = mesh("medium")
    rp, ci = O.csr_build(m.n, m.elem_v)
    a = shifted_laplacian(rp, ci)
    drp, dci, da = dev(rp, torch.int32), dev(ci, torch.int32), dev(a)
    amg = cfa.AmgPreconditioner(ctx, precision=precision)
    amg.setup(m.n, ci.size, drp, dci, da)
    r = dev(np.sin(0.37 * np.arange(m.n)) + 0.2)
    z0 = torch.zeros(m.n, dtype=torch.float64, device="cuda")
    amg.apply(r, z0)
    amg.remap(m.n, ci.size, drp, dci, da, rp, ci, np.arange(m.n))
    assert amg.remaps == 1
    z1 = torch.zeros_like(z0)
    amg.apply(r, z1)
    assert torch.equal(z0, z1)
    m2, n2o = F.refine_blob(m, radius=0.08, rounds=3)
    rp2, ci2 = O.csr_build(m2.n, m2.elem_v)
    a2 = shifted_laplacian(rp2, ci2)
    drp2, dci2, da2 = dev(rp2, torch.int32), dev(ci2, torch.int32), dev(a2)
    amg.remap(m2.n, ci2.size, drp2, dci2, da2, rp2, ci2, n2o)
    assert amg.remaps == 2
    oa = O.Amg(rp, ci, a)
    assert oa.remap(rp2, ci2, a2, n2o)
    want, got = oa.level(0), amg.level(0)
    for name in ("P", "R"):
        wr, wc, (wrp, wci, wv) = want[name][0], want[name][1], want[name][2:]
        grp, gci, gv = (host(t) for t in got[name])
        assert np.array_equal(grp, wrp) and np.array_equal(gci, wci) and np.array_equal(gv, wv)
    r2 = np.sin(0.29 * np.arange(m2.n)) + 0.1
    z = torch.zeros(m2.n, dtype=torch.float64, device="cuda")
    amg.apply(dev(r2), z)
    zo = oa.apply(r2)
    tol = 1e-12 if precision == cfa.FP64 else 1e-6
    assert np.abs(host(z) - zo).max() <= tol * np.abs(zo).max()
    s = cfa.GpuLinearSolver(ctx)
    b = dev(np.cos(0.11 * np.arange(m2.n)))
    x = torch.zeros(m2.n, dtype=torch.float64, device="cuda")
    it_remap = s.solve_pcg(m2.n, drp2, dci2, da2, b, x, 400, 1e-10, None, amg)
    assert s.converged
    fresh = cfa.AmgPreconditioner(ctx, precision=precision)
    fresh.setup(m2.n, ci2.size, drp2, dci2, da2)
    x.zero_()
    it_setup = s.solve_pcg(m2.n, drp2, dci2, da2, b, x, 400, 1e-10, None, fresh)
    assert s.converged and it_remap <= 3 * it_setup + 5


def test_amg_coarse_not_spd_is_an_error(ctx):
    m = mesh("tiny")
    rp, ci = O.csr_build(m.n, m.elem_v)
    a = -laplacian(rp, ci)            # negative definite: the coarse Cholesky must fail
    amg = cfa.AmgPreconditioner(ctx)
    with pytest.raises(cfa.CfaError) as e:
        amg.setup(m.n, ci.size, dev(rp, torch.int32), dev(ci, torch.int32), dev(a))
    assert e.value.status == cfa.CFA_COARSE_NOT_SPD


# ------------------------------------------------------------------------------------------------
# a10-a13: PCG (+ OSS + AMG)
# ------------------------------------------------------------------------------------------------
def pressure_system(m, rp, ci):
    u, v, p = fields(m)
    A, ru, rv, mass = O.assemble_momentum(m, rp, ci, u, v, u, v, p, O.bdf2_params())
    dt_proj = 2e-3 / 3
    s = O.oss_weights(m, u, v, dt_proj, 1.0, 1e-3, 0.3)
    gx, gy = O.scalar_gradient(m, p, s)
    Kp, rhs, div = O.assemble_ppe(m, rp, ci, u, v, p, gx, gy, mass, s, dt_proj, 1.0, 0.3)
    dp = np.zeros(m.n)
    O.apply_bc_pressure(m, rp, ci, Kp, rhs, dp, mass)
    oss, inv_m = O.assemble_oss(m, rp, ci, s, mass)
    return Kp, rhs, oss, inv_m


@pytest.mark.parametrize("use_oss,use_amg", [(True, True), (False, True), (True, False), (False, False)])
def test_pcg_matches_oracle(ctx, use_oss, use_amg):
    m = mesh("small")
    dm = cfa.DeviceMesh(ctx, m)
    rp, ci = dm.host_pattern()
    Kp, rhs, oss, inv_m = pressure_system(m, rp, ci)
    oa = O.Amg(rp, ci, Kp) if use_amg else None
    xo, rep = O.pcg(rp, ci, Kp, rhs, np.zeros(m.n), 4000, 1e-10, oss if use_oss else None,
                    inv_m if use_oss else None, m.tag, oa)
    dK, db, doss, dinv = dev(Kp), dev(rhs), dev(oss), dev(inv_m)
    amg = None
    if use_amg:
        amg = cfa.AmgPreconditioner(ctx)
        amg.setup(m.n, ci.size, dm.rp, dm.ci, dK)
    s = cfa.GpuLinearSolver(ctx)
    dx = torch.zeros(m.n, dtype=torch.float64, device="cuda")
    it = s.solve_pcg(m.n, dm.rp, dm.ci, dK, db, dx, 4000, 1e-10, cfa.oss_operator(dm, doss, dinv) if use_oss else None,
                     amg)
    assert s.converged and rep.converged
    assert abs(it - rep.iterations) <= max(2, rep.iterations // 50)
    assert np.abs(host(dx) - xo).max() < 1e-8 * np.abs(xo).max()
    # true residual with the oracle operator
    x = host(dx)
    Ax = O.spmv(rp, ci, Kp, x)
    if use_oss:
        O.oss_apply(m, rp, ci, oss, inv_m, x, Ax)
    assert np.linalg.norm(rhs - Ax) <= 1.5e-10 * np.linalg.norm(rhs)


@pytest.mark.parametrize("name", ["c0", "113k"])
@pytest.mark.parametrize("prec", [cfa.FP64, cfa.MIXED])
def test_pcg_update_folded_into_vcycle_matches_update_kernel(ctx, name, prec, monkeypatch):
    """The CG's update (x += alpha pn, r -= alpha q, p = pn, |r| and the stopping test) folded into
    the V-cycle's level-0 pre-smoothing and residual passes, against the separate update kernel:
    the same arithmetic per row (up to where the compiler contracts the update into a fused
    multiply-add), so iteration counts within 1, solutions within 1e-8, and the true residual of
    the folded solve below 1.5e-10. (By default c0 folds it into the ring tiles' kernel, the larger
    mesh runs the update kernel.)"""
    m = mesh(name)
    dm = cfa.DeviceMesh(ctx, m)
    rp, ci = dm.host_pattern()
    Kp, rhs, oss, inv_m = pressure_system(m, rp, ci)
    dK, db, doss, dinv = dev(Kp), dev(rhs), dev(oss), dev(inv_m)
    out = {}
    for fold in ("1", "0"):
        monkeypatch.setenv("CFA_CG_FUSE_UPDATE", fold)
        amg = cfa.AmgPreconditioner(ctx, prec)
        amg.setup(m.n, ci.size, dm.rp, dm.ci, dK)
        s = cfa.GpuLinearSolver(ctx)
        x = torch.zeros(m.n, dtype=torch.float64, device="cuda")
        it = s.solve_pcg(m.n, dm.rp, dm.ci, dK, db, x, 4000, 1e-10, cfa.oss_operator(dm, doss, dinv), amg)
        assert s.converged
        out[fold] = (it, host(x))
    assert abs(out["1"][0] - out["0"][0]) <= 1
    assert np.abs(out["1"][1] - out["0"][1]).max() <= 1e-8 * np.abs(out["0"][1]).max()
    x = out["1"][1]
    Ax = O.spmv(rp, ci, Kp, x)
    O.oss_apply(m, rp, ci, oss, inv_m, x, Ax)
    assert np.linalg.norm(rhs - Ax) <= 1.5e-10 * np.linalg.norm(rhs)


@pytest.mark.parametrize("name", ["c0", "113k"])
@pytest.mark.parametrize("prec", [cfa.FP64, cfa.MIXED])
def test_pcg_prescaled_residual_gives_the_same_bits(ctx, name, prec, monkeypatch):
    """The CG update writing c = omega0 D0^-1 r (in the V-cycle's vector type) for the level-0
    pre-smoothing, which then gathers c instead of D0^-1 and r: the products are formed in the
    same order, so the solve is bit-identical to the one that forms them inside the V-cycle."""
    m = mesh(name)
    dm = cfa.DeviceMesh(ctx, m)
    rp, ci = dm.host_pattern()
    Kp, rhs, oss, inv_m = pressure_system(m, rp, ci)
    dK, db, doss, dinv = dev(Kp), dev(rhs), dev(oss), dev(inv_m)
    out = {}
    for pre in ("1", "0"):
        monkeypatch.setenv("CFA_PRESCALE", pre)
        amg = cfa.AmgPreconditioner(ctx, prec)
        amg.setup(m.n, ci.size, dm.rp, dm.ci, dK)
        s = cfa.GpuLinearSolver(ctx)
        x = torch.zeros(m.n, dtype=torch.float64, device="cuda")
        it = s.solve_pcg(m.n, dm.rp, dm.ci, dK, db, x, 4000, 1e-10, cfa.oss_operator(dm, doss, dinv), amg)
        assert s.converged
        out[pre] = (it, host(x))
    assert out["1"][0] == out["0"][0]
    assert np.array_equal(out["1"][1], out["0"][1])


@pytest.mark.parametrize("graphs", ["1", "0"])
def test_pcg_fp64_phase_of_a_mixed_hierarchy(ctx, graphs, monkeypatch):
    """A mixed-precision hierarchy whose solves run their V-cycles in FP64 down to a relative
    residual of 1e-2 and in FP32 after: the switch keeps the flexible CG's state, so the solve
    reaches the FP64 hierarchy's iteration count (within 1) where FP32 throughout needs more, and
    its true residual meets the tolerance; with and without the solve graphs."""
    monkeypatch.setenv("CFA_GRAPHS", graphs)
    m = mesh("c0")
    dm = cfa.DeviceMesh(ctx, m)
    rp, ci = dm.host_pattern()
    Kp, rhs, oss, inv_m = pressure_system(m, rp, ci)
    dK, db, doss, dinv = dev(Kp), dev(rhs), dev(oss), dev(inv_m)
    its = {}
    for label, prec, phase in (("fp64", cfa.FP64, -1.0), ("fp32", cfa.MIXED, 0.0), ("phase", cfa.MIXED, 1e-2)):
        amg = cfa.AmgPreconditioner(ctx, prec)
        amg.set_fp64_phase(phase)
        amg.setup(m.n, ci.size, dm.rp, dm.ci, dK)
        s = cfa.GpuLinearSolver(ctx)
        x = torch.zeros(m.n, dtype=torch.float64, device="cuda")
        its[label] = s.solve_pcg(m.n, dm.rp, dm.ci, dK, db, x, 4000, 1e-10, cfa.oss_operator(dm, doss, dinv), amg)
        assert s.converged, label
        xh = host(x)
        Ax = O.spmv(rp, ci, Kp, xh)
        O.oss_apply(m, rp, ci, oss, inv_m, xh, Ax)
        assert np.linalg.norm(rhs - Ax) <= 1.5e-10 * np.linalg.norm(rhs), label
    assert abs(its["phase"] - its["fp64"]) <= 1, its
    assert its["phase"] <= its["fp32"], its
    # a warm start below the switch: the first phase stops at its initial residual, the second
    # iterates to the tolerance
    x0 = xh + 1e-8 * np.abs(xh).max() * np.sin(0.37 * np.arange(m.n))
    r0 = O.spmv(rp, ci, Kp, x0)
    O.oss_apply(m, rp, ci, oss, inv_m, x0, r0)
    assert 1e-9 < np.linalg.norm(rhs - r0) / np.linalg.norm(rhs) < 1e-2
    x = dev(x0)
    it = s.solve_pcg(m.n, dm.rp, dm.ci, dK, db, x, 4000, 1e-10, cfa.oss_operator(dm, doss, dinv), amg)
    assert s.converged and it >= 1
    xh = host(x)
    Ax = O.spmv(rp, ci, Kp, xh)
    O.oss_apply(m, rp, ci, oss, inv_m, xh, Ax)
    assert np.linalg.norm(rhs - Ax) <= 1.5e-10 * np.linalg.norm(rhs)
    with pytest.raises(cfa.CfaError):
        cfa.AmgPreconditioner(ctx, cfa.MIXED).set_fp64_phase(1.0)


@pytest.mark.parametrize("host_prec", [False, True])
def test_pcg_host_ops_match_handles(ctx, host_prec):
    """solve_pcg with the OSS term (and optionally the preconditioner) as host callbacks, the way
    the reference's std::function hooks call them, against the solve with handles."""
    import ctypes as C
    m = mesh("small")
    dm = cfa.DeviceMesh(ctx, m)
    rp, ci = dm.host_pattern()
    Kp, rhs, oss, inv_m = pressure_system(m, rp, ci)
    dK, db, doss, dinv = dev(Kp), dev(rhs), dev(oss), dev(inv_m)
    amg = cfa.AmgPreconditioner(ctx)
    amg.setup(m.n, ci.size, dm.rp, dm.ci, dK)
    s = cfa.GpuLinearSolver(ctx)
    x0 = torch.zeros(m.n, dtype=torch.float64, device="cuda")
    it0 = s.solve_pcg(m.n, dm.rp, dm.ci, dK, db, x0, 4000, 1e-10, cfa.oss_operator(dm, doss, dinv), amg)
    cb = cfa.Context(stream=ctx.stream)   # the callbacks' own context, on the same stream
    L = cfa.lib()
    calls = {"extra": 0, "prec": 0}

    def extra(i, o):
        calls["extra"] += 1
        cb.check(L.cfa_oss_apply(cb.h, dm.h, cfa.ptr(doss), cfa.ptr(dinv), C.c_void_p(i), C.c_void_p(o)))

    def prec(i, o):
        calls["prec"] += 1
        cb.check(L.cfa_amg_apply(cb.h, amg.h, C.c_void_p(i), C.c_void_p(o)))

    x1 = torch.zeros(m.n, dtype=torch.float64, device="cuda")
    it1 = s.solve_pcg_host_ops(m.n, dm.rp, dm.ci, dK, db, x1, 4000, 1e-10, extra_op=extra,
                               amg=None if host_prec else amg, precond=prec if host_prec else None)
    assert s.converged and abs(it1 - it0) <= 2
    assert calls["extra"] >= it1 + 1 and (calls["prec"] >= it1 if host_prec else calls["prec"] == 0)
    assert torch.abs(x1 - x0).max().item() <= 1e-8 * torch.abs(x0).max().item()


def test_pcg_new_pattern_at_the_same_addresses(ctx):
    """A different pattern with the same n and nnz written into the same device arrays (a remesh
    that lands on recycled buffers) is solved with its own tile plan, not the cached one."""
    import scipy.sparse as sp
    import scipy.sparse.linalg as spl
    m = mesh("small")
    rp, ci = O.csr_build(m.n, m.elem_v)
    perm = np.random.default_rng(5).permutation(m.n).astype(np.int32)
    rp2, ci2 = O.csr_build(m.n, perm[m.elem_v])
    assert ci2.size == ci.size and not np.array_equal(rp, rp2)
    drp, dci = dev(rp, torch.int32), dev(ci, torch.int32)
    dval = torch.zeros(ci.size, dtype=torch.float64, device="cuda")
    b = F.fourier_field(m.x, m.y, 4)
    db = dev(b)
    s = cfa.GpuLinearSolver(ctx)
    for r, c in ((rp, ci), (rp2, ci2)):
        rows = np.repeat(np.arange(m.n), np.diff(r))
        val = np.where(c == rows, np.diff(r)[rows].astype(np.float64), -1.0)   # SPD, diagonally dominant
        drp.copy_(torch.from_numpy(r))
        dci.copy_(torch.from_numpy(c))
        dval.copy_(torch.from_numpy(val))
        x = torch.zeros(m.n, dtype=torch.float64, device="cuda")
        s.solve_pcg(m.n, drp, dci, dval, db, x, 2000, 1e-12)
        assert s.converged
        want = spl.spsolve(sp.csr_matrix((val, c, r), shape=(m.n, m.n)).tocsc(), b)
        assert np.abs(host(x) - want).max() <= 1e-9 * np.abs(want).max()


@pytest.mark.parametrize("name,outlet_dirichlet", [("small", 0), ("medium", 0), ("medium", 1)])
def test_pressure_operator_fused_oss_matches_oracle(name, outlet_dirichlet, monkeypatch):
    """K - B^T M^-1 B assembled into one two-ring matrix (the default) and the two-pass apply
    against the oracle's K x and apply_oss_projection: 1e-13 of the largest entry."""
    m = mesh(name)
    results = []
    for fused in ("1", "0"):
        monkeypatch.setenv("CFA_OSS_FUSED", fused)
        c = cfa.Context(stream=cfa.default_context().stream)   # a fresh context plans its operator anew
        dm = cfa.DeviceMesh(c, m)
        pin = int(np.argmax(m.x)) if outlet_dirichlet else -1
        if outlet_dirichlet:
            dm.set_outlet(1, pin, 1.0)
        rp, ci = dm.host_pattern()
        Kp, rhs, oss, inv_m = pressure_system(m, rp, ci)
        x = np.sin(0.3 * np.arange(m.n)) + 0.1
        want = O.spmv(rp, ci, Kp, x)
        O.oss_apply(m, rp, ci, oss, inv_m, x, want, outlet_dirichlet=outlet_dirichlet, pin=pin)
        dK, doss, dinv = dev(Kp), dev(oss), dev(inv_m)
        op = cfa.oss_operator(dm, doss, dinv)
        cfa.pressure_operator_prepare(c, dm.rp, dm.ci, dK, op)
        y = torch.zeros(m.n, dtype=torch.float64, device="cuda")
        cfa.pressure_operator(c, dm.rp, dm.ci, dK, dev(x), y, op)
        got = host(y)
        assert np.abs(got - want).max() <= 1e-13 * np.abs(want).max()
        results.append(got)
    assert np.abs(results[0] - results[1]).max() <= 1e-13 * np.abs(results[1]).max()


def test_pcg_mixed_precision_reaches_tolerance(ctx):
    m = mesh("medium")
    dm = cfa.DeviceMesh(ctx, m)
    rp, ci = dm.host_pattern()
    Kp, rhs, oss, inv_m = pressure_system(m, rp, ci)
    dK, db, doss, dinv = dev(Kp), dev(rhs), dev(oss), dev(inv_m)
    op = cfa.oss_operator(dm, doss, dinv)
    res = {}
    for prec in (cfa.FP64, cfa.MIXED):
        amg = cfa.AmgPreconditioner(ctx, prec)
        amg.setup(m.n, ci.size, dm.rp, dm.ci, dK)
        s = cfa.GpuLinearSolver(ctx)
        dx = torch.zeros(m.n, dtype=torch.float64, device="cuda")
        it = s.solve_pcg(m.n, dm.rp, dm.ci, dK, db, dx, 4000, 1e-10, op, amg)
        assert s.converged
        x = host(dx)
        Ax = O.spmv(rp, ci, Kp, x)
        O.oss_apply(m, rp, ci, oss, inv_m, x, Ax)
        assert np.linalg.norm(rhs - Ax) <= 1.5e-10 * np.linalg.norm(rhs)
        res[prec] = (it, x)
    assert np.abs(res[cfa.MIXED][1] - res[cfa.FP64][1]).max() < 1e-7 * np.abs(res[cfa.FP64][1]).max()
    # the FP32 V-cycle (values, vectors and arithmetic) is a preconditioner accurate to ~1e-7; at a
    # 1e-10 tolerance the flexible CG takes up to about an eighth more iterations
    assert res[cfa.MIXED][0] <= 1.15 * res[cfa.FP64][0] + 3


def test_pcg_zero_rhs_and_breakdown(ctx):
    m = mesh("tiny")
    rp, ci = O.csr_build(m.n, m.elem_v)
    a = laplacian(rp, ci)
    s = cfa.GpuLinearSolver(ctx)
    drp, dci, da = dev(rp, torch.int32), dev(ci, torch.int32), dev(a)
    dx = torch.ones(m.n, dtype=torch.float64, device="cuda")
    it = s.solve_pcg(m.n, drp, dci, da, torch.zeros(m.n, dtype=torch.float64, device="cuda"), dx, 100, 1e-10)
    assert it == 0 and s.converged and float(dx.abs().max()) == 0.0     # reference: x = 0 for |b| < 1e-14
    # zero operator: p.q = 0 -> breakdown guard, not converged
    dx.zero_()
    it = s.solve_pcg(m.n, drp, dci, torch.zeros_like(da), dev(np.ones(m.n)), dx, 100, 1e-10)
    assert not s.converged and it == 0


def test_pcg_matches_reference_gpu_golden(ctx):
    g = golden("ref_gpu_small.npz")
    h = golden("ref_host_small.npz")
    rp, ci = h["rp"], h["ci"]
    n = rp.size - 1
    amg = cfa.AmgPreconditioner(ctx)
    drp, dci, da = dev(rp, torch.int32), dev(ci, torch.int32), dev(h["lap_val"])
    amg.setup(n, ci.size, drp, dci, da)
    s = cfa.GpuLinearSolver(ctx)
    dx = torch.zeros(n, dtype=torch.float64, device="cuda")
    it = s.solve_pcg(n, drp, dci, da, dev(np.cos(0.11 * np.arange(n))), dx, 400, 1e-10, None, amg)
    assert s.converged and abs(it - g["lap_pcg_info"][0]) <= 1
    assert np.abs(host(dx) - g["lap_pcg_x"]).max() < 1e-8 * np.abs(g["lap_pcg_x"]).max()


# ------------------------------------------------------------------------------------------------
# the whole step
# ------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("precision", [cfa.FP64, cfa.MIXED])
def test_step_matches_oracle(ctx, precision):
    import step as S
    m = mesh("medium")
    u, v, p = fields(m)
    st = S.SolveStep(m, u, v, p, precision=precision, ctx=ctx)
    st.amg_setup()
    # the solutions copied to pinned host memory by the step itself (u, v during the pressure
    # solve), one synchronisation of the context's stream
    outs = [torch.empty(m.n, dtype=torch.float64).pin_memory() for _ in range(3)]
    st.run(host_out=outs)
    ctx.stream.synchronize()
    rep = st.report()
    assert all(rep["conv"]), rep
    for o, d in zip(outs, (st.u, st.v, st.dp)):
        assert np.array_equal(o.numpy(), host(d))
    rp, ci = st.dm.host_pattern()
    A, ru, rv, mass = O.assemble_momentum(m, rp, ci, u, v, u, v, p, O.bdf2_params())
    uu, vv = u.copy(), v.copy()
    O.apply_bc_momentum(m, rp, ci, A, ru, rv, uu, vv)
    oi = O.Ilu(rp, ci)
    oi.factor(A)
    xu, xv, reps = O.bicgstab2(rp, ci, A, ru, rv, uu, vv, oi, 1000, 1e-10)
    assert np.abs(host(st.u) - xu).max() < 1e-8 * np.abs(xu).max()
    assert np.abs(host(st.v) - xv).max() < 1e-8 * np.abs(xv).max()
    us, vs = host(st.u), host(st.v)
    dt_proj = 2e-3 / 3
    s = O.oss_weights(m, us, vs, dt_proj, 1.0, 1e-3, 0.3)
    gx, gy = O.scalar_gradient(m, p, s)
    Kp, rhs, div = O.assemble_ppe(m, rp, ci, us, vs, p, gx, gy, mass, s, dt_proj, 1.0, 0.3)
    dp = np.zeros(m.n)
    O.apply_bc_pressure(m, rp, ci, Kp, rhs, dp, mass)
    oss, inv_m = O.assemble_oss(m, rp, ci, s, mass)
    oa = O.Amg(rp, ci, Kp)
    xo, repo = O.pcg(rp, ci, Kp, rhs, dp, 4000, 1e-10, oss, inv_m, m.tag, oa)
    assert np.abs(host(st.dp) - xo).max() < 1e-7 * np.abs(xo).max()


def test_step_matches_reference_gpu_golden(ctx):
    import step as S
    g = golden("ref_gpu_small.npz")
    h = golden("ref_host_small.npz")
    m = MeshFromGolden(h)
    st = S.SolveStep(m, h["u"], h["v"], h["p"], ctx=ctx)
    st.amg_setup()
    st.run()
    rep = st.report()
    assert all(rep["conv"])
    for k, t in (("step_u", st.u), ("step_v", st.v), ("step_dp", st.dp)):
        ref = g[k]
        assert np.abs(host(t) - ref).max() < 1e-7 * np.abs(ref).max(), k
    assert abs(rep["it_p"] - int(g["step_its"][2])) <= 2


def test_step_live_reference_harness(ctx):
    """When the reference's CUDA build is present (oracle/_ref), run one of its steps on the same
    inputs in this process and compare the solutions."""
    import ctypes as C
    import os
    from oracle import build as B
    if not os.path.exists(B.REF_LIB):
        pytest.skip("reference harness not built")
    import step as S
    R = O.ref()
    m = mesh("medium")
    u, v, p = fields(m)
    ev = np.ascontiguousarray(m.elem_v, np.int32)
    tag = np.ascontiguousarray(m.tag, np.int32)
    h = C.c_void_p(R.ref_step_create(m.n, m.ne, O._p(ev), O._p(m.x), O._p(m.y), O._p(tag), O._p(u), O._p(v), O._p(p),
                                     C.c_double(1e-3), C.c_double(1e-3), C.c_double(1.0), C.c_double(1.5),
                                     C.c_double(1.0), C.c_double(1e-3), C.c_double(0.3), C.c_double(1e-10), 1000, 4000))
    R.ref_step_amg_setup(h)
    its, conv, rel = np.zeros(3, np.int32), np.zeros(3, np.int32), np.zeros(3)
    ru, rv, rdp = np.zeros(m.n), np.zeros(m.n), np.zeros(m.n)
    R.ref_step_run(h, O._p(its), O._p(conv), O._p(rel), O._p(ru), O._p(rv), O._p(rdp))
    R.ref_step_free(h)
    st = S.SolveStep(m, u, v, p, ctx=ctx)
    st.amg_setup()
    st.run()
    assert all(conv) and all(st.report()["conv"])
    assert np.abs(host(st.u) - ru).max() < 1e-8 * np.abs(ru).max()
    assert np.abs(host(st.dp) - rdp).max() < 1e-7 * np.abs(rdp).max()


# ------------------------------------------------------------------------------------------------
# f1: after the solves (Steps C and D) and the time loop
# ------------------------------------------------------------------------------------------------
def test_post_solve_kernels_match_oracle(ctx):
    m = mesh("medium")
    dm = cfa.DeviceMesh(ctx, m)
    u, v, p = fields(m)
    rng = np.random.default_rng(5)
    dp = rng.uniform(-1, 1, m.n)
    mass = O.lumped_mass(m)
    # stiffness (adds into out)
    base = rng.uniform(-1, 1, m.n)
    want = base.copy()
    O.stiffness_apply(m, dp, -0.37, want)
    got = dev(base)
    cfa.stiffness_apply(ctx, dm, dev(dp), -0.37, got)
    assert np.abs(host(got) - want).max() <= 1e-12 * np.abs(want).max()
    # grad dp and vorticity numerators
    gdx, gdy, vn = O.grad_dp_vorticity(m, dp, u, v)
    dgx, dgy, dvn = (torch.zeros(m.n, dtype=torch.float64, device="cuda") for _ in range(3))
    cfa.grad_dp_vorticity(ctx, dm, dev(dp), dev(u), dev(v), dgx, dgy, dvn)
    for g, w in ((dgx, gdx), (dgy, gdy), (dvn, vn)):
        assert np.abs(host(g) - w).max() <= 1e-12 * np.abs(w).max()
    # correction
    div_num = rng.uniform(-1, 1, m.n) * mass
    uo, vo, po = u.copy(), v.copy(), p.copy()
    vort = O.velocity_pressure_correction(m, 2e-3 / 3, 1.0, 1.0, 1e-3, div_num, mass, gdx, gdy, vn, dp, uo, vo, po)
    du, dv, dpp, dvort = dev(u), dev(v), dev(p), torch.zeros(m.n, dtype=torch.float64, device="cuda")
    cfa.velocity_pressure_correction(ctx, dm, 2e-3 / 3, 1.0, 1.0, 1e-3, dev(div_num), dev(mass), dev(gdx), dev(gdy),
                                     dev(vn), dev(dp), du, dv, dpp, dvort)
    for g, w in ((du, uo), (dv, vo), (dpp, po), (dvort, vort)):
        assert np.abs(host(g) - w).max() <= 1e-13 * np.abs(w).max()
    # the fused Step C
    div2 = np.zeros(m.n)
    O.stiffness_apply(m, dp, -(2e-3 / 3), div2)
    u2, v2, p2 = u.copy(), v.copy(), p.copy()
    vort2 = O.velocity_pressure_correction(m, 2e-3 / 3, 1.0, 1.0, 1e-3, div2, mass, gdx, gdy, vn, dp, u2, v2, p2)
    du, dv, dpp = dev(u), dev(v), dev(p)
    bufs = [torch.zeros(m.n, dtype=torch.float64, device="cuda") for _ in range(5)]
    cfa.project_step(ctx, dm, 2e-3 / 3, 1.0, 1e-3, True, dev(mass), dev(dp), *bufs[:4], du, dv, dpp, bufs[4])
    for g, w in ((du, u2), (dv, v2), (dpp, p2), (bufs[4], vort2)):
        assert np.abs(host(g) - w).max() <= 1e-12 * np.abs(w).max()
    # volume forces
    up, vp = 0.9 * u, 0.8 * v
    want = O.volume_forces(m, u, v, 0.95 * u, 0.9 * v, up, vp, p, 1.5e3, -2e3, 0.5e3, 1e-3, 1.0)
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    cfa.volume_forces(ctx, dm, dev(u), dev(v), dev(0.95 * u), dev(0.9 * v), dev(up), dev(vp), dev(p), 1.5e3, -2e3,
                      0.5e3, 1e-3, 1.0, out)
    assert np.abs(host(out) - want).max() <= 1e-12 * np.abs(want).max()


def test_amr_indicators_match_oracle(ctx):
    m = mesh("medium")
    dm = cfa.DeviceMesh(ctx, m)
    u, v, _ = fields(m)
    mass = O.lumped_mass(m)
    g, err = O.amr_indicators(m, u, v, 1.5, 1.0, mass)
    dg = torch.zeros(4 * m.n, dtype=torch.float64, device="cuda")
    de = torch.zeros(2 * m.ne, dtype=torch.float64, device="cuda")
    cfa.amr_indicators(ctx, dm, dev(u), dev(v), 1.5, 1.0, dev(mass), dg, de)
    assert np.abs(host(dg) - g).max() <= 1e-12 * np.abs(g).max()
    assert np.abs(host(de) - err).max() <= 1e-11 * np.abs(err).max()


@pytest.mark.parametrize("precision", [cfa.FP64, cfa.MIXED])
def test_time_stepper_matches_oracle(ctx, precision):
    """The device time loop against the oracle's (same steps and options) over 12 BDF2 steps from
    rest, solves at 1e-12: drag and lift histories within 1e-9 of the drag scale."""
    import step as S
    m = mesh("small")
    z = np.zeros(m.n)
    kw = dict(dt=5e-3, tol_mom=1e-12, tol_p=1e-12, max_it_mom=400, amg_rebuild=5)
    ref = O.Stepper(m, z, z, z, **kw)
    st = S.TimeStepper(m, z, z, z, precision=precision, ctx=ctx, **kw)
    for k in range(12):
        want = ref.step()
        got = st.step()
        scale = max(1.0, abs(want[0]))
        assert abs(got[0] - want[0]) <= 1e-9 * scale and abs(got[1] - want[1]) <= 1e-9 * scale, (k, got, want)
    assert np.abs(host(st.u) - ref.u).max() <= 1e-9 * np.abs(ref.u).max()
    assert np.abs(host(st.p) - ref.p).max() <= 1e-9 * np.abs(ref.p).max()


@pytest.mark.parametrize("precision", [cfa.FP64, cfa.MIXED])
def test_time_stepper_400_steps_forces_within_1e9(ctx, precision):
    """400 BDF2 steps (dt 1e-3, from rest, the reference's defaults: OSS 0.3, AMG rebuilt every
    50 steps) on the ~22.5k-vertex uniform mesh, solves at 1e-10 so that the stopping tolerance
    does not set the size of the difference: the device loop's drag and lift histories against
    the oracle's within 1e-9 of the force scale (the largest |C_D| past the impulsive start,
    step 20 on) at every step. The disc sits on the channel's centre line, so the lift is zero
    in exact arithmetic (|C_L| stays below 1e-3 here) and is measured against the drag's scale,
    not its own."""
    import step as S
    m = mesh("c0")
    z = np.zeros(m.n)
    kw = dict(dt=1e-3, tol_mom=1e-10, tol_p=1e-10, max_it_mom=400, amg_rebuild=50)
    ref = O.Stepper(m, z, z, z, **kw)
    st = S.TimeStepper(m, z, z, z, precision=precision, ctx=ctx, **kw)
    want = np.array([ref.step() for _ in range(400)])
    got = np.array([st.step() for _ in range(400)])
    scale = np.abs(want[20:, 0]).max()
    d = np.abs(got - want) / scale
    print(f"400 steps: max |dC_D|/scale {d[:, 0].max():.3e} (step {d[:, 0].argmax() + 1}), "
          f"max |dC_L|/scale {d[:, 1].max():.3e} (step {d[:, 1].argmax() + 1}), scale {scale:.4f}, "
          f"max |C_L| {np.abs(want[20:, 1]).max():.3e}")
    assert d.max() <= 1e-9, d.max(axis=0)


# ------------------------------------------------------------------------------------------------
# f2: re-projection of transferred velocities after a remesh
# ------------------------------------------------------------------------------------------------
def test_reprojection_matches_oracle(ctx):
    import step as S
    m = mesh("small")
    dm = cfa.DeviceMesh(ctx, m)
    rp, ci = dm.host_pattern()
    u, v, p = fields(m)
    # divergence-free projection (plain PPE), p unchanged
    uo, vo = u.copy(), v.copy()
    O.project_divergence_free(m, rp, ci, 1e-3, uo, vo, tol=1e-12)
    du, dv, dpp = dev(u), dev(v), dev(p)
    mass = torch.zeros(m.n, dtype=torch.float64, device="cuda")
    it, vort = S.project_divergence_free(ctx, dm, 1e-3, du, dv, dpp, mass, amg=cfa.AmgPreconditioner(ctx), tol=1e-12)
    assert it > 0
    assert np.abs(host(du) - uo).max() <= 1e-9 * np.abs(uo).max()
    assert np.abs(host(dv) - vo).max() <= 1e-9 * np.abs(vo).max()
    assert np.array_equal(host(dpp), p)
    # scheme-consistent projection of both levels with the OSS operator
    u1, v1 = 0.9 * u, 0.9 * v
    lv = [(u1.copy(), v1.copy()), (u.copy(), v.copy())]
    O.project_scheme_consistent(m, rp, ci, 2e-3 / 3, 0.3, 1e-3, lv, p, tol=1e-12)
    du1, dv1, du, dv = dev(u1), dev(v1), dev(u), dev(v)
    S.project_scheme_consistent(ctx, dm, 2e-3 / 3, 0.3, 1e-3, du1, dv1, du, dv, dev(p),
                                amg=cfa.AmgPreconditioner(ctx), tol=1e-12)
    for g, w in ((du1, lv[0][0]), (dv1, lv[0][1]), (du, lv[1][0]), (dv, lv[1][1])):
        assert np.abs(host(g) - w).max() <= 1e-9 * np.abs(w).max()
