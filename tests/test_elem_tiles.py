"""Assembly on element tiles (a block's elements computed once) and its row-gather form for tiles
too large, against the oracle: meshes of one element to several tile heights, orders that scatter
a tile's elements, and a node of more elements than a tile holds."""
import numpy as np
import pytest

import fixtures as F

pytestmark = pytest.mark.gpu


def _shuffled(m, seed=1):
    """Vertices and elements in random order: a tile of rows touches almost only its own elements."""
    rng = np.random.default_rng(seed)
    perm, eperm = rng.permutation(m.n), rng.permutation(m.ne)
    new = np.empty_like(perm)
    new[perm] = np.arange(m.n)
    return F.Mesh(m.x[perm].copy(), m.y[perm].copy(), m.tag[perm].copy(),
                  new[m.tri][eperm].astype(np.int32), m.gen[eperm].copy())


def _wheel(spokes):
    """A disc of `spokes` elements around vertex 0, its rim in [0, 1] x [0, 1]."""
    th = 2 * np.pi * np.arange(spokes) / spokes
    x = np.concatenate([[0.5], 0.5 + 0.5 * np.cos(th)])
    y = np.concatenate([[0.5], 0.5 + 0.5 * np.sin(th)])
    k = np.arange(spokes)
    tri = np.stack([np.zeros(spokes, np.int64), 1 + k, 1 + (k + 1) % spokes], 1).astype(np.int32)
    tag = np.zeros(spokes + 1, np.int32)
    tag[1::7], tag[2::7], tag[3::11] = F.BC_INLET, F.BC_OUTLET, F.BC_WALL
    return F.Mesh(x, y, tag, tri, np.zeros(spokes, np.int32))


def _target(n, seed):
    import batch as B
    return B.batch_system(seed, n, n).mesh


def _one():
    return F.Mesh(np.array([0.0, 1.0, 0.3]), np.array([0.0, 0.2, 0.9]), np.array([0, 2, 1], np.int32),
                  np.array([[0, 1, 2]], np.int32), np.zeros(1, np.int32))


CASES = {
    "one": _one,
    "tiny": lambda: F.make_mesh("tiny"),
    "small": lambda: F.make_mesh("small"),
    "small_shuffled": lambda: _shuffled(F.make_mesh("small")),
    "c0_rows64": lambda: F.make_mesh("c0"),
    "37k_rows96": lambda: _target(31_001, 5),
    "medium_rows96": lambda: F.make_mesh("medium"),
    "wheel_24": lambda: _wheel(24),              # one thread plans the row
    "wheel_25": lambda: _wheel(25),              # the whole block does
    "wheel_127": lambda: _wheel(127),
    "wheel_255": lambda: _wheel(255),            # 256 entries in the row, as many as threads
    "wheel_256": lambda: _wheel(256),
    "wheel_1200": lambda: _wheel(1200),          # one tile with nearly all of a block's shared memory
    "wheel_2000_gather": lambda: _wheel(2000),   # records beyond it: the row gathers
    "wheel_3100_gather": lambda: _wheel(3100),   # incidences beyond the plan's sort
}


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("outlet_dirichlet", [0, 1])
def test_assembly_matches_the_oracle(name, outlet_dirichlet):
    import torch
    import cfa_b200 as cfa
    from oracle import oracle as O
    m = CASES[name]()
    ctx = cfa.default_context()
    rp, ci = O.csr_build(m.n, m.elem_v)
    dm = cfa.DeviceMesh(ctx, m, torch.from_numpy(rp).to("cuda"), torch.from_numpy(ci).to("cuda"))
    pin = int(np.flatnonzero(m.tag == F.BC_OUTLET)[0])
    if outlet_dirichlet:
        dm.set_outlet(1, pin, 1.25)
    n, nnz = m.n, len(ci)
    u, v, p = (F.fourier_field(m.x, m.y, 1), F.fourier_field(m.x, m.y, 2), 0.3 * F.fourier_field(m.x, m.y, 3))
    up, vp = 0.9 * u, 1.1 * v
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float64)).to("cuda")
    z = lambda k: torch.full((k,), float("nan"), dtype=torch.float64, device="cuda")
    # momentum without its boundary rows, then the library's own boundary rows on both
    A, ru, rv, mass = z(nnz), z(n), z(n), z(n)
    prm = cfa.bdf2_params()
    cfa.assemble_momentum(ctx, dm, t(u), t(v), t(up), t(vp), t(p), prm, A, ru, rv, mass)
    oA, oru, orv, omass = O.assemble_momentum(m, rp, ci, u, v, up, vp, p, O.bdf2_params())
    # every value is a sum of at most a few hundred terms of its own size in the same order; the
    # element formulas differ by reciprocals and contractions: a few hundred roundings of 1.1e-16
    for got, want in ((A, oA), (ru, oru), (rv, orv), (mass, omass)):
        assert np.abs(got.cpu().numpy() - want).max() <= 1e-12 * np.abs(want).max()
    A2, ru2, rv2, mass2, uu, vv = z(nnz), z(n), z(n), z(n), t(u), t(v)
    cfa.assemble_momentum(ctx, dm, t(u), t(v), t(up), t(vp), t(p), prm, A2, ru2, rv2, mass2, uu, vv, u_max=1.5)
    uu1, vv1 = t(u), t(v)
    cfa.apply_bc_momentum(ctx, dm, A, ru, rv, uu1, vv1, 1.5)
    for a, b in ((A, A2), (ru, ru2), (rv, rv2), (uu, uu1), (vv, vv1)):
        assert torch.equal(a, b)
    # pressure: values, right-hand side and OSS operator without boundary rows, then with them
    dt = 2e-3 / 3
    s = O.oss_weights(m, u, v, dt, 1.0, 1e-3, 0.3)
    gx, gy = z(n), z(n)
    cfa.scalar_gradient(ctx, dm, t(p), t(s), gx, gy)
    ogx, ogy = O.scalar_gradient(m, p, s)
    for got, want in ((gx, ogx), (gy, ogy)):
        assert np.abs(got.cpu().numpy() - want).max() <= 1e-12 * max(np.abs(ogx).max(), np.abs(ogy).max())
    K, rhs, div = z(nnz), z(n), z(n)
    cfa.assemble_ppe(ctx, dm, t(u), t(v), t(p), t(ogx), t(ogy), t(omass), t(s), dt, 1.0, 0.3, K, rhs, div,
                     apply_bc=False)
    oK, orhs, odiv = O.assemble_ppe(m, rp, ci, u, v, p, ogx, ogy, omass, s, dt, 1.0, 0.3)
    for got, want in ((K, oK), (rhs, orhs), (div, odiv)):
        assert np.abs(got.cpu().numpy() - want).max() <= 1e-11 * np.abs(want).max()
    oss, im = z(4 * nnz), z(n)
    cfa.assemble_oss(ctx, dm, t(s), t(omass), oss, im)
    ooss, oim = O.assemble_oss(m, rp, ci, s, omass)
    for got, want in ((oss, ooss), (im, oim)):
        assert np.abs(got.cpu().numpy() - want).max() <= 1e-12 * np.abs(want).max()
    K2, rhs2, div2, dp2, oss2, im2 = z(nnz), z(n), z(n), t(p), z(4 * nnz), z(n)
    cfa.assemble_pressure_system(ctx, dm, t(u), t(v), t(p), t(ogx), t(ogy), t(omass), t(s), dt, 1.0, 0.3, K2, rhs2,
                                 div2, dp2, oss2, im2)
    dp1 = t(p)
    cfa.apply_bc_pressure(ctx, dm, K, rhs, dp1, t(omass))
    for a, b in ((K, K2), (rhs, rhs2), (div, div2), (dp1, dp2), (oss, oss2), (im, im2)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("name", list(CASES))
def test_node_gradients_match_the_formulas(name):
    import torch
    import cfa_b200 as cfa
    from oracle import oracle as O
    m = CASES[name]()
    ctx = cfa.default_context()
    rp, ci = O.csr_build(m.n, m.elem_v)
    dm = cfa.DeviceMesh(ctx, m, torch.from_numpy(rp).to("cuda"), torch.from_numpy(ci).to("cuda"))
    n, t = m.n, m.tri.astype(np.int64)
    X, Y = m.x[t], m.y[t]
    area = 0.5 * np.abs((X[:, 1] - X[:, 0]) * (Y[:, 2] - Y[:, 0]) - (X[:, 2] - X[:, 0]) * (Y[:, 1] - Y[:, 0]))
    gx = np.stack([Y[:, 1] - Y[:, 2], Y[:, 2] - Y[:, 0], Y[:, 0] - Y[:, 1]], 1) / (2 * area)[:, None]
    gy = np.stack([X[:, 2] - X[:, 1], X[:, 0] - X[:, 2], X[:, 1] - X[:, 0]], 1) / (2 * area)[:, None]

    def nodes(e):          # e: one value per element, or per element and vertex
        out, size = np.zeros(n), np.zeros(n)
        e = np.broadcast_to(e if e.ndim == 2 else e[:, None], t.shape)
        np.add.at(out, t.ravel(), e.ravel())
        np.add.at(size, t.ravel(), np.abs(e).ravel())
        return out, size.max()

    grad = lambda f: ((f[t] * gx).sum(1), (f[t] * gy).sum(1))
    u, v, dp = (F.fourier_field(m.x, m.y, k) for k in (1, 2, 3))
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float64)).to("cuda")
    z = lambda k: torch.full((k,), float("nan"), dtype=torch.float64, device="cuda")

    def close(got, want):  # sums of at most 3100 terms, each a few dozen roundings
        assert np.abs(got.cpu().numpy() - want[0]).max() <= 1e-12 * want[1]

    w = area / 3
    (dx, dy), curl = grad(dp), grad(v)[0] - grad(u)[1]
    a, b, c = z(n), z(n), z(n)
    cfa.grad_dp_vorticity(ctx, dm, d(dp), d(u), d(v), a, b, c)
    for got, e in ((a, w * dx), (b, w * dy), (c, w * curl)):
        close(got, nodes(e))
    s0 = np.linspace(-1, 1, n)
    s = d(s0)
    cfa.stiffness_apply(ctx, dm, d(dp), -0.37, s)
    want, size = nodes(-0.37 * area[:, None] * (gx * dx[:, None] + gy * dy[:, None]))
    close(s, (want + s0, max(size, 1.0)))
    mass, rec, err = d(nodes(w)[0]), z(4 * n), z(2 * m.ne)
    cfa.amr_indicators(ctx, dm, d(u), d(v), 1.5, 1.0, mass, rec, err)
    ud = u - 6.0 * m.y * (1 - m.y)
    for k, e in enumerate((*grad(ud), *grad(v))):
        close(rec[k * n:(k + 1) * n], nodes(w * e))


# ----------------------------------------------------------------------------------------------
# the two forms give the same bits
# ----------------------------------------------------------------------------------------------
HUB = 2000   # elements around one vertex, whose records exceed a tile: the whole mesh takes the row gathers


def _with_hub(m, spokes=HUB):
    """`m` and, apart from it, a disc of elements: with HUB of them, m's rows as the gathers form them."""
    w = _wheel(spokes)
    return F.Mesh(np.concatenate([m.x, w.x]), np.concatenate([m.y, w.y]), np.concatenate([m.tag, 0 * w.tag]).astype(np.int32),
                  np.concatenate([m.tri, w.tri + m.n]).astype(np.int32), np.concatenate([m.gen, w.gen]))


class _Pair:
    """A mesh on the device alone (element tiles) and with the hub (row gathers), the same fields on both."""

    def __init__(self, m):
        import torch
        import cfa_b200 as cfa
        from oracle import oracle as O
        self.m, self.ctx, self.dms = m, cfa.default_context(), []
        for mesh in (m, _with_hub(m)):
            rp, ci = O.csr_build(mesh.n, mesh.elem_v)
            self.dms.append(cfa.DeviceMesh(self.ctx, mesh, torch.from_numpy(rp).to("cuda"), torch.from_numpy(ci).to("cuda")))
        self.n, self.nnz, self.ne = m.n, self.dms[0].nnz, m.ne

    def fields(self, k, *values):
        """The values (per vertex, or per element) as device arrays of mesh k, filled up for the hub."""
        import torch
        dm, out = self.dms[k], []
        for a in values:
            size = dm.ne if len(a) == self.ne else dm.n
            out.append(torch.from_numpy(np.concatenate([a, np.full(size - len(a), 0.7)])).to("cuda"))
        return out

    def same(self, call):
        """call(dm, k) -> output tensors, for both forms; their parts that belong to m are compared."""
        import torch
        outs = [call(dm, k) for k, dm in enumerate(self.dms)]
        for q, (a, b) in enumerate(zip(*outs)):
            blocks = 4 if a.numel() in (4 * self.n, 4 * self.nnz) else 1
            a, b = a.view(blocks, -1), b.view(blocks, -1)
            assert torch.isfinite(a).all()
            assert torch.equal(a, b[:, :a.shape[1]]), q


BIT_MESHES = {"one": _one, "tiny": lambda: F.make_mesh("tiny"), "small": lambda: F.make_mesh("small"),
              "small_shuffled": lambda: _shuffled(F.make_mesh("small")), "c0": lambda: F.make_mesh("c0"),
              "37k": lambda: _target(31_001, 5), "medium": lambda: F.make_mesh("medium")}


def _empty(k):
    import torch
    return torch.full((k,), float("nan"), dtype=torch.float64, device="cuda")


@pytest.mark.parametrize("with_nu", [False, True])
@pytest.mark.parametrize("name", list(BIT_MESHES))
def test_momentum_tiles_give_the_gathers_bits(name, with_nu):
    import cfa_b200 as cfa
    p = _Pair(BIT_MESHES[name]())
    f = [F.fourier_field(p.m.x, p.m.y, k) for k in range(1, 5)]
    for prm in (cfa.bdf2_params(), cfa.bdf2_params(bdf2=False, skew=0.3, rho=1.3)):
        for u_max in (None, 1.5):
            def call(dm, k):
                u, v, um, vm, pr, nu = p.fields(k, f[0], f[1], 0.9 * f[0], 1.1 * f[1], 0.3 * f[2], 1e-3 * (1 + 0.1 * f[3]))
                out = [_empty(dm.nnz), _empty(dm.n), _empty(dm.n), _empty(dm.n)]
                bc = {} if u_max is None else {"u": u.clone(), "v": v.clone(), "u_max": u_max}
                cfa.assemble_momentum(p.ctx, dm, u, v, um, vm, pr, prm, *out, nu_node=nu if with_nu else None, **bc)
                return out
            p.same(call)


@pytest.mark.parametrize("stab", [0.3, 0.0])
@pytest.mark.parametrize("name", list(BIT_MESHES))
def test_pressure_tiles_give_the_gathers_bits(name, stab):
    import cfa_b200 as cfa
    from oracle import oracle as O
    p = _Pair(BIT_MESHES[name]())
    m, dt = p.m, 2e-3 / 3
    f = [F.fourier_field(m.x, m.y, k) for k in range(1, 4)]
    s = O.oss_weights(m, f[0], f[1], dt, 1.0, 1e-3, 0.3)
    mass = np.zeros(m.n)
    np.add.at(mass, m.tri.ravel(), 1e-3 * (1.0 + np.arange(3 * m.ne) % 7))
    g = [0.1 * mass * F.fourier_field(m.x, m.y, k) for k in (5, 6)]

    def ppe(dm, k):
        u, v, pr, gx, gy, ms, es = p.fields(k, *f, *g, mass, s)
        out = [_empty(dm.nnz), _empty(dm.n), _empty(dm.n)]
        cfa.assemble_ppe(p.ctx, dm, u, v, pr, gx, gy, ms, es, dt, 1.3, stab, *out, apply_bc=False)
        return out

    def oss(dm, k):
        ms, es = p.fields(k, mass, s)
        out = [_empty(4 * dm.nnz), _empty(dm.n)]
        cfa.assemble_oss(p.ctx, dm, es, ms, *out)
        return out

    def system(dm, k):   # Dirichlet rows and columns in the same pass
        u, v, pr, gx, gy, ms, es, dp = p.fields(k, *f, *g, mass, s, f[2])
        out = [_empty(dm.nnz), _empty(dm.n), _empty(dm.n), dp, _empty(4 * dm.nnz), _empty(dm.n)]
        cfa.assemble_pressure_system(p.ctx, dm, u, v, pr, gx, gy, ms, es, dt, 1.3, stab, *out)
        return out if stab > 0.0 else out[:4]   # no OSS operator without stabilisation

    for call in (ppe, oss, system):
        p.same(call)


@pytest.mark.parametrize("weighted", [True, False])
@pytest.mark.parametrize("name", list(BIT_MESHES))
def test_gradient_tiles_give_the_gathers_bits(name, weighted):
    import cfa_b200 as cfa
    p = _Pair(BIT_MESHES[name]())
    m = p.m
    f = [F.fourier_field(m.x, m.y, k) for k in range(1, 4)]
    s = 0.5 + 0.4 * np.sin(np.arange(m.ne))

    def scalar(dm, k):
        q, es = p.fields(k, f[2], s)
        out = [_empty(dm.n), _empty(dm.n)]
        cfa.scalar_gradient(p.ctx, dm, q, es if weighted else None, *out)
        return out

    def node(dm, k):
        u, v, dp = p.fields(k, *f)
        out = [_empty(dm.n) for _ in range(3)]
        cfa.grad_dp_vorticity(p.ctx, dm, dp, u, v, *out)
        return out

    def stiffness(dm, k):
        out, dp = p.fields(k, f[0], f[2])
        cfa.stiffness_apply(p.ctx, dm, dp, -0.37, out)
        return [out]

    def recovered(dm, k):
        u, v, ms = p.fields(k, f[0], f[1], 1.0 + 0 * f[0])
        rec = _empty(4 * dm.n)
        cfa.amr_indicators(p.ctx, dm, u, v, 1.5, 1.0, ms, rec, _empty(2 * dm.ne))
        return [rec]

    for call in (scalar, node, stiffness, recovered):
        p.same(call)


# ----------------------------------------------------------------------------------------------
# which form a mesh takes
# ----------------------------------------------------------------------------------------------
def _renumbered(m, perm):
    new = np.empty_like(perm)
    new[perm] = np.arange(m.n)
    tri = new[m.tri]
    e = np.argsort(tri.min(1), kind="stable")
    return F.Mesh(m.x[perm].copy(), m.y[perm].copy(), m.tag[perm].copy(), tri[e].astype(np.int32), m.gen[e].copy())


def _sorted_by_x(m):
    return _renumbered(m, np.lexsort((m.y, m.x)))


def _appended(m, share=0.05):
    """A share of the vertices at the end, in random order."""
    q = np.random.default_rng(1).permutation(m.n)[:int(share * m.n)]
    return _renumbered(m, np.concatenate([np.setdiff1d(np.arange(m.n), q), q]))


KERNELS = {"mom": "k_momentum", "press": "k_pressure", "grad": "k_scalar_gradient", "node": "k_node_gradients",
           "rec": "k_recovered_gradient"}
# kernels on tiles (148 SMs): one wave of both forms; two waves of tiles against one of gathers; the same
# with the gathers' second wave begun; little sharing; none; none in a mesh of 64-row tiles; a hub
ROUTES = {
    "37k": (lambda: _target(31_001, 5), {"mom", "press", "grad", "node", "rec"}),
    "56k": (lambda: _target(45_001, 2), {"press", "grad", "node", "rec"}),
    "76k": (lambda: _target(60_001, 5), {"mom", "press", "node", "rec"}),
    "76k_appended": (lambda: _appended(_target(60_001, 5)), {"press", "node", "rec"}),
    "37k_sorted_by_x": (lambda: _sorted_by_x(_target(31_001, 5)), {"press"}),
    "37k_shuffled": (lambda: _shuffled(_target(31_001, 5)), set()),
    "c0_shuffled": (lambda: _shuffled(F.make_mesh("c0")), {"mom", "press", "grad", "node", "rec"}),
    "56k_hub": (lambda: _with_hub(_target(45_001, 2), 200), {"mom", "press", "grad", "node", "rec"}),
}


@pytest.mark.parametrize("name", list(ROUTES))
def test_route(name):
    import torch
    import cfa_b200 as cfa
    from oracle import oracle as O
    from torch.profiler import ProfilerActivity, profile
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the sizes are those of 148 SMs")
    make, tiles = ROUTES[name]
    m = make()
    ctx = cfa.default_context()
    rp, ci = O.csr_build(m.n, m.elem_v)
    dm = cfa.DeviceMesh(ctx, m, torch.from_numpy(rp).to("cuda"), torch.from_numpy(ci).to("cuda"))
    n, nnz = dm.n, dm.nnz
    z = lambda k: torch.ones(k, dtype=torch.float64, device="cuda")
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        cfa.assemble_momentum(ctx, dm, z(n), z(n), z(n), z(n), z(n), cfa.bdf2_params(), z(nnz), z(n), z(n), z(n))
        cfa.assemble_ppe(ctx, dm, z(n), z(n), z(n), z(n), z(n), z(n), z(m.ne), 1e-3, 1.0, 0.3, z(nnz), z(n), z(n),
                         apply_bc=False)
        cfa.scalar_gradient(ctx, dm, z(n), z(m.ne), z(n), z(n))
        cfa.grad_dp_vorticity(ctx, dm, z(n), z(n), z(n), z(n), z(n), z(n))
        cfa.amr_indicators(ctx, dm, z(n), z(n), 1.5, 1.0, z(n), z(4 * n), z(2 * m.ne))
        torch.cuda.synchronize()
    names = [e.name for e in p.events()]
    if not any("k_" in q for q in names):
        pytest.skip("kernels cannot be recorded here")
    took = {k for k, v in KERNELS.items() if any(v + "_tiles" in q for q in names)}
    assert took == tiles
    for k, v in KERNELS.items():
        assert any(v in q for q in names), k
