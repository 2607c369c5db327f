"""Level 0's sweeps in pairs over ring tiles against the one-sweep kernels: the same bits of the
V-cycle (every row sums in the same order), over tile heights, partial last tiles and orderings
whose rings do not fit."""
import numpy as np
import pytest

import fixtures as F

pytestmark = pytest.mark.gpu


def _shuffled(m, seed=1):
    perm = np.random.default_rng(seed).permutation(m.n)
    new = np.empty_like(perm)
    new[perm] = np.arange(m.n)
    return F.Mesh(m.x[perm].copy(), m.y[perm].copy(), m.tag[perm].copy(), new[m.tri].astype(np.int32), m.gen.copy())


def _target(n, seed=2):
    import batch as B
    return B.batch_system(seed, n, n).mesh


MESHES = {
    "small": lambda: F.make_mesh("small"),
    "small_shuffled": lambda: _shuffled(F.make_mesh("small")),
    "c0": lambda: F.make_mesh("c0"),
    "60k": lambda: _target(60_001),
    "160k": lambda: _target(160_001),
}


@pytest.mark.parametrize("name", list(MESHES))
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_vcycle_bits(name, precision, monkeypatch):
    import torch
    import cfa_b200 as cfa
    m = MESHES[name]()
    ctx = cfa.default_context()
    dm = cfa.DeviceMesh(ctx, m)
    n, nnz = dm.n, dm.nnz
    z = lambda k: torch.zeros(k, dtype=torch.float64, device="cuda")
    K, rhs, div, dp = z(nnz), z(n), z(n), z(n)
    t = lambda a: torch.from_numpy(a).to("cuda")
    u, v, p, g, mass, es = t(F.fourier_field(m.x, m.y, 1)), t(F.fourier_field(m.x, m.y, 2)), z(n), z(n), z(n), z(m.ne)
    cfa.assemble_ppe(ctx, dm, u, v, p, g, g, mass, es, 1e-3, 1.0, 0.0, K, rhs, div, dp)
    got = []
    for fused in ("0", "1"):     # 1: the hierarchy is set up without ring tiles
        monkeypatch.setenv("CFA_CG_FUSE_UPDATE", fused)
        amg = cfa.AmgPreconditioner(ctx, cfa.MIXED if precision == "mixed" else cfa.FP64)
        amg.setup(n, nnz, dm.rp, dm.ci, K)
        out = z(n)
        amg.apply(rhs, out)
        amg.apply(out.clone(), out)
        torch.cuda.synchronize()
        assert torch.isfinite(out).all() and float(out.abs().max()) > 0.0
        got.append(out)
    assert torch.equal(got[0], got[1])
