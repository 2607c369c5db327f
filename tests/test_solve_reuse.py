"""The Krylov loops' graphs and tile plans serve several handles and arrays on one context: every
solve gives the bits of the same solve on a context of its own."""
import numpy as np
import pytest

import fixtures as F

pytestmark = pytest.mark.gpu


def _step(cfa, S, ctx, m, seed, precision):
    f = lambda k: F.fourier_field(m.x, m.y, 10 * seed + k)
    st = S.SolveStep(m, f(1), f(2), 0.3 * f(3), precision=precision, ctx=ctx)
    st.amg_setup()
    return st


def _bits(st):
    import torch
    st.run()
    torch.cuda.synchronize()
    assert all(st.report()["conv"])
    return [t.cpu().numpy().copy() for t in (st.u, st.v, st.dp)]


def _renumbered(m, seed=3):
    """The same mesh with its vertices in another order: n and nnz stay, the pattern changes."""
    perm = np.random.default_rng(seed).permutation(m.n)
    new = np.empty_like(perm)
    new[perm] = np.arange(m.n)
    return F.Mesh(m.x[perm].copy(), m.y[perm].copy(), m.tag[perm].copy(), new[m.tri].astype(np.int32), m.gen.copy())


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_alternating_states_and_patterns_give_the_bits_of_their_own_context(precision):
    import cfa_b200 as cfa
    import step as S
    prec = cfa.MIXED if precision == "mixed" else cfa.FP64
    m = F.make_mesh("small")
    # two patterns of equal size, more handles than the context keeps loops for
    systems = [(m, 1), (_renumbered(m), 2), (m, 3), (m, 4), (_renumbered(m), 5), (m, 6)]
    own = []
    for mesh, seed in systems:
        ctx = cfa.Context()
        own.append(_bits(_step(cfa, S, ctx, mesh, seed, prec)))
        ctx.sync()
    ctx = cfa.Context()
    states = [_step(cfa, S, ctx, mesh, seed, prec) for mesh, seed in systems]
    for order in (range(6), (0, 1, 0, 2, 1, 5, 3, 4, 0)):
        for k in order:
            for got, want in zip(_bits(states[k]), own[k]):
                assert np.array_equal(got, want)


def test_tolerance_and_arrays_change_between_solves():
    import cfa_b200 as cfa
    import step as S
    import torch
    ctx = cfa.Context()
    st = _step(cfa, S, ctx, F.make_mesh("small"), 1, cfa.MIXED)
    st.run()
    want = st.dp.clone()
    for tol in (1e-3, 1e-10, 1e-6, 1e-10):
        b, x = st.rhs_p.clone(), torch.zeros_like(st.dp)     # new arrays each time
        st.solver.solve_pcg(st.n, st.dm.rp, st.dm.ci, st.Kp, b, x, 4000, tol, st.oss, st.amg)
        assert st.solver.converged and st.solver.last_rel_residual < tol
        if tol == 1e-10:
            assert torch.equal(x, want)
        else:
            assert not torch.equal(x, want)
    zero = torch.zeros_like(st.dp)
    x = torch.ones_like(st.dp)
    st.solver.solve_pcg(st.n, st.dm.rp, st.dm.ci, st.Kp, zero, x, 4000, 1e-10, st.oss, st.amg)
    assert st.solver.converged and float(x.abs().max()) == 0.0
