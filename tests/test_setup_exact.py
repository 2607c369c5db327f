"""The AMG setup's sparse products (hash tables per warp), aggregation and power iteration against
the oracle, bit for bit, on matrices whose rows meet every table size: few products, more than the
first and the second table's, and a row with more columns than the largest table holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(rows):
    """Sorted CSR arrays of a list of {column: value} rows."""
    rp = np.zeros(len(rows) + 1, np.int32)
    rp[1:] = np.cumsum([len(r) for r in rows])
    ci = np.concatenate([np.fromiter(sorted(r), np.int32, len(r)) for r in rows])
    v = np.concatenate([np.array([r[c] for c in sorted(r)]) for r in rows])
    return rp, ci, v


def _graph(n, degree, seed, weight=lambda rng: rng.uniform(0.5, 1.5)):
    """A weighted Laplacian plus identity of a random graph with neighbours close in index."""
    rng = np.random.default_rng(seed)
    rows = [dict() for _ in range(n)]
    for i in range(n):
        for j in (i + 1 + rng.choice(4 * degree, size=degree // 2, replace=False)):
            if j < n:
                w = weight(rng)
                rows[i][int(j)] = rows[int(j)][i] = -w
    for i in range(n):
        rows[i][i] = 1e-3 - sum(rows[i].values())
    return rows


def _arrow(n, seed):
    """A chain graph and one row weakly coupled to every other: its products fill no table."""
    rows = _graph(n, 4, seed)
    for j in range(1, n):
        w = 1e-4 if j not in rows[0] else -rows[0][j]
        rows[0][j] = rows[j][0] = -w
    for i in range(n):
        rows[i][i] = 0.0
        rows[i][i] = 1e-3 - sum(rows[i].values())
    return rows


CASES = {
    "first_table": (lambda: _graph(2000, 6, 1), "1", 300),
    "second_table": (lambda: _graph(3000, 16, 2), "1", 300),
    # many weak couplings beside a few strong ones, so that the graph still coarsens
    "largest_table": (lambda: _graph(3000, 60, 3, lambda rng: 1.0 if rng.random() < 0.1 else 0.01), "1", 300),
    # 1.9k columns in a row, too long for the V-cycle's tiles; its dense next level is the coarsest
    "beyond_the_tables": (lambda: _arrow(10_500, 4), "0", 2200),
}


@pytest.mark.parametrize("name", list(CASES))
def test_hierarchy_bits(name, monkeypatch):
    import torch
    import cfa_b200 as cfa
    from oracle import oracle as O
    make, tiles, coarse_target = CASES[name]
    monkeypatch.setenv("CFA_TILES", tiles)
    rp, ci, v = _csr(make())
    n = len(rp) - 1
    want = O.Amg(rp, ci, v, coarse_target=coarse_target)
    t = lambda a: torch.from_numpy(a).to("cuda")
    d = (t(rp), t(ci), t(v))
    amg = cfa.AmgPreconditioner(cfa.default_context(), coarse_target=coarse_target)
    for _ in range(2):     # the second setup on the first one's workspaces
        amg.setup(n, len(ci), *d)
        assert amg.num_levels() - 1 == want.nlev and want.nlev >= 1
        for lv in range(want.nlev):
            got, ref = amg.level(lv), want.level(lv)
            assert got["omega"] == ref["omega"]
            for k in ("A", "P", "R"):
                _, _, orp, oci, ov = ref[k]
                assert np.array_equal(got[k][0].cpu().numpy(), orp), (lv, k)
                assert np.array_equal(got[k][1].cpu().numpy(), oci), (lv, k)
                assert np.array_equal(got[k][2].cpu().numpy(), ov), (lv, k)


def test_aggregation_wait_runs_out(monkeypatch):
    """A path graph in its natural order decides node after node. With no time allowed the waiting threads
    give up, the setup reports it, and the same handle sets the same matrix up afterwards."""
    import torch
    import cfa_b200 as cfa
    from oracle import oracle as O
    n = 20_000
    rows = [{j: -1.0 for j in (i - 1, i + 1) if 0 <= j < n} | {i: 2.001} for i in range(n)]
    rp, ci, v = _csr(rows)
    t = lambda a: torch.from_numpy(a).to("cuda")
    d = (t(rp), t(ci), t(v))
    amg = cfa.AmgPreconditioner(cfa.default_context())
    amg.set_aggregation(1)
    monkeypatch.setenv("CFA_AGG_WAIT_MS", "0")
    with pytest.raises(cfa.CfaError) as e:
        amg.setup(n, len(ci), *d)
    assert e.value.status == cfa.CFA_TIMEOUT
    monkeypatch.delenv("CFA_AGG_WAIT_MS")
    amg.setup(n, len(ci), *d)
    want = O.Amg(rp, ci, v).level(0)
    assert np.array_equal(amg.level(0)["agg"].cpu().numpy(), want["agg"])
