"""Solves on matrices whose rows are longer than a tetrahedral lattice's 15 entries: the solver takes any
CSR pattern with a diagonal (quadratic elements, a refined node, matrices assembled elsewhere).

Tolerances: the matrices are diagonally dominant with condition numbers below 1e4, so at a relative
residual below 1e-11 (mixed) or a recursive one below 1e-12 (FP64) the solutions are within 1e-7 of the
sparse-direct ones; held here to the 1e-6 bar of the mixed solves and 1e-8."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as sla

pytestmark = pytest.mark.gpu

HARM = [0, 2, 9]


def _matrix(kind):
    rng = np.random.default_rng(17)
    n = 1400
    band = 7 if kind == "hubs" else 15
    rows = np.repeat(np.arange(n), band)
    cols = rows + np.tile(np.arange(1, band + 1), n)
    keep = cols < n
    rows, cols = rows[keep], cols[keep]
    if kind == "hubs":  # rows of 90 to 400 entries among rows of 15; in G^T too (low numbers)
        for hub, deg in ((3, 400), (40, 150), (41, 90), (700, 120), (n - 2, 80)):
            o = np.setdiff1d(rng.choice(n, deg, replace=False), np.arange(hub - band, hub + band + 1))
            rows, cols = np.append(rows, np.minimum(o, hub)), np.append(cols, np.maximum(o, hub))
    W = sp.coo_matrix((rng.uniform(0.2, 1.0, rows.size), (rows, cols)), shape=(n, n)).tocsr()
    W.data = np.minimum(W.data, 1.0)
    W = W + W.T
    d = np.asarray(W.sum(1)).ravel()
    K = (sp.diags(d + 0.2) - W).tocsr()
    M = (0.1 * (sp.diags(d + 1.0) + 0.5 * W)).tocsr()
    K.sort_indices()
    M.sort_indices()
    assert np.array_equal(K.indices, M.indices)
    return K, M


@pytest.fixture(scope="module", params=["band30", "hubs"])
def matrix(request):
    import torch
    K, M = _matrix(request.param)
    dev = lambda a: torch.as_tensor(a, device="cuda")  # noqa: E731
    args = (dev(K.indptr.astype(np.int32)), dev(K.indices.astype(np.int32)), dev(K.data), dev(M.data))
    lu = [sla.splu((K + 0.3j * h * M).tocsc()) for h in HARM]
    return K, args, lu


@pytest.mark.parametrize("precision,tol,bar", [("mixed", 1e-11, 1e-6), ("fp64", 1e-12, 1e-8)])
@pytest.mark.parametrize("ns", [1, 2, 4, 8, 11, 16, 32, 128])
def test_solution(matrix, ns, precision, tol, bar):
    import torch
    from dogpup_b200 import api
    K, args, lu = matrix
    n = K.shape[0]
    rng = np.random.default_rng(ns)
    nodes = np.stack([rng.choice(n, 4, replace=False) for _ in range(ns)]).astype(np.int32)
    nodes[0] = [3, 40, 700, n - 1]
    w = rng.uniform(0.1, 1.0, (ns, 4))
    fpsf = np.exp(0.2j * np.arange(len(HARM)))
    S = api.Solver(*args, 0.3, len(HARM), ns, harmonics=HARM)
    opts = api.make_opts(precision=precision, tol=tol)
    X, rep = S.solve_sources(torch.as_tensor(nodes, device="cuda"), torch.as_tensor(w, device="cuda"),
                             torch.as_tensor(fpsf, device="cuda"), opts)
    B = np.zeros((n, ns))
    for s in range(ns):
        B[nodes[s], s] = w[s]
    Bd = torch.as_tensor(B * fpsf[:, None, None], device="cuda")
    Y, rep2 = S.solve(Bd, opts)
    for r in (rep, rep2):
        assert r.n_not_converged == 0 and r.max_rel_residual < 1e-10
    for k in range(len(HARM)):
        x = lu[k].solve(B.astype(complex)) * fpsf[k]
        for got in (X, Y):
            err = np.linalg.norm(got[k].cpu().numpy() - x, axis=0) / np.linalg.norm(x, axis=0)
            assert err.max() <= bar, (k, err.max())
