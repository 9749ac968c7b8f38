"""The FP64 BiCGSTAB on fused sweeps at the edges of its layouts.

Tolerances: fluence within 1e-9 of the sparse-direct solution at tol = 1e-12 (condition numbers below
1e4; the bar of the FP64 solver's other tests); repeated solves bit for bit (every sum is ordered)."""
import numpy as np
import pytest

from test_gpu_fused_solver import DFC, _check, case  # noqa: F401

pytestmark = pytest.mark.gpu


def _solve(case, ns, harm, loop=True, seed=3, **kw):  # noqa: F811
    import torch
    from dogpup_b200 import api
    m = case["m"]
    rng = np.random.default_rng(seed)
    nodes = m.elem[rng.choice(m.ne, ns, replace=False)].astype(np.int32)
    w = rng.random((ns, 4))
    S = api.Solver(case["fem"].rowptr, case["fem"].col, case["Kd"], case["Md"], DFC, len(harm), ns, harmonics=harm)
    S.set_device_loop(loop)
    status = torch.full((len(harm) * ns,), -1, dtype=torch.int32, device="cuda")
    X, rep = S.solve_sources(torch.as_tensor(nodes, device="cuda"), torch.as_tensor(w, device="cuda"),
                             torch.ones(len(harm), dtype=torch.complex128, device="cuda"),
                             api.make_opts(precision="fp64", tol=1e-12, **kw), status=status)
    return nodes, w, X.cpu().numpy(), rep, status.cpu().numpy()


@pytest.mark.parametrize("ns", [1, 4, 5, 8, 9, 11, 16, 33, 47, 128])
def test_source_counts(case, ns):  # noqa: F811
    """Rows of 2 to 32 lanes with idle lanes and padded columns; few columns (one block takes every
    harmonic's scalars) and many (one per harmonic)."""
    harm = [0, 4, 19, 2, 40]
    nodes, w, X, rep, st = _solve(case, ns, harm)
    assert (st == 0).all() and rep.max_rel_residual < 1e-11
    _check(case, nodes, w, X, harm, np.ones(len(harm)), range(len(harm)))


@pytest.mark.parametrize("ns,nf", [(3, 4), (64, 40), (20, 128)])
def test_same_bits_every_time(case, ns, nf):  # noqa: F811
    """Many chunks per block and harmonics that leave the sweeps early; host-polled and device-driven."""
    runs = [_solve(case, ns, list(range(nf)), loop=loop, check_every=3) for loop in (True, True, False)]
    assert len({r[3].iterations for r in runs}) == 1 and all((r[4] == 0).all() for r in runs)
    assert np.array_equal(runs[0][2], runs[1][2]) and np.array_equal(runs[0][2], runs[2][2])
    nodes, w, X, _, _ = runs[0]
    _check(case, nodes, w, X, list(range(nf)), np.ones(nf), [0, nf // 2, nf - 1])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_node_ids_behind_a_header(case, precision):  # noqa: F811
    """Node ids at a 4-byte offset in their buffer: int32 data needs no wider alignment."""
    import torch
    from dogpup_b200 import api
    m, ns, harm = case["m"], 6, [0, 5]
    rng = np.random.default_rng(2)
    nodes = m.elem[rng.choice(m.ne, ns, replace=False)].astype(np.int32)
    w = rng.random((ns, 4))
    S = api.Solver(case["fem"].rowptr, case["fem"].col, case["Kd"], case["Md"], DFC, 2, ns, harmonics=harm)
    for skip in (1, 2, 3):
        buf = torch.zeros(skip + 4 * ns, dtype=torch.int32, device="cuda")
        ids = buf[skip:].view(ns, 4)
        ids.copy_(torch.as_tensor(nodes))
        X, rep = S.solve_sources(ids, torch.as_tensor(w, device="cuda"),
                                 torch.ones(2, dtype=torch.complex128, device="cuda"),
                                 api.make_opts(precision=precision, tol=1e-12 if precision == "fp64" else 1e-11))
        assert rep.n_not_converged == 0
        _check(case, nodes, w, X.cpu().numpy(), harm, np.ones(2), range(2))


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-11)])
@pytest.mark.parametrize("ns,nf", [(1, 1), (1, 40), (2, 1), (2, 21)])
def test_one_or_two_sources(case, precision, tol, ns, nf):  # noqa: F811
    """Two columns per harmonic: a row's records in halves on two lanes; several levels and one."""
    import torch
    from dogpup_b200 import api
    m, harm = case["m"], list(range(nf))
    nodes = m.elem[[11, 500][:ns]].astype(np.int32)
    w = np.random.default_rng(6).random((ns, 4))
    S = api.Solver(case["fem"].rowptr, case["fem"].col, case["Kd"], case["Md"], DFC, nf, ns)
    X, rep = S.solve_sources(torch.as_tensor(nodes, device="cuda"), torch.as_tensor(w, device="cuda"),
                             torch.ones(nf, dtype=torch.complex128, device="cuda"),
                             api.make_opts(precision=precision, tol=tol))
    assert rep.n_not_converged == 0 and rep.max_rel_residual < 1e-10
    _check(case, nodes, w, X.cpu().numpy(), harm, np.ones(nf), [0, nf // 2, nf - 1])
