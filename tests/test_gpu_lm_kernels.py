"""The one-call LM update and the Cholesky chain at the edges of their tiles.

Tolerances: the update from split-BF16 Gram matrices against FP64, 1e-3 of its norm (the Gram
entries carry ~2^-16 relative error, the damped systems here have condition numbers below 1e2);
Cholesky residual |H x - b| / |b| at most 64 n eps with well-conditioned H: 64 * 16500 * 1.1e-16 < 1e-9."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _v(t):
    return None if t is None else C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("nv,nm", [(1, 1), (1, 5), (7, 3), (63, 127), (64, 128), (65, 129), (129, 65), (200, 2048),
                                   (130, 2049), (500, 31)])
@pytest.mark.parametrize("weighted", [False, True])
def test_lm_update_both_forms(nv, nm, weighted):
    """Odd and aligned rows, both operand layouts (form 1: unknowns, 2: measurements), zero weights."""
    import torch
    from dogpup_b200._lib import lib, check
    rng = np.random.default_rng(nv * 7 + nm)
    J = torch.as_tensor(rng.standard_normal((nv, nm)), dtype=torch.float32, device="cuda")
    y = torch.as_tensor(rng.standard_normal(nm), device="cuda")
    W = rng.uniform(0.5, 2.0, nm)
    W[nm // 3] = 0.0 if nm > 3 else 1.0
    Wd = torch.as_tensor(W, device="cuda") if weighted else None
    Jd, w = J.double(), (Wd if weighted else torch.ones(nm, dtype=torch.float64, device="cuda"))
    H = (Jd * w) @ Jd.T
    H.diagonal().add_(0.3 * H.diagonal().max())
    x0 = torch.linalg.solve(H, (Jd * w) @ y)
    for form in (1, 2):
        x = torch.full((nv,), float("nan"), dtype=torch.float64, device="cuda")
        check(lib.dgp_lm_update(_v(J), nv, nm, _v(Wd), _v(y), 0.3, _v(x), form, None, None))
        assert float((x - x0).norm() / x0.norm()) < 1e-3, form


@pytest.mark.parametrize("n", [16500])
def test_cholesky_wide_panels(n):
    """From 16,384 rows on the outer panels are 1536 columns wide (1024 below, 3333 in the other tests)."""
    import torch
    from dogpup_b200._lib import lib, check
    g = torch.Generator(device="cuda").manual_seed(1)
    B = torch.randn((n, 2 * n), generator=g, device="cuda")
    H0 = (B @ B.T).double() / n
    H0.diagonal().add_(1.0)
    del B
    b = torch.randn(n, generator=g, dtype=torch.float64, device="cuda")
    H, x = H0.clone(), b.clone()
    check(lib.dgp_cholesky_solve(_v(H), n, n, _v(x), None))
    S = torch.tril(H0) + torch.tril(H0, -1).T
    assert float((S @ x - b).norm() / b.norm()) < 1e-9


def test_lm_update_from_several_host_threads():
    """Calls on their own streams share the library's scratch memory and Cholesky streams: each gives what
    it gives alone, bit for bit (no atomics in its sums)."""
    import threading
    import torch
    from dogpup_b200._lib import lib
    sizes = [(300, 700), (900, 400), (513, 2100), (1700, 1600)]
    g = torch.Generator(device="cuda").manual_seed(5)
    data = [(torch.randn((nv, nm), generator=g, device="cuda"),
             torch.randn(nm, generator=g, dtype=torch.float64, device="cuda")) for nv, nm in sizes]

    def call(i, x, stream):
        J, y = data[i]
        return lib.dgp_lm_update(_v(J), J.shape[0], J.shape[1], None, _v(y), 0.2, _v(x), 0, None, stream)

    alone = [torch.empty(nv, dtype=torch.float64, device="cuda") for nv, _ in sizes]
    for i, x in enumerate(alone):
        assert call(i, x, None) == 0
    torch.cuda.synchronize()
    out = [[torch.empty_like(x) for _ in range(4)] for x in alone]
    rcs = []

    def work(i):
        s = torch.cuda.Stream()
        for x in out[i]:
            rcs.append(call(i, x, s.cuda_stream))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert rcs == [0] * 16
    for a, xs in zip(alone, out):
        assert all(torch.equal(a, x) for x in xs)
