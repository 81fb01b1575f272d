"""Solves by one launch for both triangular phases (refinement and condition estimate) at the edges of its 32-row
blocks, against LAPACK.

Refined solutions: hbem_refine stops at a relative residual of 1e-7 and keeps x in FP32 (2^-24 of each entry); the
matrices' condition numbers stay below 30 (diagonally dominant), so 30 * 1e-7 + 6e-8 < 4e-6.  Condition estimates:
cgecon's own on the same matrix, 1 % apart as the estimator's vectors are rounded differently."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("needs a CUDA device", allow_module_level=True)

from scipy.linalg import lapack  # noqa: E402

from hornlab_metal_bem_b200.native import HBEM_PREC_TF32X3, _stream_ptr, _t_ptr, check, load_library  # noqa: E402


def _parts(z):
    return (torch.tensor(np.ascontiguousarray(z.real), dtype=torch.float32).cuda(),
            torch.tensor(np.ascontiguousarray(z.imag), dtype=torch.float32).cuda())


@pytest.mark.parametrize("n,batch", [(1, 2), (2, 1), (31, 3), (32, 1), (33, 2), (64, 1), (129, 5), (160, 1), (161, 2),
                                     (513, 3)])
def test_refined_solution_and_condition_estimate(n, batch):
    lib = load_library()
    rng = np.random.default_rng(n)
    A = (rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))).astype(np.complex64)
    A += (4.0 * np.sqrt(n)) * np.eye(n, dtype=np.complex64)[rng.permutation(n)]   # interchanges off the diagonal
    b = (rng.standard_normal((batch, n)) + 1j * rng.standard_normal((batch, n))).astype(np.complex64)
    A0r, A0i = _parts(A)
    Ar, Ai = A0r.clone(), A0i.clone()
    br, bi = _parts(b)
    xr, xi = torch.zeros_like(br), torch.zeros_like(bi)
    piv = torch.empty((batch, n), dtype=torch.int32, device="cuda")
    info = torch.empty(batch, dtype=torch.int32, device="cuda")
    anorm = torch.empty(batch, dtype=torch.float32, device="cuda")
    rcond = torch.empty(batch, dtype=torch.float64, device="cuda")
    st = _stream_ptr()
    check(lib.hbem_matrix_norm1(n, batch, _t_ptr(Ar), _t_ptr(Ai), n, n * n, _t_ptr(anorm), st), "hbem_matrix_norm1")
    check(lib.hbem_lu_factor(n, batch, _t_ptr(Ar), _t_ptr(Ai), n, n * n, _t_ptr(piv), n, _t_ptr(info), HBEM_PREC_TF32X3,
                             st), "hbem_lu_factor")
    check(lib.hbem_lu_rcond(n, batch, _t_ptr(Ar), _t_ptr(Ai), n, n * n, _t_ptr(anorm), _t_ptr(rcond), st),
          "hbem_lu_rcond")
    # from x = 0 the first pass solves for b itself
    check(lib.hbem_refine(n, batch, _t_ptr(A0r), _t_ptr(A0i), n, n * n, _t_ptr(Ar), _t_ptr(Ai), n * n, _t_ptr(piv), n,
                          _t_ptr(br), _t_ptr(bi), n, _t_ptr(xr), _t_ptr(xi), n, 1e-7, 6, None, None, st), "hbem_refine")
    assert not info.cpu().numpy().any()
    x = xr.double().cpu().numpy() + 1j * xi.double().cpu().numpy()
    for m in range(batch):
        ref = np.linalg.solve(A[m].astype(np.complex128), b[m].astype(np.complex128))
        assert np.linalg.norm(x[m] - ref) <= 4e-6 * np.linalg.norm(ref)
        lu, _, _ = lapack.cgetrf(A[m])
        want, _ = lapack.cgecon(lu, np.abs(A[m]).sum(0).max().astype(np.float32), norm="1")
        assert abs(float(rcond[m]) - want) <= 1e-2 * want


HBEM_TUNE_LU_SOLVE, HBEM_TUNE_WAVE_SPIN = 2, 7
HBEM_ERR_STATE = -4


@pytest.mark.parametrize("mode", [1, 2, 3])
def test_forced_solve_schemes_take_the_condition_estimate(mode):
    """HBEM_TUNE_LU_SOLVE: every solve of the estimate is the forced scheme's (a copy and at least one launch of its
    own, 13 times), not the built-in one; the same 1 % to cgecon."""
    lib = load_library()
    n, batch = 161, 2
    rng = np.random.default_rng(3)
    A = (rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))).astype(np.complex64)
    Ar, Ai = _parts(A)
    piv = torch.empty((batch, n), dtype=torch.int32, device="cuda")
    info = torch.empty(batch, dtype=torch.int32, device="cuda")
    anorm = torch.tensor(np.abs(A).sum(1).max(1), device="cuda")
    rcond = torch.empty(batch, dtype=torch.float64, device="cuda")
    st = _stream_ptr()
    check(lib.hbem_lu_factor(n, batch, _t_ptr(Ar), _t_ptr(Ai), n, n * n, _t_ptr(piv), n, _t_ptr(info), HBEM_PREC_TF32X3,
                             st), "hbem_lu_factor")
    launches = {}
    try:
        for m in (0, mode):
            check(lib.hbem_set_tuning(HBEM_TUNE_LU_SOLVE, m), "hbem_set_tuning")
            before = int(lib.hbem_launch_count())
            check(lib.hbem_lu_rcond(n, batch, _t_ptr(Ar), _t_ptr(Ai), n, n * n, _t_ptr(anorm), _t_ptr(rcond), st),
                  "hbem_lu_rcond")
            launches[m] = int(lib.hbem_launch_count()) - before
            for i in range(batch):
                lu, _, _ = lapack.cgetrf(A[i])
                want, _ = lapack.cgecon(lu, np.abs(A[i]).sum(0).max().astype(np.float32), norm="1")
                assert abs(float(rcond[i]) - want) <= 1e-2 * want
    finally:
        lib.hbem_set_tuning(HBEM_TUNE_LU_SOLVE, 0)
    assert launches[mode] >= launches[0] + 13


def test_wait_that_runs_out_is_reported_and_leaves_the_context_usable():
    """The built-in refinement and condition estimate with their waits bounded to one poll
    (HBEM_TUNE_WAVE_SPIN = 1): both give up, say so once, and are right again with the built-in bound."""
    lib = load_library()
    n = 2048
    rng = np.random.default_rng(9)
    A = (rng.standard_normal((1, n, n)) + 1j * rng.standard_normal((1, n, n))).astype(np.complex64)
    A += (4.0 * np.sqrt(n)) * np.eye(n, dtype=np.complex64)
    b = (rng.standard_normal((1, n)) + 1j * rng.standard_normal((1, n))).astype(np.complex64)
    A0r, A0i = _parts(A)
    Ar, Ai = A0r.clone(), A0i.clone()
    br, bi = _parts(b)
    piv = torch.empty((1, n), dtype=torch.int32, device="cuda")
    info = torch.empty(1, dtype=torch.int32, device="cuda")
    norm = np.abs(A[0]).sum(0).max().astype(np.float32)
    anorm = torch.tensor([norm], device="cuda")
    rcond = torch.empty(1, dtype=torch.float64, device="cuda")
    st = _stream_ptr()
    check(lib.hbem_lu_factor(n, 1, _t_ptr(Ar), _t_ptr(Ai), n, n * n, _t_ptr(piv), n, _t_ptr(info), HBEM_PREC_TF32X3,
                             st), "hbem_lu_factor")

    def estimate():
        check(lib.hbem_lu_rcond(n, 1, _t_ptr(Ar), _t_ptr(Ai), n, n * n, _t_ptr(anorm), _t_ptr(rcond), st),
              "hbem_lu_rcond")
        return lib.hbem_solve_status(st)

    def refine():
        xr, xi = torch.zeros_like(br), torch.zeros_like(bi)
        rc = lib.hbem_refine(n, 1, _t_ptr(A0r), _t_ptr(A0i), n, n * n, _t_ptr(Ar), _t_ptr(Ai), n * n, _t_ptr(piv), n,
                             _t_ptr(br), _t_ptr(bi), n, _t_ptr(xr), _t_ptr(xi), n, 1e-7, 6, None, None, st)
        return rc, xr.double().cpu().numpy() + 1j * xi.double().cpu().numpy()

    try:
        check(lib.hbem_set_tuning(HBEM_TUNE_WAVE_SPIN, 1), "hbem_set_tuning")
        assert estimate() == HBEM_ERR_STATE
        assert refine()[0] == HBEM_ERR_STATE
        assert lib.hbem_solve_status(st) == 0   # reported once
    finally:
        lib.hbem_set_tuning(HBEM_TUNE_WAVE_SPIN, 0)
    assert estimate() == 0
    want, _ = lapack.cgecon(lapack.cgetrf(A[0])[0], norm, norm="1")
    assert abs(float(rcond[0]) - want) <= 1e-2 * want
    rc, x = refine()
    ref = np.linalg.solve(A[0].astype(np.complex128), b[0].astype(np.complex128))
    assert rc == 0 and np.linalg.norm(x[0] - ref) <= 4e-6 * np.linalg.norm(ref)
