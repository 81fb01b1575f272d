"""Column blocks factored by one launch (single CTA up to 384 rows, clusters above) and the row moves and
triangular solve that follow: P A = L U at the edges of sub-blocks, blocks and CTAs.

Tolerance: the backward error of LU with partial pivoting is at most about n 2^-24 times the growth of the
entries (below 10 here); 1e-5 leaves a factor of ten at n = 1200, where rounding errors average out instead."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("needs a CUDA device", allow_module_level=True)

from hornlab_metal_bem_b200.native import HBEM_PREC_TF32X3, _stream_ptr, _t_ptr, check, load_library  # noqa: E402

HBEM_TUNE_LU_PANEL, HBEM_TUNE_LU_UPDATE, HBEM_TUNE_LU_PANEL_KERNEL = 1, 8, 10


def _factor(A, ld, panel=0, kernel=0):
    lib = load_library()
    F, n = A.shape[:2]
    planes = np.zeros((2, F, n, ld), np.float32)
    planes[0, :, :, :n], planes[1, :, :, :n] = A.real, A.imag
    re, im = torch.tensor(planes[0]).cuda(), torch.tensor(planes[1]).cuda()
    piv = torch.empty((F, n), dtype=torch.int32, device="cuda")
    info = torch.empty(F, dtype=torch.int32, device="cuda")
    check(lib.hbem_set_tuning(HBEM_TUNE_LU_UPDATE, 1), "hbem_set_tuning")   # exact FP32 products in the bulk
    try:
        check(lib.hbem_set_tuning(HBEM_TUNE_LU_PANEL, panel), "hbem_set_tuning")
        check(lib.hbem_set_tuning(HBEM_TUNE_LU_PANEL_KERNEL, kernel), "hbem_set_tuning")
        check(lib.hbem_lu_factor(n, F, _t_ptr(re), _t_ptr(im), ld, n * ld, _t_ptr(piv), n, _t_ptr(info), HBEM_PREC_TF32X3,
                                 _stream_ptr()), "hbem_lu_factor")
    finally:
        for knob in (HBEM_TUNE_LU_UPDATE, HBEM_TUNE_LU_PANEL, HBEM_TUNE_LU_PANEL_KERNEL):
            lib.hbem_set_tuning(knob, 0)
    check(lib.hbem_solve_status(_stream_ptr()), "hbem_solve_status")
    LU = (re.double() + 1j * im.double())[:, :, :n].cpu().numpy()
    return LU, piv.cpu().numpy(), info.cpu().numpy()


def _permuted(A, piv):
    P = A.copy()
    for j, p in enumerate(piv):
        P[[j, p]] = P[[p, j]]
    return P


@pytest.mark.parametrize("n,pad", [(1, 0), (15, 0), (16, 0), (17, 3), (48, 0), (63, 1), (64, 0), (65, 0), (80, 0),
                                   (130, 2), (384, 0), (385, 3), (449, 3), (769, 3), (1200, 0)])
def test_block_panel_factors(n, pad):
    rng = np.random.default_rng(n)
    A = (rng.standard_normal((2, n, n)) + 1j * rng.standard_normal((2, n, n))).astype(np.complex64)
    # columns whose pivots' squares leave the FP32 range, or lie at the ends of the unscaled reciprocal's
    for col, scale in zip([n // 2, n // 3, n - 1, 0], [1e-20, 1e16, 1e-16, 1e18]):
        A[1, :, col] *= np.float32(scale)
    LU, piv, info = _factor(A, n + pad)
    assert not info.any()
    for m in range(2):
        L, U = np.tril(LU[m], -1) + np.eye(n), np.triu(LU[m])
        assert np.abs(np.tril(LU[m], -1)).max(initial=0.0) <= np.sqrt(2.0) * (1 + 1e-5)
        # each column over its own norm, so that the scaled ones count as the others
        ref = _permuted(A[m].astype(np.complex128), piv[m])
        size = np.linalg.norm(ref, axis=0)
        assert np.linalg.norm((L @ U - ref) / size) <= 1e-5 * np.sqrt(n)


@pytest.mark.parametrize("n,col", [(40, 0), (200, 17), (500, 70)])
def test_zero_column_is_reported_and_ties_take_the_first_row(n, col):
    rng = np.random.default_rng(n)
    A = (rng.standard_normal((1, n, n)) + 1j * rng.standard_normal((1, n, n))).astype(np.complex64)
    Z = A.copy()
    Z[0, :, col] = 0.0
    assert _factor(Z, n)[2][0] == col + 1
    T = A.copy()
    T[0, :, 0] = 3.0   # every row ties in the first column: icamax keeps row 0
    assert _factor(T, n)[1][0, 0] == 0


def test_block_panel_is_bitwise_stable_under_concurrent_work():
    rng = np.random.default_rng(5)
    A = (rng.standard_normal((8, 1043, 1043)) + 1j * rng.standard_normal((8, 1043, 1043))).astype(np.complex64)
    quiet = _factor(A, 1044)
    side = torch.cuda.Stream()
    X = torch.randn(4096, 4096, device="cuda")
    for _ in range(2):
        with torch.cuda.stream(side):
            for _ in range(60):
                X @ X
        busy = _factor(A, 1044)
        assert all(np.array_equal(a, b) for a, b in zip(quiet, busy))
    torch.cuda.synchronize()


def test_register_sub_panels_stay_selectable_for_refined_factors():
    """HBEM_TUNE_LU_PANEL_KERNEL = 1 takes the register sub-panels, whose factors are the shared-memory ones' bits
    (HBEM_TUNE_LU_PANEL = 64), in place of the whole-block launch."""
    rng = np.random.default_rng(6)
    A = (rng.standard_normal((2, 300, 300)) + 1j * rng.standard_normal((2, 300, 300))).astype(np.complex64)
    registers, shared = _factor(A, 300, kernel=1), _factor(A, 300, panel=64)
    assert all(np.array_equal(a, b) for a, b in zip(registers, shared))


def test_multipliers_use_a_correctly_rounded_reciprocal():
    """Column 0: multipliers x * conj(d) (1 / |d|^2) with every operation rounded once to FP32 (longdouble holds the
    exact products and, but for a tie's last bit, the sums), bit for bit over 400 pivots."""
    rng = np.random.default_rng(8)
    A = (rng.standard_normal((400, 20, 20)) + 1j * rng.standard_normal((400, 20, 20))).astype(np.complex64)
    LU, piv, _ = _factor(A, 20)
    f32, wide = np.float32, np.longdouble
    fma = lambda a, b, c: (wide(a) * wide(b) + wide(c)).astype(f32)  # noqa: E731
    for m in range(400):
        x = _permuted(A[m], piv[m])[:, 0]
        xr, xi, dr, di = x.real[1:], x.imag[1:], x.real[:1], x.imag[:1]
        den = f32(1.0) / fma(dr, dr, di * di)
        ir, ii = dr * den, -di * den
        assert np.array_equal(LU[m, 1:, 0].real.astype(f32), fma(xr, ir, -(xi * ii)))
        assert np.array_equal(LU[m, 1:, 0].imag.astype(f32), fma(xr, ii, xi * ir))
