"""The TF32x3 trailing update at the edges of its 64 x 64 complex tiles and of the factorisation."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from hornlab_metal_bem_b200.native import (  # noqa: E402
    HBEM_PREC_TF32X3, HBEM_TRANS_N, _stream_ptr, _t_ptr, check, load_library, matrix_ld,
)

SIZES = [129, 191, 193, 256, 257, 321, 449, 1025]


@pytest.mark.parametrize("n,batch", [(n, 3) for n in SIZES] + [(385, 40)])
def test_factors_solve_to_the_split_product_error(n, batch):
    """Backward error within n 2^-22: both operands keep 22 significant bits, and a system of
    independent normal entries has no element growth beyond sqrt(n)."""
    lib = load_library()
    rng = np.random.default_rng(n)
    ld = matrix_ld(n)
    A = (rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))).astype(np.complex64)
    b = (rng.standard_normal((batch, n)) + 1j * rng.standard_normal((batch, n))).astype(np.complex64)
    planes = torch.zeros((2, batch, n, ld), device="cuda")
    planes[0, :, :, :n] = torch.from_numpy(A.real.copy()).cuda()
    planes[1, :, :, :n] = torch.from_numpy(A.imag.copy()).cuda()
    br, bi = torch.from_numpy(b.real.copy()).cuda(), torch.from_numpy(b.imag.copy()).cuda()
    piv = torch.zeros((batch, n), dtype=torch.int32, device="cuda")
    info = torch.ones(batch, dtype=torch.int32, device="cuda")
    check(lib.hbem_lu_factor(n, batch, _t_ptr(planes[0]), _t_ptr(planes[1]), ld, n * ld, _t_ptr(piv), n, _t_ptr(info),
                             HBEM_PREC_TF32X3, _stream_ptr()), "hbem_lu_factor", lib)
    check(lib.hbem_lu_solve(n, 1, batch, _t_ptr(planes[0]), _t_ptr(planes[1]), ld, n * ld, _t_ptr(piv), n, _t_ptr(br),
                            _t_ptr(bi), 1, n, HBEM_TRANS_N, _stream_ptr()), "hbem_lu_solve", lib)
    torch.cuda.synchronize()
    assert int(info.abs().sum()) == 0
    x = br.cpu().numpy().astype(np.complex128) + 1j * bi.cpu().numpy()
    for m in range(batch):
        r = b[m] - A[m].astype(np.complex128) @ x[m]
        scale = np.linalg.norm(A[m].astype(np.complex128), 2) * np.linalg.norm(x[m])
        assert np.linalg.norm(r) <= n * 2.0**-22 * scale
