"""Assembly gradients: one frequency against FP64 central differences of the oracle's matrix and right-hand side, and
more frequencies than one launch stages, and an odd count, against one frequency a call.

Tolerance 2e-5 relative: a launch's FP32 sums over the frequencies are rounded per term (2^-24), and the touching
pairs' lane sums cancel by up to two orders of magnitude (2^-24 * 100 = 6e-6) in either grouping."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("needs a CUDA device", allow_module_level=True)

from oracle.oracle import Oracle  # noqa: E402

from hornlab_metal_bem_b200 import generators as G  # noqa: E402
from hornlab_metal_bem_b200.geometry import build_geometry_buffers  # noqa: E402
from hornlab_metal_bem_b200.mesh import make_pure_function_spaces  # noqa: E402
from hornlab_metal_bem_b200.native import NativeSession, _np_ptr, _stream_ptr, _t_ptr, check  # noqa: E402


@pytest.mark.parametrize("freqs", [2, 3, 21])
@pytest.mark.parametrize("level", [0, 1])
def test_assembly_gradient_sums_over_frequencies(freqs, level):
    mesh = G.icosphere(level, 0.1)   # 20 triangles: less than a tile; 80: ragged
    p1, dp0 = make_pure_function_spaces(mesh.grid)
    b = build_geometry_buffers(mesh.grid, mesh.physical_tags, p1, dp0)
    n, T, V = b.p1_dof_count, b.n_triangles, np.asarray(b.vertices_3xn_f32).shape[1]
    rng = np.random.default_rng(freqs)
    k = np.linspace(5.0, 60.0, freqs).astype(np.float32)
    dev = torch.device("cuda")
    lam, p = (torch.tensor(rng.standard_normal((2, freqs, n)), dtype=torch.float32, device=dev) for _ in range(2))
    q = torch.tensor(rng.standard_normal((2, freqs, T)), dtype=torch.float32, device=dev)
    q[:, :, T // 2:] = 0.0
    with NativeSession(b, check_open_edges=False) as s:
        def grad(f0, f1):
            out = torch.zeros((3, V), dtype=torch.float64, device=dev)
            cut = [x[f0:f1].contiguous() for z in (lam, p, q) for x in z]
            kk = np.ascontiguousarray(k[f0:f1])
            check(s.lib.hbem_assemble_backward(
                s.handle, f1 - f0, _np_ptr(kk), None, _t_ptr(cut[0]), _t_ptr(cut[1]), n, _t_ptr(cut[2]), _t_ptr(cut[3]),
                n, _t_ptr(cut[4]), _t_ptr(cut[5]), T, _t_ptr(out), _stream_ptr()), "hbem_assemble_backward")
            torch.cuda.synchronize()
            return out.cpu().numpy()

        whole = grad(0, freqs)
        single = sum(grad(f, f + 1) for f in range(freqs))
    assert np.linalg.norm(whole - single) <= 2e-5 * np.linalg.norm(single)


@pytest.mark.parametrize("k", [5.0, 60.0])
@pytest.mark.parametrize("level", [0, 1])
def test_assembly_gradient_matches_central_differences(level, k):
    """d/dX of Re lam^H (b - A p) for every coordinate.  Tolerance 1e-3: a sample's phase and 1/r^3 are right to 5e-6,
    and the touching pairs' sums cancel by up to two orders of magnitude.  Step 1e-6 on edges of 0.05 and more:
    truncation (1e-6 / 0.05)^2, rounding 2^-53 / 1e-6 of a sum that its derivative exceeds by 1 / 0.1."""
    mesh = G.icosphere(level, 0.1)
    p1, dp0 = make_pure_function_spaces(mesh.grid)
    b = build_geometry_buffers(mesh.grid, mesh.physical_tags, p1, dp0)
    n, T = b.p1_dof_count, b.n_triangles
    base = np.asarray(b.vertices_3xn_f32, dtype=np.float64)
    rng = np.random.default_rng(level)
    dev = torch.device("cuda")
    lam, p, q = ((rng.standard_normal(m) + 1j * rng.standard_normal(m)).astype(np.complex64) for m in (n, n, T))
    q[T // 2:] = 0.0
    parts = [torch.tensor(np.ascontiguousarray(x), device=dev) for z in (lam, p, q) for x in (z.real, z.imag)]
    out = torch.zeros(base.shape, dtype=torch.float64, device=dev)
    kk = np.array([k], np.float32)
    with NativeSession(b, check_open_edges=False) as s:
        check(s.lib.hbem_assemble_backward(
            s.handle, 1, _np_ptr(kk), None, _t_ptr(parts[0]), _t_ptr(parts[1]), n, _t_ptr(parts[2]), _t_ptr(parts[3]), n,
            _t_ptr(parts[4]), _t_ptr(parts[5]), T, _t_ptr(out), _stream_ptr()), "hbem_assemble_backward")
        torch.cuda.synchronize()

    def value(v):
        A, rhs = Oracle(b, 0, "g64", vertices_3xv=v).corrected(float(kk[0]), q)
        return float(np.vdot(lam.astype(np.complex128), rhs - A @ p.astype(np.complex128)).real)

    ref, h = np.zeros_like(base), 1e-6
    for c in np.ndindex(*base.shape):
        step = np.zeros_like(base)
        step[c] = h
        ref[c] = (value(base + step) - value(base - step)) / (2 * h)
    assert np.linalg.norm(out.cpu().numpy() - ref) <= 1e-3 * np.linalg.norm(ref)


@pytest.mark.parametrize("missing", ["real", "imaginary"])
def test_neumann_data_of_one_part_only(missing):
    """A NULL part of the Neumann data is a part of zeros, for regular and touching pairs alike."""
    mesh = G.icosphere(1, 0.1)
    p1, dp0 = make_pure_function_spaces(mesh.grid)
    b = build_geometry_buffers(mesh.grid, mesh.physical_tags, p1, dp0)
    n, T, V = b.p1_dof_count, b.n_triangles, np.asarray(b.vertices_3xn_f32).shape[1]
    rng = np.random.default_rng(7)
    k = np.array([5.0, 30.0], np.float32)
    dev = torch.device("cuda")
    lam, p = (torch.tensor(rng.standard_normal((2, 2, n)), dtype=torch.float32, device=dev) for _ in range(2))
    q = torch.tensor(rng.standard_normal((2, T)), dtype=torch.float32, device=dev)
    with NativeSession(b, check_open_edges=False) as s:
        def grad(q_re, q_im):
            out = torch.zeros((3, V), dtype=torch.float64, device=dev)
            check(s.lib.hbem_assemble_backward(
                s.handle, 2, _np_ptr(k), None, _t_ptr(lam[0]), _t_ptr(lam[1]), n, _t_ptr(p[0]), _t_ptr(p[1]), n,
                _t_ptr(q_re), _t_ptr(q_im), T, _t_ptr(out), _stream_ptr()), "hbem_assemble_backward")
            torch.cuda.synchronize()
            return out.cpu().numpy()

        zero = torch.zeros_like(q)
        one, both = (grad(None, q), grad(zero, q)) if missing == "real" else (grad(q, None), grad(q, zero))
        without = grad(None, None)
    assert np.linalg.norm(both - without) > 0.01 * np.linalg.norm(both)   # the Neumann data matter
    assert np.linalg.norm(one - both) <= 2e-5 * np.linalg.norm(both)
