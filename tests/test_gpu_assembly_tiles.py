"""Unordered pair assembly and its right-hand sides at the edges of their tiles, against the FP64 oracle.

Tolerance 2e-5 relative L2: the FP32 product k r (at most 20 here) is off by 2^-24 of itself, 1.2e-6, the fast
sine and cosine by 2^-21 and 1/r by 2^-22.9 relative; the differences y - x of FP32 points (coordinates up to
0.3, triangles down to 0.02 apart) by 2^-25 * 0.3 / 0.02 = 5e-7, three times that in 1/r^3.  The sum of these
at their worst is 5e-6, with room for near pairs that weigh more than their share."""
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
from hornlab_metal_bem_b200.mesh import make_pure_function_spaces, mesh_from_arrays  # noqa: E402
from hornlab_metal_bem_b200.native import (  # noqa: E402
    HBEM_ASM_REGULAR, HBEM_ASM_ZERO, NativeSession, _np_ptr, _stream_ptr, _t_ptr, check, load_library,
)


def _buffers(mesh):
    p1, dp0 = make_pure_function_spaces(mesh.grid)
    return build_geometry_buffers(mesh.grid, mesh.physical_tags, p1, dp0)


def _fan(n):
    """Two n-gon pyramids: apexes shared by n triangles, more than a row list's packed eight."""
    a = 2.0 * np.pi * np.arange(n) / n
    v = np.vstack([np.stack([0.2 * np.cos(a), 0.2 * np.sin(a), 0.0 * a], 1), [[0, 0, 0.15], [0, 0, -0.15]]])
    f = [(i, (i + 1) % n, n) for i in range(n)] + [((i + 1) % n, i, n + 1) for i in range(n)]
    return mesh_from_arrays(v, np.array(f, np.int32), np.ones(2 * n, np.int32))


def _apart(n):
    """n triangles without a common vertex: 96 dofs a test tile, planes that two wavenumbers overflow."""
    rng = np.random.default_rng(3)
    c = np.stack(np.meshgrid(np.arange(4), np.arange(4), np.arange(3), indexing="ij"), -1).reshape(-1, 3)[:n] * 0.1
    v = (c[:, None] + 0.02 * rng.standard_normal((n, 3, 3))).reshape(-1, 3)
    return mesh_from_arrays(v, np.arange(3 * n, dtype=np.int32).reshape(n, 3), np.ones(n, np.int32))


def _scattered():
    """70 triangles without a common vertex: more dofs in a 64-triangle tile than the ordered kernel can stage, which
    is no limit of the unordered one.  k r reaches 26 here, 1.6e-6 of the tolerance."""
    rng = np.random.default_rng(4)
    c = np.stack(np.meshgrid(np.arange(4), np.arange(4), np.arange(5), indexing="ij"), -1).reshape(-1, 3)[:70] * 0.1
    v = (c[:, None] + 0.02 * rng.standard_normal((70, 3, 3))).reshape(-1, 3)
    return mesh_from_arrays(v, np.arange(210, dtype=np.int32).reshape(70, 3), np.ones(70, np.int32))


def _half(axes):
    """Half horn (x >= 0), its axes exchanged in a cycle."""
    mesh = G.horn(G.HornSpec(edge=0.03), quarter=False, half=True)
    v = np.asarray(mesh.grid.vertices, dtype=np.float64)[axes].T
    return mesh_from_arrays(v, np.asarray(mesh.grid.elements).T, np.asarray(mesh.physical_tags))


MESHES = {"one_tile": (lambda: G.icosphere(0, 0.1), None, 0), "ragged": (lambda: G.icosphere(1, 0.1), None, 0),
          "fan": (lambda: _fan(37), None, 0), "apart": (lambda: _apart(38), None, 0),
          "scattered": (_scattered, None, 0),
          "quarter": (lambda: G.horn(G.HornSpec(edge=0.02), quarter=True), "yz+xz", 3),
          "half": (lambda: _half([0, 1, 2]), "yz", 1), "half_xz": (lambda: _half([2, 0, 1]), "xz", 2),
          "half_xy": (lambda: _half([1, 2, 0]), "xy", 4)}
HBEM_TUNE_ASM_PAIRS = 3


def _check(name, freqs, sources, robin, damped=False):
    make, plane, sym = MESHES[name]
    b = _buffers(make())
    n, T = b.p1_dof_count, b.n_triangles
    rng = np.random.default_rng(11)
    k = np.linspace(4.0, 40.0, freqs).astype(np.float32)
    ki = np.linspace(0.1, 2.0, freqs).astype(np.float32) if damped else None
    q = (rng.standard_normal((sources, freqs, T)) + 1j * rng.standard_normal((sources, freqs, T))).astype(np.complex64)
    q[:, :, rng.random(T) < 0.5] = 0.0
    beta = np.where(rng.random(T) < 0.6, 0.3 - 0.1j, 0.0).astype(np.complex64) if robin else None
    dev = torch.device("cuda")
    parts = lambda z: (torch.tensor(np.ascontiguousarray(z.real), device=dev),  # noqa: E731
                       torch.tensor(np.ascontiguousarray(z.imag), device=dev))
    qr, qi = parts(q)
    br_, bi_ = parts(beta) if robin else (None, None)
    A = torch.empty((2, freqs, n, n), device=dev)
    rhs = torch.empty((2, sources, freqs, n), device=dev)
    with NativeSession(b, symmetry_plane=plane, check_open_edges=False) as s:
        check(s.lib.hbem_assemble_multi(
            s.handle, freqs, _np_ptr(k), _np_ptr(ki), sources, _t_ptr(qr), _t_ptr(qi), T, freqs * T, _t_ptr(br_),
            _t_ptr(bi_), _t_ptr(A[0]), _t_ptr(A[1]), n, n * n, _t_ptr(rhs[0]), _t_ptr(rhs[1]), n, freqs * n,
            HBEM_ASM_REGULAR | HBEM_ASM_ZERO, _stream_ptr()), "hbem_assemble_multi")
    A, rhs = (z.double().cpu().numpy() for z in (A, rhs))
    A, rhs = A[0] + 1j * A[1], rhs[0] + 1j * rhs[1]
    o = Oracle(b, sym, "f64")
    for f in range(freqs):
        for sv in range(sources):
            A_ref, b_ref = o.regular(float(k[f]), q[sv, f], k_imag=float(ki[f]) if damped else 0.0, beta=beta)
            assert np.linalg.norm(A[f] - A_ref) <= 2e-5 * np.linalg.norm(A_ref)
            assert np.linalg.norm(rhs[sv, f] - b_ref) <= 2e-5 * np.linalg.norm(b_ref)


@pytest.mark.parametrize("freqs,sources,robin", [(1, 1, False), (2, 3, False), (3, 1, False), (3, 2, True)])
@pytest.mark.parametrize("name", sorted(MESHES))
def test_regular_assembly_at_tile_edges(name, freqs, sources, robin):
    _check(name, freqs, sources, robin)


@pytest.mark.parametrize("freqs,sources,robin", [(2, 1, False), (3, 3, False), (3, 1, True)])
@pytest.mark.parametrize("name", sorted(MESHES))
def test_complex_wavenumbers(name, freqs, sources, robin):
    """exp(-Im k r) is 2^-22 off, its argument (below 1.5) 2^-23."""
    _check(name, freqs, sources, robin, damped=True)


@pytest.mark.parametrize("freqs,robin,damped", [(1, False, False), (3, True, False), (2, True, True)])
@pytest.mark.parametrize("name", sorted(set(MESHES) - {"scattered"}))
def test_ordered_pairs(name, freqs, robin, damped):
    lib = load_library()
    check(lib.hbem_set_tuning(HBEM_TUNE_ASM_PAIRS, 1), "hbem_set_tuning")
    try:
        _check(name, freqs, 1, robin, damped)
    finally:
        lib.hbem_set_tuning(HBEM_TUNE_ASM_PAIRS, 0)
