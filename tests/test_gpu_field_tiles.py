"""The exterior field's two tile widths: the same bits on either side of their line, and no call that is slower than
one with more points."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("needs a CUDA device", allow_module_level=True)

from hornlab_metal_bem_b200 import generators as G  # noqa: E402
from hornlab_metal_bem_b200.geometry import build_geometry_buffers  # noqa: E402
from hornlab_metal_bem_b200.mesh import make_pure_function_spaces  # noqa: E402
from hornlab_metal_bem_b200.native import NativeSession, _np_ptr, _stream_ptr, _t_ptr, check  # noqa: E402

MESHES = {"sphere": (lambda: G.icosphere(2, 0.1), None),
          "half": (lambda: G.horn(G.HornSpec(edge=0.02), quarter=False, half=True), "yz"),
          "quarter": (lambda: G.horn(G.HornSpec(edge=0.007), quarter=True), "yz+xz")}


def _session(name):
    make, plane = MESHES[name]
    mesh = make()
    p1, dp0 = make_pure_function_spaces(mesh.grid)
    return NativeSession(build_geometry_buffers(mesh.grid, mesh.physical_tags, p1, dp0), symmetry_plane=plane,
                         check_open_edges=False)


def _field(s, data, n_obs):
    p, q, obs = data
    k = np.array([37.0], np.float32)
    o = obs[:, :n_obs].contiguous()
    out = torch.empty((2, n_obs), device="cuda")
    args = (s.handle, 1, _np_ptr(k), _t_ptr(p[0]), _t_ptr(p[1]), s.n_dof, _t_ptr(q[0]), _t_ptr(q[1]), s.n_triangles,
            _t_ptr(o), n_obs, _t_ptr(out[0]), _t_ptr(out[1]), n_obs, _stream_ptr())
    return (lambda: check(s.lib.hbem_field(*args), "hbem_field")), out, (o, k)


def _data(s):
    g = torch.Generator(device="cuda").manual_seed(1)
    rand = lambda *shape: torch.randn(shape, device="cuda", generator=g)  # noqa: E731
    return rand(2, s.n_dof), rand(2, s.n_triangles), 2.0 + rand(3, 6000)


@pytest.mark.parametrize("name", sorted(MESHES))
def test_either_tile_gives_the_same_bits(name):
    with _session(name) as s:
        data = _data(s)
        run, whole, keep = _field(s, data, 6000)   # eight points a CTA
        run()
        for n in (1, 2, 7, 8, 1041, 2071, 2073):
            run, part, keep2 = _field(s, data, n)
            run()
            assert torch.equal(part, whole[:, :n])


def test_fewer_points_take_no_longer():
    """Quarter horn, one frequency: just below two CTAs of eight points an SM against just there.  The fastest of
    15 timings of 8 calls each, in turn; they repeat within 1 %."""
    with _session("quarter") as s:
        data = _data(s)
        sm = torch.cuda.get_device_properties(0).multi_processor_count
        calls = [_field(s, data, n) for n in (16 * sm - 8, 16 * sm)]
        times = [[], []]
        for rep in range(17):
            for i, (run, _, _) in enumerate(calls):
                e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
                torch.cuda._sleep(200000)
                e0.record()
                for _ in range(8):
                    run()
                e1.record()
                torch.cuda.synchronize()
                if rep >= 2:
                    times[i].append(e0.elapsed_time(e1))
        fewer, more = (min(t) for t in times)
        assert fewer <= 1.03 * more
