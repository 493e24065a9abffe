"""A heat source that is switched off does not enter the temperature, whatever its scale holds: the bits of a
scale of 1, for grids of whole float4 rows and others, thermal and fused substeps."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [np.inf, -np.inf, np.nan, 3e38])
@pytest.mark.parametrize("shape", [(6, 10, 16), (6, 10, 15)])
def test_scale_of_an_inactive_source(gpu, shape, scale):
    import torch
    from bug_defense_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(3)
    rand = lambda lo, hi: torch.rand(shape, device="cuda", generator=g) * (hi - lo) + lo
    T0, K, R = rand(25.0, 120.0), rand(2e-4, 6e-4), rand(2e-3, 4e-3)
    flags = (rand(0.0, 1.0) < 0.3).to(torch.uint8) * _lib.FLAG_ABLATED

    def run(name, q_scale):
        a, b, H = T0.clone(), torch.empty_like(T0), torch.zeros_like(T0)
        p = (_lib.ThermalParams if name == "thermal" else _lib.AblationParams)()
        p.nx, p.ny, p.nz = shape
        p.dx = p.dy = p.dz = 0.015
        p.dt, p.h_eff, p.t_ambient, p.q_scale, p.is_active = 5e-6, 1e-5, 25.0, q_scale, 0
        if name == "thermal":
            _lib.call("bd_thermal_advance", ctypes.byref(p), _lib.ptr(a), _lib.ptr(b), 4, None, _lib.ptr(K), _lib.ptr(R),
                      _lib.stream_ptr())
        else:
            p.t_abl, p.t_void, p.zero_src_in_ablated = 100.0, 350.0, 1
            _lib.call("bd_ablation_advance", ctypes.byref(p), _lib.ptr(a), _lib.ptr(b), 4, _lib.ptr(H), None, None,
                      _lib.ptr(flags), None, _lib.ptr(K), _lib.ptr(R), _lib.stream_ptr())
        return a

    for name in ("thermal", "ablation"):
        want, got = run(name, 1.0), run(name, float(scale))
        assert torch.isfinite(want).all() and not torch.equal(want, T0)
        assert torch.equal(got, want), name
