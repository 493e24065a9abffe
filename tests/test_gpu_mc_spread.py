"""Few photons are spread over half of the resident warps, some lanes of each: the launch's grid follows from the
photon count, and the maps do not depend on it (photons cut into launches of other sizes, exact tally: each launch
rounds a voxel once to FP32, so b launches differ by at most (b + 1) 2^-24 relative)."""
import json

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _trace(props, shape, n, offset=0):
    import torch
    from bug_defense_b200 import voxel_mc
    A = torch.zeros(int(np.prod(shape)), device="cuda")
    p = voxel_mc.make_params(Nx=shape[0], Ny=shape[1], Nz=shape[2], Lx=0.5, Ly=0.5, Lz=0.6, n_photons=n, spot_dia=0.2,
                             theta_inc_deg=15.0, seed=5, tally_fluence=False, photon_offset=offset)
    voxel_mc.trace(p, props, A)
    return A


@pytest.mark.parametrize("n", [0, 1, 5, 2367, 2369, 9473, 40_000, 75_777, 151_553])
def test_spread_of_few_photons(gpu, tmp_path, n):
    import torch
    from bug_defense_b200 import voxel_mc
    from torch.profiler import ProfilerActivity, profile
    shape = (18, 20, 24)
    full = lambda v: np.full(shape, v)
    props = voxel_mc.pack_props(full(2.0), full(15.0), full(0.85), full(1.4), torch.device("cuda"))
    _trace(props, shape, 10)
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        A = _trace(props, shape, n)
        torch.cuda.synchronize()
    path = tmp_path / "trace.json"
    prof.export_chrome_trace(str(path))
    grids = [e["args"]["grid"][0] for e in json.loads(path.read_text())["traceEvents"]
             if "k_mc_trace" in e.get("name", "") and "grid" in e.get("args", {})]
    parts = [_trace(props, shape, b - a, a) for a, b in zip((0, n // 3, n // 2), (n // 3, n // 2, n))]
    np.testing.assert_allclose(sum(q.double() for q in parts).cpu().numpy(), A.double().cpu().numpy(),
                               rtol=4 * 2.0 ** -24, atol=0)
    if not prof.events():          # where another tool already traces the process, the profiler records nothing
        return
    assert len(grids) == 1
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    occ = 8                                            # resident CTAs of the kernel per SM
    lanes = min(32, max(1, -(-n // (2 * sms * occ))))
    assert grids[0] == max(1, min(sms * occ, -(-n // (4 * lanes))))
    if lanes < 32:                                     # half of the warps at most while a warp has lanes to spare
        assert grids[0] <= sms * occ // 2 + 1
