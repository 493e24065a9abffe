"""Photons that leave a grid with an axis of more than 2^24 voxels, where a voxel index in FP32 no longer
counts: every deposit lies inside the grid and the ledger closes.

The launch without fluence gives the map of the launch with it to the bit (both step whole-number indices);
the map's sum and the ledger's absorbed weight are the same deposits, rounded to the tally's 2^-36 steps and
once to FP32 a voxel: 1e-6 relative."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, FROM_END, D = 2 ** 24 + 84, 50, 2.0 ** -10       # voxels of the long axis, launch point, voxel size (mm)


@pytest.mark.parametrize("axis,launch,phi", [(0, "z", 0.0), (1, "z", 90.0), (2, "x", 90.0)])
def test_photons_leave_a_long_axis_at_its_end(gpu, axis, launch, phi):
    import torch
    from bug_defense_b200 import _lib, voxel_mc
    shape, size = [1, 1, 1], [1.0, 1.0, 1.0]
    shape[axis], size[axis] = N, N * D
    at = N * D - FROM_END * D
    centre = {(0, "z"): (at, 0.5), (1, "z"): (0.5, at), (2, "x"): (0.5, at)}[(axis, launch)]
    props = torch.empty((N, 4), device="cuda")
    props[:] = torch.tensor([3.0, 1.0 / 3.0, 0.5, 1.0], device="cuda")      # mu_t, mu_a / mu_t, g, n
    out = []
    for fluence in (False, True):
        A = torch.zeros(N, device="cuda")
        L = torch.zeros(N, device="cuda") if fluence else None
        led = torch.zeros(_lib.LEDGER_LEN, dtype=torch.float64, device="cuda")
        p = voxel_mc.make_params(Nx=shape[0], Ny=shape[1], Nz=shape[2], Lx=size[0], Ly=size[1], Lz=size[2],
                                 n_photons=3000, spot_dia=2.0 ** -6, theta_inc_deg=60.0, phi_inc_deg=phi,
                                 beam_center=centre, launch_axis=launch, seed=3, tally_fluence=fluence)
        voxel_mc.trace(p, props, A, L=L, ledger=led)
        out.append((A, led.cpu().numpy()))
    (A, led), (A1, led1) = out
    assert torch.equal(A, A1)
    np.testing.assert_allclose(led, led1, rtol=1e-12, atol=1e-9)
    closure = led[1:7].sum() + led[8] + led[9] - led[7]
    assert abs(closure / 3000 - 1.0) < 1e-12
    assert led[_lib.LEDGER_LATERAL] > 0 and led[_lib.LEDGER_ABSORBED] > 0
    assert abs(float(A.double().sum()) / led[_lib.LEDGER_ABSORBED] - 1.0) < 1e-6
