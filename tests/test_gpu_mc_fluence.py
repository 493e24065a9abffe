"""The tracer of the fluence launches follows the same photon histories as the one without: the exact absorbed
tally gives the same map to the bit, the ledger counts the same events, and its FP64 weight channels differ by
the order of their sums only (1e-12 relative)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("semantics,axis", [("cpu", "z"), ("metal", "z"), ("cpu", "x"), ("metal", "x")])
@pytest.mark.parametrize("n,profile,r_max,max_events", [(1, "gaussian", 0.0, None), (33, "tophat", 0.0, None),
                                                        (20_001, "gaussian", 0.21, None), (5000, "gaussian", 0.0, 40),
                                                        (160_001, "kim_exp_disk", 0.0, None)])
def test_same_histories_with_and_without_fluence(gpu, n, profile, r_max, max_events, semantics, axis):
    import torch
    from bug_defense_b200 import _lib, voxel_mc
    dev = torch.device("cuda")
    shape = (18, 20, 24)
    z = np.arange(shape[2])
    mu_a = np.broadcast_to(np.where(z < 6, 8.0, 0.4), shape).copy()
    mu_s = np.broadcast_to(np.where(z < 6, 20.0, 12.0), shape).copy()
    idx = np.broadcast_to(np.where(z < 6, 1.56, 1.40), shape).copy()
    props = voxel_mc.pack_props(mu_a, mu_s, np.full(shape, 0.88), idx, dev)
    flags = torch.zeros(shape, dtype=torch.uint8, device=dev)
    flags[:, :, 3] = _lib.FLAG_ABLATED
    nv = int(np.prod(shape))
    out = []
    for fluence in (False, True):
        A, L = torch.zeros(nv, device=dev), torch.zeros(nv, device=dev)
        led = torch.zeros(_lib.LEDGER_LEN, dtype=torch.float64, device=dev)
        p = voxel_mc.make_params(Nx=shape[0], Ny=shape[1], Nz=shape[2], Lx=0.5, Ly=0.5, Lz=0.6, n_photons=n,
                                 spot_dia=0.2, theta_inc_deg=15.0, launch_axis=axis, seed=9, semantics=semantics,
                                 beam_profile=profile, r_max=r_max, tally_fluence=fluence, photon_offset=0,
                                 max_events=max_events)
        voxel_mc.trace(p, props, A, L=L if fluence else None, ledger=led, flags=flags)
        out.append((A.cpu().numpy(), led.cpu().numpy(), L.cpu().numpy()))
    (a0, l0, _), (a1, l1, track) = out
    np.testing.assert_array_equal(a0, a1)
    whole = [_lib.LEDGER_COLLISIONS, _lib.LEDGER_CROSSINGS]
    np.testing.assert_array_equal(l0[whole], l1[whole])
    np.testing.assert_allclose(l1, l0, rtol=1e-12, atol=1e-12 * n)
    assert a0.sum() > 0 and track.sum() > 0 and np.all(track >= 0)
