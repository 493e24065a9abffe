"""Photon histories do not depend on how many lanes of a warp trace photons: n photons in one launch
(spread over all resident warps when they are few) give the sums of the same photons traced in launches
of other sizes. The absorbed tally is exact integers per launch, rounded once to FP32: with b launches
the sums differ by at most (b + 1) roundings, (b + 1) 2^-24 relative per voxel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("semantics,axis", [("cpu", "z"), ("metal", "z"), ("cpu", "x")])
@pytest.mark.parametrize("n,parts", [(1, 1), (33, 3), (4737, 5), (20_000, 4), (160_001, 2)])
def test_maps_do_not_depend_on_the_launch_size(gpu, n, parts, semantics, axis):
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

    def run(count, offset):
        A, led = torch.zeros(nv, device=dev), torch.zeros(_lib.LEDGER_LEN, dtype=torch.float64, device=dev)
        p = voxel_mc.make_params(Nx=shape[0], Ny=shape[1], Nz=shape[2], Lx=0.5, Ly=0.5, Lz=0.6, n_photons=count,
                                 spot_dia=0.2, theta_inc_deg=15.0, launch_axis=axis, seed=9, semantics=semantics,
                                 tally_fluence=False, photon_offset=offset)
        voxel_mc.trace(p, props, A, ledger=led, flags=flags)
        return A.double().cpu().numpy(), led.cpu().numpy()

    A, led = run(n, 0)
    cuts = np.linspace(0, n, parts + 1).astype(int)
    split = [run(int(b - a), int(a)) for a, b in zip(cuts[:-1], cuts[1:])]
    np.testing.assert_allclose(sum(s[0] for s in split), A, rtol=(parts + 1) * 2.0 ** -24, atol=0)
    np.testing.assert_allclose(sum(s[1] for s in split), led, rtol=1e-12, atol=1e-12 * n)
    assert led[_lib.LEDGER_LAUNCHED] == n and A.sum() > 0
    if n > 1000:
        assert led[_lib.LEDGER_ABSORBED_VOID] > 0
    closure = led[1:7].sum() + led[8] + led[9] - led[7]
    assert abs(closure / n - 1.0) < 1e-12
