"""The chained plume kernel (four steps per pass over the field) against the FP64 oracle, where its
tiling can go wrong: 16-row tiles and their remainders, runs of void longer than a window of 32 z
groups, rows that are no multiple of four voxels, step counts that leave a remainder of the four, and
more blocks of steps than one launch holds.

Tolerance: FP32 against FP64, each step a convex combination rounded a few times: the relative error
stays below (steps) x 8 x 2^-24, 1e-6 for 2 steps and 5e-4 for 1100."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _void(rng, shape, kind):
    vd = rng.uniform(size=shape) < 0.8
    if kind == "full":
        vd[:] = True
    elif kind == "layers":                      # a bulk layer, solid, a gap layer and a deep cavity
        vd[:] = False
        n = shape[2]
        vd[:, :, :n // 3] = True
        vd[:, :, n // 2:n // 2 + 3] = True
        vd[shape[0] // 3:shape[0] // 2 + 1, shape[1] // 4:, n // 3:n - 1] = True
    return vd


CASES = [((20, 16, 24), "pores", 1), ((20, 17, 24), "pores", 2), ((7, 33, 25), "pores", 3),
         ((12, 40, 128), "full", 4), ((6, 35, 132), "full", 5), ((5, 18, 271), "full", 9),
         ((40, 37, 150), "layers", 6), ((3, 3, 3), "full", 8), ((1, 5, 9), "full", 4), ((9, 1, 9), "full", 4),
         ((64, 50, 140), "layers", 33), ((6, 6, 6), "full", 1100)]


@pytest.mark.parametrize("shape,kind,steps", CASES)
def test_chained_plume_matches_oracle(gpu, orc, shape, kind, steps):
    rng = np.random.default_rng(sum(shape) + steps)
    vd = _void(rng, shape, kind)
    C0 = (rng.uniform(0.1, 1.0, shape) * vd).astype(np.float32)
    dx, dy, dz, dt, Dxy, Dz, vz, tau = 0.03, 0.025, 0.02, 1e-5, 1.5, 2.5, 4.0, 0.02
    ctx = gpu.MetalAblationContext(*shape, dx, dy, dz, dt, 0.0, 20.0, 100.0, 300.0,
                                   plume_params={'D_xy': Dxy, 'D_z': Dz, 'vz': vz, 'tau_linger': tau},
                                   plume_dt_policy='as_given')
    z = np.zeros(shape)
    ctx.set_state(np.full(shape, 20.0), z, z, z, np.zeros(shape, np.uint8), np.zeros(shape, np.uint8), z, z,
                  np.full(shape, 1e-3), plume=C0, plume_void=vd)
    ctx.advance_substeps(steps, is_active=0)
    got = ctx.get_plume()
    C, Cn = C0.astype(np.float64), np.empty(shape)
    decay = float(np.exp(-dt / tau))
    for _ in range(steps):
        orc.diffuse_plume_step(C, Cn, vd, *shape, dx, dy, dz, dt, Dxy, Dz, vz, decay)
        C, Cn = Cn, C
    np.testing.assert_allclose(got, C, rtol=steps * 8 * 2.0 ** -24, atol=1e-12)
    assert np.all(got[~vd] == 0.0)
