"""The substep kernel at the edges of its 4-voxel groups, rows, warps and chunks of planes, against the
FP64 oracle, and its char kinetics against the closed form where temperatures straddle the limit
below which a substep's rate is nothing in FP32."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (2, 1, 3), (1, 3, 2), (5, 3, 4), (3, 5, 5), (4, 2, 7), (3, 33, 4), (9, 7, 36), (17, 19, 61),
          (6, 2, 257), (33, 40, 64)]


@pytest.mark.parametrize("shape", SHAPES)
def test_thermal_steps_match_oracle(gpu, orc, shape):
    """8 steps; FP32 against FP64: T is rounded about 20 times a step, 8 x 20 x 2^-24 = 1e-5 relative."""
    rng = np.random.default_rng(sum(shape))
    T0, Q = rng.uniform(20, 120, shape), rng.uniform(0, 900, shape)
    k, rho = rng.uniform(2e-4, 6e-4, shape), rng.uniform(1.5e-3, 4e-3, shape)
    geo = (0.03, 0.025, 0.02, 2e-5)
    got = gpu.run_thermal3d_substeps_gpu(T0, Q, k, rho, *shape, *geo, 8, 15e-6, 20.0, 1)
    T, Tn = T0.copy(), np.empty_like(T0)
    for _ in range(8):
        orc.thermal3d_step_explicit(T, Tn, Q, k, rho, *shape, *geo, 15e-6, 20.0, 1)
        T, Tn = Tn, T
    assert np.max(np.abs(got - T) / np.abs(T)) <= 1e-5


@pytest.mark.parametrize("shape", [(3, 5, 5), (5, 9, 64), (4, 3, 131)])
@pytest.mark.parametrize("dry_share", [0.05, 0.5, 1.0])
def test_char_of_scattered_dry_voxels(gpu, shape, dry_share):
    """Without conduction and source T stays, so chi after n substeps is 1 - (1 - chi0) exp(-n rate dt).
    Per substep FP32 rounds 1 - x twice (2^-24 absolute) and the exponentials to a few ulp of the rate:
    an exponent of up to 40 in FP32 carries 40 x 2^-23 relative into it, 5e-6; 10 substeps of a chi below 1
    stay within 10 x 2^-24 + 1e-5."""
    A, E, dt, n = 1.0e11, 1.75e5 / 8.314, 5e-5, 10
    rng = np.random.default_rng(int(100 * dry_share) + sum(shape))
    T0 = rng.uniform(20.0, 600.0, shape).astype(np.float32).astype(np.float64)
    cold = rng.uniform(size=shape) < 0.5
    T0[cold] = 25.0
    dry = rng.uniform(size=shape) < dry_share
    chi0 = rng.uniform(0, 0.9, shape).astype(np.float32).astype(np.float64) * dry
    z = np.zeros(shape)
    ctx = gpu.MetalAblationContext(*shape, 0.015, 0.015, 0.015, dt, 0.0, 20.0, 1e9, 1e9, char_params=(A, E))
    ctx.set_state(T0, z, z, chi0, dry, np.zeros(shape, np.uint8), z, z, np.full(shape, 3e-3))
    ctx.advance_substeps(n, is_active=0)
    T, _, _, chi = ctx.get_state()
    assert np.array_equal(T, T0)
    want = np.where(dry, 1.0 - (1.0 - chi0) * np.exp(-n * dt * A * np.exp(-E / (T0 + 273.15))), chi0)
    assert np.max(np.abs(chi - want)) <= n * 2.0 ** -24 + 1e-5
    assert np.array_equal(chi[~dry], chi0[~dry])
    if dry.sum() > 50:                     # the draw holds dry voxels that char (1.7e-3 at 600 C)
        assert np.any(want - chi0 > 1e-4)
