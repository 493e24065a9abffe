"""Which kernel runs a plume stage: a chain only where it is the shorter way, a launch per step for stages of few
steps; and the chain at the edges of its tiling with enough steps to be chosen, against the FP64 oracle.

Tolerance: FP32 against FP64, each step a convex combination rounded a few times: the relative error stays below
(steps) x 8 x 2^-24."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ARGS = (0.03, 0.025, 0.02, 1e-5, 1.5, 2.5, 4.0)
DECAY = float(np.exp(-1e-5 / 0.02))


def _advance(shape, vd, C0, steps):
    import torch
    from bug_defense_b200 import _lib
    from bug_defense_b200.ablation import plume_params_struct
    a = torch.from_numpy(C0).cuda()
    b = torch.full_like(a, 7.0)
    flags = torch.from_numpy((vd * _lib.FLAG_VOID).astype(np.uint8)).cuda()
    p = plume_params_struct(shape, *ARGS, 0.02, "as_given")
    in_b = ctypes.c_int(0)
    _lib.call("bd_plume_advance", ctypes.byref(p), _lib.ptr(a), _lib.ptr(b), steps, _lib.ptr(flags), ctypes.byref(in_b),
              _lib.stream_ptr())
    return (b if in_b.value else a).cpu().numpy()


def _kernels(fn):
    import torch
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        out = fn()
        torch.cuda.synchronize()
    keys = [e.key for e in prof.key_averages()]
    names = ("k_plume_direct", "k_plume_direct_c", "k_plume_chain", "k_plume_step")
    ran = {n for n in names if any(f"::{n}(" in key or f"::{n}<" in key for key in keys)}
    return out, ran if keys else None      # where another tool already traces the process, the profiler records nothing


# few steps; a long x axis, where a chain's first block takes longer than all the launches; rows of no whole float4
@pytest.mark.parametrize("shape,steps,kernel", [((120, 40, 64), 1, "k_plume_direct"), ((120, 40, 64), 6, "k_plume_direct"),
                                                ((120, 40, 64), 300, "k_plume_chain"),
                                                ((900, 16, 32), 40, "k_plume_direct"),
                                                ((120, 40, 63), 5, "k_plume_step"), ((120, 40, 63), 300, "k_plume_chain")])
def test_kernel_of_a_stage(gpu, orc, shape, steps, kernel):
    rng = np.random.default_rng(sum(shape) + steps)
    vd = rng.uniform(size=shape) < 0.8
    C0 = rng.uniform(0.1, 1.0, shape).astype(np.float32)
    got, ran = _kernels(lambda: _advance(shape, vd, C0, steps))
    assert ran in ({kernel}, None)
    C, Cn = np.where(vd, C0, 0.0).astype(np.float64), np.empty(shape)
    for _ in range(steps):
        orc.diffuse_plume_step(C, Cn, vd, *shape, *ARGS, DECAY)
        C, Cn = Cn, C
    np.testing.assert_allclose(got, C, rtol=steps * 8 * 2.0 ** -24, atol=1e-12)
    assert np.all(got[~vd] == 0.0)


# tiles and their remainders, windows of z groups, remainders of 1, 2 and 3 steps
@pytest.mark.parametrize("shape,kind,steps", [((20, 17, 24), "pores", 121), ((7, 33, 25), "pores", 122),
                                              ((12, 40, 128), "full", 123), ((6, 35, 132), "full", 120),
                                              ((5, 18, 271), "pores", 121), ((40, 37, 150), "layers", 202),
                                              ((3, 3, 3), "full", 123), ((1, 5, 9), "full", 60), ((9, 1, 9), "full", 61)])
def test_chain_matches_oracle_and_the_launches_per_step(gpu, orc, shape, kind, steps):
    rng = np.random.default_rng(sum(shape) + steps)
    vd = rng.uniform(size=shape) < 0.8
    if kind == "full":
        vd[:] = True
    elif kind == "layers":
        vd[:] = False
        n = shape[2]
        vd[:, :, :n // 3] = True
        vd[:, :, n // 2:n // 2 + 3] = True
        vd[shape[0] // 3:shape[0] // 2 + 1, shape[1] // 4:, n // 3:n - 1] = True
    C0 = rng.uniform(0.1, 1.0, shape).astype(np.float32)
    got, ran = _kernels(lambda: _advance(shape, vd, C0, steps))
    assert ran in ({"k_plume_chain"}, None)
    C, Cn = np.where(vd, C0, 0.0).astype(np.float64), np.empty(shape)
    one = np.where(vd, C0, 0.0).astype(np.float32)
    for _ in range(steps):
        orc.diffuse_plume_step(C, Cn, vd, *shape, *ARGS, DECAY)
        C, Cn = Cn, C
        one = _advance(shape, vd, one, 1)
    np.testing.assert_allclose(got, C, rtol=steps * 8 * 2.0 ** -24, atol=1e-12)
    np.testing.assert_array_equal(got, one)
