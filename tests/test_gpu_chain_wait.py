"""The chained plume kernel's bounded wait on progress in global memory: when nobody advances it, the wait gives up
after its polls, raises the error flag that the host turns into BD_ERR_TIMEOUT, and the context stays usable; when
the progress is there, it does not."""
import ctypes
import time

import pytest

pytestmark = pytest.mark.gpu


def _stage():
    import torch
    from bug_defense_b200 import _lib
    from bug_defense_b200.ablation import plume_params_struct
    shape = (12, 20, 24)
    g = torch.Generator(device="cuda").manual_seed(2)
    a = torch.rand(shape, device="cuda", generator=g)
    b = torch.zeros_like(a)
    flags = torch.full(shape, _lib.FLAG_VOID, dtype=torch.uint8, device="cuda")
    p = plume_params_struct(shape, 0.03, 0.025, 0.02, 1e-5, 1.5, 2.5, 4.0, 0.02, "as_given")
    in_b = ctypes.c_int(0)
    _lib.call("bd_plume_advance", ctypes.byref(p), _lib.ptr(a), _lib.ptr(b), 120, _lib.ptr(flags), ctypes.byref(in_b),
              _lib.stream_ptr())
    return (b if in_b.value else a).clone()


def test_chain_wait_times_out_and_the_context_survives(gpu):
    import torch
    from bug_defense_b200 import _lib
    before = _stage()
    t0 = time.perf_counter()
    for polls in (1, 300, 4000):       # below and above the polls between two looks at the error flag
        with pytest.raises(_lib.BugdefError) as exc:
            _lib.call("bd_selftest_chain_wait_timeout", polls, 0, _lib.stream_ptr())
        assert exc.value.code == _lib.BD_ERR_TIMEOUT and "gave up" in str(exc.value)
        _lib.call("bd_selftest_chain_wait_timeout", polls, 1, _lib.stream_ptr())
    assert time.perf_counter() - t0 < 10.0
    with pytest.raises(ValueError):
        _lib.call("bd_selftest_chain_wait_timeout", 0, 0, _lib.stream_ptr())
    assert torch.equal(before, _stage())
