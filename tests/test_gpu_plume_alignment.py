"""Plume fields that are not 16-byte aligned (views into a larger buffer): rows of whole float4 groups must
then not be moved as such. Same bits as the aligned fields, which every kernel gives; the batched stage, which
has no scalar form, refuses them."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _at(t, off):
    """The tensor's values in a buffer that starts `off` floats past a 256-byte boundary."""
    import torch
    buf = torch.zeros(t.numel() + 64, device=t.device)
    v = buf[off:off + t.numel()].view(t.shape)
    v.copy_(t)
    return v


@pytest.mark.parametrize("kernel", [4, 6])
@pytest.mark.parametrize("shape", [(9, 35, 24), (5, 20, 1028)])
def test_unaligned_fields_give_the_aligned_bits(gpu, shape, kernel):
    import torch
    from bug_defense_b200 import _lib
    from bug_defense_b200.ablation import plume_params_struct
    g = torch.Generator(device="cuda").manual_seed(4)
    vd = (torch.rand(shape, device="cuda", generator=g) < 0.8).to(torch.uint8) * _lib.FLAG_VOID
    c0 = torch.rand(shape, device="cuda", generator=g) * (vd > 0)
    p = plume_params_struct(shape, 0.03, 0.025, 0.02, 1e-5, 1.5, 2.5, 4.0, 0.02, "as_given")
    was = ctypes.c_int(0)
    _lib.call("bd_tune_get", _lib.TUNE_PLUME_KERNEL, ctypes.byref(was))
    _lib.call("bd_tune_set", _lib.TUNE_PLUME_KERNEL, kernel)
    try:
        for steps in (1, 7, 90):
            ref = None
            for off_a, off_b in ((0, 0), (1, 0), (0, 2), (3, 3), (2, 1)):
                a, b = _at(c0, off_a), _at(torch.zeros_like(c0), off_b)
                in_b = ctypes.c_int(0)
                _lib.call("bd_plume_advance", ctypes.byref(p), _lib.ptr(a), _lib.ptr(b), steps, _lib.ptr(vd),
                          ctypes.byref(in_b), _lib.stream_ptr())
                got = (b if in_b.value else a).clone()
                ref = got if ref is None else ref
                assert torch.equal(got, ref), (steps, off_a, off_b)
    finally:
        _lib.call("bd_tune_set", _lib.TUNE_PLUME_KERNEL, was.value)


def test_engine_with_unaligned_plume(gpu, monkeypatch):
    from bug_defense_b200 import _lib, campaign, plume
    inst = dict(campaign.campaign_instances(1, grid=(24, 24, 128), n_plume_air=8)[22], n_photons=20_000, pulse_ms=12.0)
    made = plume.PlumeField.__init__

    def unaligned(self, *args, **kw):
        made(self, *args, **kw)
        self.raw = _at(self.raw, 1)

    runs = []
    for patch in (False, True):
        if patch:
            monkeypatch.setattr(plume.PlumeField, "__init__", unaligned)
        eng = campaign.make_engine(inst)
        assert (eng.plume.raw.data_ptr() % 16 != 0) == patch
        eng.step_epochs(14)
        runs.append((eng.T.copy(), eng.plume.raw.cpu().numpy(), eng.ablated.copy()))
    assert np.any(runs[0][1] > 0) and runs[0][2].sum() > 0
    assert all(np.array_equal(x, y) for x, y in zip(*runs))
    batch = ctypes.c_void_p()
    with pytest.raises(ValueError):
        _lib.call("bd_plume_batch_create", (ctypes.c_void_p * 1)(eng._handle), 1, ctypes.byref(batch))
