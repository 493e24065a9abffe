"""Chained plume stages of few units beside each other: on streams of their own, the bits of each alone, and the
CTAs without work leave the chip to the others. A stage of 64x64x144 keeps some 40 CTAs busy; when every CTA
of a launch stayed, eight such stages took as long beside each other as one after the other."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _engines(n):
    from bug_defense_b200 import campaign
    out = []
    for inst in campaign.campaign_instances(1, grid=(64, 64, 128), n_plume_air=16)[:n]:
        eng = campaign.make_engine(dict(inst, n_photons=20_000, pulse_ms=3.0))
        eng.power = eng.laser_power
        eng.step_epochs(3)
        eng.power = 0.0
        out.append(eng)
    return out


def test_small_stages_share_the_chip(gpu):
    import torch

    def epochs(engines, streams, n):
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(streams[0])
        for st in streams[1:]:
            st.wait_event(e0)
        for _ in range(n):
            for eng, st in zip(engines, streams):
                with torch.cuda.stream(st):
                    eng._enqueue(0)
        for st in streams[1:]:
            done = torch.cuda.Event()
            done.record(st)
            streams[0].wait_event(done)
        e1.record(streams[0])
        e1.synchronize()
        return e0.elapsed_time(e1) / n

    fields = []
    for beside in (False, True):
        engines = _engines(8)
        one = torch.cuda.Stream()
        streams = [torch.cuda.Stream() for _ in engines] if beside else [one] * len(engines)
        epochs(engines, streams, 2)
        t = min(epochs(engines, streams, 4) for _ in range(3))
        fields.append((t, [(e.T.copy(), e.plume.raw.cpu().numpy()) for e in engines]))
    (serial, a), (together, b) = fields
    for (Ta, Ca), (Tb, Cb) in zip(a, b):
        assert np.array_equal(Ta, Tb) and np.array_equal(Ca, Cb)
    assert together < 0.75 * serial, (together, serial)


def test_chains_of_many_tiles_on_two_streams(gpu, orc):
    """More than 32 y tiles (a second pass of the unit list) and two stages at a time."""
    import torch
    from bug_defense_b200 import _lib
    from bug_defense_b200.ablation import plume_params_struct
    shape, steps = (5, 530, 24), 130
    rng = np.random.default_rng(8)
    args = (0.03, 0.025, 0.02, 1e-5, 1.5, 2.5, 4.0)
    p = plume_params_struct(shape, *args, 0.02, "as_given")
    cases = []
    for _ in range(2):
        vd = rng.uniform(size=shape) < 0.8
        C0 = (rng.uniform(0.1, 1.0, shape) * vd).astype(np.float32)
        cases.append((vd, C0, torch.from_numpy(C0).cuda(), torch.zeros(shape, device="cuda"),
                      torch.from_numpy((vd * _lib.FLAG_VOID).astype(np.uint8)).cuda(), torch.cuda.Stream()))
    torch.cuda.synchronize()
    import threading
    outs = [None, None]

    def advance(i):
        _, _, a, b, fl, st = cases[i]
        in_b = ctypes.c_int(0)
        _lib.call("bd_plume_advance", ctypes.byref(p), _lib.ptr(a), _lib.ptr(b), steps, _lib.ptr(fl),
                  ctypes.byref(in_b), _lib.stream_ptr(st))
        outs[i] = (b if in_b.value else a).cpu().numpy()

    threads = [threading.Thread(target=advance, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for (vd, C0, *_), got in zip(cases, outs):
        C, Cn = C0.astype(np.float64), np.empty(shape)
        for _ in range(steps):
            orc.diffuse_plume_step(C, Cn, vd, *shape, *args, float(np.exp(-1e-5 / 0.02)))
            C, Cn = Cn, C
        np.testing.assert_allclose(got, C, rtol=steps * 8 * 2.0 ** -24, atol=1e-12)
        assert np.all(got[~vd] == 0.0)
