"""Renders into pinned host images are resolved over the link, others copied;
a resolved frame leaves the key buffer empty for the next. Frames of changing
sizes (partial last words, smaller and larger than the one before), into
pinned, misaligned and single outputs, must equal the pageable render of a
fresh handle, bit for bit."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(640, 360), (1, 1), (3, 1), (5, 7), (321, 243), (64, 64), (1280, 720), (33, 500)]


def test_pinned_frames_equal_pageable(gpu_lib):
    import torch
    import fluidsim
    from fluidsim import render, scenes
    sc = scenes.dam_break_16k()

    def fresh():
        sim = fluidsim.FluidSimulation(sc["params"])
        sim.InitializeData(sc["pos"].shape[0], sc["pos"], sc["vel"])
        return sim
    sim = fresh()
    drawn = 0
    for k, (w, h) in enumerate(SIZES):
        eye = (2.0 + 0.1 * k, 3.0, 9.0)
        v = render.view(eye, (-2.0, -1.5, -1.0), w, h)
        ref = fresh()
        want_img, want_depth = ref.render(v)
        ref.close()
        drawn += int((want_depth < 1.0).sum())
        off = k % 2  # every other frame a depth image that is not 16-byte aligned
        img = torch.zeros(w * h * 4, dtype=torch.uint8, pin_memory=True)
        depth = torch.zeros(w * h + off, dtype=torch.float32, pin_memory=True)[off:]
        for outs in ((img, depth), (img, None), (None, depth), (None, None)):
            img.zero_()
            depth.zero_()
            ptrs = [None if o is None else ctypes.c_void_p(o.data_ptr()) for o in outs]
            assert gpu_lib.sph_render(sim.handle, ctypes.byref(v), *ptrs, None) == 0
            if outs[0] is not None:
                assert np.array_equal(img.numpy().reshape(h, w, 4), want_img), (w, h)
            if outs[1] is not None:
                assert np.array_equal(depth.numpy().reshape(h, w), want_depth), (w, h)
    sim.close()
    assert drawn > 1000
