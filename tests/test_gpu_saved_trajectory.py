"""Backward passes of the libtorch operators and the context's trajectory."""
import importlib

import numpy as np
import pytest

from test_gpu_grad import wave_case

pytestmark = pytest.mark.gpu


def test_backward_uses_the_forward_trajectory(gpu_lib, cgs, synth, oracle_mod):
    """The backward pass reuses the coordinates that its forward pass left on
    the context only while no other trajectory was set in between: with one in
    between, the gradients are those of the saved trajectory all the same."""
    import torch
    ag = importlib.import_module("4d_lung_gb300.autograd")
    img, grid, nch = (16, 16, 12), (32, 32, 24), 3
    w, lines, r, smaps, x, y, p, _, _ = wave_case(cgs, synth, oracle_mod, img, grid, nch)
    k1 = torch.from_numpy(synth.wave_trajectory(w, synth.perturbed_wave(w, 0.05, 1), lines=lines)).cuda()
    k2 = torch.from_numpy(synth.wave_trajectory(w, synth.perturbed_wave(w, 0.05, 2), lines=lines)).cuda()
    v = torch.from_numpy(x.reshape(1, -1)).cuda()
    grads = []
    for between in (False, True):
        k = k1.clone().requires_grad_(True)
        q = ag.apply_a(r, v, k)
        if between:
            ag.apply_a(r, v, k2)
        q.backward(v)
        grads.append(k.grad.cpu().numpy())
    assert np.abs(grads[0]).max() > 0
    assert np.array_equal(grads[0], grads[1])
