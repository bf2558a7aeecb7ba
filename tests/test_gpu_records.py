"""Tap records over the kernel shapes: the power series of the Bessel factor on
float pairs (up to b = 19 or so) and the library function beyond, against the
FP64 oracle.  The weights are rounded to float in either form, as the oracle
rounds its own, so the tolerance is that of the forward operator (FP32 FFT)."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kb_w,kb_b", [(4.0, 0.0), (4.0, 0.5), (3.0, 5.0), (4.0, 8.9962), (4.25, 14.9086),
                                       (4.9, 18.5), (4.9, 24.0)])
def test_forward_and_gradient_over_kernel_shapes(gpu_lib, cgs, oracle_mod, o64, kb_w, kb_b):
    import torch
    img, grid, nch = (16, 16, 12), (32, 32, 24), 3
    rng = np.random.default_rng(4)
    k = rng.uniform(0.05, 0.95, (400, 3))
    x = (rng.standard_normal((nch,) + img) + 1j * rng.standard_normal((nch,) + img)).astype(np.complex64)
    p = oracle_mod.make_params(img, grid, nch, kb_w=kb_w, kb_b=kb_b)
    r = cgs.Reco(img, grid, nch, kb_w=kb_w, kb_b=kb_b)
    r.set_trajectory(k)
    kft = o64.kernel_ft(p)
    assert rel_l2(r.nufft_fwd(x), o64.nufft_fwd(p, o64.taps(p, k), kft, x)) < 2e-5
    # derivative records: dL/dk against the FP64 form of the same library, whose
    # distances are not rounded to float (2e-3, as the gradient tests)
    if kb_b < 10:
        return
    maps = x / np.sqrt(np.sum(np.abs(x) ** 2, axis=0))
    r.set_smaps(maps.astype(np.complex64))
    xt = torch.from_numpy(x[0]).cuda()
    y = torch.zeros((nch, 400), dtype=torch.complex64, device="cuda")
    g32 = torch.zeros((400, 3), dtype=torch.float32, device="cuda")
    g64 = torch.zeros((400, 3), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    l32 = r.loss_grad_tensor(xt, y, grad_k=g32)
    l64 = r.loss_grad_fp64_tensor(xt.to(torch.complex128), y, grad_k=g64)
    assert abs(l32 - l64) / l64 < 1e-4
    assert rel_l2(g32.cpu().numpy(), g64.cpu().numpy()) < 2e-3
