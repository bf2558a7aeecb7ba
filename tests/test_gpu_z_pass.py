"""The pipelined z passes (coil maps; the half-line form and the general one)
against the plain ones (per-coil images): with a map of ones on one coil and
zeros on the others, E^H E of an image is that coil's forward and adjoint
transform, every product exact, so the results must agree bit for bit.  And
the solve whose forward z pass applies the CG updates against the solve with a
kernel per update."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

Z = [  # image and line length along z: split of the line
    (8, 16),      # 4 x 4, half of the line
    (20, 40),     # 8 x 5, odd split: half of the line in the general form
    (16, 32),     # 4 x 8
    (24, 48),     # 8 x 6, general form
    (50, 128),    # 8 x 16, less than half
    (32, 32),     # the whole line
    (96, 192),    # 16 x 12
    (98, 192),    # 16 x 12, more than half
    (160, 320),   # 16 x 20, 8 lines per block
    (176, 352),   # 32 x 11
    (224, 448),   # 16 x 28
]


def make(cgs, iz, gz, nch, seed):
    rng = np.random.default_rng(seed)
    img, grid = (7, 9, iz), (16, 24, gz)     # lines left over in the last block
    k = rng.uniform(0, 1, (400, 3))
    r = cgs.Reco(img, grid, nch, kb_w=4.0, kb_b=9.0)
    r.set_trajectory(k)
    return r, rng, img


@pytest.mark.parametrize("iz,gz", Z)
@pytest.mark.parametrize("coil", [0, 2])
def test_pipelined_z_passes_equal_plain_ones_bitwise(gpu_lib, cgs, iz, gz, coil):
    nch = 3
    r, rng, img = make(cgs, iz, gz, nch, 31)
    maps = np.zeros((nch,) + img, np.complex64)
    maps[coil] = 1
    r.set_smaps(maps)
    x = (rng.standard_normal(img) + 1j * rng.standard_normal(img)).astype(np.complex64)
    xs = np.zeros_like(maps)
    xs[coil] = x
    want = r.nufft_adj(r.nufft_fwd(xs))[coil]
    got = r.apply_ehde(x)
    assert np.abs(want).max() > 0
    assert np.array_equal(got, want)


@pytest.mark.parametrize("iz,gz", [z for z in Z if z[1] in (16, 32, 192, 320)])
def test_fused_cg_updates_in_the_half_line_form(gpu_lib, cgs, iz, gz):
    import torch
    nch, iters = 2, 5
    r, rng, img = make(cgs, iz, gz, nch, 32)
    r.set_smaps((rng.standard_normal((nch,) + img) + 1j * rng.standard_normal((nch,) + img)).astype(np.complex64))
    r.set_bins([np.arange(0, 250), np.arange(250, 400)])
    stream = torch.cuda.Stream()
    r.set_stream(stream.cuda_stream)
    with torch.cuda.stream(stream):
        d = torch.from_numpy((rng.standard_normal((nch, 400)) + 1j * rng.standard_normal((nch, 400))).astype(np.complex64)).cuda()
        xf = torch.zeros((2,) + img, dtype=torch.complex64, device="cuda")
        xs = torch.zeros_like(xf)
        tr = torch.zeros((iters, 2) + img, dtype=torch.complex64, device="cuda")
    stream.synchronize()
    resf, _ = r.cg_sense_batched_tensor(d, xf, 0.0, iters)
    ress, _ = r.cg_sense_trace_tensor(d, xs, 0.0, iters, tr)
    stream.synchronize()
    assert np.array_equal(resf, ress)
    assert torch.equal(xf, xs) and torch.count_nonzero(xf[1]) > 0
    r.close()
