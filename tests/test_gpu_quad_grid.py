"""The forward grid in quads of coils (three coils or more) against coil
planes (one coil): every coil goes through the same operations in the same
order in either form, so the samples must agree bit for bit.  Sizes at the
edges of the quad x pass: one padded and one full quad, image lines in one and
two copies, 4- and 8-column units, half-pruned lines and general ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [
    ((16, 16, 12), (32, 32, 24), 3, 4.0),      # the smallest line, 3 of 4 coils
    ((32, 24, 20), (64, 48, 40), 4, 4.25),     # 5 candidates on some axes
    ((33, 17, 13), (64, 32, 24), 5, 4.0),      # odd image, a quad of one coil
    ((75, 16, 12), (128, 32, 24), 9, 4.25),    # general line, three quads
    ((128, 16, 12), (256, 32, 24), 4, 4.0),    # half-pruned, 8-column units
    ((160, 16, 12), (320, 32, 24), 6, 4.0),    # half-pruned, 4-column units
    ((300, 16, 12), (320, 32, 24), 3, 4.0),    # input rows in two copies
    ((88, 16, 12), (176, 32, 24), 4, 4.0),     # R2 odd
    ((176, 16, 12), (352, 32, 24), 3, 4.0),    # R1 = 32
]


@pytest.mark.parametrize("img,grid,nch,kb_w", CASES)
@pytest.mark.parametrize("pruned", [True, False])
def test_quads_equal_coil_planes_bitwise(gpu_lib, cgs, img, grid, nch, kb_w, pruned):
    rng = np.random.default_rng(5)
    # a cluster of samples, some at the faces of the grid
    k = np.concatenate([0.5 + 0.2 * rng.standard_normal((700, 3)).clip(-2, 2), rng.uniform(0, 1, (100, 3))])
    k[:6] = [[0, 0, 0], [1, 1, 1], [0, 1, 0.5], [1, 0, 0.5], [0.5, 0, 1], [0.5, 1, 0]]
    x = (rng.standard_normal((nch,) + img) + 1j * rng.standard_normal((nch,) + img)).astype(np.complex64)
    kw = dict(kb_w=kb_w, kb_b=9.0)
    r = cgs.Reco(img, grid, nch, **kw)
    r.set_trajectory(k)
    r.set_support_pruning(pruned)
    one = cgs.Reco(img, grid, 1, **kw)
    one.set_trajectory(k)
    one.set_support_pruning(pruned)
    y = r.nufft_fwd(x)
    assert np.isfinite(y).all() and np.abs(y).max() > 0
    for c in range(nch):
        assert np.array_equal(y[c], one.nufft_fwd(x[c:c + 1])[0]), c
    # every coils-per-thread form
    for cc in (1, 2, 4):
        r.set_launch_shape(0, 8, cc)
        assert np.array_equal(r.nufft_fwd(x), y), cc


@pytest.mark.parametrize("img,grid,nch,kb_w", CASES)
@pytest.mark.parametrize("compensated", [False, True])
def test_sliced_gather_equals_tiled_kernel_bitwise(gpu_lib, cgs, img, grid, nch, kb_w, compensated):
    """The gather over the sliced matrix and the adjoint x pass from the quad
    grid against the tiled spreading kernel and the pass from coil planes, with
    a crowded spot (slices of very different lengths) and two bins."""
    rng = np.random.default_rng(6)
    k = np.concatenate([0.5 + 0.15 * rng.standard_normal((500, 3)).clip(-3, 3), rng.uniform(0, 1, (100, 3)),
                        0.5 + 0.002 * rng.standard_normal((300, 3))])
    k[:6] = [[0, 0, 0], [1, 1, 1], [0, 1, 0.5], [1, 0, 0.5], [0.5, 0, 1], [0.5, 1, 0]]
    y = (rng.standard_normal((nch, len(k))) + 1j * rng.standard_normal((nch, len(k)))).astype(np.complex64)
    maps = (rng.standard_normal((nch,) + img) + 1j * rng.standard_normal((nch,) + img)).astype(np.complex64)
    r = cgs.Reco(img, grid, nch, kb_w=kb_w, kb_b=9.0)
    r.set_trajectory(k)
    r.set_smaps(maps)
    r.set_precision(compensated)
    got = r.nufft_adj(y)
    r.set_launch_shape(0, 6, 2)
    assert np.array_equal(got, r.nufft_adj(y))
    r.set_launch_shape(0, 1, 2)
    assert np.abs(got).max() > 0
    assert np.array_equal(got, r.nufft_adj(y))
    r.set_bins([np.arange(0, 450), np.arange(450, 900)])
    r.set_launch_shape(0, 6, 2)
    x6, res6, _ = r.cg_sense_batched(y, 0.0, 3)
    r.set_launch_shape(0, 1, 2)
    x1, res1, _ = r.cg_sense_batched(y, 0.0, 3)
    assert np.array_equal(x6, x1) and np.array_equal(res6, res1)


@pytest.mark.parametrize("nch,coil", [(3, 2), (4, 1), (5, 4), (9, 6)])
@pytest.mark.parametrize("kb_w", [4.0, 4.25])
@pytest.mark.parametrize("ns", [1, 33, 800])
def test_quad_loss_gradients_equal_coil_planes(gpu_lib, cgs, nch, coil, kb_w, ns):
    """Loss, dL/dk and dL/dx with one coil's map and data non-zero against a
    single-coil reconstruction (coil planes): warps whose samples all hold four
    candidates an axis and others, at the grid's faces, part-filled warps and
    blocks.  The residual and the derivative sums are the same bits; the loss
    adds them in FP64 in another order (1e-12) and dL/dk rounds two products and
    their sum per coil (a few 6e-8: 1e-6)."""
    import torch
    rng = np.random.default_rng(8)
    img, grid = (16, 16, 12), (32, 32, 24)
    k = rng.uniform(0, 1, (ns, 3))
    k[:6] = np.array([[0, 0, 0], [1, 1, 1], [0, 1, 0.5], [1, 0, 0.5], [0.5, 0, 1], [0.5, 1, 0]])[:min(ns, 6)]
    one = (rng.standard_normal(img) + 1j * rng.standard_normal(img)).astype(np.complex64)
    maps = np.zeros((nch,) + img, np.complex64)
    maps[coil] = one
    y = np.zeros((nch, ns), np.complex64)
    y[coil] = rng.standard_normal(ns) + 1j * rng.standard_normal(ns)
    x = torch.from_numpy((rng.standard_normal(img) + 1j * rng.standard_normal(img)).astype(np.complex64)).cuda()
    dcf = rng.uniform(0.5, 1.5, ns).astype(np.float32)
    got = []
    for n, m, d in ((nch, maps, y), (1, maps[coil:coil + 1], y[coil:coil + 1])):
        r = cgs.Reco(img, grid, n, kb_w=kb_w, kb_b=9.0)
        r.set_trajectory(k)
        r.set_dcf(dcf)
        r.set_smaps(m)
        gx = torch.zeros_like(x)
        gk = torch.zeros((ns, 3), dtype=torch.float32, device="cuda")
        loss = r.loss_grad_tensor(x, torch.from_numpy(np.ascontiguousarray(d)).cuda(), gx, gk)
        got.append((loss, gx.cpu().numpy(), gk.cpu().numpy()))
    (la, xa, ka), (lb, xb, kb) = got
    assert lb > 0 and np.abs(kb).max() > 0
    assert abs(la - lb) < 1e-12 * lb
    assert np.array_equal(xa, xb)
    assert np.linalg.norm(ka - kb) < 1e-6 * np.linalg.norm(kb)
