"""Set-ups in which the sliced tap matrix does not fit: the rows take its place."""
import glob
import importlib
import os
import subprocess
import sys
import textwrap

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fake_lib(gpu_lib, cgs, tmp_path_factory):
    """The library's objects linked with an allocator that can be told to fail."""
    build = importlib.import_module("4d_lung_gb300.build")
    d = tmp_path_factory.mktemp("fake")
    shim, out = str(d / "shim.o"), str(d / "libcgsense.so")
    subprocess.run(["g++", "-O1", "-fPIC", "-I", "/usr/local/cuda/include", "-c",
                    os.path.join(ROOT, "tests", "drivers", "fake_malloc.cpp"), "-o", shim], check=True)
    objs = [o for o in glob.glob(os.path.join(build.BUILD, "*.o")) if not o.endswith("torch_ops.o")]
    subprocess.run([build.NVCC] + build.ARCH + ["-shared", "-o", out, shim] + objs +
                   ["-cudart", "static", "-lcufft", "-lgomp", "-ldl", "-Xlinker", "--wrap=cudaMalloc",
                    "-Xlinker", "-rpath,/usr/local/cuda/lib64"], check=True)
    return out


_RUN = textwrap.dedent("""
    import importlib, sys
    import numpy as np
    sys.path.insert(0, sys.argv[1])
    cgs = importlib.import_module("4d_lung_gb300")
    cgs.LIB_PATH = sys.argv[2]
    L = cgs.lib()
    nch = int(sys.argv[3])
    rng = np.random.default_rng(12)
    img, grid = (32, 16, 12), (64, 32, 24)
    k = np.concatenate([rng.uniform(0, 1, (600, 3)), 0.5 + 0.02 * rng.standard_normal((200, 3))])
    maps = (rng.standard_normal((nch,) + img) + 1j * rng.standard_normal((nch,) + img)).astype(np.complex64)
    x = (rng.standard_normal(img) + 1j * rng.standard_normal(img)).astype(np.complex64)
    y = (rng.standard_normal((nch, 800)) + 1j * rng.standard_normal((nch, 800))).astype(np.complex64)

    def ready():
        L.fake_malloc_fail(-1)
        r = cgs.Reco(img, grid, nch, kb_w=4.0, kb_b=9.0)
        r.set_trajectory(k)
        r.set_smaps(maps)
        L.fake_malloc_fail(-1)
        return r

    def outputs(r):
        return [r.apply_ehde(x), r.nufft_adj(y), r.cg_sense(y, 0.0, 3)[0], r.pipe_menon_dcf(4)]

    r = ready()
    r.apply_ehde(x)
    n = L.fake_malloc_count()
    want = outputs(r)
    points = r.spread_matrix_stats()
    survived = 0
    for i in range(n):
        r = ready()
        L.fake_malloc_fail(i)
        try:
            q = r.apply_ehde(x)
        except cgs.CGSError:
            continue
        L.fake_malloc_fail(-1)
        assert np.array_equal(q, want[0]), i
        assert all(np.array_equal(a, b) for a, b in zip(outputs(r), want)), i
        r.set_launch_shape(0, 1, 2)
        r.set_launch_shape(0, 6, 2)
        assert all(np.array_equal(a, b) for a, b in zip(outputs(r), want)), i
        survived += 1
    print("allocations", n, "survived", survived)
    assert survived >= 5
""")


@pytest.mark.parametrize("nch", [3, 4])
def test_a_failed_allocation_of_the_slices_falls_back_to_rows(fake_lib, nch):
    """Each allocation of a set-up fails once in turn: with those of the slices
    (offsets, order, headers, line masks, entries) the call still succeeds, over
    rows (fused with the adjoint x pass at 4 coils, unfused at 3), and all results
    keep their bits, as any spreading does."""
    r = subprocess.run([sys.executable, "-c", _RUN, ROOT, fake_lib, str(nch)], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_slices_that_are_mostly_padding_give_way_to_rows(gpu_lib, cgs):
    """All samples at one place: 64 points hold all taps, 8 of them in a tile, and
    slices of 32 points would take four times the rows' memory."""
    rng = np.random.default_rng(13)
    img, grid, nch, n = (32, 16, 12), (64, 32, 24), 4, 1500
    y = (rng.standard_normal((nch, n)) + 1j * rng.standard_normal((nch, n))).astype(np.complex64)
    # four taps an axis, those along z in two tiles of 8 columns (14, 15 and 16, 17)
    at = np.array([31.5, 15.5, 15.5]) / (np.array(grid) - 1)
    maps = (rng.standard_normal((nch,) + img) + 0j).astype(np.complex64)
    out = []
    for variant in (0, 1):
        r = cgs.Reco(img, grid, nch, kb_w=4.0, kb_b=9.0)
        r.set_trajectory(np.tile(at, (n, 1)))
        r.set_smaps(maps)
        if variant:
            r.set_launch_shape(0, variant, 2)
        out.append(r.nufft_adj(y))
        if not variant:
            assert r.spread_fused()
    assert np.abs(out[0]).max() > 0
    assert np.array_equal(out[0], out[1])
    # the next trajectory gets its slices again
    r = cgs.Reco(img, grid, nch, kb_w=4.0, kb_b=9.0)
    r.set_trajectory(np.tile(at, (n, 1)))
    r.nufft_adj(y)
    assert r.spread_fused()
    r.set_trajectory(rng.uniform(0, 1, (n, 3)))
    r.nufft_adj(y)
    assert not r.spread_fused()
