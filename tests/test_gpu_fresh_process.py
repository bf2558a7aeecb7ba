"""A context sets up the passes of its own line lengths only: a process whose first
context has lengths 192, 32 and 24 builds its Toeplitz spectra over lines of 384
(more than 48 KiB of shared memory), and a second context brings 512."""
import subprocess
import sys
import textwrap

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

_RUN = textwrap.dedent("""
    import importlib, sys
    import numpy as np
    sys.path.insert(0, sys.argv[1])
    cgs = importlib.import_module("4d_lung_gb300")
    rng = np.random.default_rng(2)
    c64 = lambda *d: (rng.standard_normal(d) + 1j * rng.standard_normal(d)).astype(np.complex64)
    rel = lambda a, b: np.linalg.norm(a - b) / np.linalg.norm(b)
    img, nch = (96, 8, 6), 3
    r = cgs.Reco(img, (192, 32, 24), nch, kb_w=4.0, kb_b=9.0)
    r.set_trajectory(rng.uniform(0.1, 0.9, (500, 3)))
    r.set_smaps(c64(nch, *img))
    x = c64(*img)
    r.set_toeplitz(1)
    a = r.apply_ehde(x)
    assert r.toeplitz_spectrum_method() == 1
    r.set_toeplitz_spectrum(1)
    b = r.apply_ehde(x)
    assert r.toeplitz_spectrum_method() == 2
    assert rel(a, b) < 1e-5, rel(a, b)     # the two builds of the spectrum, as in the Toeplitz tests
    r = cgs.Reco((300, 8, 6), (512, 16, 16), nch, kb_w=4.0, kb_b=9.0)
    k = rng.uniform(0, 1, (500, 3))
    r.set_trajectory(k)
    y = c64(nch, 500)
    v = r.nufft_adj(y)
    r.set_launch_shape(0, 1, 2)
    assert np.array_equal(v, r.nufft_adj(y)) and np.abs(v).max() > 0
""")


def test_lengths_are_set_up_where_they_are_first_used(gpu_lib):
    r = subprocess.run([sys.executable, "-c", _RUN, ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
