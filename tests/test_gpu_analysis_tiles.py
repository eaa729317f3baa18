"""The field analysis where its grouping of cells can go wrong.

Labelling takes four consecutive cells per thread or four rows of 32 per warp (the larger boxes' merge):
random masks put several drops into one group of four and dozens into one warp.  The diagnostics march 32 x 16 tiles and the spectrum
sums runs of equal shells in a warp: boxes that leave partial tiles, rows shorter than a warp and
more shells than eight warps' histograms hold.  Sums of N terms in FP64 against numpy's: 1e-12.
"""
import math

import numpy as np
import pytest

from mhit36_mixedp_b200 import Params, Solver, synth
from oracle import mhit_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("conn", [6, 26])
@pytest.mark.parametrize("shape,fill", [((16, 16, 16), 0.1), ((64, 16, 32), 0.3), ((192, 16, 16), 0.05),
                                        ((256, 64, 256), 0.05)])
def test_labels_of_random_masks(gpu, shape, fill, conn):
    nx, ny, nz = shape
    rng = np.random.default_rng(11)
    phi = (rng.random((nz, ny, nx)) < fill).astype(np.float64)
    u, v, w = (rng.standard_normal((nz, ny, nx)) for _ in range(3))
    with Solver(Params(nx=nx, ny=ny, nz=nz, phiflag=1)) as s:
        s.upload(u, v, w, phi)
        got = s.label_drops(0.5, conn, labels=True)
    lab = orc.label_components(phi, 0.5, conn)
    ref = orc.drop_statistics(lab, u, v, w)
    expect = np.where(lab >= 0, np.searchsorted(ref["label"], lab) + 1, 0)  # roots in index order
    np.testing.assert_array_equal(got["labels"], expect)
    np.testing.assert_array_equal(got["cells"], ref["cells"])
    for key in ("u", "v", "w"):
        assert np.max(np.abs(got[key] - ref[key])) < 1e-12, key


def test_every_masked_cell_is_counted_in_every_call(gpu):
    n = 256
    z = np.zeros((n, n, n))
    with Solver(Params(nx=n, phiflag=1)) as s:
        s.upload(z, z, z, z)
        s.init_drops(synth.drop_centres(64, 3), 0.3)
        mask = int((s.download(("phi",))["phi"] >= 0.5).sum())
        first = s.label_drops(0.5, 6)["cells"]
        assert int(first.sum()) == mask
        for _ in range(30):
            np.testing.assert_array_equal(s.label_drops(0.5, 6)["cells"], first)


@pytest.mark.parametrize("shape", [(16, 16, 16), (32, 64, 16), (192, 16, 64)])
def test_diagnostics_and_spectrum_of_ragged_boxes(gpu, shape):
    nx, ny, nz = shape
    dx = 2 * math.pi / nx
    u, v, w = synth.solenoidal_velocity(nx, 3, ny=ny, nz=nz)
    with Solver(Params(nx=nx, ny=ny, nz=nz, mu=0.004)) as s:
        s.upload(u, v, w)
        d = s.diagnostics()
        E, E8 = s.energy_spectrum(4096), s.energy_spectrum(8)
    div = ((orc.xp(u) - u) + (orc.yp(v) - v) + (orc.zp(w) - w)) / dx
    scale = np.max(np.abs(u)) / dx
    assert abs(d["maxdiv"] - np.max(np.abs(div))) <= 1e-12 * scale
    ke = 0.5 * np.mean(u * u + v * v + w * w)
    assert abs(d["ke"] - ke) <= 1e-12 * ke
    eps = orc.dissipation(u, v, w, 0.004, dx)
    assert abs(d["dissipation"] - eps) <= 1e-12 * eps
    ref = orc.energy_spectrum(u, v, w, 4096)
    assert np.max(np.abs(E - ref)) <= 1e-12 * ref.sum()
    assert np.max(np.abs(E8 - ref[:8])) <= 1e-12 * ref.sum()
