"""Phase and momentum stages on boxes whose tiles and z chunks do not divide the grid.

The stencils march tiles of x-y cells over chunks of z planes chosen from the grid size; these boxes
leave a partial last tile in x or y, a short last chunk, or a chunk of two planes.  Each stage is one
FP64 evaluation of the oracle's expressions, so the usual 1e-12 of the buffer's maximum applies.  The
stages run twice: the first step is an Euler step with an empty history, the second (Adams-Bashforth)
reads the right-hand sides of the first.
"""
import numpy as np
import pytest

from mhit36_mixedp_b200 import Params, Solver, _lib, synth
from oracle import mhit_oracle as orc

pytestmark = pytest.mark.gpu
TOL = 1e-12


def rel(a, b):
    return float(np.max(np.abs(a - b)) / np.max(np.abs(b)))


@pytest.mark.parametrize("clamp", [0, 1])
@pytest.mark.parametrize("shape", [(16, 16, 16), (16, 64, 16), (64, 16, 128), (192, 64, 128), (32, 192, 64), (64, 128, 16),
                                   (128, 32, 64), (192, 16, 32), (256, 32, 16)])
def test_stencil_stages_on_ragged_boxes(gpu, shape, clamp):
    nx, ny, nz = shape
    dx = 2 * np.pi / nx
    u, v, w = synth.solenoidal_velocity(nx, 3, ny=ny, nz=nz)
    # one smooth interface that crosses every tile and chunk boundary, phi strictly inside (0, 1),
    # its critical points (where the normal has no direction) off the grid points; on boxes with an
    # axis of few cells it is wider, or phi leaves (0, 1) in the first step and psi becomes NaN
    z, y, x = np.meshgrid(*(np.arange(n) * 2 * np.pi / n for n in (nz, ny, nx)), indexing="ij")
    width = dx * max(1.0, nx / (4 * min(ny, nz)))
    phi = 0.5 * (1 - np.tanh((np.cos(x + 0.1) + np.cos(y + 0.13) + np.cos(z + 0.17)) / (2 * width)))
    prm = dict(nx=nx, ny=ny, nz=nz, dt=2e-4, mu=0.004, phiflag=1, sigma=0.3, acdi_clamp=clamp)
    op = orc.Params(**prm)
    st = orc.new_state(op, u, v, w, phi=phi)
    with Solver(Params(**prm)) as s:
        s.upload(u, v, w, phi)
        for step in range(2):
            orc.phase_step(op, st)
            s.run_stage("phase")
            assert rel(s.buffer("phin"), st.phi) < TOL, step
            assert rel(s.buffer("rphi"), st.rhsphi_o) < TOL, step
            orc.momentum_step(op, st, orc.forcing_tables(op))
            s.run_stage("momentum")
            for f, name in (("un", "u"), ("vn", "v"), ("wn", "w"), ("ru", "rhsu_o"), ("rv", "rhsv_o"), ("rw", "rhsw_o")):
                assert rel(s.buffer(f), getattr(st, name)) < TOL, (step, f)
            s.commit_step()


@pytest.mark.parametrize("tma", [1, 0])
def test_momentum_of_a_large_box_without_the_phase_field(gpu, tma):
    """From 2^25 cells on the single-phase momentum step has a kernel of its own; a flat box of that
    size, its rings filled by TMA boxes (where they need no wrap) and by copies."""
    nx, ny, nz = 1024, 1024, 32
    u, v, w = synth.solenoidal_velocity(nx, 3, ny=ny, nz=nz)
    prm = dict(nx=nx, ny=ny, nz=nz, dt=5e-5, mu=0.004)
    op = orc.Params(**prm)
    st = orc.new_state(op, u, v, w)
    with Solver(Params(**prm)) as s:
        assert _lib.load().mhit_debug_set_mom_tma(s._ctx, tma) == 0
        s.upload(u, v, w)
        s.run_stage("momentum")
        orc.momentum_step(op, st, orc.forcing_tables(op))
        for f, name in (("un", "u"), ("vn", "v"), ("wn", "w")):
            assert rel(s.buffer(f), getattr(st, name)) < TOL
        for f, name in (("ru", "rhsu_o"), ("rv", "rhsv_o"), ("rw", "rhsw_o")):
            assert rel(s.buffer(f), getattr(st, name)) < TOL


@pytest.mark.parametrize("tma", [1, 0])
def test_momentum_of_a_large_box_over_two_chunks(gpu, tma):
    """The large boxes' kernel over two z chunks and an Adams-Bashforth step: against the oracle, and
    bit for bit against the general kernel.  Without forcing, and periodic in half the box's y length,
    the box holds two copies of a box of half its cells, which takes the general kernel."""
    nx, ny, nz = 512, 512, 128
    u, v, w = synth.solenoidal_velocity(nx, 3, ny=ny // 2, nz=nz)
    prm = dict(nx=nx, nz=nz, dt=1e-4, mu=0.004, f1=0.0, f2=0.0, f3=0.0)
    op = orc.Params(ny=ny // 2, **prm)
    st = orc.new_state(op, u, v, w)
    twice = [np.concatenate([a, a], axis=1) for a in (u, v, w)]
    with Solver(Params(ny=ny, **prm)) as s, Solver(Params(ny=ny // 2, **prm)) as half:
        assert _lib.load().mhit_debug_set_mom_tma(s._ctx, tma) == 0
        s.upload(*twice)
        half.upload(u, v, w)
        for step in range(2):
            orc.momentum_step(op, st, orc.forcing_tables(op))
            for one in (s, half):
                one.run_stage("momentum")
            for f, name in (("un", "u"), ("vn", "v"), ("wn", "w"), ("ru", "rhsu_o"), ("rv", "rhsv_o"), ("rw", "rhsw_o")):
                h, got = half.buffer(f), s.buffer(f)
                assert rel(h, getattr(st, name)) < TOL, (step, f)
                np.testing.assert_array_equal(got[:, : ny // 2], h, err_msg=f)
                np.testing.assert_array_equal(got[:, ny // 2 :], h, err_msg=f)
            for one in (s, half):
                one.commit_step()


def test_phase_field_at_the_ends_of_the_logarithm(gpu):
    """Without the clamp, phi = -1e-16 makes psi = log(0) = -inf and a smaller one NaN, as in the
    reference; phi = 0, 1 and beyond 1 stay finite.  The stage must give NaN where the oracle does (the
    normal of an infinite psi difference) and the oracle's values everywhere else."""
    n = 32
    u, v, w = synth.solenoidal_velocity(n, 3)
    z, y, x = np.meshgrid(*(np.arange(n) * 2 * np.pi / n,) * 3, indexing="ij")
    dx = 2 * np.pi / n
    phi = 0.5 * (1 - np.tanh((np.cos(x + 0.1) + np.cos(y + 0.13) + np.cos(z + 0.17)) / (2 * dx)))
    for q, val in enumerate((-1e-16, -1e-15, -0.5, 0.0, 1.0, 1.0 + 2.0**-52, 1.5, 1e-300, 1e-17, 1.0 - 2.0**-53)):
        phi[16, 3 * q + 1, 7] = val
    op = orc.Params(nx=n, ny=n, nz=n, dt=2e-4, phiflag=1)
    st = orc.new_state(op, u, v, w, phi=phi)
    with np.errstate(all="ignore"):
        orc.phase_step(op, st)
    bad = np.isnan(st.rhsphi_o)
    assert 0 < bad.sum() < bad.size // 8
    with Solver(Params(nx=n, dt=2e-4, phiflag=1)) as s:
        s.upload(u, v, w, phi)
        s.run_stage("phase")
        for f, name in (("rphi", "rhsphi_o"), ("phin", "phi")):
            got, ref = s.buffer(f), getattr(st, name)
            np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
            assert rel(got[~bad], ref[~bad]) < TOL, f
