"""The staged sweeps at the edges of their tiles and z chunks, and kinematic
sources that fill several thread blocks, against the FP32 oracle."""
import numpy as np
import pytest

import awp_inputs as ai
import awpsgt
import oracle

from test_gpu_parity import Case, assert_same_state, kinematic_rupture, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz,igreen", [
    (8, 8, 8, (1,)), (31, 15, 9, (1,)), (32, 16, 10, (1, 2)), (33, 17, 11, (1, 2, 3)), (34, 31, 12, (3,)),
    (63, 33, 8, (1, 2)), (65, 18, 21, (2,)), (95, 47, 14, (1, 2, 3)),
])
def test_tile_and_chunk_edges_are_bit_exact(nx, ny, nz, igreen):
    """Pairs of cells cut by the grid's edge, partial tiles in x and y, chunks
    of the automatic rule down to five levels: every field, CHKJ and the SGT
    image bit for bit."""
    c = Case(nx=nx, ny=ny, nz=nz, nt=12, igreen=igreen, nd=3, npts=20,
             srcs=[[(nx // 2 + 1, ny // 2 + 1, nz // 2)]] * len(igreen), ntiskp=3, write_step=2)
    s = c.gpu(kernel="staged")
    for q in range(len(igreen)):
        assert_same_state(s, c.oracle(q), q)
    s.close()


@pytest.mark.parametrize("n", [1, 128, 129, 400])
def test_kinematic_subfaults_over_several_blocks(n):
    """One thread per cell that holds subfaults: block edges, and cells shared
    by many subfaults (every third one falls on one of four cells).  The
    tolerance is the kinematic parity test's: the CUDA and C-library sines and
    exponentials differ in the last bits."""
    nx, ny, nz, nt, dt = 48, 40, 32, 40, 0.01
    xyz = [(10 + k % 28, 12 + (k // 28) % 14, 6 + k % 9) for k in range(n)]
    xyz = [(20 + (k // 3) % 4, 20, 12) if k % 3 == 2 else c for k, c in enumerate(xyz)]
    tab = kinematic_rupture(n, dt=dt)
    media = ai.layered_media(nx, ny, nz, 200.0, seed=3, pert_std=0.05, corr_len=1000.0)
    pts = ai.sgt_points(nx, ny, 20, 50, seed=0)
    kw = dict(nd=8, socalq=1, ntiskp_sgt=5, write_step=4, fl=0.01, fh=25.0, fp=0.5)
    p = awpsgt.make_params(nx, ny, nz, 200.0, dt, nt, nst=2, igreen=(1,), kinematic=1, **kw)
    with awpsgt.Solver(p) as s:
        s.load_media(media)
        s.set_source(0, xyz, tab)
        s.set_points(pts)
        s.run(nt)
        g, gxx = s.sgt(0), s.field("xx")
    o = oracle.Oracle(nx=nx, ny=ny, nz=nz, dh=200.0, dt=dt, nt=nt, nst=2, igreen=1, kinematic=1, precision="f32", **kw)
    o.load_media(media)
    o.set_source(xyz, tab)
    o.set_points(pts)
    o.run(nt)
    assert np.abs(g).max() > 0
    assert rel_l2(g, o.sgt()) <= 1e-5
    assert rel_l2(gxx, o.field("xx")) <= 1e-5


@pytest.mark.parametrize("precision", ["f16", "bf16"])
@pytest.mark.parametrize("nx,ny,nz,igreen,nve", [
    (33, 17, 11, (1,), 1), (65, 18, 21, (1, 2), 1), (48, 40, 32, (1, 2, 3), 1), (31, 24, 9, (2, 3), 0),
])
def test_16bit_media_staged_equals_two_sweep(precision, nx, ny, nz, igreen, nve):
    """The default (staged) stepper with 16-bit media tiles against the plain
    two-sweep one, which reads the same arrays cell by cell: bit-identical."""
    c = Case(nx=nx, ny=ny, nz=nz, nt=12, igreen=igreen, nd=3, npts=20, nve=nve,
             srcs=[[(nx // 2 + 1, ny // 2 + 1, nz // 2)]] * len(igreen), ntiskp=3, write_step=2)
    a = c.gpu(precision=precision)
    b = c.gpu(precision=precision, kernel="two_sweep")
    assert "k_vel_tma" in a.profile(1) and "k_vel" in b.profile(1)
    for q in range(len(igreen)):
        for f in oracle.FIELDS:
            if f in ("qp", "qs") or (nve == 0 and f.startswith("r")):
                continue
            assert np.array_equal(a.field(f, q).view(np.uint32), b.field(f, q).view(np.uint32)), (f, q)
        assert np.array_equal(a.sgt(q), b.sgt(q))
    a.close()
    b.close()
