"""Failure detection without a GPU fault.

* A bounded barrier wait that runs out: with AWP_TEST_TMA_WITHHOLD the producer
  warp of block 0 in the staged stress sweep issues no copies (and no arrival)
  for one ring use, so the consumers waiting on that slot give up after the
  wait limit (AWP_TEST_WAIT_US, here 20 ms).  The block's other copies land
  before it exits; the solve reports AWP_ERR_TIMEOUT; the context stays usable
  and the next solve is bit-exact with the oracle.
* A device allocation that fails (AWP_TEST_FAIL_ALLOC = n: the n-th allocation
  of a solver): AWP_ERR_OOM, everything allocated so far is released, and
  the next solver works.
* A device on which a solve just fits (AWP_TEST_DEVICE_BYTES: allocations fail
  once the process's blocks would pass that many bytes): it runs without
  padded rows, wherever the memory runs out.
Nothing here traps, faults or hangs a GPU, or fills its memory.
"""
import gc

import numpy as np
import pytest

import awpsgt

from test_gpu_parity import Case, assert_same_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncomp,kernel_name", [(3, "k_str_tmab"), (1, "k_str_tma")])
def test_withheld_tile_copy_times_out_then_next_solve_is_exact(monkeypatch, ncomp, kernel_name):
    c = Case(nt=30, igreen=(1, 2, 3)[:ncomp], srcs=[[(24, 20, 10)]] * ncomp)
    monkeypatch.setenv("AWP_TEST_TMA_WITHHOLD", "5")
    monkeypatch.setenv("AWP_TEST_WAIT_US", "20000")
    with pytest.raises(awpsgt.AwpError) as e:
        c.gpu(kernel="staged")
    assert awpsgt.STATUS[e.value.status] == "AWP_ERR_TIMEOUT"
    assert "barrier wait ran out" in str(e.value)
    monkeypatch.delenv("AWP_TEST_TMA_WITHHOLD")
    monkeypatch.delenv("AWP_TEST_WAIT_US")
    s = c.gpu(steps=5, kernel="staged")
    assert s.profile(1)[kernel_name]["launches"] == 1       # the stress sweep the injection exercised
    s.close()
    s = c.gpu(kernel="staged")
    for q in range(ncomp):
        assert_same_state(s, c.oracle(q), q)


@pytest.mark.parametrize("nth", [1, 7, 20])
def test_failed_allocation_is_oom_and_releases_everything(monkeypatch, nth):
    c = Case(nt=20)
    gc.collect()                                      # solvers of earlier tests released first
    live0, _ = awpsgt.device_memory(0)
    monkeypatch.setenv("AWP_TEST_FAIL_ALLOC", str(nth))
    p = awpsgt.make_params(c.nx, c.ny, c.nz, c.dh, c.dt, c.nt, igreen=c.igreen, **c.kw())
    with pytest.raises(awpsgt.AwpError) as e:
        awpsgt.Solver(p)
    assert awpsgt.STATUS[e.value.status] == "AWP_ERR_OOM"
    assert "AWP_TEST_FAIL_ALLOC" in str(e.value)
    assert awpsgt.device_memory(0)[0] == live0          # every block of the failed solver released
    monkeypatch.delenv("AWP_TEST_FAIL_ALLOC")
    s = c.gpu()
    assert awpsgt.device_memory(0)[0] > live0
    assert_same_state(s, c.oracle())
    assert np.abs(s.sgt()).max() > 0
    s.close()
    assert awpsgt.device_memory(0)[0] == live0


def test_failed_sgt_staging_is_oom(monkeypatch):
    """The staging block of awp_get_sgt_rwg is the first allocation after a
    solve is set up: made to fail there, the call reports AWP_ERR_OOM and the
    next one works."""
    c = Case(nt=20)
    want = c.gpu().sgt_rwg(0, z_source=False)
    for nth in range(10, 200):
        monkeypatch.setenv("AWP_TEST_FAIL_ALLOC", str(nth))
        try:
            s = c.gpu()
        except awpsgt.AwpError as e:
            assert awpsgt.STATUS[e.status] == "AWP_ERR_OOM"
            continue
        try:                                # a set-up call may have tried again without row padding
            s.sgt_rwg(0, z_source=False)
            continue
        except awpsgt.AwpError as e:
            assert awpsgt.STATUS[e.status] == "AWP_ERR_OOM"
        assert np.array_equal(s.sgt_rwg(0, z_source=False), want)
        return
    raise AssertionError("no allocation of a solve was made to fail")


def device_pitch(s):
    return s.device_field("u1", 0)[1].pitch


# where the padded rows no longer fit: in awp_create, in the media, in the SGT images
@pytest.mark.parametrize("nx,ny,nz,npts,nt,kw", [
    (14, 280, 260, 10, 12, {}),
    (100, 200, 100, 50, 12, {}),
    (100, 200, 100, 50, 12, dict(precision="f16")),
    (100, 200, 100, 12000, 240, {}),
    (100, 200, 100, 12000, 240, dict(precision="bfp")),
    (100, 200, 100, 12000, 240, dict(npc=1, nd=10)),
])
def test_solve_that_just_fits_runs_without_row_padding(monkeypatch, nx, ny, nz, npts, nt, kw):
    kw = dict(kw)
    prm = dict(igreen=(1, 2, 3), nst=nt - 1, ntiskp_sgt=1, write_step=10, nd=3)
    prm.update(kw)
    p = awpsgt.make_params(nx, ny, nz, 200.0, 0.01, nt, **prm)
    rng = np.random.default_rng(3)
    media = np.empty((nz, ny, nx, 3), np.float32)
    media[..., 0], media[..., 1], media[..., 2] = 4800.0, 2800.0, 2500.0
    media *= 1.0 + 0.05 * rng.random((nz, ny, nx, 1), dtype=np.float32)
    pts = np.stack([rng.integers(1, n + 1, npts) for n in (nx, ny, nz)], 1)
    stf = rng.standard_normal((1, nt - 1, 6)).astype(np.float32)

    def solve(points_first):
        s = awpsgt.Solver(p)
        if points_first:
            s.set_points(pts)
        s.load_media(media)
        for q in range(3):
            s.set_source(q, [(nx // 2, ny // 2, 20)], stf)
        if not points_first:
            s.set_points(pts)
        s.run(12)
        return s

    gc.collect()
    awpsgt.release_cached_memory()
    live0, _ = awpsgt.device_memory(0)
    s = solve(False)
    narrow = (nx + 10 + 7) // 8 * 8
    assert device_pitch(s) == (nx + 10 + 31) // 32 * 32 > narrow
    want = [(s.sgt(q), s.chkj(q), s.field("xy", q)) for q in range(3)]
    s.close()
    awpsgt.release_cached_memory()
    # the footprint's allowance for media staging and small buffers is 64 MiB; two slabs are 46 MiB at most here,
    # and the padding adds 54 MiB at least
    monkeypatch.setenv("AWP_TEST_DEVICE_BYTES", str(live0 + awpsgt.footprint_bytes(p, npts) - (12 << 20)))
    for points_first in (False, True):
        s = solve(points_first)
        assert device_pitch(s) == narrow
        for q in range(3):
            for a, b in zip((s.sgt(q), s.chkj(q), s.field("xy", q)), want[q]):
                assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
        s.close()
        awpsgt.release_cached_memory()
    assert awpsgt.device_memory(0) == (live0, 0)


def test_solver_goes_on_after_a_refused_allocation():
    """SGT images of 7 TB: cudaMalloc refuses them at once.  The call reports
    it, and the solver (its rows no longer padded) and later launches are not
    affected by the error."""
    c = Case(nx=100, ny=40, nz=32, nt=30, srcs=[[(50, 20, 10)]])
    p = awpsgt.make_params(c.nx, c.ny, c.nz, c.dh, c.dt, 300000, igreen=c.igreen,
                           **dict(c.kw(), nst=c.nt, ntiskp_sgt=1, write_step=10))
    s = awpsgt.Solver(p)
    s.load_media(c.media)
    s.set_source(0, c.srcs[0], c.stfs[0])
    with pytest.raises(awpsgt.AwpError) as e:
        s.set_points(np.ones((1000000, 3), np.int32))
    assert awpsgt.STATUS[e.value.status] == "AWP_ERR_OOM"
    s.run(c.nt)
    ref = c.gpu()
    for f in ("u1", "xx", "xy", "r4"):
        assert np.array_equal(s.field(f).view(np.uint32), ref.field(f).view(np.uint32)), f


@pytest.mark.parametrize("how", ["set_field", "device_field"])
def test_written_fields_survive_the_change_of_rows(monkeypatch, how):
    """A wavefield set before the SGT images no longer fit keeps its values;
    after a device pointer has been handed out the arrays stay where they are
    and the failure is reported."""
    c = Case(nx=100, ny=60, nz=40, nt=240, igreen=(1,), srcs=[[(50, 30, 10)]])
    npts = 12000
    pts = np.stack([np.random.default_rng(5).integers(1, n + 1, npts) for n in (c.nx, c.ny, c.nz)], 1)
    p = awpsgt.make_params(c.nx, c.ny, c.nz, c.dh, c.dt, c.nt, igreen=c.igreen,
                           **dict(c.kw(), ntiskp_sgt=1, write_step=10))
    u = np.random.default_rng(6).standard_normal((c.nz + 4, c.ny + 4, c.nx + 4)).astype(np.float32)

    def solve():
        s = awpsgt.Solver(p)
        s.load_media(c.media)
        s.set_source(0, c.srcs[0], c.stfs[0])
        if how == "set_field":
            s.set_field("u1", u, 0)
        else:
            device_pitch(s)
        live = awpsgt.device_memory(0)[0]
        s.set_points(pts)
        s.run(10)
        return s, live

    gc.collect()
    awpsgt.release_cached_memory()
    s, live = solve()
    want, after = [s.field(f) for f in ("u1", "xx", "r1")], awpsgt.device_memory(0)[0]
    s.close()
    awpsgt.release_cached_memory()
    # room for the narrow arrays and the SGT images, less than the padding short of the padded ones
    monkeypatch.setenv("AWP_TEST_DEVICE_BYTES", str(after - (1 << 20)))
    if how == "device_field":
        with pytest.raises(awpsgt.AwpError) as e:
            solve()
        assert awpsgt.STATUS[e.value.status] == "AWP_ERR_OOM"
        return
    s, _ = solve()
    assert device_pitch(s) == 112 and after > live
    for a, b in zip([s.field(f) for f in ("u1", "xx", "r1")], want):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
