"""Failure detection on the GPU without a fault: a bounded wait that runs out.

With MPCF_TEST_DROP_LAST_COPY a non-persistent stage launch arms the
mbarrier of each z-chunk's last bulk copy without issuing the copy (a flag
that nothing sets).  The CTA's final bounded wait gives up, the kernel
records MPCF_ERRBIT_TMA_TIMEOUT and returns with no copy in flight, the
host reads the status, and the same context then runs a clean stage whose
results equal a fresh solver's."""
import numpy as np
import pytest

from conftest import cloud_state
from test_gpu_parity import assert_bitwise

pytestmark = pytest.mark.gpu


def test_bulk_copy_wait_runs_out_and_the_context_stays_usable(mpcf):
    dims = (32, 8, 12)             # one 32x8 tile, rows of 128 bytes: bulk copies
    U0 = cloud_state(dims, nb=1)
    with mpcf.Solver([dims], precision="fp32_ref") as s:
        s.set_tiling(8, 6, persistent=False, tma=True)
        s.set_state(U0)
        s.set_test_flags(mpcf._lib.TEST_DROP_LAST_COPY)
        s.stage(0.0, 0.25, 0.05)
        w = s.error_word(clear=True)
        assert w & mpcf._lib.ERRBIT_TMA_TIMEOUT, hex(w)
        # the context is usable: a clean stage from the same state
        s.set_test_flags(0)
        s.set_state(U0)
        s.stage(0.0, 0.25, 0.05)
        assert s.error_word() == 0
        U, R = s.get_state()
    with mpcf.Solver([dims], precision="fp32_ref") as f:
        f.set_tiling(8, 6, persistent=False, tma=True)
        f.set_state(U0)
        f.stage(0.0, 0.25, 0.05)
        Uf, Rf = f.get_state()
    assert_bitwise(U, Uf, "state after the timed-out stage")
    assert_bitwise(R, Rf, "register after the timed-out stage")


def test_no_copy_is_issued_after_a_give_up_and_none_is_left_in_flight(mpcf):
    """The chunk's first copy after the prologue is dropped: the wait one slab
    in runs out, the CTA issues no further copy (the count stops at the 3
    copies issued before: the prologue's two and the halo box issued with
    the dropped one), waits for that halo box before it exits (no
    MPCF_ERRBIT_TMA_INFLIGHT), and the context stays usable."""
    dims = (32, 8, 12)             # one 32x8 tile, two 6-slab chunks
    U0 = cloud_state(dims, nb=1)
    with mpcf.Solver([dims], precision="fp32_ref") as s:
        s.set_tiling(8, 6, persistent=False, tma=True)
        s.set_state(U0)
        # a clean launch with the counter on (the last copy dropped: one
        # copy fewer than the 13 per chunk of a full chunk)
        s.set_test_flags(mpcf._lib.TEST_DROP_LAST_COPY)
        s.test_copy_count(clear=True)
        s.stage(0.0, 0.25, 0.05)
        assert s.test_copy_count(clear=True) == 2 * 12
        s.error_word(clear=True)
        s.set_state(U0)
        s.set_test_flags(mpcf._lib.TEST_DROP_MID_COPY)
        s.stage(0.0, 0.25, 0.05)
        w = s.error_word(clear=True)
        assert w & mpcf._lib.ERRBIT_TMA_TIMEOUT, hex(w)
        assert not (w & mpcf._lib.ERRBIT_TMA_INFLIGHT), hex(w)
        assert s.test_copy_count(clear=True) == 2 * 3
        s.set_test_flags(0)
        s.set_state(U0)
        s.stage(0.0, 0.25, 0.05)
        assert s.error_word() == 0
        U, R = s.get_state()
    with mpcf.Solver([dims], precision="fp32_ref") as f:
        f.set_tiling(8, 6, persistent=False, tma=True)
        f.set_state(U0)
        f.stage(0.0, 0.25, 0.05)
        Uf, Rf = f.get_state()
    assert_bitwise(U, Uf, "state after the given-up stage")
    assert_bitwise(R, Rf, "register after the given-up stage")


def test_persistent_launches_ignore_the_test_flag(mpcf):
    dims = (32, 8, 12)
    with mpcf.Solver([dims], precision="mixed") as s:
        s.set_tiling(8, 6, persistent=True, tma=True)
        s.set_state(cloud_state(dims, nb=1))
        s.set_test_flags(mpcf._lib.TEST_DROP_LAST_COPY)
        s.stage(0.0, 0.25, 0.05)
        assert s.error_word() == 0
    with pytest.raises(mpcf.MpcfError):
        with mpcf.Solver([dims], precision="mixed") as s:
            s.set_test_flags(4)    # unknown flag


@pytest.mark.parametrize("prec", ["mixed", "fp32_ref"])
def test_copy_count_of_overlapping_persistent_launches(mpcf, prec):
    """A test flag on a streamed and on a windowed run of persistent launches:
    no copy is dropped, no tile is skipped (the result is that of the run
    without the flag, bit for bit), and the count covers every launch of all
    three stages: 2 d + 1 slab copies for a tile d planes deep (its d halo
    boxes and d + 1 interiors)."""
    dims, dz, steps = (64, 24, 30), 5, 2
    U0 = [np.ascontiguousarray(a) for a in cloud_state(dims, nb=1)]
    tiles = 2 * 3
    got = []
    for flag in (0, mpcf._lib.TEST_DROP_LAST_COPY):
        with mpcf.Solver([dims], precision=prec) as s:
            s.set_tiling(8, dz, persistent=True, tma=True)
            s.set_test_flags(flag)
            host = [a.copy() for a in U0]
            s.run_host(host, steps, cfl=0.3, nchunks=3)
            assert s.error_word() == 0
            got.append(host)
            assert s.test_copy_count() == (3 * steps * tiles * 6 * (2 * dz + 1) if flag else 0)
    assert_bitwise(got[1], got[0], "streamed run with the flag")
    got = []
    for flag in (0, mpcf._lib.TEST_DROP_LAST_COPY):
        with mpcf.WindowSolver(dims, 6, nslots=5, precision=prec) as w:
            w.set_tiling(8, 3, persistent=True, tma=True)
            w.set_test_flags(flag)
            host = [a.copy() for a in U0]
            w.run(host, steps, cfl=0.3)
            assert w.error_word() == 0
            got.append(host)
            assert w.test_copy_count() == (3 * steps * tiles * 10 * (2 * 3 + 1) if flag else 0)
    assert_bitwise(got[1], got[0], "windowed run with the flag")


def test_the_wait_for_a_planes_register_and_state_runs_out(mpcf):
    """The copy that a chunk's first plane is finalised from is dropped: the
    wait before the finalisation runs out one slab later.  Six slab copies
    were issued until then (the prologue's two and two slabs' pairs), none
    after it; those pending are waited for (no MPCF_ERRBIT_TMA_INFLIGHT), and
    the context stays usable.  Persistent launches ignore the flag."""
    dims = (32, 8, 12)             # one 32x8 tile, two 6-slab chunks
    U0 = cloud_state(dims, nb=1)
    with mpcf.Solver([dims], precision="fp32_ref") as s:
        s.set_tiling(8, 6, persistent=False, tma=True)
        s.set_state(U0)
        s.set_test_flags(mpcf._lib.TEST_DROP_PLANE_COPY)
        s.test_copy_count(clear=True)
        s.stage(0.0, 0.25, 0.05)
        w = s.error_word(clear=True)
        assert w & mpcf._lib.ERRBIT_TMA_TIMEOUT, hex(w)
        assert not (w & mpcf._lib.ERRBIT_TMA_INFLIGHT), hex(w)
        assert s.test_copy_count(clear=True) == 2 * 6
        s.set_tiling(8, 6, persistent=True, tma=True)
        s.set_state(U0)
        s.stage(0.0, 0.25, 0.05)
        assert s.error_word() == 0
        s.set_test_flags(0)
        s.set_tiling(8, 6, persistent=False, tma=True)
        s.set_state(U0)
        s.stage(0.0, 0.25, 0.05)
        assert s.error_word() == 0
        U, R = s.get_state()
    with mpcf.Solver([dims], precision="fp32_ref") as f:
        f.set_tiling(8, 6, persistent=False, tma=True)
        f.set_state(U0)
        f.stage(0.0, 0.25, 0.05)
        Uf, Rf = f.get_state()
    assert_bitwise(U, Uf, "state after the given-up stage")
    assert_bitwise(R, Rf, "register after the given-up stage")


def test_a_give_up_with_a_helper_warp(mpcf):
    """The same at 7 rows in the reference form, whose helper warp waits for
    the halo boxes alone: a dropped interior makes the columns' wait run out,
    and the helper's own runs out at the next box, which is not issued."""
    dims = (32, 7, 12)             # one 32x7 tile, two 6-slab chunks
    U0 = cloud_state(dims, nb=1)
    got = []
    for flag in (mpcf._lib.TEST_DROP_MID_COPY, 0):
        with mpcf.Solver([dims], precision="fp32_ref") as s:
            s.set_tiling(7, 6, persistent=False, tma=True)
            s.set_state(U0)
            if flag:
                s.set_test_flags(flag)
                s.stage(0.0, 0.25, 0.05)
                w = s.error_word(clear=True)
                assert w & mpcf._lib.ERRBIT_TMA_TIMEOUT and not w & mpcf._lib.ERRBIT_TMA_INFLIGHT, hex(w)
                assert s.test_copy_count() == 2 * 3
                s.set_test_flags(0)
                s.set_state(U0)
            s.stage(0.0, 0.25, 0.05)
            assert s.error_word() == 0
            got.append(s.get_state())
    for a, b, what in zip(*got, ("state", "register")):
        assert_bitwise(a, b, what + " after the given-up stage")
