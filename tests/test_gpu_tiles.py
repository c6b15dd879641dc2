"""The stage kernel where its tiles, its fluxes' upwind choice and its
branch-free weights can go wrong."""
import numpy as np
import pytest

import oracle_lib as O
from conftest import cloud_state
from test_gpu_parity import assert_bitwise, rel_linf

pytestmark = pytest.mark.gpu

ABS, REF = 0, 1


@pytest.mark.parametrize("dims", [(5, 5, 3), (32, 8, 1 + 2), (33, 9, 4), (64, 8, 8), (36, 7, 23), (65, 17, 19)])
def test_default_tiling_matches_oracle(mpcf, dims):
    """A new solver's tiling (its chunk depth follows the sizes; last chunks
    and tiles are ragged) and depths 1 and 2: one step, bit for bit."""
    bc = (REF, ABS, ABS, REF, REF, ABS)
    U = cloud_state(dims, nb=1)
    R = [np.zeros_like(a) for a in U]
    U0 = [a.copy() for a in U]
    dt_o, _ = O.step(dims, bc, U, R, cfl=0.3)
    for dz in (None, 1, 2):
        for persistent in (False, True):
            with mpcf.Solver([dims], bc=[bc], precision="fp32_ref") as s:
                if dz is not None:
                    s.set_tiling(8, dz, persistent, True)
                s.set_state(U0)
                assert s.step(cfl=0.3)[0] == dt_o
                Ug, Rg = s.get_state()
                assert s.error_word() == 0
            assert_bitwise(Ug, U, f"state, dz {dz}")
            assert_bitwise(Rg, R, f"register, dz {dz}")


def test_contact_at_rest_and_nan_velocity(mpcf):
    """s* = 0 on every face (uniform pressure, no velocity, a density jump):
    both sides' fluxes are blended, as in the reference.  A NaN transverse
    momentum in one cell reaches the same cells as in the reference's
    two-sided sum."""
    dims = (40, 16, 12)
    n = dims[0] * dims[1] * dims[2]
    x = np.arange(n) % dims[0]
    rho = np.where(x < 17, 1000.0, 1.0).astype(np.float32)
    zero = np.zeros(n, np.float32)
    G = np.full(n, 2.5, np.float32)
    E = np.full(n, 250.0, np.float32)
    for nan in (False, True):
        v = zero.copy()
        if nan:
            v[:] = 3.0 * rho                       # s* != 0 in y: upwind fluxes
            v[20 + dims[0] * (7 + dims[1] * 5)] = np.nan
        U = [rho.copy(), (2.0 * rho if nan else zero).copy(), v, zero.copy(), E + 20 * rho, G.copy(), zero.copy()]
        U = [np.ascontiguousarray(a, np.float32) for a in U]
        R = [np.zeros_like(a) for a in U]
        U0 = [a.copy() for a in U]
        O.stage(dims, (ABS,) * 6, U, R, 0.0, 0.25, 0.01)
        with mpcf.Solver([dims], precision="fp32_ref") as s:
            s.set_state(U0)
            s.stage(0.0, 0.25, 0.01)
            Ug, Rg = s.get_state()
        assert_bitwise(Ug, U, f"state, nan {nan}")
        assert_bitwise(Rg, R, f"register, nan {nan}")


@pytest.mark.parametrize("prec", ["fp64", "fp64_fast"])
@pytest.mark.parametrize("scale", [1.0, 1e16, 1e22, 1e60, 1e70, 1e74])
def test_fp64_weights_over_the_range_of_scales(mpcf, prec, scale):
    """Pressures from 1 to 1e74: above about 1e18 the fast form's shared
    reciprocal leaves its range (1e22), and above about 1e67 the sums of the
    reference form's weights, of order 1 / (10 p^4), fall below 2^-900 (1e70);
    both then take their general forms.  Random cells, so
    the indicators do not cancel; one stage against the FP64 oracle, whose
    1/6 of the extra terms is the reference's float literal, 5e-9 off: with
    dt/h divU of order 0.1 that moves G by less than 1e-8 (all else differs
    by contraction, 2^-53 times a few hundred operations)."""
    dims = (34, 18, 9)
    rng = np.random.default_rng(5)
    n = dims[0] * dims[1] * dims[2]
    p = scale * rng.uniform(0.5, 2.0, n)
    U = [rng.uniform(1.0, 2.0, n), np.zeros(n), np.zeros(n), np.zeros(n), 2.5 * p, np.full(n, 2.5), np.zeros(n)]
    R = [np.zeros(n) for _ in range(7)]
    U0 = [a.copy() for a in U]
    dtinvh = 0.1 / np.sqrt(1.4 * 2 * scale)
    O.stage(dims, (ABS,) * 6, U, R, 0.0, 0.25, dtinvh)
    with mpcf.Solver([dims], precision=prec) as s:
        s.set_state(U0)
        s.stage(0.0, 0.25, dtinvh)
        Ug, _ = s.get_state()
    for q in range(7):
        assert np.isfinite(Ug[q]).all()
        assert rel_linf(Ug[q], U[q]) <= 1e-8, (q, rel_linf(Ug[q], U[q]))


@pytest.mark.parametrize("persistent", [False, True])
@pytest.mark.parametrize("dims", [[(36, 9, 7), (33, 8, 5)], [(36, 9, 7), (64, 8, 5)]])
def test_ensemble_rows_with_and_without_bulk_copies(mpcf, dims, persistent):
    """Bulk copies are used by the domains whose rows are multiples of 16
    bytes.  One step of every domain, bit for bit."""
    want, U0 = [], []
    for i, d in enumerate(dims):
        U = cloud_state(d, nb=1 + i)
        U0.append([a.copy() for a in U])
        R = [np.zeros_like(a) for a in U]
        dt, _ = O.step(d, (ABS,) * 6, U, R, cfl=0.3)
        want.append((dt, U, R))
    with mpcf.Solver(dims, precision="fp32_ref") as s:
        s.set_tiling(8, 3, persistent, True)
        for i, U in enumerate(U0):
            s.set_state(U, dom=i)
        dts = s.step(cfl=0.3)
        for i, (dt, U, R) in enumerate(want):
            Ug, Rg = s.get_state(dom=i)
            assert dts[i] == dt
            assert_bitwise(Ug, U, f"domain {i}")
            assert_bitwise(Rg, R, f"register of domain {i}")


@pytest.mark.parametrize("prec", ["fp32_ref", "mixed", "fp64_fast"])
def test_overlapping_stage_streams_match_resident_run(mpcf, prec):
    """Streamed and windowed runs put each stage on its own stream: chunks
    thinner than the stencil's reach and whole-depth ones, persistent and not,
    against the resident run, bit for bit."""
    dims = (40, 24, 30)
    dt = mpcf.dtype_of(mpcf.PRECISIONS[prec])
    U0 = [np.asarray(a, dt) for a in cloud_state(dims, nb=2)]
    with mpcf.Solver([dims], precision=prec) as s:
        s.set_state(U0)
        s.run(3, cfl=0.3)
        want = s.get_state(with_reg=False)
    for dz, nchunks, persistent in ((2, 15, False), (2, 15, True), (5, 3, True), (30, 8, False)):
        with mpcf.Solver([dims], precision=prec) as s:
            s.set_tiling(8, dz, persistent, True)
            host = [a.copy() for a in U0]
            s.run_host(host, 3, cfl=0.3, nchunks=nchunks)
        assert_bitwise(host, want, f"streamed, dz {dz}, persistent {persistent}")
    for nslices, nslots in ((3, 5), (5, 6), (10, 3)):
        with mpcf.WindowSolver(dims, nslices, nslots=nslots, precision=prec) as w:
            host = [a.copy() for a in U0]
            w.run(host, 3, cfl=0.3)
        assert_bitwise(host, want, f"windowed, {nslices} planes")


def test_autotune_tries_fifteen_rows_in_the_reference_form(mpcf):
    """240 rows of tiles at height 8 and at 15, but half the CTAs at 15 fit
    one round of the device's slots: 15 rows are 9 % faster here, and the
    autotuner finds a tiling as fast."""
    dims = (21, 235, 109)
    with mpcf.Solver([dims], precision="fp32_ref") as s:
        s.set_state(cloud_state(dims, nb=2))
        _, best = s.autotune(reps=3)
        s.set_tiling(15, 6, False, False)
        s.time_stages(2)
        assert best <= 1.05 * min(s.time_stages(2) for _ in range(3))


@pytest.mark.parametrize("prec", ["fp32_ref", "mixed", "fp64_fast"])
def test_bulk_copy_and_other_domains_of_one_ensemble(mpcf, prec):
    """Domains with and without rows of 16-byte multiples, in turn: each kind
    keeps its way to load (slab copies are counted for the first alone), and
    every domain, its conservation sums and its dt equal those of a solver of
    its own, bit for bit, launched plainly, persistently and as a graph."""
    dims = [(33, 8, 5), (36, 9, 7), (41, 17, 6), (64, 8, 12), (32, 8, 9), (38, 25, 5)]
    bulk = [d for d in dims if d[0] * (8 if prec.startswith("fp64") else 4) % 16 == 0]
    assert 0 < len(bulk) < len(dims)
    dt = mpcf.dtype_of(mpcf.PRECISIONS[prec])
    U0 = [[np.asarray(a, dt) for a in cloud_state(d, nb=1 + i)] for i, d in enumerate(dims)]
    want = []
    for d, U in zip(dims, U0):
        with mpcf.Solver([d], precision=prec) as s:
            s.set_tiling(8, 3, False, False)
            s.track_conservation(True)
            s.set_state(U)
            t = s.run(3, cfl=0.3)
            want.append((t, s.get_state(), s.conserved_sums()))
    copies = sum((-(-d[0] // 32)) * (-(-d[1] // 8)) * (2 * d[2] + -(-d[2] // 3)) for d in bulk)
    for persistent in (False, True):
        for graph in (False, True):
            with mpcf.Solver(dims, precision=prec) as s:
                s.set_tiling(8, 3, persistent, True)
                assert s.tiling() == (8, 3, persistent, True)
                s.track_conservation(True)
                if persistent:
                    s.set_test_flags(mpcf._lib.TEST_DROP_LAST_COPY)     # (counts; persistent launches drop none)
                for i, U in enumerate(U0):
                    s.set_state(U, dom=i)
                t = s.run(3, cfl=0.3, graph=graph)
                sums = s.conserved_sums()
                assert s.error_word() == 0
                for i, (tw, (Uw, Rw), sw) in enumerate(want):
                    Ug, Rg = s.get_state(dom=i)
                    assert t[i] == tw[0]
                    assert np.array_equal(sums[i], sw[0])
                    assert_bitwise(Ug, Uw, f"domain {i}, persistent {persistent}")
                    assert_bitwise(Rg, Rw, f"register of domain {i}, persistent {persistent}")
                if persistent:
                    assert s.test_copy_count() == 9 * copies


def test_signs_of_zeros(mpcf):
    """Gas (P = 0) in blocks of equal velocities with zeros of both signs and
    pressure jumps that expand against slow inflow (u < 0 < s*): many fluxes
    are zeros, whose sign the reference's blend of the two sides decides.
    Every bit of state and register over three stages."""
    dims = (40, 17, 12)
    rng = np.random.default_rng(8)
    block = np.stack(np.meshgrid(*[np.arange(n) // 2 for n in dims[::-1]], indexing="ij")).reshape(3, -1)
    pick = lambda v: np.asarray(v)[rng.integers(0, len(v), (dims[2], dims[1], dims[0]))[tuple(block)]]   # noqa: E731
    speeds = [0.0, -0.0, 1e-2, -1e-2, -1e-2]
    rho, p = pick([1.0, 1.25, 2.0]), pick([1.0, 1.0, 8.0])
    u, v, w = pick(speeds), pick(speeds), pick(speeds)
    G = np.full_like(rho, 2.5)
    U = [np.ascontiguousarray(a, np.float32) for a in (rho, rho * u, rho * v, rho * w, G * p + 0.5 * rho * (u * u + v * v + w * w), G, 0 * rho)]
    R = [np.zeros_like(a) for a in U]
    stages = ((0.0, 0.25, 0.05), (-17.0 / 32, 8.0 / 9, 0.05), (-32.0 / 27, 0.75, 0.05))
    with mpcf.Solver([dims], precision="fp32_ref") as s:
        s.set_state(U, R)
        for st in stages:
            s.stage(*st)
        Ug, Rg = s.get_state()
    for a, b, dtinvh in stages:
        O.stage(dims, (ABS,) * 6, U, R, a, b, dtinvh)
    for q in range(7):
        for got, want, what in ((Ug[q], U[q], "state"), (Rg[q], R[q], "register")):
            assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), (what, q, int((got.view(np.uint32) != want.view(np.uint32)).sum()))


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("prec", ["fp32", "mixed", "fp64_fast"])
def test_a_state_without_sound_speed_spreads_in_the_fast_forms(mpcf, prec, axis):
    """Supersonic flow (Mach 8, along each axis and both ways) into a cell
    whose pressure is below -pc: no real sound speed and no star speed, so
    every flux of its faces is NaN, the supersonic neighbour's included.  All
    seven fields lose the same cells as in the oracle, and the error word
    says so."""
    dims = (36, 12, 9)
    shape = dims[::-1]
    for way in (1.0, -1.0):
        dt = np.float64 if prec == "fp64_fast" else np.float32
        rho, p = np.ones(shape), np.ones(shape)
        p[4, 6, 17] = -3.0
        G, mom = np.full(shape, 2.5), [np.zeros(shape) for _ in range(3)]
        mom[axis][:] = 10.0 * way
        E = G * p + 0.5 * sum(m * m for m in mom)
        U = [np.ascontiguousarray(a.reshape(-1), dt) for a in (rho, *mom, E, G, 0 * rho)]
        R = [np.zeros_like(a) for a in U]
        with mpcf.Solver([dims], precision=prec) as s:
            s.set_state(U, R)
            s.stage(0.0, 0.25, 0.01)
            Ug, Rg = s.get_state()
            assert s.error_word() & mpcf._lib.ERRBIT_NONPHYSICAL
        O.stage(dims, (ABS,) * 6, U, R, 0.0, 0.25, 0.01)
        for q in range(7):
            assert np.isnan(U[q]).any()
            assert np.array_equal(np.isnan(Ug[q]), np.isnan(U[q])), (q, int(np.isnan(Ug[q]).sum()), int(np.isnan(U[q]).sum()))
            assert np.array_equal(np.isnan(Rg[q]), np.isnan(R[q])), q


def reciprocals(mpcf, x, rn):
    import ctypes
    x = np.ascontiguousarray(x, np.float64)
    y = np.empty_like(x)
    pd = ctypes.POINTER(ctypes.c_double)
    mpcf._lib.check(mpcf.lib().mpcf_probe_rcp64(0, int(rn), x.size, x.ctypes.data_as(pd), y.ctypes.data_as(pd)))
    return y


def reciprocal_arguments():
    """What the stage kernel takes reciprocals of, and the edges of the
    mantissa: powers of two and their neighbours, at exponents over +-900."""
    rng = np.random.default_rng(3)
    p = np.exp(rng.uniform(np.log(1e-6), np.log(1e38), (3, 1 << 20)))          # indicators + eps
    p32 = p.astype(np.float32).astype(np.float64)
    sums = []
    for q in (1.0 / (10.0 * p * p), 1.0 / (10.0 * p32 * p32)):
        sums += [q[0] + 6.0 * q[1] + 3.0 * q[2], q[2] + 6.0 * q[1] + 3.0 * q[0]]
    scale = np.ldexp(1.0, rng.integers(-900, 900, 1 << 20).astype(np.int32))
    k = rng.integers(0, 1 << 10, 1 << 20)
    ulp = 2.0 ** -52
    return np.concatenate([10.0 * p.ravel() * p.ravel(), 10.0 * p32.ravel() * p32.ravel(), *sums,
                           scale * rng.uniform(1.0, 2.0, scale.size), scale * (1.0 + k * ulp),
                           scale * (2.0 - (k + 2) * ulp)])


def test_reference_form_reciprocal_rounds_like_division(mpcf):
    """rcp_rn equals IEEE division on 1.3e7 arguments; for a mantissa of all
    ones, where Markstein's theorem does not hold, it is at most one unit in
    the last place off."""
    x = reciprocal_arguments()
    y = reciprocals(mpcf, x, True)
    bad = y != 1.0 / x
    assert not bad.any(), (int(bad.sum()), x[bad][:4].tolist())
    ones = np.ldexp(2.0 - 2.0 ** -52, np.arange(-900, 900).astype(np.int32))
    y, want = reciprocals(mpcf, ones, True), 1.0 / ones
    assert (np.abs(y.view(np.int64) - want.view(np.int64)) <= 1).all()


def test_fast_form_reciprocal_error(mpcf):
    """rcp_f64: the approximation's error e (below 2^-19) becomes e^4 after
    two Newton steps, below the rounding of the last, of relative size 2^-53,
    plus the residual's own rounding times e^2: within one unit in the last
    place of division."""
    x = reciprocal_arguments()
    y, want = reciprocals(mpcf, x, False), 1.0 / x
    assert (np.abs(y.view(np.int64) - want.view(np.int64)) <= 1).all()


@pytest.mark.parametrize("tma", [False, True])
@pytest.mark.parametrize("prec,ty", [("fp32_ref", 3), ("fp32_ref", 7), ("fp32_ref", 15), ("fp64", 3), ("fp64", 7)])
def test_heights_with_a_helper_warp(mpcf, prec, ty, tma):
    """The reference forms' tiles of 2^n - 1 rows have a warp without columns:
    state, register, dt and conservation sums over ragged tiles.  FP32: the
    oracle's bits.  FP64: within 1e-12 of the 8-row tiles (whose instances
    contract their expressions for themselves)."""
    dims = (44, 2 * ty + 1, 9)
    bc = (REF, ABS, ABS, REF, REF, ABS)
    U0 = [np.asarray(a, mpcf.dtype_of(mpcf.PRECISIONS[prec])) for a in cloud_state(dims, nb=1)]
    if prec == "fp32_ref":
        U, R = [a.copy() for a in U0], [np.zeros_like(a) for a in U0]
        dts = [O.step(dims, bc, U, R, cfl=0.3)[0] for _ in range(2)]
    else:
        with mpcf.Solver([dims], bc=[bc], precision=prec) as s:
            s.set_tiling(8, 4, False, tma)
            s.set_state(U0)
            dts = [s.step(cfl=0.3)[0] for _ in range(2)]
            U, R = s.get_state()
    for persistent in (False, True):
        with mpcf.Solver([dims], bc=[bc], precision=prec) as s:
            s.set_tiling(ty, 4, persistent, tma)
            assert s.launch_shape()[2] == 32 * (ty + 1)
            s.track_conservation(True)
            s.set_state(U0)
            got = [s.step(cfl=0.3)[0] for _ in range(2)]
            Ug, Rg = s.get_state()
            sums = s.conserved_sums()[0]
            assert s.error_word() == 0
        for q in range(5):
            assert abs(sums[q] - Ug[q].astype(np.float64).sum()) <= 1e-12 * np.abs(Ug[q].astype(np.float64)).sum()
        if prec == "fp32_ref":
            assert got == dts
            assert_bitwise(Ug, U, f"state, {ty} rows, persistent {persistent}")
            assert_bitwise(Rg, R, f"register, {ty} rows, persistent {persistent}")
        else:
            assert np.allclose(got, dts, rtol=1e-12, atol=0)
            for q in range(7):
                assert rel_linf(Ug[q], U[q]) <= 1e-12, (q, rel_linf(Ug[q], U[q]))
