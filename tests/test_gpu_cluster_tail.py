"""The coarse levels on one thread-block cluster against the per-level kernels: every level's u and b
(ghosts included) bit for bit after a fixed schedule, and the refinement solver's pressure against
its single-CTA tail's; which hierarchies the cluster takes, by their launch counts."""
import os
import subprocess
import sys

import numpy as np
import pytest

import opencurrent_b200 as ocu
from oracle import oracle_ctypes as O
from tests.helpers import DIR as D, NEU as N, PER as P, bc_from, mg_params, npdt
from tests.test_gpu_parity import assert_same, dev_grid, to_ocu_bc

pytestmark = pytest.mark.gpu

NEU, DIR, PER = (ocu.BoundaryCondition(t) for t in (ocu.BC_NEUMANN, ocu.BC_DIRICHELET, ocu.BC_PERIODIC))
NONE = ocu.BoundaryCondition(ocu.BC_NONE)
BCS = {"neumann": ocu.BoundaryConditionSet(NEU), "dirichlet": ocu.BoundaryConditionSet(DIR),
       "periodic": ocu.BoundaryConditionSet(PER),
       "mixed": ocu.BoundaryConditionSet(NEU, xpos=PER, xneg=PER, zpos=DIR),
       "open": ocu.BoundaryConditionSet(DIR, ypos=NONE, zneg=NEU)}
# coarse levels held by one CTA only; split over few and over all 16 ranks; uneven planes per rank; a
# coarsest level (4x32x48, four ranks of one plane) with more than one pair per thread
SHAPES = [(16, 16, 16), (64, 64, 64), (40, 24, 56), (96, 80, 48), (72, 64, 36), (68, 16, 20), (8, 64, 96)]
SYMMETRIC = [(40, 24, 56), (72, 64, 36)]


def solver(cls, dims, bc, b, **knobs):
    s = cls
    s.bc = bc
    for k, v in knobs.items():
        setattr(s, k, v)
    rhs = ocu.Grid3DDevice(b[1])
    rhs.init(*dims)
    host = rhs.empty_host()
    L = rhs.layout
    v = np.lib.stride_tricks.as_strided(host[int(L.shift):], dims,
                                        tuple(q * host.itemsize for q in (L.xstride, L.ystride, 1)))
    v[:] = b[0]
    rhs.copy_from_host(host)
    h = 1.0 / max(dims)
    s.initialize_storage(*dims, h, 1.25 * h if dims[1] == 24 else h, h, rhs)
    return s


def bits(a):
    return a.view(np.int64 if a.dtype == np.float64 else np.int32)


def launches(f):
    n = ocu.kernel_launch_count()
    f()
    return ocu.kernel_launch_count() - n


@pytest.mark.parametrize("dtype", [ocu.F32, ocu.F64])
@pytest.mark.parametrize("bc", list(BCS))
@pytest.mark.parametrize("dims", SHAPES)
@pytest.mark.parametrize("level_arithmetic", [False, True])  # of the coarsest level: the host routine's or the others'
def test_levels_bit_identical(level_arithmetic, dims, bc, dtype):
    b = np.random.default_rng(3).uniform(-1, 1, dims)
    got, counts = [], []
    for knobs in (dict(), dict(tail_cells=-1)):
        s = solver(ocu.Sol_MultigridPressure3DDevice(dtype), dims, BCS[bc], (b, dtype),
                   make_symmetric_operator=dims in SYMMETRIC, disable_relax_on_host=level_arithmetic,
                   nu2=1 if dims == (64, 64, 64) else 2, **knobs)
        counts.append(launches(lambda: (s.run_fmg(1), s.run_vcycles(2))))
        got.append([g(l).copy_to_host() for l in range(s.stats.num_levels) for g in (s.read_u, s.read_b)])
    # the cluster took its levels (a coarsest level alone is one launch by the host routine's arithmetic too)
    assert counts[0] < counts[1] or (s.stats.num_levels == 2 and not level_arithmetic)
    for one, other in zip(*got):
        assert np.all(np.isfinite(other))
        assert np.array_equal(bits(one), bits(other))


# (8, 8, 8): the whole hierarchy in the tail, its ramp ending with level 0's own V-cycle
@pytest.mark.parametrize("dims", SHAPES + [(8, 8, 8)])
@pytest.mark.parametrize("bc", ["neumann", "mixed", "periodic"])
def test_refinement_levels_bit_identical(dims, bc, monkeypatch):
    b = np.random.default_rng(4).uniform(-1, 1, dims)
    b -= b.mean()
    got, counts = [], []
    for env in (None, "512"):
        if env:
            monkeypatch.setenv("OCU_B200_CHQ_TAIL", env)
        s = solver(ocu.Sol_MultigridPressureMixed3DDeviceD(), dims, BCS[bc], (b, ocu.F64))
        counts.append(launches(lambda: s.solve(1e-9, 3)))
        got.append(s.pressure().copy_to_host())
    assert counts[0] < counts[1] or s.stats.num_levels == 2  # two levels: the coarsest is one launch either way
    assert np.all(np.isfinite(got[1]))
    assert np.array_equal(*map(bits, got))


# An axis periodic on one face only: each face keeps its own rule on every level.
ONE_SIDED = {f"{a}{per}_{'dirichlet' if other == D else 'neumann'}": (f"{a}{per}", f"{a}{'neg' if per == 'pos' else 'pos'}",
                                                                       other)
             for a in "xyz" for per in ("pos", "neg") for other in (D, N)}


@pytest.mark.parametrize("dtype", [ocu.F32, ocu.F64])
@pytest.mark.parametrize("name", list(ONE_SIDED))
@pytest.mark.parametrize("rest", [N, P])
def test_one_sided_periodic_axes(name, rest, dtype):
    dims, h = (32, 24, 40), (0.03, 0.04, 0.03)
    per, other, kind = ONE_SIDED[name]
    faces = {f: (rest, 0.0) for f in ("xpos", "xneg", "ypos", "yneg", "zpos", "zneg")}
    faces[per], faces[other] = (P, 0.0), (kind, 0.0)
    bc = bc_from(faces)
    L = O.layout(*dims)
    rhs = np.zeros(int(L.allocated), npdt(dtype))
    O.interior(rhs, L)[:] = np.random.default_rng(5).uniform(-1, 1, dims)
    om = O.OracleMG("d" if dtype == ocu.F64 else "f", mg_params(bc), *dims, *h, rhs, L)
    s = ocu.Sol_MultigridPressure3DDevice(dtype)
    s.bc = to_ocu_bc(bc)
    g = dev_grid(rhs, dtype, L)
    s.initialize_storage(*dims, *h, g)
    for one in (om, s):
        one.run_fmg(1)
        one.run_vcycles(2)
    for l in range(om.num_levels):
        for which, mine in (("u", s.read_u), ("b", s.read_b)):
            want = om.grid(which, l)[0]
            assert np.all(np.isfinite(want))
            assert_same(mine(l).copy_to_host(), want, f"{which} of level {l}")


@pytest.mark.parametrize("dtype", [ocu.F32, ocu.F64])
@pytest.mark.parametrize("dims, clustered", [((60, 60, 60), True), ((20, 100, 100), True), ((8, 128, 128), False),
                                             ((76, 76, 76), False)])
def test_large_coarsest_level_stays_with_the_launches(dims, clustered, dtype):
    """Relaxed by the level kernels' arithmetic, a coarsest level of more pairs than three trips of a
    rank's threads is faster as launches: 900, 1250 pairs a rank below that line, 2048 and 2166 above."""
    b = np.random.default_rng(7).uniform(-1, 1, dims)
    counts = []
    for knobs in (dict(), dict(tail_cells=-1)):
        s = solver(ocu.Sol_MultigridPressure3DDevice(dtype), dims, BCS["dirichlet"], (b, dtype),
                   disable_relax_on_host=True, **knobs)
        counts.append(launches(lambda: s.run_vcycles(1)))
    assert (counts[0] < counts[1]) if clustered else (counts[0] == counts[1])


EARLIER_ERROR = """
import opencurrent_b200 as ocu
from opencurrent_b200._capi import ERR_ALLOC, ERR_CUDA
for attempt in range(2):  # the device is asked for its cluster size in the first solve only
    rhs = ocu.Grid3DDevice(ocu.F32)
    rhs.init(32, 32, 32)
    s = ocu.Sol_MultigridPressure3DDevice(ocu.F32)
    s.bc = ocu.BoundaryConditionSet(ocu.BoundaryCondition(ocu.BC_NEUMANN))
    s.initialize_storage(32, 32, 32, 1 / 32, 1 / 32, 1 / 32, rhs)
    try:
        ocu.Grid3DDevice(ocu.F32).init(20000, 20000, 20000)  # 32 TB
        raise SystemExit("allocated")
    except ocu.OcuError as e:
        assert e.status == ERR_ALLOC, e
    try:
        s.run_vcycles(1)
        print("taken")
    except ocu.OcuError as e:
        assert e.status == ERR_CUDA and "out of memory" in str(e), e
        print("reported")
    s.run_vcycles(1)
"""


def test_asking_for_the_cluster_size_keeps_an_earlier_error():
    """A refused allocation leaves its error with the thread, and the next launch reports it, in a
    program's first solve as in any other."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", EARLIER_ERROR], capture_output=True, text=True, timeout=300, cwd=root)
    assert r.returncode == 0 and r.stdout.split() == ["reported", "reported"], r.stdout + r.stderr
