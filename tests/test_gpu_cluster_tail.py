"""The coarse levels on one thread-block cluster against the per-level kernels: every level's u and b
(ghosts included) bit for bit after a fixed schedule, and the refinement solver's pressure against
its single-CTA tail's."""
import numpy as np
import pytest

import opencurrent_b200 as ocu

pytestmark = pytest.mark.gpu

NEU, DIR, PER = (ocu.BoundaryCondition(t) for t in (ocu.BC_NEUMANN, ocu.BC_DIRICHELET, ocu.BC_PERIODIC))
NONE = ocu.BoundaryCondition(ocu.BC_NONE)
BCS = {"neumann": ocu.BoundaryConditionSet(NEU), "dirichlet": ocu.BoundaryConditionSet(DIR),
       "periodic": ocu.BoundaryConditionSet(PER),
       "mixed": ocu.BoundaryConditionSet(NEU, xpos=PER, xneg=PER, zpos=DIR),
       "open": ocu.BoundaryConditionSet(DIR, ypos=NONE, zneg=NEU)}
# coarse levels held by one CTA only; split over few and over all 16 ranks; uneven planes per rank; a
# coarsest level with more than one pair per thread; two planes along x
SHAPES = [(16, 16, 16), (64, 64, 64), (40, 24, 56), (96, 80, 48), (72, 64, 36), (68, 16, 20), (8, 64, 96)]


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


@pytest.mark.parametrize("dtype", [ocu.F32, ocu.F64])
@pytest.mark.parametrize("bc", list(BCS))
@pytest.mark.parametrize("dims", SHAPES)
def test_levels_bit_identical(dims, bc, dtype):
    b = np.random.default_rng(3).uniform(-1, 1, dims)
    sym = dims == (40, 24, 56)
    got = []
    for knobs in (dict(), dict(tail_cells=-1)):
        s = solver(ocu.Sol_MultigridPressure3DDevice(dtype), dims, BCS[bc], (b, dtype), make_symmetric_operator=sym,
                   disable_relax_on_host=dims == (96, 80, 48), nu2=1 if dims == (64, 64, 64) else 2, **knobs)
        s.run_fmg(1)
        s.run_vcycles(2)
        got.append([g(l).copy_to_host() for l in range(s.stats.num_levels) for g in (s.read_u, s.read_b)])
    for one, other in zip(*got):
        assert np.array_equal(one, other, equal_nan=True)


@pytest.mark.parametrize("dims", SHAPES)
@pytest.mark.parametrize("bc", ["neumann", "mixed", "periodic"])
def test_refinement_levels_bit_identical(dims, bc, monkeypatch):
    b = np.random.default_rng(4).uniform(-1, 1, dims)
    b -= b.mean()
    got = []
    for env in (None, "512"):
        if env:
            monkeypatch.setenv("OCU_B200_CHQ_TAIL", env)
        s = solver(ocu.Sol_MultigridPressureMixed3DDeviceD(), dims, BCS[bc], (b, ocu.F64))
        s.solve(1e-9, 3)
        got.append(s.pressure().copy_to_host())
    assert np.array_equal(*got, equal_nan=True)
