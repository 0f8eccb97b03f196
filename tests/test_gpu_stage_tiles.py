"""The FP64 stage kernel at the edges of its tiles (32 x 11 cells, any number of
planes): what a cell gets must not depend on where in a tile, a segment of
planes or a halo it lies."""
import numpy as np
import pytest

from m2c_b200 import abi, cases

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (2, 3, 4), (31, 10, 2), (32, 11, 1), (33, 12, 3), (34, 22, 5), (64, 23, 2), (65, 21, 17),
          (5, 34, 9), (30, 9, 33)]


def periodic_box(shape, seed, **scheme):
    g = abi.grid(*shape, bc=(abi.BC_PERIODIC,) * 6)
    s = abi.scheme(cfl=0.3, **scheme)
    r = np.random.default_rng(seed)
    V = cases.empty_state(g)
    inner = V[1:-1, 1:-1, 1:-1]
    n = inner.shape[:3]
    inner[..., 0] = 1.0 + 0.05 * r.uniform(-1, 1, n)
    inner[..., 1:4] = 0.1 * r.uniform(-1, 1, n + (3,))
    inner[..., 4] = 1.0 + 0.05 * r.uniform(-1, 1, n)
    return g, s, [abi.material(1.4, 0.0)], V


@pytest.mark.parametrize("flux,limiter,rec_var", [(abi.FLUX_HLLC, abi.LIM_VANALBADA, 0), (abi.FLUX_ROE, abi.LIM_GENMINMOD, 0),
                                                  (abi.FLUX_LLF, abi.LIM_VANALBADA, 3)])
@pytest.mark.parametrize("shape", SHAPES)
def test_periodic_box_does_not_see_its_tiles(gpu, shape, flux, limiter, rec_var):
    """FP64 in a fully periodic box: shifting the field shifts residual and
    steps with it, bit for bit."""
    g, s, mats, V = periodic_box(shape, 3, flux=flux, limiter=limiter, rec_var=rec_var, rk_order=3)
    inner = V[1:-1, 1:-1, 1:-1].copy()
    got = []
    for shift in ((0, 0, 0), (1, 3, 7), (2, 5, 19)):
        V[1:-1, 1:-1, 1:-1] = np.roll(inner, shift, axis=(0, 1, 2))
        sol = gpu.Solver(g, s, mats)
        sol.upload(V)
        R = sol.residual()[1:-1, 1:-1, 1:-1]
        sol.run(2)
        W, _, _ = sol.download()
        back = tuple(-q for q in shift)
        got.append((np.roll(R, back, axis=(0, 1, 2)), np.roll(W[1:-1, 1:-1, 1:-1], back, axis=(0, 1, 2)), sol.t))
        sol.close()
    for R, W, t in got[1:]:
        assert np.array_equal(R, got[0][0]) and np.array_equal(W, got[0][1]) and t == got[0][2]


@pytest.mark.parametrize("shape", SHAPES)
def test_walls_and_inlets_match_reference(gpu, ref, shape):
    bc = (abi.BC_INLET, abi.BC_OUTLET, abi.BC_SLIPWALL, abi.BC_STICKWALL, abi.BC_SYMMETRY, abi.BC_SYMMETRY)
    g, s, mats, V = cases.random_box(*shape, bc=bc)
    sol = gpu.Solver(g, s, mats)
    sol.upload(V)
    oracle = ref.RefCase(g, s, mats)
    oracle.set_state(V)
    Rg, Rr = cases.interior(sol.residual()), cases.interior(oracle.residual())
    assert np.abs(Rg - Rr).max() <= 1e-12 * np.abs(Rr).max()
