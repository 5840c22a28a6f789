"""The single-pass step of the two-density and D3Q27 models against the two passes it fuses.

lbx_step runs k_cg_march; the kernel-level entries lbx_init_rho and lbx_time_step_cg run the phase-field /
density pass and the collision pass with the same helpers in the same order, so every population must agree bit
for bit: on boxes smaller than a column, with columns that wrap, cut columns, segments of one plane (the plan of
small boxes) and segments that go round the four-plane window several times, on every storage the models take.
"""
import numpy as np
import pytest

from lbcuda_b200 import LBSim, make_params
from lbcuda_b200.inputs import seeded_noise_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", ["cg-diffdens", "cg-d3q27", "cg-diffdens-d3q27"])
@pytest.mark.parametrize("storage", ["f32", "f16", "bf16", "f64"])
@pytest.mark.parametrize("shape", [(3, 3, 3), (32, 8, 5), (33, 9, 40), (70, 23, 17)])
def test_single_pass_equals_two_passes(model, storage, shape):
    nx, ny, nz = shape
    rR, rB = seeded_noise_fields(nx, ny, nz, seed=3, amp=0.05)
    a, b = (LBSim(make_params(nx, ny, nz, model=model, storage=storage, sigma=0.02, beta=0.7, tauB=0.8, densR=2.0,
                              densB=1.0)) for _ in range(2))
    for s in (a, b):
        s.set_fields(rR, rB, (0.01, -0.02, 0.005))
    a.step(5)
    for _ in range(5):
        assert b._L.lbx_init_rho(b._h) == 0 and b._L.lbx_time_step_cg(b._h) == 0
    for p, q in zip(a.get_pops(), b.get_pops()):
        assert np.isfinite(p).all() and np.array_equal(p, q)
    assert a.status()[0] == 0 and a.steps_taken == b.steps_taken == 5
    a.close()
    b.close()


@pytest.mark.parametrize("model", ["cg-diffdens", "cg-d3q27", "cg-diffdens-d3q27"])
@pytest.mark.parametrize("storage", ["f32", "f16", "bf16", "f64"])
@pytest.mark.parametrize("shape,zlen", [((39, 15, 17), 7), ((21, 27, 19), 6), ((65, 20, 24), 24), ((16, 16, 9), 5)])
def test_window_reused_over_long_segments(model, storage, shape, zlen):
    """Segments of at least five planes write every slot of the window again, with a whole column, an even split
    and a shorter last segment; widths and heights that cut the last column in x, in y and in both."""
    nx, ny, nz = shape
    rR, rB = seeded_noise_fields(nx, ny, nz, seed=5, amp=0.05)
    a, b = (LBSim(make_params(nx, ny, nz, model=model, storage=storage, sigma=0.02, beta=0.7, tauB=0.8, densR=2.0,
                              densB=1.0)) for _ in range(2))
    a.set_lean_shape(0, zlen)
    for s in (a, b):
        s.set_fields(rR, rB, (0.01, -0.02, 0.005))
    a.step(4)
    for _ in range(4):
        assert b._L.lbx_init_rho(b._h) == 0 and b._L.lbx_time_step_cg(b._h) == 0
    for p, q in zip(a.get_pops(), b.get_pops()):
        assert np.isfinite(p).all() and np.array_equal(p, q)
    assert a.status()[0] == 0
    a.close()
    b.close()


@pytest.mark.parametrize("model,storage", [("cg-diffdens", "bf16"), ("cg-d3q27", "f16"), ("cg-d3q27", "bf16"),
                                           ("cg-diffdens", "f16")])
@pytest.mark.parametrize("nx", [40, 41])
def test_both_sides_of_the_small_box_rule(model, storage, nx):
    """64,000 cells and a few more: some 16-bit models go back to two passes there; the step is the same."""
    rR, rB = seeded_noise_fields(nx, 40, 40, seed=8, amp=0.05)
    a, b = (LBSim(make_params(nx, 40, 40, model=model, storage=storage, sigma=0.02, beta=0.7, densR=2.0, densB=1.0))
            for _ in range(2))
    for s in (a, b):
        s.set_fields(rR, rB)
    a.step(3)
    for _ in range(3):
        assert b._L.lbx_init_rho(b._h) == 0 and b._L.lbx_time_step_cg(b._h) == 0
    for p, q in zip(a.get_pops(), b.get_pops()):
        assert np.isfinite(p).all() and np.array_equal(p, q)
    assert a.status()[0] == 0 and a.steps_taken == 3
    a.close()
    b.close()
