"""The rounding of solver paths whose operations are fixed: states after a few
steps, bit for bit. The stored states come from the kernels that divide and
take square roots in IEEE arithmetic, in the reference's order of operations
(float32: of the same expressions with the fast divide of the primitives)."""
import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu


def _field(n, dtype, seed):
    """A rough supersonic field, the same as the stored states started from."""
    r = np.random.default_rng(seed)
    rho = 1 + 0.3 * r.random(n)
    u = 2 + 0.5 * r.standard_normal(n)
    v = 0.5 * r.standard_normal(n)
    p = 1 + 0.5 * r.random(n)
    W = np.stack([rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)], 1)
    return W.astype(dtype).astype(np.float64)


def _steps(mesh, slots=1, steps=4, **options):
    from eulersr_b200.solver import FlowCase, Solver
    dtype = np.float64 if options["precision"] == "f64" else np.float32
    s = Solver(mesh, slots, **options)
    for g in range(slots):
        s.set_case(g, FlowCase(mach=1.5 + g, aoa_deg=2.0, cfl=0.5, tf=100.0, dtype=dtype),
                   W_init=_field(mesh.n_cells, dtype, g))
    s.step(steps)
    states = [s.get_state(g) for g in range(slots)]
    s.close()
    return states


@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_constant_reconstruction_local_time_step(diamond02, precision):
    """The local time step of constant reconstruction: an IEEE square root and
    one division a cell, also in the fast float32 mode."""
    want = np.load(GOLDEN / "constant_local_dt.npz")[precision]
    got = _steps(diamond02, precision=precision, reconstruction="constant", dt_mode="local")[0]
    assert np.array_equal(got, want.astype(np.float64))
