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


@pytest.mark.parametrize("exponent", [-60, 240, 280])
def test_float64_limiter_far_from_unit_scale(diamond02, exponent):
    """Density and pressure in units 2^exponent: the limiter's fractions have
    squares of state differences above and below, whose cross products leave
    float64's range from 2^256 on although each fraction is ordinary. Held to
    the float64 parity tolerance against the oracle (field-scaled 1e-12)."""
    from conftest import oracle_mesh, rel_err
    from eulersr_b200.solver import FlowCase, Solver
    from oracle import euler_oracle as O
    scale = 2.0 ** exponent
    om = oracle_mesh(diamond02, np.float64)
    W, inlet = O.initialize(diamond02.n_cells, dict(rho_inf=scale, p_inf=scale, gamma=1.4, Mach=2.5, aoa=5.0,
                                                    case=diamond02.metadata["case"]), np.float64)
    dt = O.get_dt(W, om, CFL=0.6)
    for _ in range(20):
        W = O.time_step_srk2(W, om, dt, inlet)
    s = Solver(diamond02, 1, precision="f64")
    s.set_case(0, FlowCase(mach=2.5, aoa_deg=5.0, cfl=0.6, tf=100.0, rho_inf=scale, p_inf=scale))
    assert abs(s.dt()[0] - dt) <= 1e-14 * dt
    s.step(20)
    assert rel_err(s.get_state(0), W) <= 1e-12
    s.close()


@pytest.mark.parametrize("run", ["diamond_hllc_global_SRK2", "naca0012_rusanov_local_RK2", "naca0012_hllc_local_EE"])
def test_float64_reference_fidelity_keeps_the_sequence(diamond02, naca02, run):
    """Float64 with fidelity 'reference' computes the reference's sequence of
    operations, not the fast mode's formulas (third slot of three)."""
    geom, flux, dt_mode, scheme = run.split("_")
    got = _steps(diamond02 if geom == "diamond" else naca02, slots=3, precision="f64", fidelity="reference", flux=flux,
                 dt_mode=dt_mode, time_scheme=scheme)[2]
    assert np.array_equal(got, np.load(GOLDEN / "float64_sequence.npz")[run])
