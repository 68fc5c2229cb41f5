"""Parity at the bench's full size: the NACA0012 h=0.025 mesh (25,049 cells)
and its 256-case batch.

* float64 kernels against the NumPy oracle (10 SRK2 steps, 1e-12) and the
  C/OpenMP restatement (100 steps, 1e-12) on the full mesh, transonic case;
* the fast float32 path's accuracy: within 1e-5 of the float64 oracle after
  20 steps, closer to it than the reference's own float32 (float32 parity
  with the reference is tests/test_gpu_hr_parity.py);
* the 256-case batch of the bench (default_rng(1) draws): sampled slots equal
  their single-case solves bitwise after a 50-step chunk, and the batch's
  states stay finite with positive density and pressure.
"""
import numpy as np
import pytest

from conftest import oracle_mesh, rel_err

pytestmark = pytest.mark.gpu

MACH, AOA = 0.8, 1.25


@pytest.fixture(scope="module")
def naca_hr():
    from eulersr_b200.meshing.generate import cached_mesh
    return cached_mesh("naca0012", 0.025)


def _gpu(mesh, prec, steps, mach=MACH, aoa=AOA):
    from eulersr_b200.solver import Solver, FlowCase
    dtype = np.float64 if prec == "f64" else np.float32
    s = Solver(mesh, 1, precision=prec)
    s.set_case(0, FlowCase(mach=mach, aoa_deg=aoa, cfl=0.6, tf=100.0, dtype=dtype))
    s.step(steps)
    W = s.get_state(0)
    s.close()
    return W


def _oracle(mesh, dtype, steps, mach=MACH, aoa=AOA):
    from oracle import euler_oracle as O
    om = oracle_mesh(mesh, dtype)
    W, inlet = O.initialize(mesh.n_cells, dict(rho_inf=1.0, p_inf=1.0, gamma=1.4, Mach=mach, aoa=aoa,
                                               case="naca0012"), dtype)
    dt = O.get_dt(W, om, CFL=0.45 if 0.6 < mach < 1.1 else 0.6)
    for _ in range(steps):
        W = O.time_step_srk2(W, om, dt, inlet)
    return W


def test_full_mesh_f64_matches_oracle(naca_hr):
    assert naca_hr.n_cells > 25000
    assert rel_err(_gpu(naca_hr, "f64", 10), _oracle(naca_hr, np.float64, 10)) <= 1e-12


def test_full_mesh_f64_100_steps_matches_c_restatement(naca_hr):
    from oracle.cport import CpuCase
    cc = CpuCase(naca_hr, MACH, AOA, np.float64)
    ref = cc.srk2(cc.W0, 100)
    assert rel_err(_gpu(naca_hr, "f64", 100), ref) <= 1e-12


def test_full_mesh_f32_fast_fidelity_accuracy(naca_hr):
    """Accuracy of the fast float32 path at full size (not its parity, which
    tests/test_gpu_hr_parity.py holds with the reference fidelity): 20 steps
    land within 1e-5 of the float64 oracle, closer to it than the reference's
    own float32 (the oracle's float32), because the fast path forms the
    geometry in float64 and rounds it once where the reference forms
    barycentre differences and face offsets in float32 on cells ~3e-3 across
    at coordinates ~2."""
    W64 = _oracle(naca_hr, np.float64, 20)
    e_gpu = rel_err(_gpu(naca_hr, "f32", 20), W64)
    e_ref32 = rel_err(_oracle(naca_hr, np.float32, 20), W64)
    print(f"full-size float32 vs float64 oracle after 20 steps: fast path {e_gpu:.3e}, reference float32 {e_ref32:.3e}")
    assert e_gpu <= 1e-5
    assert e_gpu < e_ref32


def test_full_batch_slots_equal_single_solves(naca_hr):
    """The bench's batch: 256 cases, Mach ~ U[0.7, 3] and alpha on the 0.5-degree
    grid from default_rng(1); a 50-step chunk of the whole batch (K2 by
    patches) leaves every sampled slot bitwise equal to the same case advanced
    alone (per-cell K2)."""
    from eulersr_b200.solver import DeviceMesh, FlowCase, Solver
    rng = np.random.default_rng(1)
    mach = rng.uniform(0.7, 3.0, 256)
    aoa = rng.choice(np.arange(-5, 5.01, 0.5), 256)
    cases = [FlowCase(mach=float(m), aoa_deg=float(a), cfl=0.6, tf=1e9, dtype=np.float32) for m, a in zip(mach, aoa)]
    dm = DeviceMesh(naca_hr)
    s = Solver(dm, 256, precision="f32", block_size="patches")   # K2 by patches; the single solves per cell
    s.set_cases(list(range(256)), cases)
    s.step(50)
    states = s.get_states(list(range(256)), dtype=np.float32)
    for W in states:
        assert np.isfinite(W).all()
        assert (W[:, 0] > 0).all()
        rho = W[:, 0].astype(np.float64)
        p = (W[:, 3] - 0.5 * (W[:, 1].astype(np.float64) ** 2 + W[:, 2].astype(np.float64) ** 2) / rho) * 0.4
        assert (p > 0).all()
    for b in (0, 97, 255):
        one = Solver(dm, 1, precision="f32")
        one.set_case(0, cases[b])
        one.step(50)
        assert np.array_equal(one.get_state(0).astype(np.float32), states[b]), b
        one.close()
    s.close()


@pytest.mark.parametrize("counts", [(8,), (9,), (16, 3), (17, 1), (1, 40), (3, 64), (2, 2)])
@pytest.mark.parametrize("options", [dict(), dict(time_scheme="RK2", dt_mode="local"), dict(stop_rule="density_l2"),
                                     dict(flux="rusanov", time_scheme="EE")],
                         ids=["srk2", "rk2-local", "density-l2", "rusanov-ee"])
def test_slot_groups_of_full_size_solves_equal_single_solves(naca_hr, diamond02, counts, options):
    """What a full-size float32 batch runs (64-cell tiles; groups of 8 slots, of
    4 where 8 would leave a fifth of them empty, each mesh its own width where
    single-slot meshes prevail) on one mesh and on two of unequal slot counts,
    with an idle slot in the first group: every sampled slot ends bitwise equal
    to the same case advanced alone."""
    from eulersr_b200.solver import DeviceMesh, FlowCase, Solver
    meshes = [DeviceMesh(naca_hr), DeviceMesh(diamond02)][:len(counts)]
    n = sum(counts)
    r = np.random.default_rng(n)
    cases = [FlowCase(mach=float(r.uniform(0.7, 3.0)), aoa_deg=float(r.uniform(-5, 5)), cfl=0.6, tf=1e9, dtype=np.float32,
                      threshold=1e-30) for _ in range(n)]
    s = Solver(meshes, list(counts), precision="f32", **options)
    run = [g for g in range(n) if counts[0] < 3 or g != 1]
    s.set_cases(run, [cases[g] for g in run])
    s.step(9)
    for g in sorted({0, counts[0] // 2, counts[0] - 1, n - 1} & set(run)):
        one = Solver(meshes[0 if g < counts[0] else 1], 1, precision="f32", **options)
        one.set_case(0, cases[g])
        one.step(9)
        want, got = one.get_state(0), s.get_state(g)
        assert np.isfinite(want).all() and np.array_equal(want, got), g
        one.close()
    s.close()


@pytest.mark.parametrize("counts", [(4,), (6,), (3, 20)])
@pytest.mark.parametrize("dt_mode", ["global", "local"])
def test_float64_slot_groups_of_full_size_solves_equal_single_solves(naca_hr, diamond02, counts, dt_mode):
    """The same for the float64 stage kernel's 64-cell tiles and groups of 4."""
    from eulersr_b200.solver import DeviceMesh, FlowCase, Solver
    meshes = [DeviceMesh(naca_hr), DeviceMesh(diamond02)][:len(counts)]
    n = sum(counts)
    r = np.random.default_rng(n)
    cases = [FlowCase(mach=float(r.uniform(0.7, 3.0)), aoa_deg=float(r.uniform(-5, 5)), cfl=0.6, tf=1e9) for _ in range(n)]
    s = Solver(meshes, list(counts), precision="f64", dt_mode=dt_mode)
    s.set_cases(list(range(n)), cases)
    s.step(6)
    for g in sorted({0, counts[0] - 1, n - 1}):
        one = Solver(meshes[0 if g < counts[0] else 1], 1, precision="f64", dt_mode=dt_mode)
        one.set_case(0, cases[g])
        one.step(6)
        assert np.array_equal(one.get_state(0), s.get_state(g)), g
        one.close()
    s.close()
