"""Panel QR and short Jacobi rounds against the oracle's column loops (needs a B200).

The one-site and dynamic sweeps factor every site of a saturated chain; the
bond dimensions put the factored matrices on both sides of a panel (16
columns) and of the row counts that change a warp's share (32, 64, 128, 256
rows).  A digital circuit with non-unitary noise and a tight threshold walks
and splits bonds of every size up to its cap.  Bound: 1e-10 of the largest
value, the bar of the trajectory parity tests, for two time indices.
"""
import numpy as np
import pytest

from yaqs_julia_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chi,tdvp", [(3, "1site"), (8, "dynamic"), (16, "1site"), (17, "dynamic"), (33, "1site"),
                                      (70, "1site")])
def test_saturated_sweeps_match_oracle(oracle, chi, tdvp):
    L = 8 if chi <= 8 else 13
    obs = [api.Observable(f"Z{i}", api.Z, i) for i in range(1, L + 1)]
    obs.append(api.Observable("S", None, L // 2, kind="entropy"))
    cfg = api.TimeEvolutionConfig(obs, 0.05, dt=0.05, num_traj=2, max_bond_dim=chi)
    nm = api.NoiseModel([{"name": "lowering", "sites": [i], "strength": 0.3} for i in range(1, L + 1)], L)
    d = api.Descriptors(api.random_mps(L, chi, seed=chi), api.init_general_hamiltonian(L, 1, 0.8, 0.6, 0.1, 0, 0.3),
                        cfg, nm, seed=3, tdvp_mode=api.TDVP_MODES[tdvp])
    ref, chi_ref, _ = oracle.analog_run(d)
    got = api.run_descriptors(d)
    assert np.abs(got.trajectories - ref).max() <= 1e-10 * max(1.0, np.abs(ref).max())
    assert np.array_equal(got.max_bond, chi_ref)


@pytest.mark.parametrize("chi", [33, 70])
def test_entropy_of_wide_bonds_matches_oracle(oracle, chi):
    """Singular values of 2 chi x chi centre tensors: 66 rows take 16 lanes a
    pair, 140 rows a whole warp."""
    L = 15
    obs = [api.Observable("S7", None, 7, kind="entropy"), api.Observable("S8", None, 8, kind="entropy")]
    cfg = api.TimeEvolutionConfig(obs, 0.0, dt=0.05, num_traj=1, max_bond_dim=chi, order=1)
    nm = api.NoiseModel([{"name": "pauli_z", "sites": [1], "strength": 0.1}], L)
    d = api.Descriptors(api.random_mps(L, chi, seed=1), api.init_ising(L, 1.0, 0.5), cfg, nm, seed=3,
                        tdvp_mode=api.TDVP_MODES["1site"])
    ref, _, _ = oracle.analog_run(d)
    got = api.run_descriptors(d)
    assert np.abs(got.trajectories - ref).max() <= 1e-10 * np.abs(ref).max()


@pytest.mark.parametrize("threads", ["128", "256"])
def test_circuit_bonds_match_oracle(oracle, threads, monkeypatch):
    monkeypatch.setenv("YAQS_DIGITAL_THREADS", threads)
    L = 9
    rng = np.random.default_rng(5)
    c = api.DigitalCircuit(L)
    for _ in range(4):
        for i in list(range(1, L, 2)) + list(range(2, L, 2)):
            c.add_gate(api.Rzz(rng.uniform(0.2, 1.5)), [i, i + 1])
            c.add_gate(api.Rxx(rng.uniform(0.2, 1.5)), [i, i + 1])
        for i in range(1, L + 1):
            c.add_gate(api.Rx(rng.uniform(0.2, 1.5)), [i])
        c.add_gate(api.Barrier(), [])
    obs = [api.Observable(f"Z{i}", api.Z, i) for i in range(1, L + 1)]
    cfg = api.TimeEvolutionConfig(obs, 3.0, dt=1.0, num_traj=6, max_bond_dim=32, truncation_threshold=1e-12)
    nm = api.NoiseModel([{"name": "lowering", "sites": [i], "strength": 0.05} for i in range(1, L + 1)] +
                        [{"name": "pauli_x", "sites": [i], "strength": 0.02} for i in range(1, L + 1)], L)
    d = api.CircuitDescriptors(api.MPS(L), c, cfg, nm, seed=9)
    ref, chi_ref, _ = oracle.digital_run(d)
    got = api.run_circuit_descriptors(d)
    assert np.abs(got.trajectories - ref).max() <= 1e-10
    assert np.array_equal(got.max_bond, chi_ref)
