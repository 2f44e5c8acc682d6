"""Served FP64 requests against the same request run directly (needs a B200).

One-site and dynamic sweeps and circuits with bonds up to 32, in a server that
admits mixed requests (its batches run in the tensor-core kernel).  FP64
analog requests and circuits on 256-thread programs give the same bits; the
default direct circuit runs 128-thread programs, whose block sums add in
another order: 1e-12 for some thousand roundings of values up to 1.
"""
import numpy as np
import pytest

from yaqs_julia_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("start", ["random", "Neel"])
@pytest.mark.parametrize("tdvp", ["1site", "dynamic"])
def test_sweeps(tdvp, start):
    with api.Server(max_L=11, max_bond_dim=33, max_mpo_width=5, chunk=2) as srv:
        for chi in (8, 16, 33):
            L = 11
            obs = [api.Observable(f"Z{i}", api.Z, i) for i in range(1, L + 1)]
            obs.append(api.Observable("S", None, L // 2, kind="entropy"))
            cfg = api.TimeEvolutionConfig(obs, 0.2, dt=0.05, num_traj=6, max_bond_dim=chi)
            nm = api.NoiseModel([{"name": "lowering", "sites": [i], "strength": 0.1} for i in range(1, L + 1)], L)
            psi = api.random_mps(L, chi, seed=1) if start == "random" else api.MPS(L, state="Neel")
            problem = (psi, api.init_general_hamiltonian(L, 1, 0.8, 0.6, 0, 0, 0.3), cfg, nm)
            served = srv.result(srv.submit(*problem, seed=5, tdvp=tdvp), timeout=300)
            direct = api.run_descriptors(api.Descriptors(*problem, seed=5, tdvp_mode=api.TDVP_MODES[tdvp]))
            assert np.array_equal(served.trajectories, direct.trajectories)
            assert np.array_equal(served.max_bond, direct.max_bond)


@pytest.mark.parametrize("noise", ["pauli_x", "lowering"])
def test_circuits(noise, monkeypatch):
    L, rng = 11, np.random.default_rng(3)
    c = api.DigitalCircuit(L)
    for _ in range(4):
        for i in list(range(1, L, 2)) + list(range(2, L, 2)):
            c.add_gate(api.Rzz(rng.uniform(0.2, 1.2)), [i, i + 1])
            c.add_gate(api.Rxx(rng.uniform(0.2, 1.2)), [i, i + 1])
        for i in range(1, L + 1):
            c.add_gate(api.Rx(rng.uniform(0.2, 1.2)), [i])
        c.add_gate(api.Barrier(), [])
    obs = [api.Observable(f"Z{i}", api.Z, i) for i in range(1, L + 1)]
    cfg = api.TimeEvolutionConfig(obs, 3.0, dt=1.0, num_traj=12, max_bond_dim=32)
    nm = api.NoiseModel([{"name": noise, "sites": [i], "strength": 0.05} for i in range(1, L + 1)], L)
    problem = (api.MPS(L), c, cfg, nm)
    with api.Server(max_L=11, max_bond_dim=32, max_mpo_width=5, chunk=2) as srv:
        served = srv.result(srv.submit(*problem, seed=5), timeout=300)
    assert served.max_bond.max() == 32
    for threads, bound in (("256", 0.0), ("128", 1e-12)):
        monkeypatch.setenv("YAQS_DIGITAL_THREADS", threads)
        direct = api.run_circuit_descriptors(api.CircuitDescriptors(*problem, seed=5))
        assert np.abs(served.trajectories - direct.trajectories).max() <= bound
        assert np.array_equal(served.max_bond, direct.max_bond)
