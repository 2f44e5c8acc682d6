"""FP64 TDVP sweeps keep the order of their sums (needs a B200).

Where a bond's basis holds directions that rounding decides (after a
non-unitary jump, after growth from a product state, in a chain with a
symmetry), a sweep follows those directions, and another order of the sums
moves the records by 1e-9 to 1e-4.  golden/kept_order.json holds the records
of the general path (plain products, column QR, projections on the whole
basis, full environments) on a B200 for five such problems, one of them a
circuit of TDVP windows; its order gives the same states.  Bound: 1e-12, about
100 roundings of a contraction over 128 values.  One more problem has records
that a symmetry makes zero: they are nothing but rounding and are equal only
if every sum is.
"""
import json
import os

import numpy as np
import pytest

from yaqs_julia_b200 import _abi as A
from yaqs_julia_b200 import api

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "kept_order.json")


def _desc(psi, H, procs, steps, nt, chi, tdvp, **kw):
    L = psi.length
    obs = [api.Observable(f"Z{i}", api.Z, i) for i in range(1, L + 1)]
    obs.append(api.Observable("S", None, L // 2, kind="entropy"))
    cfg = api.TimeEvolutionConfig(obs, steps * 0.05, dt=0.05, num_traj=nt, max_bond_dim=chi)
    return api.Descriptors(psi, H, cfg, api.NoiseModel(procs, L), tdvp_mode=api.TDVP_MODES[tdvp], **kw)


def _procs(name, sites, strength=0.1):
    return [{"name": name, "sites": [i], "strength": strength} for i in sites]


def _evolved_xy():
    """A saturated state with the chain's symmetry: 2-site sweeps from Neel."""
    L, H = 12, api.init_general_hamiltonian(12, 1, 1, 0, 0, 0, 0.3)
    cfg = api.TimeEvolutionConfig([api.Observable("Z1", api.Z, 1)], 0.6, dt=0.1, num_traj=1, max_bond_dim=16,
                                  truncation_threshold=1e-24)
    s = api.Session(api.Descriptors(api.MPS(L, state="Neel"), H, cfg, api.NoiseModel(_procs("pauli_z", [1], 1e-12), L),
                                    seed=1))
    s.advance(s.remaining)
    psi = s.state(0)
    s.finish()
    return psi, H


def _problem(name):
    if name == "jump_right_of_the_middle":  # trajectory 0 jumps at every chance, trajectory 1 never
        u = np.zeros((2, 16))
        u[1] = 0.999999
        return _desc(api.random_mps(16, 128, seed=5), api.init_general_hamiltonian(16, 1, 1, 1, 0, 0, 0.5),
                     _procs("lowering", [9], 0.3), 2, 2, 128, "1site", rng_mode=A.YAQS_RNG_INJECTED, uniforms=u)
    if name == "dynamic_from_a_product":
        return _desc(api.MPS(11, state="Neel"), api.init_general_hamiltonian(11, 1.4, 0.6, 0, 0, 0, 0),
                     _procs("pauli_z", range(1, 12)), 6, 4, 16, "dynamic", seed=11)
    if name == "padded_start":
        return _desc(api.MPS(10, state="Neel", pad=16), api.init_general_hamiltonian(10, 1, 1, 1, 0, 0, 0.5),
                     _procs("lowering", range(1, 11)), 6, 4, 16, "1site", seed=3)
    if name == "zero_by_symmetry":
        L = 3
        obs = [api.Observable(f"Z{i}", api.Z, i) for i in range(1, L + 1)]
        cfg = api.TimeEvolutionConfig(obs, 0.8, dt=0.1, num_traj=8, max_bond_dim=16, order=1)
        return api.Descriptors(api.MPS(L, state="x+"), api.init_ising(L, 1.0, 0.7), cfg,
                               api.NoiseModel(_procs("pauli_z", range(1, L + 1)), L), seed=4)
    if name == "tdvp_windows":
        L, c = 12, api.DigitalCircuit(12)
        for _ in range(5):
            for i in list(range(1, L, 2)) + list(range(2, L, 2)):
                c.add_gate(api.RzzGate(0.1), [i, i + 1])
            for i in range(1, L + 1):
                c.add_gate(api.Rx(0.1), [i])
            c.add_gate(api.Barrier(), [])
        obs = [api.Observable(f"{n}{i}", op, i) for i in range(1, L + 1) for n, op in (("Z", api.Z), ("X", api.X))]
        cfg = api.TimeEvolutionConfig(obs, 4.0, dt=1.0, num_traj=12, max_bond_dim=64, truncation_threshold=1e-6)
        nm = api.NoiseModel([{"name": n, "sites": [i], "strength": 0.01} for i in range(1, L + 1)
                             for n in ("pauli_x", "pauli_y", "pauli_z")], L)
        return api.CircuitDescriptors(api.MPS(L, state="x+"), c, cfg, nm, seed=4, local_method="tdvp",
                                      long_range_method="tdvp")
    psi, H = _evolved_xy()
    return _desc(psi, H, _procs("pauli_z", range(1, 13)), 12, 4, 16, "1site", seed=2)


NAMES = ["jump_right_of_the_middle", "dynamic_from_a_product", "padded_start", "evolved_symmetric_start", "tdvp_windows"]


def _run(d):
    return (api.run_circuit_descriptors if isinstance(d, api.CircuitDescriptors) else api.run_descriptors)(d)


def _golden(name):
    return np.array(json.load(open(GOLDEN))[name])


@pytest.mark.parametrize("name", NAMES)
def test_records_of_the_general_path(name):
    res = _run(_problem(name))
    ref = _golden(name)
    assert res.trajectories.shape == ref.shape
    assert np.abs(res.trajectories - ref).max() <= 1e-12
    if name == "jump_right_of_the_middle":
        assert res.stats["jumps"] >= 2


def test_records_of_pure_rounding():
    res = _run(_problem("zero_by_symmetry"))
    ref = _golden("zero_by_symmetry")
    assert 0 < np.abs(ref).max() < 1e-14
    assert np.array_equal(res.trajectories, ref)
