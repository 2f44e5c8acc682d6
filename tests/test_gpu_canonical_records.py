"""One-site records read from the canonical form (needs a B200).

The values must equal the oracle's centre sweep wherever the centre stands,
with observables on some sites only, and a run whose gates or restored
tensors leave the canonical form must fall back to full environments.
Bound: 1e-10, the parity bar of the trajectory tests.
"""
import numpy as np
import pytest

from yaqs_julia_b200 import api

pytestmark = pytest.mark.gpu


def _circuit(L, gates):
    c = api.DigitalCircuit(L)
    for op, sites in gates:
        c.add_gate(op, sites)
    c.add_gate(api.Barrier(), [])
    return c


@pytest.mark.parametrize("last", [1, 3, 6])
@pytest.mark.parametrize("where", [[1], [6, 7], [2, 5], list(range(1, 8))])
def test_centre_and_sites(oracle, last, where):
    """The last two-qubit gate puts the centre on site last + 1."""
    L = 7
    gates = [(api.Rx(0.3 + 0.2 * i), [i]) for i in range(1, L + 1)]
    gates += [(api.Rzz(0.7), [i, i + 1]) for i in (1, 3, 5, 2, 4, 6)] + [(api.Rxx(0.4), [last, last + 1])]
    obs = [api.Observable(f"{n}{i}", op, i) for i in where for n, op in (("Z", api.Z), ("X", api.X))]
    cfg = api.TimeEvolutionConfig(obs, 0.0, dt=1.0, num_traj=3, max_bond_dim=16)
    nm = api.NoiseModel([{"name": "pauli_x", "sites": [i], "strength": 0.1} for i in range(1, L + 1)], L)
    d = api.CircuitDescriptors(api.MPS(L), _circuit(L, gates), cfg, nm, seed=2)
    ref, _, _ = oracle.digital_run(d)
    got = api.run_circuit_descriptors(d)
    assert np.abs(got.trajectories - ref).max() <= 1e-10


def test_restored_tensors_in_another_gauge():
    """A similarity on a bond leaves the state and its records unchanged but
    not the canonical form; the restored run records the same values."""
    L = 6
    obs = [api.Observable(f"Z{i}", api.Z, i) for i in range(1, L + 1)]
    gates = [(api.Rx(0.4 * i), [i]) for i in range(1, L + 1)] + [(api.Rzz(0.9), [i, i + 1]) for i in (1, 3, 5, 2, 4)]
    c = _circuit(L, gates)
    c.add_gate(api.Rx(0.3), [2])
    c.add_gate(api.Barrier(), [])
    cfg = api.TimeEvolutionConfig(obs, 1.0, dt=1.0, num_traj=1, max_bond_dim=16)
    out = []
    for skew in (False, True):
        s = api.Session(api.CircuitDescriptors(api.MPS(L), c, cfg, None, seed=1))
        s.advance(s.remaining - 1)
        cp = s.checkpoint()
        if skew:
            psi = cp["states"][0]
            g = np.diag(np.linspace(0.5, 2.0, psi.tensors[3].shape[2])).astype(complex)
            psi.tensors[3] = np.einsum("lpr,rs->lps", psi.tensors[3], g)
            psi.tensors[4] = np.einsum("sr,rpt->spt", np.linalg.inv(g), psi.tensors[4])
        s.restore(cp)
        s.advance(s.remaining)
        out.append(s.finish().trajectories)
    assert np.abs(out[0] - out[1]).max() <= 1e-10
