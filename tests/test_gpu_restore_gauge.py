"""Restoring checkpoints: the look at the restored gauge (needs a B200).

Mixed runs and circuits read records from the canonical form.  A restored
trajectory in another gauge takes the run's records off it; restoring a
canonical one brings them back, bit for bit; and the look costs no more than
the copies beside it.
"""
import time

import numpy as np
import pytest

from yaqs_julia_b200 import _abi as A
from yaqs_julia_b200 import api

pytestmark = pytest.mark.gpu


def _desc(L, chi, nt, steps, start):
    obs = [api.Observable(f"Z{i}", api.Z, i) for i in range(1, L + 1)]
    cfg = api.TimeEvolutionConfig(obs, steps * 0.05, dt=0.05, num_traj=nt, max_bond_dim=chi)
    nm = api.NoiseModel([{"name": "pauli_z", "sites": [i], "strength": 0.2} for i in range(1, L + 1)], L)
    psi = api.random_mps(L, chi, seed=2) if start == "random" else api.MPS(L, state="Neel")
    return api.Descriptors(psi, api.init_general_hamiltonian(L, 1, 1, 1, 0, 0, 0.4), cfg, nm, seed=6,
                           tdvp_mode=api.TDVP_MODES["1site" if start == "random" else "2site"],
                           precision=A.YAQS_PREC_MIXED)


def _skew(psi, b):
    """The same state with bond b (between sites b and b + 1) in another gauge."""
    g = np.diag(np.linspace(0.5, 2.0, psi.tensors[b - 1].shape[2])).astype(complex)
    psi.tensors[b - 1] = np.einsum("lpr,rs->lps", psi.tensors[b - 1], g)
    psi.tensors[b] = np.einsum("sr,rpt->spt", np.linalg.inv(g), psi.tensors[b])


@pytest.mark.parametrize("which,b", [(0, 1), (4, 5), (2, 7)])
def test_canonical_records_return_with_a_canonical_checkpoint(which, b):
    d = _desc(8, 16, 5, 4, "Neel")
    straight = api.run_descriptors(d)
    s = api.Session(d)
    s.advance(2)
    cp, other = s.checkpoint(), s.checkpoint()
    _skew(other["states"][which], b)
    s.restore(other)
    s.advance(1)
    s.restore(cp)
    s.advance(s.remaining)
    got = s.finish()
    assert np.array_equal(got.trajectories, straight.trajectories)


def test_restoring_costs_no_more_than_copying():
    s = api.Session(_desc(16, 128, 12, 1, "random"))
    s.advance(1)
    cp = s.checkpoint()
    s.restore(cp)
    best = [1e9, 1e9]
    for _ in range(3):
        t0 = time.perf_counter()
        s.checkpoint()
        t1 = time.perf_counter()
        s.restore(cp)
        best = [min(best[0], t1 - t0), min(best[1], time.perf_counter() - t1)]
    s.finish()
    assert best[1] <= 4 * best[0]
