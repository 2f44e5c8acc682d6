"""Device memory held between runs is given back on request (needs a B200)."""
import pytest
import torch

from yaqs_julia_b200 import _lib, api

pytestmark = pytest.mark.gpu


def _problem(L=24, chi=32, nt=200):
    obs = [api.Observable("Z1", api.Z, 1)]
    cfg = api.TimeEvolutionConfig(obs, 0.0, dt=0.05, num_traj=nt, max_bond_dim=chi, order=1)
    nm = api.NoiseModel([{"name": "pauli_z", "sites": [1], "strength": 0.1}], L)
    return api.random_mps(L, chi, seed=1), api.init_ising(L, 1.0, 0.5), cfg, nm


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info(0)[0]


def test_context_gives_its_memory_back_and_runs_on():
    ctx = _lib.Context(0)
    before = _free()
    a = api.run_descriptors(api.Descriptors(*_problem(), seed=1), ctx)
    held = before - _free()
    ctx.trim()
    left = before - _free()
    b = api.run_descriptors(api.Descriptors(*_problem(), seed=1), ctx)
    ctx.close()
    assert held >= 64 << 20  # the states alone take 170 MB
    assert left <= 8 << 20
    assert (a.trajectories == b.trajectories).all()


def test_server_gives_its_memory_back_and_serves_on():
    with api.Server(max_L=24, max_bond_dim=32, max_mpo_width=3, mixed=False) as srv:
        srv.trim()
        before = _free()
        a = srv.result(srv.submit(*_problem(), seed=1), timeout=300)
        held = before - _free()
        srv.trim()
        left = before - _free()
        b = srv.result(srv.submit(*_problem(), seed=1), timeout=300)
    assert held >= 64 << 20
    assert left <= 8 << 20
    assert (a.trajectories == b.trajectories).all()
