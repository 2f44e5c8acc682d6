"""Hamiltonians that carry an operator across a site, and states that spoil the
identity channels (needs a B200).

An XX coupling over two sites beside a ZZ one keeps an MPO channel open through
a site, so the structured products of the mixed form have pass-through terms;
odd bonds of 17 and 33 lie above the shared-memory solves.  The oracle runs
the same problems in FP64: 1e-10 for the FP64 sweeps, 1e-5 for the mixed ones,
the bounds of the trajectory parity tests.
"""
import numpy as np
import pytest

from yaqs_julia_b200 import _abi as A
from yaqs_julia_b200 import api

pytestmark = pytest.mark.gpu
BOUND = {"fp64": 1e-10, "mixed": 1e-5}


def next_nearest(L, j1, j2, h, decay=None):
    """sum j1 Z Z + j2 X_i X_(i+2) + h Z as an MPO; with decay, X X at every
    distance r, j2 decay^(r-2), through a channel that feeds itself."""
    w = 5  # 0: not started, 1: Z waits, 2: X waits for one site, 3: X may end, 4: ended
    eye, x, z = np.eye(2), api.X, api.Z
    W = np.zeros((w, 2, 2, w), dtype=complex)
    W[0, :, :, 0] = W[4, :, :, 4] = eye
    W[0, :, :, 1], W[1, :, :, 4] = z, j1 * z
    W[0, :, :, 2], W[2, :, :, 3], W[3, :, :, 4] = x, eye, j2 * x
    if decay:
        W[3, :, :, 3] = decay * eye
    W[0, :, :, 4] = h * z
    ts = [W.copy() for _ in range(L)]
    ts[0], ts[-1] = W[:1].copy(), W[..., -1:].copy()
    return api.MPO(L, ts)


def _dense(L, j1, j2, h):
    def on(*ops):
        out = np.ones((1, 1))
        for i in range(L):
            out = np.kron(out, dict(ops).get(i, np.eye(2)))
        return out
    H = sum(h * on((i, api.Z)) for i in range(L))
    H = H + sum(j1 * on((i, api.Z), (i + 1, api.Z)) for i in range(L - 1))
    return H + sum(j2 * on((i, api.X), (i + 2, api.X)) for i in range(L - 2))


def test_the_mpo_is_the_operator():
    assert np.abs(next_nearest(5, 0.8, 0.6, 0.3).to_matrix() - _dense(5, 0.8, 0.6, 0.3)).max() < 1e-14


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("tdvp", ["1site", "dynamic"])
@pytest.mark.parametrize("chi,decay", [(17, None), (33, None), (17, 0.5)])
def test_pass_through_terms_match_oracle(oracle, chi, decay, tdvp, precision):
    L = 11
    obs = [api.Observable(f"{n}{i}", op, i) for i in range(1, L + 1) for n, op in (("Z", api.Z), ("X", api.X))]
    cfg = api.TimeEvolutionConfig(obs, 0.1, dt=0.05, num_traj=3, max_bond_dim=chi)
    nm = api.NoiseModel([{"name": "pauli_z", "sites": [i], "strength": 0.4} for i in range(1, L + 1)], L)
    d = api.Descriptors(api.random_mps(L, chi, seed=chi), next_nearest(L, 0.8, 0.6, 0.3, decay), cfg, nm, seed=3,
                        tdvp_mode=api.TDVP_MODES[tdvp],
                        precision=A.YAQS_PREC_MIXED if precision == "mixed" else A.YAQS_PREC_FP64)
    ref, chi_ref, _ = oracle.analog_run(d)
    got = api.run_descriptors(d)
    assert got.stats["jumps"] > 0
    assert np.abs(got.trajectories - ref).max() <= BOUND[precision]
    assert np.array_equal(got.max_bond, chi_ref)


@pytest.mark.parametrize("spoilt", [2, 6, 9])
def test_a_spoilt_channel_takes_the_general_product(spoilt):
    """A restored state in another gauge left or right of its centre has no
    identity in the environments beyond that bond.  The same sweep with the
    structured products switched off by hidden channels (scaled MPO bonds) gives
    the same records to FP32 rounding."""
    L, chi = 11, 17
    H = next_nearest(L, 0.8, 0.6, 0.3)
    hidden = [t.copy() for t in H.tensors]
    for b in range(1, L):
        g = np.linspace(0.5, 2.0, 5)
        hidden[b - 1], hidden[b] = hidden[b - 1] * g, hidden[b] / g[:, None, None, None]
    obs = [api.Observable(f"Z{i}", api.Z, i) for i in range(1, L + 1)]
    cfg = api.TimeEvolutionConfig(obs, 0.1, dt=0.05, num_traj=2, max_bond_dim=chi, order=1)
    nm = api.NoiseModel([{"name": "pauli_z", "sites": [1], "strength": 0.01}], L)
    out = []
    for op in (H, api.MPO(L, hidden)):
        s = api.Session(api.Descriptors(api.random_mps(L, chi, seed=4), op, cfg, nm, seed=3,
                                        tdvp_mode=api.TDVP_MODES["1site"], precision=A.YAQS_PREC_MIXED))
        s.advance(1)
        cp = s.checkpoint()
        for psi in cp["states"]:
            g = np.diag(np.linspace(0.6, 1.4, psi.tensors[spoilt - 1].shape[2])).astype(complex)
            psi.tensors[spoilt - 1] = np.einsum("lpr,rs->lps", psi.tensors[spoilt - 1], g)
            psi.tensors[spoilt] = np.einsum("sr,rpt->spt", np.linalg.inv(g), psi.tensors[spoilt])
        s.restore(cp)
        s.advance(s.remaining)
        out.append(s.finish().trajectories)
    assert np.abs(out[0] - out[1]).max() <= 1e-5
