"""The autotuner keeps Hamiltonians apart whose products take different forms
(needs a B200).

Scaling the channels of every bond of an MPO leaves the operator and its
widths as they are but hides the identity channels, so its tcgen05 product is the
general one: it is measured for itself, and both runs agree with the FP64
oracle to the mixed bound of test_gpu_mixed.py (1e-5).
"""
import ctypes as C

import numpy as np
import pytest

from yaqs_julia_b200 import _abi as A
from yaqs_julia_b200 import _lib, api

pytestmark = pytest.mark.gpu


def _shapes(ctx):
    n = C.c_int32(0)
    ctx.check(ctx._lib.yaqs_autotune_results(ctx.handle, None, 0, C.byref(n)))
    rows = np.zeros((max(n.value, 1), 8))
    ctx.check(ctx._lib.yaqs_autotune_results(ctx.handle, A.dptr(rows), n.value, C.byref(n)))
    return [tuple(int(x) for x in r[:5]) for r in rows[:n.value]]


def _scaled_channels(H):
    ts = [t.copy() for t in H.tensors]
    for b in range(1, H.length):
        g = np.linspace(0.5, 2.5, H.bond_dims[b])
        ts[b - 1] = ts[b - 1] * g
        ts[b] = ts[b] / g[:, None, None, None]
    return api.MPO(H.length, ts)


def test_equal_widths_with_and_without_identity_channels(oracle):
    L, chi = 9, 13  # widths 5 at bonds no other test tunes
    plain = api.init_general_hamiltonian(L, 1, 0.8, 0.6, 0, 0, 0.3)
    obs = [api.Observable(f"Z{i}", api.Z, i) for i in range(1, L + 1)]
    nm = api.NoiseModel([{"name": "pauli_z", "sites": [i], "strength": 0.1} for i in range(1, L + 1)], L)
    ctx = _lib.default_context()
    counts = []
    for H in (plain, _scaled_channels(plain)):
        assert H.bond_dims == plain.bond_dims
        cfg = api.TimeEvolutionConfig(obs, 0.1, dt=0.05, num_traj=3, max_bond_dim=chi)
        d = api.Descriptors(api.random_mps(L, chi, seed=2), H, cfg, nm, seed=1, precision=A.YAQS_PREC_MIXED,
                            tdvp_mode=api.TDVP_MODES["1site"])
        ref, _, _ = oracle.analog_run(d)
        assert np.abs(api.run_descriptors(d, ctx).trajectories - ref).max() <= 1e-5
        counts.append(_shapes(ctx).count((chi, 2, chi, 5, 5)))
    assert counts == [1, 2]
