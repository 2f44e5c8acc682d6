"""The work that users of this engine have it do, as cases that can be timed.

A case is a dict of plain values; ``prepare`` makes from it and a seed what a
program holds before its call, ``run`` makes the call through the public entry
points and returns everything it computes, ``work`` counts what the call
cannot do without and ``exact`` gives 64-bit values where plain numpy has
them.  Kinds of case:

  analog   Simulator.run with an MPO: trajectories of a noisy spin chain
  digital  Simulator.run with a circuit (TEBD gates or TDVP windows)
  serve    requests of several sizes submitted together to one server

Every floating result is float64, except that a mixed-precision run's records
are kept as float32, which is what its FP32 products carry.
"""
from __future__ import annotations

import math

import numpy as np

from yaqs_julia_b200 import _abi as A
from yaqs_julia_b200 import api


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def _analog(name, **kw):
    c = dict(name=name, kind="analog", L=6, model="ising", start="zeros", noise="relax_deph", tdvp="2site",
             precision="fp64", chi=16, traj=200, steps=10, dt=0.1, thr=1e-9, order=2, obs="z", packed=False)
    c.update(kw)
    return c


def _digital(name, **kw):
    c = dict(name=name, kind="digital", circuit="ising", L=12, depth=4, chi=64, traj=128, noise="pauli",
             rate=0.01, method="tebd", thr=1e-9, packed=False)
    c.update(kw)
    return c


def listed():
    return [
        # a quick look at a three-spin chain: a handful of trajectories, so the
        # call's set-up, launch and read-back are what the user waits for
        _analog("analog_L3_smallest", L=3, chi=4, traj=4, steps=5),
        # the reference's own small workload: L = 6 Ising, relaxation and
        # dephasing, chi 16, dt 0.1 up to T = 5, 200 trajectories
        _analog("analog_L6_ising", thr=1e-10, steps=50),
        # an odd XY chain growing from the Neel state under the 2-site sweep,
        # with X, Z, two-site and entropy records
        _analog("analog_L13_xy_growth", L=13, model="xy", start="Neel", chi=64, traj=100, steps=12, dt=0.05,
                obs="rich"),
        # the headline configuration: L = 30 Heisenberg, chi 64, 1024
        # trajectories from a saturated start, mixed precision
        _analog("analog_L30_chi64_mixed", L=30, model="heisenberg", start="random", noise="deph", tdvp="dynamic",
                precision="mixed", chi=64, traj=1024, steps=1, dt=0.05, obs="z_entropy", packed=True),
        # the same chain in plain ComplexF64, a ragged number of trajectories
        # over two full time indices
        _analog("analog_L30_chi64_fp64", L=30, model="heisenberg", start="random", noise="deph", tdvp="dynamic",
                chi=64, traj=260, steps=2, dt=0.05, obs="z_entropy", packed=True),
        # one request of the uneven batch: a longer Ising chain, 2-site sweep,
        # bonds growing from a product state
        _analog("analog_L32_ising_2site", L=32, chi=32, traj=150, steps=6, dt=0.05),
        # the widest bonds that are served, one-site sweep
        _analog("analog_L16_chi128_1site", L=16, model="heisenberg", start="random", tdvp="1site", chi=128, traj=64,
                steps=1, dt=0.05, packed=True),
        # an ideal circuit run once without noise: the latency of one trajectory
        _digital("digital_ideal_n11", L=11, depth=6, traj=1, noise="none", thr=1e-13),
        # the digital benchmark: L = 40 Trotterised Ising, 60 layers, Pauli
        # noise after every 2-qubit gate, 512 trajectories
        _digital("digital_L40_ising", L=40, depth=60, chi=128, traj=512, packed=True),
        # a served QAOA request: ring of 20 qubits, two layers, the closing
        # edge through a SWAP chain, depolarising noise
        _digital("digital_ring20_qaoa", circuit="ring", L=20, depth=2, traj=300, rate=0.005 / 3),
        # the reference's default gate method: TDVP windows, relaxation noise
        _digital("digital_windows_n9", circuit="windows", L=9, depth=3, chi=32, traj=60, noise="relax_deph",
                 rate=0.02, method="tdvp"),
        # a server with analog and digital requests of uneven size in flight
        dict(name="serve_uneven", kind="serve", L=16, chi=32, requests=5, traj=100, steps=4, depth=2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["small", "growth", "saturated", "ising", "ring", "windows", "serve"])
    noise = rng.choice(["relax_deph", "deph"])
    model = rng.choice(["ising", "xy", "heisenberg"])
    if kind == "small":
        c = _analog("", L=rng.randint(2, 8), model=model, chi=16, traj=_log_int(rng, 1, 400),
                    start=rng.choice(["zeros", "Neel", "x+"]), noise=noise, steps=_log_int(rng, 2, 40),
                    thr=rng.choice([1e-9, 1e-10]), order=rng.choice([1, 2]))
    elif kind == "growth":
        c = _analog("", L=rng.randint(9, 40), model=model, start="zeros" if model == "ising" else "Neel", noise=noise,
                    chi=rng.choice([32, 64]), traj=_log_int(rng, 16, 150), steps=rng.randint(2, 6), dt=0.05,
                    obs=rng.choice(["z", "rich"]))
    elif kind == "saturated":
        chi = rng.choice([16, 23, 32, 48, 64])
        c = _analog("", L=rng.randint(12, 30), model=model, start="random", noise=noise,
                    tdvp=rng.choice(["dynamic", "1site"]), precision=rng.choice(["fp64", "mixed"]), chi=chi,
                    traj=_log_int(rng, 40, 300), steps=rng.randint(1, 2), dt=0.05,
                    obs=rng.choice(["z", "z_entropy"]), packed=True)
    elif kind == "ising":
        c = _digital("", L=rng.randint(8, 48), depth=_log_int(rng, 4, 30), chi=rng.choice([64, 128]),
                     traj=_log_int(rng, 16, 512), noise=rng.choice(["pauli", "relax_deph"]), rate=0.01, packed=True)
    elif kind == "ring":
        c = _digital("", circuit="ring", L=rng.randint(8, 20), depth=rng.randint(1, 2), traj=_log_int(rng, 32, 300),
                     rate=0.005 / 3)
    elif kind == "windows":
        c = _digital("", circuit="windows", L=rng.randint(4, 10), depth=rng.randint(1, 3), chi=32,
                     traj=_log_int(rng, 8, 60), noise=rng.choice(["pauli", "relax_deph"]), rate=0.02, method="tdvp")
    else:
        c = dict(kind="serve", L=rng.randint(8, 20), chi=rng.choice([16, 32]), requests=rng.randint(2, 6),
                 traj=_log_int(rng, 20, 100), steps=rng.randint(1, 4), depth=rng.randint(1, 2))
    c.pop("name", None)
    return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _noise(kind, L, rng, rate=None):
    if kind == "none":
        return None
    sites = range(1, L + 1)
    if kind == "pauli":
        return api.NoiseModel([{"name": n, "sites": [i], "strength": rate} for i in sites
                               for n in ("pauli_x", "pauli_y", "pauli_z")], L)
    g = [rate, rate] if rate is not None else rng.uniform(0.05, 0.15, 2)
    procs = [{"name": "pauli_z", "sites": [i], "strength": float(g[0])} for i in sites]
    if kind == "relax_deph":
        procs = [{"name": "lowering", "sites": [i], "strength": float(g[1])} for i in sites] + procs
    return api.NoiseModel(procs, L)


def _hamiltonian(model, L, rng):
    if model == "ising":
        return api.init_ising(L, 1.0, float(rng.uniform(0.3, 1.2)))
    if model == "xy":
        a = float(rng.uniform(0.1, 0.9))
        return api.init_general_hamiltonian(L, 1 + a, 1 - a, 0, 0, 0, 0)
    return api.init_general_hamiltonian(L, 1, 1, 1, 0, 0, float(rng.uniform(0.1, 0.9)))


def _observables(kind, L):
    obs = [api.Observable(f"Z{i}", api.Z, i) for i in range(1, L + 1)]
    if kind == "rich":
        obs += [api.Observable(f"X{i}", api.X, i) for i in range(1, L + 1)]
        obs += [api.Observable(f"ZZ{i}", np.kron(api.Z, api.Z), [i, i + 1]) for i in range(1, L, 3)]
    if kind in ("rich", "z_entropy"):
        obs.append(api.Observable("S_half", None, L // 2, kind="entropy"))
    return obs


def _analog_problem(case, seed):
    rng = np.random.default_rng(seed)
    L = case["L"]
    psi = (api.random_mps(L, case["chi"], seed=seed) if case["start"] == "random"
           else api.MPS(L, state=case["start"]))
    cfg = api.TimeEvolutionConfig(_observables(case["obs"], L), case["steps"] * case["dt"], dt=case["dt"],
                                  num_traj=case["traj"], max_bond_dim=case["chi"], truncation_threshold=case["thr"],
                                  order=case["order"])
    return psi, _hamiltonian(case["model"], L, rng), cfg, _noise(case["noise"], L, rng)


def _circuit_gates(case, seed):
    """The circuit as (generator name, angle, sites) in program order, None for a sampling barrier."""
    rng = np.random.default_rng(seed)
    L, gates = case["L"], []
    bonds = list(range(1, L, 2)) + list(range(2, L, 2))
    if case["circuit"] == "ising":
        a, b = 0.1 * rng.uniform(0.8, 1.2, 2)
        for _ in range(case["depth"]):
            gates += [("zz", a, [i, i + 1]) for i in bonds] + [("x", b, [i]) for i in range(1, L + 1)] + [None]
    elif case["circuit"] == "ring":
        for _ in range(case["depth"]):
            g, b = rng.uniform(0, np.pi, 2)
            gates += [("zz", g, [i, i + 1]) for i in bonds] + [("zz", g, [L, 1])]
            gates += [("x", b, [i]) for i in range(1, L + 1)]
    else:  # windows: nearest-neighbour XX and ZZ and one long-range ZZ a layer
        for _ in range(case["depth"]):
            t = rng.uniform(0.1, 0.4, 3)
            gates += [("xx", t[0], [i, i + 1]) for i in bonds] + [("zz", t[1], [1, min(L, 4)])]
            gates += [("x", t[2], [i]) for i in range(1, L + 1)] + [None]
    return gates


_GATES = {"zz": api.Rzz, "xx": api.Rxx, "x": api.Rx}
_WINDOW_GATES = {"zz": api.RzzGate, "xx": api.RxxGate, "x": api.Rx}


def _digital_problem(case, seed):
    L = case["L"]
    make = _WINDOW_GATES if case["method"] == "tdvp" else _GATES
    circ = api.DigitalCircuit(L)
    for g in _circuit_gates(case, seed):
        if g is None:
            circ.add_gate(api.Barrier(), [])
        else:
            circ.add_gate(make[g[0]](float(g[1])), g[2])
    n_samples = sum(g is None for g in _circuit_gates(case, seed)) or 1
    obs = [api.Observable(f"Z{i}", api.Z, i) for i in range(1, L + 1)]
    if case["circuit"] == "ring":
        obs = [api.Observable(f"ZZ{i}", np.kron(api.Z, api.Z), [i, i + 1]) for i in range(1, L)]
    cfg = api.TimeEvolutionConfig(obs, float(n_samples - 1), dt=1.0, num_traj=case["traj"],
                                  max_bond_dim=case["chi"], truncation_threshold=case["thr"])
    return api.MPS(L), circ, cfg, _noise(case["noise"], L, np.random.default_rng(seed), case["rate"])


def _requests(case, seed):
    """Uneven requests of one stream: analog FP64, QAOA ring, analog mixed, in turn."""
    rng = np.random.default_rng(case["L"])  # the sizes belong to the case, the values to the seed
    out = []
    for k in range(case["requests"]):
        L = int(rng.integers(max(4, case["L"] // 2), case["L"] + 1))
        nt = int(rng.integers(max(1, case["traj"] // 2), case["traj"] + 1))
        if k % 3 == 1:
            sub = _digital("", circuit="ring", L=L, depth=case["depth"], traj=nt, rate=0.005 / 3, chi=case["chi"])
            out.append((_digital_problem(sub, seed + k), dict(seed=seed + k)))
        elif k % 3 == 2:
            sub = _analog("", L=L, model="heisenberg", start="random", chi=case["chi"], traj=nt, dt=0.05,
                          steps=min(2, case["steps"]))
            out.append((_analog_problem(sub, seed + k), dict(seed=seed + k, precision="mixed", tdvp="dynamic")))
        else:
            sub = _analog("", L=L, model=["ising", "xy"][k % 2], start=["zeros", "Neel"][k % 2], chi=case["chi"],
                          traj=nt, dt=0.05, steps=case["steps"])
            out.append((_analog_problem(sub, seed + k), dict(seed=seed + k)))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        server = api.Server(max_L=case["L"], max_bond_dim=case["chi"], max_mpo_width=5, chunk=2,
                            hbm_budget=4 << 30)
        return dict(case=case, server=server, requests=_requests(case, seed))
    problem = _analog_problem(case, seed) if kind == "analog" else _digital_problem(case, seed)
    state = dict(case=case, seed=seed, problem=problem)
    if case["packed"]:  # the arrays as a Julia host has them, handed to the C entry point
        psi, op, cfg, nm = problem
        if kind == "analog":
            state["desc"] = api.Descriptors(
                psi, op, cfg, nm, seed=seed, tdvp_mode=api.TDVP_MODES[case["tdvp"]],
                precision=A.YAQS_PREC_MIXED if case["precision"] == "mixed" else A.YAQS_PREC_FP64)
        else:
            state["desc"] = api.CircuitDescriptors(psi, op, cfg, nm, seed=seed, local_method=case["method"],
                                                   long_range_method=case["method"])
    return state


# ---------------------------------------------------------------------------
# The calls
# ---------------------------------------------------------------------------
def _outputs(res, precision="fp64"):
    if precision == "mixed":
        return dict(trajectories=res.trajectories.astype(np.float32), mean=res.mean.astype(np.float32),
                    max_bond=res.max_bond)
    return dict(trajectories=res.trajectories, mean=res.mean, max_bond=res.max_bond)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "serve":
        server = state["server"]
        ids = [(server.submit(*problem, **kw), kw.get("precision", "fp64")) for problem, kw in state["requests"]]
        return [_outputs(server.result(rid), prec) for rid, prec in ids]
    if "desc" in state:
        go = api.run_descriptors if kind == "analog" else api.run_circuit_descriptors
        return _outputs(go(state["desc"]), case.get("precision", "fp64"))
    psi, op, cfg, nm = state["problem"]
    if kind == "analog":
        res = api.run(psi, op, cfg, nm, seed=state["seed"], tdvp=case["tdvp"], precision=case["precision"])
    else:
        res = api.run(psi, op, cfg, nm, seed=state["seed"], local_method=case["method"],
                      long_range_method=case["method"])
    return _outputs(res, case.get("precision", "fp64"))


# ---------------------------------------------------------------------------
# What a call cannot do without
# ---------------------------------------------------------------------------
_WIDTH = {"ising": 3, "xy": 4, "heisenberg": 5}


def _analog_work(L, chi, traj, steps, model, saturated, nobs, tdvp="2site"):
    """Effective-Hamiltonian products of the sweeps: a Lanczos solve takes no
    fewer than three of them, the identity blocks of the environments need no
    arithmetic (w - 1 of w blocks on each side), and a growing chain is
    counted at the bonds of its first layer."""
    b = [min(2 ** min(i, L - i, 60), chi if saturated else 2) for i in range(L + 1)]
    w = _WIDTH[model] - 1
    D = 4 if tdvp == "2site" else 2
    sites = sum(8.0 * w * D * b[i] * b[min(i + D // 2, L)] * (b[i] + b[min(i + D // 2, L)])
                for i in range(L - D // 2 + 1))
    sweeps = max(1, 2 * steps - 1)
    state = 32.0 * sum(b[i] * b[i + 1] for i in range(L))
    return {"flops": traj * sweeps * 2 * 3 * sites, "bytes": traj * (2.0 * state * steps + 8.0 * nobs * (steps + 1))}


def _digital_work(L, gates, traj, nobs, n_samples):
    """Every gate applied to sites of bond 2: merge, 4 x 4 map and a QR-sized
    factorisation of a 4 x 4 block; each trajectory's state read and written
    once a circuit."""
    return {"flops": traj * gates * 8.0 * (32 + 64 + 64), "bytes": traj * (2.0 * 128 * L + 8.0 * nobs * n_samples)}


def work(case):
    kind = case["kind"]
    if kind == "serve":
        one = _analog_work(case["L"], case["chi"], 0.75 * case["traj"], case["steps"], "ising", False, case["L"])
        return {k: v * case["requests"] for k, v in one.items()}
    if kind == "analog":
        nobs = len(_observables(case["obs"], case["L"]))
        return _analog_work(case["L"], case["chi"], case["traj"], case["steps"], case["model"],
                            case["start"] == "random", nobs, case["tdvp"])
    gates = [g for g in _circuit_gates(case, 1)]
    n2 = sum(g is not None and len(g[2]) == 2 for g in gates)
    return _digital_work(case["L"], n2, case["traj"], case["L"], sum(g is None for g in gates) or 1)


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------
_PAULI = {"z": np.diag([1.0, -1.0]).astype(complex), "x": np.array([[0, 1], [1, 0]], dtype=complex)}


def _rotate(v, name, angle, sites, L):
    """exp(-i angle/2 P) v for a Pauli string P (a Pauli on each listed site); axis k of v is site k + 1."""
    w = v
    for s in sites:
        w = np.moveaxis(np.tensordot(_PAULI[name[0]], w, axes=(1, s - 1)), 0, s - 1)
    return math.cos(angle / 2) * v - 1j * math.sin(angle / 2) * w


def exact(case, seed):
    if case["kind"] != "digital" or case["noise"] != "none" or case["circuit"] != "ising" or case["L"] > 14:
        return None  # stochastic records, or a splitting without a closed form
    L = case["L"]
    v = np.zeros((2,) * L, dtype=complex)
    v[(0,) * L] = 1.0
    rows = []
    for g in _circuit_gates(case, seed):
        if g is None:
            p = np.abs(v) ** 2
            rows.append([float(np.sum(p.take(0, axis=i)) - np.sum(p.take(1, axis=i))) for i in range(L)])
        else:
            v = _rotate(v, g[0], float(g[1]), g[2], L)
    z = np.array(rows).T
    return dict(trajectories=z[None], mean=z, max_bond=None)
