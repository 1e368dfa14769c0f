"""Measured work of the framework, through its public entry points.

A case is one thing that a program using the framework has it do over and over: an
epidemic on a resident population (whole, or a day at a time), a run from parameters
to output counts, a batch of replicates and scenarios, the simulation of intervention
scenarios for the surrogate, surrogate inference from host or device buffers, and a
training epoch of the surrogate's network.  ``listed`` names the fixed cases, ``draw``
draws one more of the same ranges.
"""
import json

import numpy as np
import torch

import pandemicthrust_gb300 as pt
from pandemicthrust_gb300 import scenarios as scn
from pandemicthrust_gb300 import surrogate as sg

PERSONS_PER_SCALE = 2.354e6   # expected persons at people_scaling 1


def listed():
    return [
        # A caller that looks at every day (pt_step_day), on the smallest population of
        # the smoke test: launches and round trips count.
        dict(name="step_24k_8d", kind="step", persons=23_540, ratio=1.0, days=8, r_p=1.8, r_s=1.3, seeds=30, iv=False),
        # The small configuration: 100,000 persons, 30 days, R 1.4 / 1.2, 10 seeds each.
        dict(name="run_100k_30d", kind="run", persons=100_000, ratio=1.0, days=30, r_p=1.4, r_s=1.2, seeds=10,
             iv=False),
        # One scenario with interventions at the surrogate's population size.
        dict(name="run_1M_interventions", kind="run", persons=1_000_003, ratio=1.0, days=100, r_p=1.8, r_s=1.6,
             seeds=100, iv=True),
        # A dense epidemic with as many locations per person as the thesis-style runs:
        # most errand buckets are read on most days.
        dict(name="run_12M_dense", kind="run", persons=12_000_000, ratio=1.0, days=60, r_p=2.0, r_s=1.7, seeds=1000,
             iv=False),
        # The headline: 50M persons, 100 days, R 1.5 / 1.2, ten times the locations.
        dict(name="run_50M_100d", kind="run", persons=50_000_000, ratio=10.0, days=100, r_p=1.5, r_s=1.2, seeds=100,
             iv=False),
        # A whole run as the executable does it: population setup, days, generation counts.
        dict(name="fresh_4M_100d", kind="fresh", persons=4_000_000, ratio=1.0, days=100, r_p=1.8, r_s=1.3, seeds=30,
             iv=False),
        # Replicates and scenarios of uneven size in one batch (sizes log-uniform, R
        # uniform in [1.1, 2.0]).
        dict(name="batch_48", kind="batch", instances=48, low=200_000, high=4_000_000, days=100),
        # Training data of the surrogate: intervention scenarios at 1M persons, from
        # scenario dicts to daily curves.
        dict(name="simulate_24x1M", kind="simulate", scenarios=24, replicates=1, persons=1_000_000),
        # The planner asking about a few scenarios: 32 rows, host arrays, shipped ensemble.
        dict(name="predict_32_host", kind="predict", rows=32, where="host", chunk=4096, members=0, hidden=256, depth=4),
        # The intervention search's scoring step: 100,000 candidates, host arrays.
        dict(name="predict_100k_host", kind="predict", rows=100_000, where="host", chunk=131_072, members=0,
             hidden=256, depth=4),
        # Bulk screening on device buffers.
        dict(name="predict_262k_device", kind="predict", rows=262_144, where="device", chunk=262_144, members=0,
             hidden=256, depth=4),
        # One epoch of the surrogate's training at its batch size (32 steps of forward,
        # backward and Adam), weights in and out.
        dict(name="train_16k", kind="train", rows=16_384, batch=512, hidden=256, depth=4, outputs=sg.OUTPUTS),
    ]


def _log_uniform(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def draw(rng):
    kind = rng.choice(["step", "run", "run", "fresh", "batch", "simulate", "predict", "predict", "train"])
    if kind in ("step", "run", "fresh"):
        most = {"step": 2e6, "run": 2e7, "fresh": 8e6}[kind]
        persons = int(_log_uniform(rng, 1e4, most)) | 1
        return dict(kind=kind, persons=persons, ratio=rng.choice([1.0, 1.0, 3.0, 10.0]),
                    days=rng.randint(8, 20 if kind == "step" else 100), r_p=round(rng.uniform(1.1, 2.0), 3),
                    r_s=round(rng.uniform(1.1, 2.0), 3), seeds=int(_log_uniform(rng, 10, 1000)),
                    iv=rng.random() < 0.4)
    if kind == "batch":
        return dict(kind=kind, instances=int(_log_uniform(rng, 2, 40)), low=int(_log_uniform(rng, 2e4, 2e5)),
                    high=int(_log_uniform(rng, 3e5, 3e6)), days=rng.randint(20, 100))
    if kind == "simulate":
        return dict(kind=kind, scenarios=int(_log_uniform(rng, 2, 20)), replicates=rng.randint(1, 3),
                    persons=int(_log_uniform(rng, 2e4, 4e5)) | 1)
    if kind == "predict":
        shipped = rng.random() < 0.6
        return dict(kind=kind, rows=int(_log_uniform(rng, 1, 250_000)) | 1, where=rng.choice(["host", "device"]),
                    chunk=rng.choice([4096, 65_536, 262_144]), members=0 if shipped else rng.randint(1, 5),
                    hidden=256 if shipped else rng.choice([32, 96, 128, 256]),
                    depth=4 if shipped else rng.randint(2, 4))
    return dict(kind="train", rows=int(_log_uniform(rng, 500, 16_000)) | 1, batch=rng.choice([32, 100, 128, 256, 512]),
                hidden=rng.choice([32, 100, 128, 256]), depth=rng.randint(1, 4), outputs=rng.choice([3, 24, sg.OUTPUTS]))


# ------------------------------------------------------------------ inputs
def _params(case):
    scale = case["persons"] / PERSONS_PER_SCALE
    return scn.scenario(max_days=case["days"], r_pandemic=case["r_p"], r_seasonal=case["r_s"],
                        initial_pandemic=case["seeds"], initial_seasonal=case["seeds"], people_scaling=scale,
                        location_scaling=scale * case["ratio"])


def _scenario_list(n, seed):
    return sg.sample_scenarios(n, np.random.default_rng(seed))


def _features(rows, seed):
    """Rows as surrogate.features makes them: seven scaled parameters and four derived inputs."""
    rng = np.random.default_rng(seed)
    X = np.empty((rows, 11), np.float32)
    X[:, :7] = rng.random((rows, 7), dtype=np.float32)
    vaccination = 0.5 * X[:, 6]
    X[:, 7] = (1.1 + 0.9 * X[:, 0]) * (1 - vaccination) / 2.0
    X[:, 8] = (1.1 + 0.9 * X[:, 1]) * (1 - vaccination) / 2.0
    start, length = np.rint(60 * X[:, 3]), np.rint(42 * X[:, 4])
    X[:, 3], X[:, 4] = start / 60, length / 42
    X[:, 9] = (start + length) / 100
    X[:, 10] = (np.minimum(start + length, 60) - start) / 60
    return X


def _weights(widths, seed):
    """He-uniform matrices rounded to BF16 (as a saved model holds them) and small biases, in the library's order."""
    rng = np.random.default_rng(seed)
    parts = []
    for a, b in zip(widths[:-1], widths[1:]):
        w = rng.uniform(-1, 1, (b, a)).astype(np.float32) * np.float32((6.0 / a) ** 0.5)
        parts += [torch.from_numpy(w).to(torch.bfloat16).float().numpy().ravel(),
                  rng.normal(0, 0.05, b).astype(np.float32)]
    return np.concatenate(parts)


def _widths(case):
    return [11] + [case["hidden"]] * case["depth"] + [case.get("outputs", sg.OUTPUTS)]


def _train_targets(X, outputs, seed):
    """Smooth curves of the inputs with some noise: values roughly in [0, 1], as the encoded targets are."""
    rng = np.random.default_rng(seed + 1)
    A = rng.normal(0, 1, (X.shape[1], outputs)).astype(np.float32)
    Y = 0.5 + 0.4 * np.tanh(X @ A - A.sum(axis=0) / 2)
    return (Y + rng.normal(0, 0.03, Y.shape)).astype(np.float32)


class _Closing:
    """What a program keeps between calls; its engines are closed when it is dropped."""

    def __init__(self, case, **kept):
        self.case = case
        self.__dict__.update(kept)

    def __del__(self):
        for name in ("sim", "batch", "surrogate", "net"):
            if name in self.__dict__:
                self.__dict__.pop(name).close()


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "run", "fresh"):
        params, core_seed = _params(case), 777 + seed
        rng = np.random.default_rng(seed)
        iv = dict(school_closure_start=int(rng.integers(0, 30)), school_closure_days=int(rng.integers(7, 43)),
                  workplace_absenteeism=float(rng.uniform(0.05, 0.3)),
                  vaccination_coverage=float(rng.uniform(0.0, 0.2))) if case["iv"] else None
        if kind == "fresh":
            return _Closing(case, params=params, core_seed=core_seed, iv=iv)
        sim = pt.PandemicSim(params, core_seed)
        if iv:
            sim.set_interventions(iv)
        sim.setupSim()
        return _Closing(case, sim=sim)
    if kind == "batch":
        params, seeds = scn.batched_workload(count=case["instances"], min_persons=case["low"],
                                             max_persons=case["high"], days=case["days"], rng_seed=20240)
        batch = pt.PandemicBatch(params, [s + 10_000 * seed for s in seeds])
        batch.setup()
        return _Closing(case, batch=batch)
    if kind == "simulate":
        return _Closing(case, scenarios=_scenario_list(case["scenarios"], seed), seed_base=100_000 + 1000 * seed)
    if kind == "predict":
        if case["members"] == 0:
            surrogate = sg.Surrogate.load(sg.SHIPPED_MODEL, max_batch=case["chunk"])
        else:
            surrogate = sg.Surrogate(1_000_000, hidden=case["hidden"], depth=case["depth"], max_batch=case["chunk"],
                                     members=case["members"])
            for k, net in enumerate(surrogate.nets):
                net.set_params(_weights(_widths(case), 100 * seed + k))
        X = _features(case["rows"], seed)
        if case["where"] == "host":
            return _Closing(case, surrogate=surrogate, X=X)
        Y = torch.empty((case["rows"], sg.OUTPUTS), dtype=torch.float32, device="cuda")
        return _Closing(case, surrogate=surrogate, X=torch.from_numpy(X).cuda(), Y=Y)
    X = _features(case["rows"], seed)
    net = sg.MLP(_widths(case), max_batch=case["batch"], seed=seed)
    net.set_data(X, _train_targets(X, case["outputs"], seed))
    return _Closing(case, net=net, params=_weights(_widths(case), seed), shuffle=seed)


# ------------------------------------------------------------------ one pass
def _table(rows, length):
    """rows in a table of a fixed length (an epidemic may stop early, a population's size depends on its seed)."""
    out = np.zeros((length,) + rows.shape[1:], rows.dtype)
    out[:len(rows)] = rows
    return out


def run(state):
    case = state.case
    kind = case["kind"]
    if kind == "run":
        state.sim.reset_epidemic()
        counts, infected = state.sim.runToCompletion()
        return _table(counts, case["days"]), _table(infected, case["days"]), state.sim.final_gen_counts()
    if kind == "step":
        sim = state.sim
        sim.reset_epidemic()
        rows = []
        while True:
            rc, counts, infected = sim.step_day()
            if rc == pt.PT_FINISHED:
                break
            rows.append(counts + [infected])
            if rc != pt.PT_OK:
                break
        people = int(1.05 * case["persons"]) + 1000
        return _table(np.array(rows, np.int32), case["days"]), {k: _table(v, people) for k, v in
                                                                sim.person_state().items()}
    if kind == "fresh":
        sim = pt.PandemicSim(state.params, state.core_seed)
        if state.iv:
            sim.set_interventions(state.iv)
        sim.setupSim()
        counts, infected = sim.runToCompletion()
        gens = sim.final_gen_counts()
        sim.close()
        return _table(counts, case["days"]), _table(infected, case["days"]), gens
    if kind == "batch":
        b = state.batch
        b.reset_epidemic()
        b.run()
        rows = [b.counts(k) for k in range(b.k)]
        return (np.stack([_table(c, case["days"]) for c, _ in rows]),
                np.stack([_table(i, case["days"]) for _, i in rows]), b.final_gen_counts())
    if kind == "simulate":
        return sg.simulate(state.scenarios, case["replicates"], case["persons"], seed_base=state.seed_base)
    if kind == "predict":
        if case["where"] == "host":
            return state.surrogate.raw_features(state.X)
        state.surrogate.raw_device(state.X.data_ptr(), case["rows"], state.Y.data_ptr())
        return state.Y
    state.net.set_params(state.params)
    loss = state.net.train(1, batch=case["batch"], lr=1e-3, seed=state.shuffle)
    return loss, state.net.get_params()


def _mlp_flops(case, rows, members=1):
    w = _widths(case)
    return 2.0 * members * rows * sum(a * b for a, b in zip(w[:-1], w[1:]))


def work(case):
    kind = case["kind"]
    if kind in ("predict", "train"):
        w = _widths(case)
        nparam = sum(a * b + b for a, b in zip(w[:-1], w[1:]))
        io = 4.0 * case["rows"] * (w[0] + w[-1])
        if kind == "predict":
            members = case["members"] or 4
            return {"bytes": io + 2.0 * members * nparam, "flops": _mlp_flops(case, case["rows"], members)}
        first = 2.0 * case["rows"] * w[0] * w[1]   # no gradient of the inputs
        return {"bytes": io + 8.0 * nparam, "flops": 3 * _mlp_flops(case, case["rows"]) - first}
    # Simulations: every day reads each person's two status and two day bytes; weekdays
    # also the age; a fresh population writes 20 bytes a person (household, workplace,
    # age, status, generations).
    if kind == "batch":
        rng_persons = scn.batched_workload(count=case["instances"], min_persons=case["low"],
                                           max_persons=case["high"], days=case["days"])[0]
        persons = sum(p["people_scaling"] for p in rng_persons) * PERSONS_PER_SCALE
        days = case["days"]
    elif kind == "simulate":
        persons, days = float(case["persons"]) * case["scenarios"] * case["replicates"], sg.DAYS
    else:
        persons, days = float(case["persons"]), case["days"]
    weekdays = sum(1 for d in range(days) if d % 7 < 5)
    setup = 20.0 if kind in ("fresh", "simulate") else 6.0
    return {"bytes": persons * (4.0 * days + weekdays + setup), "flops": 0}


# ------------------------------------------------------------------ 64-bit values
def _shipped_members():
    z = np.load(sg.SHIPPED_MODEL)
    widths = json.loads(str(z["meta"]))["widths"]
    out = []
    for bits, biases in zip(z["params"], z["biases"]):
        values = (bits.astype(np.uint32) << 16).view(np.float32)
        layers, at, b_at = [], 0, 0
        for a, b in zip(widths[:-1], widths[1:]):
            layers.append((values[at:at + a * b].reshape(b, a), biases[b_at:b_at + b]))
            at += a * b + b
            b_at += b
        out.append(layers)
    return out


def _drawn_members(case, seed):
    out = []
    for k in range(case["members"]):
        values, at, layers = _weights(_widths(case), 100 * seed + k), 0, []
        for a, b in zip(_widths(case)[:-1], _widths(case)[1:]):
            layers.append((values[at:at + a * b].reshape(b, a), values[at + a * b:at + a * b + b]))
            at += a * b + b
        out.append(layers)
    return out


def exact(case, seed):
    """Inference in 64 bits.  Simulations return whole numbers; a training epoch has no
    64-bit value here, since the order of its rows is the library's own shuffle."""
    if case["kind"] != "predict":
        return None
    members = _shipped_members() if case["members"] == 0 else _drawn_members(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    X = torch.from_numpy(_features(case["rows"], seed)).to(dev).double()
    total = 0
    for layers in members:
        h = X
        for k, (w, b) in enumerate(layers):
            z = h @ torch.from_numpy(w).to(dev).double().T + torch.from_numpy(b).to(dev).double()
            h = torch.nn.functional.gelu(z, approximate="tanh") if k + 1 < len(layers) else z
        total = total + h
    return total / len(members)
