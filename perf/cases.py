"""What the speed of this framework is measured on: the work that a user's program has it do, through the public
entry points, from the smallest calls to the largest.

A case is a dict of plain values; its "work" names the entry point:

  score        population scoring: score_columns_gpu, score_checked_gpu, score_population_gpu
  deltas       swap_deltas over a batch of moves
  partners     two_switch_scores / transposition_scores of every slot of some states
  tempering    TemperingChains.run, chains of one grid size
  epoch        TemperingChains.epoch, the tempering driver's unit of work
  mixed        TemperingChains.run over chains of several grid sizes in one launch
  learned      LearnedProposal.step: candidates, MLP inference, exact moves
  train        LearnedProposal.train: one Adam step on a batch from the ring buffer
  beam         DeviceBeam: a search of some generations, from the initial state to the status read back
  scan         best_four_cycle / best_double_switch through one anchor

States are two points per row and column, drawn at random as the framework's own seeding draws them (two permutations
that differ in every row), made on the GPU from the seed.
"""
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

PACKAGE = "no_three_in_line_b200"


def _package():
    """The package directory no-three-in-line_b200/ (its name is no identifier) imported as no_three_in_line_b200."""
    if PACKAGE not in sys.modules:
        root = Path.cwd() / "no-three-in-line_b200"
        spec = importlib.util.spec_from_file_location(PACKAGE, root / "__init__.py",
                                                      submodule_search_locations=[str(root)])
        module = importlib.util.module_from_spec(spec)
        sys.modules[PACKAGE] = module
        spec.loader.exec_module(module)
    return sys.modules[PACKAGE]


def _module(name):
    _package()
    return importlib.import_module(PACKAGE + "." + name)


# ---------------------------------------------------------------------------
# The cases.
# ---------------------------------------------------------------------------
def listed():
    return [
        # The smallest scoring call: 256 states of a 20 x 20 grid, as a search over small grids makes it all the time.
        {"name": "score_256_n20", "work": "score", "call": "columns", "n": 20, "states": 256, "badness": False},
        # The benchmark's workload: determinant and slope counts of 4096 n = 75 states, cross-checked, with badness.
        {"name": "checked_4096_n75", "work": "score", "call": "checked", "n": 75, "states": 4096, "badness": True},
        # A large population of an odd grid size, P/Q layout with badness, as a beam or genetic search rescores one.
        {"name": "population_20011_n61", "work": "score", "call": "population", "n": 61, "states": 20011,
         "badness": True},
        # A batch of proposed moves over a resident population.
        {"name": "deltas_65536_n75", "work": "deltas", "n": 75, "states": 4096, "moves": 65536, "badness": False},
        # Every 2-switch of 64 states: what a local search or the exhaustive beam asks of its elites.
        {"name": "partners_64_n75", "work": "partners", "call": "two_switch", "n": 75, "states": 64},
        # Replica exchange, 32 ladders of 64 temperatures, in the middle of a run: one block of 100 sweeps.
        {"name": "tempering_2048_n75", "work": "tempering", "n": 75, "ladders": 32, "ladder": 64, "tmin": 0.05,
         "tmax": 5.0, "sweeps": 100, "burn": 100, "bad_bias": 0},
        # The tempering driver's epoch at its default size, slots drawn by badness.
        {"name": "epoch_128_n75", "work": "epoch", "n": 75, "ladders": 8, "ladder": 16, "tmin": 0.2, "tmax": 4.0,
         "steps": 100, "burn": 50, "bad_bias": 85},
        # Uneven counts of five grid sizes in one launch, each size with its own share of sweeps.
        {"name": "mixed_2944", "work": "mixed", "ladder": 32, "l40": 32, "l52": 24, "l60": 16, "l68": 12, "l75": 8,
         "s40": 50, "s52": 30, "s60": 30, "s68": 20, "s75": 20, "tmin": 0.05, "tmax": 5.0, "burn": 50},
        # One learned step of 2048 chains: 128 candidates a chain scored by the MLP, 16 exact moves each.
        {"name": "learned_2048_n75", "work": "learned", "n": 75, "ladders": 32, "ladder": 64, "tmin": 0.05,
         "tmax": 5.0, "moves": 16, "bad_bias": 85, "ring": 1 << 21},
        # One training step of the proposal network, in the middle of a run.
        {"name": "train_4096", "work": "train", "batch": 4096, "ring": 1 << 21, "steps": 100},
        # Twenty generations of a beam search at the command line's population, elite and window.
        {"name": "beam_32768_n75", "work": "beam", "n": 75, "population": 32768, "elite": 64, "strength": 12,
         "window": 12, "bad_bias": 85, "generations": 20},
        # The best four-cycle through one anchor slot of an n = 75 state.
        {"name": "scan_n75", "work": "scan", "call": "four_cycle", "n": 75},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    work = rng.choice(("score", "score", "deltas", "partners", "tempering", "epoch", "mixed", "learned", "train",
                       "beam", "scan"))
    n = rng.randint(20, 75)
    if work == "score":
        return {"work": work, "call": rng.choice(("columns", "checked", "population")), "n": rng.randint(10, 75),
                "states": _log(rng, 64, 20011), "badness": rng.random() < 0.5}
    if work == "deltas":
        return {"work": work, "n": n, "states": _log(rng, 16, 4096), "moves": _log(rng, 256, 65536),
                "badness": rng.random() < 0.3}
    if work == "partners":
        return {"work": work, "call": rng.choice(("two_switch", "two_switch", "transposition")), "n": n,
                "states": _log(rng, 1, 64)}
    if work == "tempering":
        ladder = rng.choice((16, 32, 64))
        return {"work": work, "n": rng.randint(40, 75), "ladders": rng.randint(4, 2048 // ladder), "ladder": ladder,
                "tmin": rng.choice((0.05, 0.1, 0.2)), "tmax": rng.choice((4.0, 5.0)),
                "sweeps": 10 * rng.randint(1, 10), "burn": 50, "bad_bias": rng.choice((0, 0, 85))}
    if work == "epoch":
        return {"work": work, "n": rng.randint(40, 75), "ladders": rng.randint(2, 16), "ladder": rng.choice((8, 16)),
                "tmin": 0.2, "tmax": 4.0, "steps": rng.randint(50, 400), "burn": 50,
                "bad_bias": rng.choice((0, 50, 85))}
    if work == "mixed":
        case = {"work": work, "ladder": rng.choice((16, 32)), "tmin": 0.05, "tmax": 5.0, "burn": 20}
        for size in (40, 52, 60, 68, 75):
            case["l%d" % size] = 2 * rng.randint(1, 8)
            case["s%d" % size] = 10 * rng.randint(1, 4)
        return case
    if work == "learned":
        return {"work": work, "n": rng.randint(40, 75), "ladders": rng.randint(4, 32), "ladder": rng.choice((16, 64)),
                "tmin": 0.05, "tmax": 5.0, "moves": rng.choice((1, 4, 16)), "bad_bias": rng.choice((0, 85)),
                "ring": 1 << rng.randint(17, 20)}
    if work == "train":
        return {"work": work, "batch": _log(rng, 256, 4096), "ring": 1 << rng.randint(17, 20),
                "steps": rng.randint(10, 1000)}
    if work == "beam":
        elite = rng.randint(16, 128)
        return {"work": work, "n": n, "population": max(2 * elite, _log(rng, 2048, 32768)), "elite": elite,
                "strength": rng.randint(4, 12), "window": rng.randint(4, 16), "bad_bias": 85,
                "generations": rng.randint(5, 20)}
    return {"work": work, "call": rng.choice(("four_cycle", "double_switch")), "n": n}


# ---------------------------------------------------------------------------
# Inputs.
# ---------------------------------------------------------------------------
def _generator(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + salt)


def _states(count, n, seed, salt=0):
    """P, Q int32 [count, n] on the GPU: two permutations that differ in every row."""
    g = _generator(seed, salt)
    p = torch.argsort(torch.rand((count, n), generator=g, device="cuda"), dim=1)
    q = torch.argsort(torch.rand((count, n), generator=g, device="cuda"), dim=1)
    while True:
        clash = torch.nonzero((p == q).any(1)).flatten()
        if clash.numel() == 0:
            return p.to(torch.int32), q.to(torch.int32)
        q[clash] = torch.argsort(torch.rand((clash.numel(), n), generator=g, device="cuda"), dim=1)


def _columns(p, q):
    return torch.stack((p, q), dim=2).reshape(p.shape[0], -1).to(torch.int16).contiguous()


def _moves(states, n, count, seed):
    """(state, u, v) int32 [count, 3]: slots u, v uniform, as the walk proposes them (a few are illegal)."""
    g = _generator(seed, 2)
    b = torch.randint(0, states, (count,), generator=g, device="cuda")
    uv = torch.randint(0, 2 * n, (count, 2), generator=g, device="cuda")
    return torch.cat((b[:, None], uv), dim=1).to(torch.int32).contiguous()


def _ladder(case, ladders):
    return np.tile(np.geomspace(case["tmin"], case["tmax"], case["ladder"]), ladders)


def _chains(case, seed):
    p, q = _states(case["ladders"] * case["ladder"], case["n"], seed)
    return _module("tempering").TemperingChains(_columns(p, q).cpu().numpy(), _ladder(case, case["ladders"]),
                                                int(seed) + 1, ladder_size=case["ladder"])


SIZES = (40, 52, 60, 68, 75)
N_IN, N_H = 192, 256
W1, B1, W2, B2, W3, B3 = 0, 49152, 49408, 114944, 115200, 115456


def _params(seed):
    """A network in the middle of training: He-uniform weights, small biases, the padding inputs' weights zero."""
    g = torch.Generator().manual_seed(int(seed) + 77)
    u = lambda *shape: 2 * torch.rand(shape, generator=g) - 1  # noqa: E731
    p = torch.zeros(B3 + 4)
    w1 = u(N_H, N_IN) * math.sqrt(6.0 / 162)
    w1[:, 162:] = 0
    p[W1:B1] = w1.flatten()
    p[B1:W2] = 0.05 * u(N_H)
    p[W2:B2] = (u(N_H, N_H) * math.sqrt(6.0 / N_H)).flatten()
    p[B2:W3] = 0.05 * u(N_H)
    p[W3:B3] = u(N_H) * math.sqrt(3.0 / N_H)
    p[B3] = 0.1
    return p


def _ring(case, seed):
    """A filled ring buffer: badness of low-energy n = 75 states, moves' features, exact dE of proposed moves."""
    g = _generator(seed, 3)
    cap = case["ring"]
    bad = torch.randint(0, 8, (cap, 150), generator=g, device="cuda") * \
        torch.randint(0, 2, (cap, 150), generator=g, device="cuda")
    feat = torch.empty((cap, 12), device="cuda")
    feat[:, :4] = torch.randint(0, 8, (cap, 4), generator=g, device="cuda") / 16.0
    feat[:, 4:] = torch.randint(0, 75, (cap, 8), generator=g, device="cuda") / 75.0
    dE = (6.0 + 7.0 * torch.randn(cap, generator=g, device="cuda")).round().clamp(-60, 200)
    return feat.to(torch.bfloat16), bad.to(torch.uint8), dE.to(torch.int16)


def prepare(case, seed):
    work, s = case["work"], {"case": case}
    if work in ("score", "deltas", "partners"):
        p, q = _states(case["states"], case["n"], seed)
        s["p"], s["q"], s["columns"] = p.contiguous(), q.contiguous(), _columns(p, q)
        if work == "deltas":
            s["moves"] = _moves(case["states"], case["n"], case["moves"], seed)
        if work == "partners":
            s["scores"], s["badness"] = _module("gpu").score_columns_gpu(s["columns"], badness=True)
            m = 2 * case["n"]
            at = torch.arange(case["states"] * m, device="cuda")
            s["anchors"] = torch.stack((at // m, at % m), dim=1).to(torch.int32).contiguous()
    elif work in ("tempering", "epoch"):
        s["chains"] = ch = _chains(case, seed)
        if work == "epoch":  # the driver tunes the launch shape before its first epoch
            tune = _module("autotune").autotune(ch, probe_sweeps=2, exchange_every=2)
            ch.threads_per_chain, ch.chains_per_block = tune.threads_per_chain, tune.chains_per_block
        ch.run(case["burn"], exchange_every=10, bad_bias=case["bad_bias"])
    elif work == "mixed":
        groups = []
        for size in SIZES:
            p, q = _states(case["l%d" % size] * case["ladder"], size, seed, size)
            groups.append((size, _columns(p, q).cpu().numpy()))
        s["chains"] = ch = _module("tempering").TemperingChains.mixed(groups, _ladder(case, 1), int(seed) + 1)
        s["sweeps"] = [case["s%d" % size] for size in SIZES for _ in range(case["l%d" % size])]
        ch.run(case["burn"], exchange_every=10, chains_per_block=16)
    elif work == "learned":
        s["chains"] = _chains(case, seed)
        s["proposal"] = _module("learned").LearnedProposal(
            s["chains"], seed=int(seed) + 1, ring_capacity=case["ring"], params=_params(seed).numpy(),
            moves=case["moves"], bad_bias=case["bad_bias"])
    elif work == "train":
        p, q = _states(16, 75, seed)
        ch = _module("tempering").TemperingChains(_columns(p, q).cpu().numpy(), np.geomspace(0.05, 5.0, 16),
                                                  int(seed) + 1, ladder_size=16)
        s["proposal"] = lp = _module("learned").LearnedProposal(
            ch, seed=int(seed) + 1, ring_capacity=case["ring"], batch=case["batch"], params=_params(seed).numpy(),
            moves=16)
        feat, bad, dE = _ring(case, seed)
        lp.rb_feat.copy_(feat.view(torch.int16))
        lp.rb_bad.copy_(bad)
        lp.rb_dE.copy_(dE)
        lp.counters[0] = case["ring"] // 256 + 1  # 16 chains x 16 moves a step: the ring is full
        lp.counters[1] = case["steps"]
        lp.adam_v.fill_(1e-4)
    elif work == "beam":
        p, q = _states(1, case["n"], seed)
        s["base"] = torch.stack((p, q), dim=2).cpu().numpy()
        s["beam"] = _module("gpu_device_search").DeviceBeam(
            case["n"], seed=int(seed) + 1, population=case["population"], elite_size=case["elite"],
            max_strength=case["strength"], energy_window=case["window"], bad_bias=case["bad_bias"],
            history_len=case["generations"])
    else:
        p, q = _states(1, case["n"], seed)
        s["initial"] = _module("state").PairPermutations(tuple(p[0].tolist()), tuple(q[0].tolist()))
        s["anchor"] = int(torch.randint(0, 2 * case["n"], (1,), generator=torch.Generator().manual_seed(int(seed))))
    return s


# ---------------------------------------------------------------------------
# One pass.
# ---------------------------------------------------------------------------
def _chain_outputs(ch):
    return {"columns": ch.cols, "badness": ch.badness_dev, "energy": ch.energy, "best_energy": ch.best_energy,
            "best_columns": ch.best_cols, "temp_of": ch.temp_of, "chain_at": ch.chain_at, "counter": ch.counter,
            "accepted": ch.accepted_dev, "exchanges": ch.ladder_exchanges}


def run(state):
    case = state["case"]
    work = case["work"]
    if work == "score":
        gpu = _module("gpu")
        if case["call"] == "columns":
            got = gpu.score_columns_gpu(state["columns"], badness=case["badness"])
            return got if case["badness"] else (got,)
        if case["call"] == "checked":
            got = gpu.score_checked_gpu(state["columns"], badness=case["badness"])
            return (got.scores, got.badness) if case["badness"] else (got.scores,)
        got = gpu.score_population_gpu(state["p"], state["q"], badness=case["badness"])
        return got if case["badness"] else (got,)
    if work == "deltas":
        got = _module("gpu_delta").swap_deltas(state["columns"], state["moves"], badness=case["badness"])
        return got if case["badness"] else (got,)
    if work == "partners":
        delta = _module("gpu_delta")
        call = delta.two_switch_scores if case["call"] == "two_switch" else delta.transposition_scores
        return (call(state["columns"], state["badness"], state["scores"], state["anchors"]),)
    if work == "tempering":
        state["chains"].run(case["sweeps"], exchange_every=10, sweeps_per_launch=case["sweeps"],
                            bad_bias=case["bad_bias"])
        return _chain_outputs(state["chains"])
    if work == "epoch":
        state["chains"].epoch(case["steps"], case["bad_bias"])
        return _chain_outputs(state["chains"])
    if work == "mixed":
        state["chains"].run(max(state["sweeps"]), exchange_every=10, chains_per_block=16,
                            ladder_sweeps=state["sweeps"])
        return _chain_outputs(state["chains"])
    if work == "learned":
        lp = state["proposal"]
        lp.step()
        return {"pred": lp.pred, "candidates": lp.cand, "ring_dE": lp.rb_dE, "ring_features": lp.rb_feat,
                "ring_badness": lp.rb_bad, "stats": lp.stats, **_chain_outputs(state["chains"])}
    if work == "train":
        lp = state["proposal"]
        lp.train()
        return {"params": lp.params, "grads": lp.grads, "adam_m": lp.adam_m, "adam_v": lp.adam_v, "loss": lp.loss}
    if work == "beam":
        beam = state["beam"]
        beam.init(state["base"])
        for generation in range(1, case["generations"] + 1):
            beam.generation(generation)
        return {"status": beam.read_status(), "best_p": beam.best_p, "best_q": beam.best_q, "elite_p": beam.elite_p,
                "elite_q": beam.elite_q, "elite_scores": beam.elite_scores, "elite_badness": beam.elite_badness,
                "child_scores": beam.child_scores, "history": beam.history}
    scan = _module("gpu_neighborhood")
    call = scan.best_four_cycle if case["call"] == "four_cycle" else scan.best_double_switch
    got = call(state["initial"], state["anchor"])
    return {"p": np.asarray(got.state.P), "q": np.asarray(got.state.Q), "score": got.score,
            "evaluated": got.evaluated, "legal": got.legal}


# ---------------------------------------------------------------------------
# What a pass cannot do without.  Integer operations count as flops: one per
# pair of points of a state scored (its direction), one per point and moved
# point of a move, and for a proposal its random block (20 multiplies) and
# the test of its four positions (12).
# ---------------------------------------------------------------------------
PROPOSAL_OPS = 32


def work(case):
    kind = case["work"]
    if kind == "score":
        m, b = 2 * case["n"], case["states"]
        inputs = 2 * b * m if case["call"] != "population" else 4 * b * m
        return {"bytes": inputs + 4 * b + (4 * b * m if case["badness"] else 0), "flops": b * m * (m - 1) / 2}
    if kind == "deltas":
        m, k = 2 * case["n"], case["moves"]
        states = min(case["states"], k)
        return {"bytes": 2 * states * m + 16 * k + (4 * k * m if case["badness"] else 0), "flops": 4.0 * k * m}
    if kind == "partners":
        m, b = 2 * case["n"], case["states"]
        out = m if case["call"] == "two_switch" else case["n"]
        return {"bytes": b * (6 * m + 4) + b * m * (8 + 4 * out), "flops": b * (m * (m - 1) / 2 + 6.0 * m * out)}
    if kind in ("tempering", "epoch"):
        c, m = case["ladders"] * case["ladder"], 2 * case["n"]
        proposals = c * (case["sweeps"] * m if kind == "tempering" else case["steps"])
        return {"bytes": 2.0 * c * (6 * m + 32), "flops": float(proposals * PROPOSAL_OPS)}
    if kind == "mixed":
        chains = proposals = 0
        for size in SIZES:
            c = case["l%d" % size] * case["ladder"]
            chains += c * (12 * size + 32)
            proposals += c * case["s%d" % size] * 2 * size
        return {"bytes": 2.0 * chains, "flops": float(proposals * PROPOSAL_OPS)}
    if kind == "learned":
        c, m = case["ladders"] * case["ladder"], 2 * case["n"]
        mlp = 2.0 * c * (150 * N_H + 128 * (12 * N_H + N_H * N_H + N_H))
        return {"bytes": c * (12.0 * m + 128 * 8 + case["moves"] * 176), "flops": mlp + 8.0 * c * case["moves"] * m}
    if kind == "train":
        b = case["batch"]
        return {"bytes": 176.0 * b + 4.0 * (B3 + 4) * 8, "flops": 6.0 * b * (162 * N_H + N_H * N_H + N_H)}
    if kind == "beam":
        m, k = 2 * case["n"], case["population"] * case["generations"]
        return {"bytes": 12.0 * case["elite"] * m * case["generations"] + 4.0 * k, "flops": 8.0 * k * m}
    n = case["n"]
    return {"bytes": 24.0 * n, "flops": 9.0 * 8 * (n - 1) * (n - 2) * (n - 3) / 6}


# ---------------------------------------------------------------------------
# The same results in plain 64-bit torch and numpy.
# ---------------------------------------------------------------------------
def _pairs_through(rows, cols, r0, c0):
    """Per state, the pairs of points collinear with (r0, c0); points at (r0, c0) itself are left out.  int64 [b]."""
    dr, dc = rows[None, :] - r0[:, None], cols - c0[:, None]
    zero = (dr[:, :, None] * dc[:, None, :]) == (dc[:, :, None] * dr[:, None, :])
    here = (dr == 0) & (dc == 0)
    zero &= ~(here[:, :, None] | here[:, None, :])
    inside = (~here).sum(1)
    return (zero.sum((1, 2)) - inside) // 2  # each pair twice, each point with itself once


def _on_line(rows, cols, r0, c0, r1, c1):
    """Points other than the two themselves on the line through (r0, c0) and (r1, c1)."""
    dr, dc = rows[None, :] - r0[:, None], cols - c0[:, None]
    hit = dr * (c1 - c0)[:, None] == dc * (r1 - r0)[:, None]
    hit &= ~((dr == 0) & (dc == 0))
    hit &= ~((rows[None, :] == r1[:, None]) & (cols == c1[:, None]))
    return hit.sum(1)


def _exact_scores(columns):
    m = columns.shape[1]
    rows = torch.arange(m, device="cuda") // 2
    bad = torch.empty(columns.shape, dtype=torch.int64, device="cuda")
    for at in range(0, columns.shape[0], 2048):
        cols = columns[at:at + 2048].to(torch.int64)
        for s in range(m):
            r0 = torch.full((cols.shape[0],), s // 2, device="cuda")
            bad[at:at + 2048, s] = _pairs_through(rows, cols, r0, cols[:, s])
    return bad.sum(1) // 3, bad


def _exact_deltas(columns, moves):
    """(dE, legal as the walk tests it) of moves (state, u, v), int64 [k]."""
    m = columns.shape[1]
    rows = torch.arange(m, device="cuda") // 2
    dE = torch.empty(moves.shape[0], dtype=torch.int64, device="cuda")
    for at in range(0, moves.shape[0], 4096):
        b, u, v = moves[at:at + 4096].to(torch.int64).unbind(1)
        old = columns[b].to(torch.int64)
        k = torch.arange(b.numel(), device="cuda")
        cu, cv = old[k, u], old[k, v]
        new = old.clone()
        new[k, u], new[k, v] = cv, cu
        total = torch.zeros(b.numel(), dtype=torch.int64, device="cuda")
        for sign, cols in ((-1, old), (1, new)):
            a, c = cols[k, u], cols[k, v]
            ru, rv = u // 2, v // 2
            total += sign * (_pairs_through(rows, cols, ru, a) + _pairs_through(rows, cols, rv, c) -
                             _on_line(rows, cols, ru, a, rv, c))
        dE[at:at + 4096] = total
    return dE


def _philox(c0, c1, c2, c3, k0, k1):
    """Philox4x32-10 over numpy uint64 arrays holding 32-bit words."""
    mask = np.uint64(0xFFFFFFFF)
    c = [np.asarray(x, np.uint64) for x in (c0, c1, c2, c3)]
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & mask,
             (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & mask]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _exact_pred(case, seed):
    """The MLP's predictions for the first step's candidates."""
    c, n, m = case["ladders"] * case["ladder"], case["n"], 2 * case["n"]
    p, q = _states(c, n, seed)
    columns = _columns(p, q)
    bad = _exact_scores(columns)[1]
    cols, badness = columns.cpu().numpy().astype(np.int64), bad.cpu().numpy()
    chain, j = np.meshgrid(np.arange(c), np.arange(128), indexing="ij")
    zero = np.zeros_like(chain)
    r = _philox(zero, zero, chain, 0xC0000000 | j, int(seed) + 1, 0)
    top = lambda x, k: ((x * np.asarray(k, np.uint64)) >> np.uint64(32)).astype(np.int64)  # noqa: E731
    u, v = top(r[0], m), top(r[1], m)
    if case["bad_bias"] > 0:
        run_sum = np.cumsum(badness, axis=1)
        total = run_sum[:, -1]
        target = top(r[3], total[:, None])
        weighted = np.stack([np.searchsorted(run_sum[i], target[i], side="right") for i in range(c)])
        use = (top(r[2], 100) < case["bad_bias"]) & (total[:, None] > 0)
        u = np.where(use, weighted, u)
    x = np.zeros((c, 128, 162))
    for i, slot in enumerate((u, v, u ^ 1, v ^ 1)):
        x[:, :, i] = np.take_along_axis(badness, slot, 1) / 16.0
        x[:, :, 4 + i] = (slot >> 1) / n
        x[:, :, 8 + i] = np.take_along_axis(cols, slot, 1) / n
    x[:, :, 12:12 + m] = badness[:, None, :] / 16.0
    x, w = torch.from_numpy(x).cuda(), _params(seed).double().cuda()
    h = torch.relu(x @ w[W1:B1].view(N_H, N_IN)[:, :162].T + w[B1:W2])
    h = torch.relu(h @ w[W2:B2].view(N_H, N_H).T + w[B2:W3])
    return (h @ w[W3:B3] + w[B3]) * 16.0


def _exact_train(case, seed):
    b, t = case["batch"], case["steps"]
    feat, bad, dE = _ring(case, seed)
    key = (int(seed) + 1) ^ 0x5A5A5A5A
    r = _philox(np.full(b, t), np.zeros(b), np.arange(b), np.full(b, 0x7A000000), key & 0xFFFFFFFF, key >> 32)
    slot = (((r[0] << np.uint64(32)) | r[1]) % np.uint64(case["ring"])).astype(np.int64)
    slot = torch.from_numpy(slot).cuda()
    x = torch.zeros((b, N_IN), dtype=torch.float64, device="cuda")
    x[:, :12], x[:, 12:162] = feat[slot].double(), bad[slot].double() / 16.0
    y = dE[slot].double() / 16.0
    w = _params(seed).double().cuda().requires_grad_(True)
    h = torch.relu(x @ w[W1:B1].view(N_H, N_IN).T + w[B1:W2])
    h = torch.relu(h @ w[W2:B2].view(N_H, N_H).T + w[B2:W3])
    squares = ((h @ w[W3:B3] + w[B3] - y) ** 2).sum()
    (squares / b).backward()
    g = w.grad
    adam_m, adam_v = 0.1 * g, 0.999 * 1e-4 + 0.001 * g * g
    step = t + 1
    new = w.detach() - 1e-3 * (adam_m / (1 - 0.9 ** step)) / (torch.sqrt(adam_v / (1 - 0.999 ** step)) + 1e-8)
    return {"params": new, "grads": g, "adam_m": adam_m, "adam_v": adam_v, "loss": squares.detach().reshape(1)}


def exact(case, seed):
    kind = case["work"]
    if kind in ("score", "deltas", "partners"):
        columns = _columns(*_states(case["states"], case["n"], seed))
    if kind == "score":
        e, bad = _exact_scores(columns)
        return (e, bad) if case["badness"] else (e,)
    if kind == "deltas":
        moves = _moves(case["states"], case["n"], case["moves"], seed)
        b, u, v = moves.to(torch.int64).unbind(1)
        cu, cv = columns[b, u], columns[b, v]
        legal = (u // 2 != v // 2) & (cu != cv) & (columns[b, u ^ 1] != cv) & (columns[b, v ^ 1] != cu)
        dE = torch.where(legal, _exact_deltas(columns, moves), 1 << 30)
        return (dE, None) if case["badness"] else (dE,)
    if kind == "partners":
        m = 2 * case["n"]
        step = 1 if case["call"] == "two_switch" else 2
        at = torch.arange(case["states"] * m, device="cuda")
        b, u = (at // m)[:, None], (at % m)[:, None]
        v = torch.arange(0, m, step, device="cuda")[None, :] + (0 if step == 1 else u % 2)
        b, u, v = (x.expand(at.numel(), m // step).reshape(-1) for x in (b, u, v))
        legal = (u // 2 != v // 2) & (columns[b, v] != columns[b, u ^ 1]) & (columns[b, u] != columns[b, v ^ 1])
        e = _exact_scores(columns)[0]
        dE = torch.zeros_like(b)
        pick = torch.nonzero(legal).flatten()
        dE[pick] = _exact_deltas(columns, torch.stack((b[pick], u[pick], v[pick]), 1))
        return (torch.where(legal, e[b] + dE, 1 << 30).reshape(at.numel(), m // step),)
    if kind == "learned":
        none = ("candidates", "ring_dE", "ring_features", "ring_badness", "stats", "columns", "badness", "energy",
                "best_energy", "best_columns", "temp_of", "chain_at", "counter", "accepted", "exchanges")
        return {"pred": _exact_pred(case, seed), **{k: None for k in none}}
    if kind == "train":
        return _exact_train(case, seed)
    return None  # trajectories of a search: nothing but a replay gives them
