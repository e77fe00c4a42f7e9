"""Performance cases of the framework's public entry points.

Each case is one call that a user's program makes: ``OptimizedEngine.match`` on
host strings, and ``DFASet.run`` / ``run_all`` / ``scan``, ``NFA.run`` and
``PNFA.run`` on strings that are resident on the GPU. ``listed()`` names the
cases, ``draw()`` gives others from the same ranges, ``prepare()`` makes what
the program holds before the call (strings, automaton handle), ``run()`` is one
call, ``exact()`` the FP64 result of the probabilistic cases.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from trex_b200.engine import NFA, PNFA, DFASet
from trex_b200.optimized_engine import OptimizedEngine
from trex_b200.workloads import ACGT, random_bool_nfa, random_dfa, random_prob_nfa

DEV = "cuda:0"
PATTERN = "(a|b)*a(a|b)"


def listed():
    return [
        # the documented front door: a regex and a list of Python strings, a small batch, where
        # packing, copies and launches count
        dict(name="match_2000", kind="match", n=2000, median=48, lo=4, hi=400),
        # one 16-state pattern over ACGT on a small resident batch (4 MB): latency and launches
        dict(name="dfa_plain_4096x1024", kind="dfa", states="16", n=4096, median=1024, sigma=0.0,
             symbols="acgt", all=False),
        # the headline batch: 16 automata of 8, 12 and 16 states, a million ragged strings
        dict(name="dfa_ragged_1M", kind="dfa", states="8,8,8,8,8,12,12,12,12,12,16,16,16,16,16,16",
             n=1000000, median=2048, sigma=1.18, symbols="mixed", all=False),
        # larger automata (32 and 64 states), ragged strings
        dict(name="dfa_n32_64_100K", kind="dfa", states="32,32,64,64", n=100003, median=2048,
             sigma=1.18, symbols="bytes", all=False),
        # per-position states of a few very long strings
        dict(name="scan_8x256MiB", kind="scan", states=16, n=8, median=1 << 28, sigma=0.0),
        # per-position states of ragged strings of a small automaton, odd lengths
        dict(name="scan_ragged_3001", kind="scan", states=7, n=3001, median=20000, sigma=1.18),
        # Boolean NFA, 64 states, 20 symbols, many equal strings
        dict(name="nfa_256Kx4096", kind="nfa", states=64, symbols=20, n=262144, median=4096,
             sigma=0.0, rejects=False),
        # the same automaton on a served batch: about two thousand ragged strings
        dict(name="nfa_ragged_2048", kind="nfa", states=64, symbols=20, n=2048, median=2048,
             sigma=1.18, rejects=True),
        # probabilistic NFA, 64 states, 20 symbols: the tensor-core form on a full batch
        dict(name="pnfa_bf16_64Kx2048", kind="pnfa", mode="bf16", states=64, symbols=20, n=65536,
             median=2048, sigma=0.0),
        # the plain FP32 form of the same automaton, a smaller batch
        dict(name="pnfa_fp32_8192x512", kind="pnfa", mode="fp32", states=64, symbols=20, n=8192,
             median=512, sigma=0.0),
        # the low-latency form on a served group of a few hundred ragged strings
        dict(name="pnfa_bf16cc_300", kind="pnfa", mode="bf16cc", states=64, symbols=20, n=300,
             median=1024, sigma=1.0),
        # a two-symbol alphabet, FP16 operands, on the shape of the published numbers
        dict(name="pnfa_fp16_s2_256Kx2048", kind="pnfa", mode="fp16", states=64, symbols=2, n=262144,
             median=2048, sigma=0.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# the most characters a drawn case walks (once an automaton, so that it stays below the listed ones)
_CHARS = {"match": 1 << 20, "dfa": 1 << 31, "scan": 1 << 30, "nfa": 1 << 29, "bf16": 1 << 26,
          "fp16": 1 << 26, "bool": 1 << 26, "bool8": 1 << 26, "fp32": 1 << 22, "bf16cc": 1 << 21,
          "fp16cc": 1 << 21}


def draw(rng):
    kind = rng.choice(["match", "dfa", "dfa", "dfa", "scan", "nfa", "nfa", "pnfa", "pnfa", "pnfa"])
    sigma = rng.choice([0.0, 0.5, 1.18])
    if kind == "match":
        med = _log_int(rng, 8, 1024)
        n = min(_log_int(rng, 50, 20000), _CHARS[kind] // med)
        return dict(kind=kind, n=n, median=med, lo=1, hi=8 * med)
    if kind == "dfa":
        states = rng.choice(["5", "8", "13", "16", "8,12,16", "3,8,11,16,16,7", "32", "17,64", "100",
                             "8,40,16"])
        n_dfas = states.count(",") + 1
        every = n_dfas > 1 and rng.random() < 0.35
        med = _log_int(rng, 40, 8192)
        n = min(_log_int(rng, 200, 1000000), _CHARS[kind] // (med * (2 * n_dfas if every else 2)))
        if "100" in states or "64" in states:
            n = max(200, n // 8)
        return dict(kind=kind, states=states, n=n, median=med, sigma=sigma,
                    symbols=rng.choice(["acgt", "bytes", "mixed"]), all=every)
    if kind == "scan":
        med = _log_int(rng, 1000, 1 << 26)
        n = max(1, min(_log_int(rng, 1, 50000), _CHARS[kind] // (2 * med)))
        return dict(kind=kind, states=rng.randint(3, 16), n=n, median=med, sigma=sigma)
    if kind == "nfa":
        med = _log_int(rng, 40, 8192)
        n = max(100, min(_log_int(rng, 100, 262144), _CHARS[kind] // (2 * med)))
        return dict(kind=kind, states=rng.choice([64, 64, 17, 32, 50]),
                    symbols=rng.choice([2, 4, 20, 20, 26, 60]), n=n, median=med, sigma=sigma,
                    rejects=rng.random() < 0.5)
    mode = rng.choice(["bf16", "bf16", "fp16", "bool", "bool8", "fp32", "bf16cc", "fp16cc"])
    med = _log_int(rng, 40, 2048)
    n = max(40, min(_log_int(rng, 40, 65536), _CHARS[mode] // (2 * med)))
    return dict(kind="pnfa", mode=mode, states=rng.choice([64, 64, 40, 25]),
                symbols=rng.choice([2, 4, 20, 20, 20, 7, 12]), n=n, median=med,
                sigma=min(sigma, 1.0))


def _lens(case, seed):
    """String lengths: all equal (sigma 0), or log-normal about the median. A case's lengths are
    the same for every seed, their order is the seed's (so that outputs keep their shapes)."""
    n, med = case["n"], case["median"]
    spread = 0.8 if case["kind"] == "match" else case["sigma"]
    if not spread:
        return np.full(n, med, dtype=np.int64)
    lo, hi = {"match": (case.get("lo"), case.get("hi")),
              "pnfa": (min(16, med), 16 * med)}.get(case["kind"], (min(16, med), 32 * med))
    lens = np.rint(np.exp(np.random.default_rng(1).normal(np.log(med), spread, size=n)))
    return np.random.default_rng([seed, 1]).permutation(np.clip(lens, lo, hi).astype(np.int64))


def _offsets(lens):
    off = np.zeros(len(lens) + 1, dtype=np.int64)
    np.cumsum(lens, out=off[1:])
    return off


def _device_strings(lens, seed, symbols):
    """Random strings on the GPU: symbols = number of byte values 0.., "bytes", "acgt" or "mixed"
    (bytes, with every tenth string or so over ACGT)."""
    total = int(lens.sum())
    g = torch.Generator(device=DEV)
    g.manual_seed(seed * 7 + 3)
    high = symbols if isinstance(symbols, int) else 4 if symbols == "acgt" else 256
    data = torch.randint(0, high, (total,), dtype=torch.uint8, device=DEV, generator=g)
    if isinstance(symbols, int) or symbols == "bytes":
        return data
    lut = torch.from_numpy(ACGT.copy()).to(DEV)
    off = _offsets(lens)
    sub = np.ones(len(lens), dtype=bool)
    if symbols == "mixed":
        sub = np.random.default_rng([seed, 2]).random(len(lens)) < 0.1
    step = max(1, int(len(lens) * (1 << 27) / max(total, 1)))   # about 128 MiB at a time
    for i in range(0, len(lens), step):
        j = min(len(lens), i + step)
        part = data[off[i]:off[j]]
        letters = lut[(part & 3).int()]
        if symbols == "mixed":
            flag = torch.repeat_interleave(torch.from_numpy(sub[i:j]).to(DEV),
                                           torch.from_numpy(lens[i:j]).to(DEV))
            letters = torch.where(flag, letters, part)
        part.copy_(letters)
    return data


def _nfa_tables(case, seed):
    rng = np.random.default_rng([seed, 3])
    return random_bool_nfa(rng, case["states"], case["symbols"], min(0.5, 3.2 / case["states"]))


def _pnfa_tables(case, seed):
    rng = np.random.default_rng([seed, 4])
    T, start, accept = random_prob_nfa(rng, case["states"], case["symbols"])
    return T.astype(np.float32), start.astype(np.float32), accept.astype(np.float32)


def prepare(case, seed):
    lens = _lens(case, seed)
    kind = case["kind"]
    if kind == "match":
        rng = np.random.default_rng([seed, 5])
        blob = np.frombuffer(b"ab", dtype=np.uint8)[rng.integers(0, 2, int(lens.sum()))]
        text, off = blob.tobytes().decode("latin-1"), _offsets(lens)
        return dict(case=case, engine=OptimizedEngine(pattern=PATTERN, config="auto"),
                    strings=[text[off[i]:off[i + 1]] for i in range(len(lens))])
    offsets = torch.from_numpy(_offsets(lens)).to(DEV)
    state = dict(case=case, offsets=offsets)
    if kind in ("dfa", "scan"):
        rng = np.random.default_rng([seed, 6])
        sizes = [int(s) for s in str(case["states"]).split(",")]
        symbols = case.get("symbols", "bytes")
        alphabet = ACGT if symbols == "acgt" else np.arange(256)
        state["engine"] = DFASet([random_dfa(s, alphabet, rng) for s in sizes])
        state["data"] = _device_strings(lens, seed, symbols)
        if kind == "dfa" and not case["all"] and len(sizes) > 1:
            state["ids"] = torch.arange(case["n"], device=DEV, dtype=torch.int32) % len(sizes)
        return state
    # every NFA case meets a few bytes outside its alphabet when they are skipped
    skipped = kind == "nfa" and not case["rejects"] and case["sigma"] > 0
    state["data"] = _device_strings(lens, seed, case["symbols"] + (1 if skipped else 0))
    if kind == "nfa":
        T, start, accept = _nfa_tables(case, seed)
        state["engine"] = NFA(T, start, accept, unknown_rejects=case["rejects"])
    else:
        state["engine"] = PNFA(*_pnfa_tables(case, seed))
    return state


def run(state):
    case, engine = state["case"], state["engine"]
    kind = case["kind"]
    if kind == "match":
        return np.array(engine.match(state["strings"]))
    data, offsets = state["data"], state["offsets"]
    if kind == "dfa":
        if case["all"]:
            return engine.run_all(data, offsets)
        return engine.run(data, offsets, state.get("ids"))[:2]
    if kind == "scan":
        return engine.scan(data, offsets)[:3]
    if kind == "nfa":
        return engine.run(data, offsets)
    return engine.run(data, offsets, case["mode"])


def work(case):
    """Every character read once, offsets and ids read, results written; 2 N^2 operations a
    character for the probabilistic forms."""
    n = case["n"]
    total = int(_lens(case, 0).sum())
    kind = case["kind"]
    if kind == "match":
        return {"bytes": total + 9 * n, "flops": 0}
    out = {"dfa": 2, "scan": 2, "nfa": 9, "pnfa": 9}[kind]
    size = total + 8 * (n + 1)
    if kind == "dfa":
        n_dfas = case["states"].count(",") + 1
        size += out * n * (n_dfas if case["all"] else 1) + (4 * n if n_dfas > 1 and not case["all"] else 0)
    else:
        size += out * n + (total if kind == "scan" else 0)
    tensor = kind == "pnfa" and not case["mode"].startswith("bool")
    return {"bytes": size, "flops": 2 * case["states"] ** 2 * total if tensor else 0}


# largest relative error of the log-likelihoods against FP64 seen over the ranges above, brought
# to 2048 symbols a string: it falls with the root of the length (the steps' rounding errors are
# independent, the value grows with the length)
_ERROR = {"bf16": 2.5e-5, "bf16cc": 2.5e-5, "fp16": 5e-6, "fp16cc": 5e-6, "fp32": 5e-10}


def tolerance(case):
    """States, masks and flags are exact; log-likelihoods differ by at most four times the error
    of the 16-bit operands (or FP32 sums) that the form rounds to at every step."""
    if case["kind"] != "pnfa" or case["mode"].startswith("bool"):
        return "exact"
    rel = 4 * _ERROR[case["mode"]] * math.sqrt(2048 / min(2048, case["median"]))
    return {"rel": rel, "max": 20 * rel}


def exact(case, seed):
    """(log-likelihoods, None) of a probabilistic case in FP64: every symbol's product, then the
    string's own; strings in order of length, so that those still running are a prefix."""
    if case["kind"] != "pnfa" or case["mode"].startswith("bool"):
        return None
    lens = _lens(case, seed)
    off = torch.from_numpy(_offsets(lens)).to(DEV)
    data = _device_strings(lens, seed, case["symbols"])
    T, start, accept = (torch.from_numpy(x).double().to(DEV) for x in _pnfa_tables(case, seed))
    sym, N, _ = T.shape
    W = T.permute(2, 0, 1).reshape(N, sym * N).contiguous()   # [source, symbol x destination]
    order = np.argsort(-lens, kind="stable")
    out = torch.empty(case["n"], dtype=torch.float64, device=DEV)
    for i in range(0, case["n"], 16384):
        ids = order[i:i + 16384]
        ln = lens[ids]
        first = off[torch.from_numpy(ids).to(DEV)]
        x = start.repeat(len(ids), 1)
        e = torch.zeros(len(ids), dtype=torch.float64, device=DEV)
        live = np.searchsorted(-ln, -np.arange(ln[0]), side="left")   # strings longer than t
        for t in range(int(ln[0])):
            k = int(live[t])
            c = data[first[:k] + t].long()
            y = (x[:k] @ W).view(k, sym, N)[torch.arange(k, device=DEV), c]
            if t % 8 == 7:
                m = y.abs().amax(1, keepdim=True).clamp_min(1e-300)
                y = y / m
                e[:k] += m[:, 0].log()
            x[:k] = y
        out[torch.from_numpy(ids).to(DEV)] = (x @ accept).log() + e
    return out, None
