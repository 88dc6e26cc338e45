"""Performance cases of the matching framework, through its public entry points.

A case names a rule set (the automata), an input and the options of one call:

  match     one input cut into segments against one rule set (`Engine.match`),
            as the command line and `class Ngap` do it;
  batch     many streams of uneven length against several rule sets in one
            call (`batch_match_async`), alone or as the bursts of a server;
  features  byte features of input regions and the cost model's predictions
            on them (`cost_model.byte_features`, `LearnedModel`).

A program loads its rules once and matches many inputs against them, so the
tables and the engine are kept per rule set and set of options; the inputs are
made from the seed alone, on the GPU: bytes drawn from the rule set's own
symbol law with occurrences of its patterns planted at a fixed distance, as
the generators of `ngap_b200/workloads.py` do it. Reports are copied into a
buffer that the program keeps (rows past the last report stay -1).
"""
import ctypes
import functools
import math
import random

import numpy as np
import torch

import ngap_b200 as nb
from ngap_b200 import cost_model, workloads

KINDS = ("literal", "hamming", "levenshtein", "dotstar")
OCC = 48            # bytes of a planted occurrence (the longest pattern and its surroundings)
SAMPLE_EVERY = 128  # distance of the occurrences in a rule set's sample input


def listed():
    return [
        # the quick start: one short line against a handful of rules, bytes in
        # host memory; nothing but latency and launches
        _match("quickstart_81b", "literal", 8, 1, 81, "nonblockingallgroups", 3, 1, where="bytes"),
        # plain single stream: 64 regexes on 1 MiB of printable text
        _match("literal64_1m", "literal", 64, 1, 1 << 20, "nonblockingallgroups", -1, 1),
        # the same with the blocking algorithm it is compared with, default options
        _match("literal64_blocking_1m", "literal", 64, 1, 1 << 20, "blockinggroups", 0, 10),
        # Hamming k-mer search, 166k states, the headline benchmark
        _match("hamming1000_16m", "hamming", 1000, 16, 1 << 20, "nonblockingpcgroups", -1, 10),
        # k-mer search with the reference's usual options (three table levels,
        # ten groups) on segments of odd length
        _match("hamming200_p3_3m", "hamming", 200, 3, 1000003, "nonblockingallgroups", 3, 10),
        # edit-distance search with every option left at its default
        _match("levenshtein50_default_1m", "levenshtein", 50, 1, 999999, "nonblockingallgroups", 0,
               10),
        # the largest single input: edit distance on DNA, then dot-star
        # regexes on text, 32 segments
        _match("mix_32m", "mix", 2500, 32, 1 << 20, "nonblockingpcgroups", -1, 10),
        # log scanning: dot-star regexes on ragged segments in pinned host memory
        _match("dotstar300_ragged_4m", "dotstar", 300, 5, 777777, "nonblockingallgroups", -1, 1,
               where="pinned"),
        # motif search with very many hits: about one report per five bytes,
        # so sorting and copying the reports weigh as much as matching
        _match("motifs500_dense_8m", "motif", 500, 4, 2000000, "nonblockingpcgroups", -1, 1),
        # a server's burst: four batches of one to six requests, log-normal
        # lengths around 64 KiB, from pinned memory
        {"name": "serving_burst", "kind": "batch", "rules": 8, "scale": 1.0, "law": "lognormal",
         "streams": 6, "batches": 4, "layout": 5, "where": "pinned",
         "algorithm": "nonblockingpcgroups", "depth": -1},
        # bulk batch: 512 streams of 1 KiB to 4 MiB against eight rule sets
        {"name": "batch_512", "kind": "batch", "rules": 8, "scale": 1.0, "law": "loguniform",
         "streams": 512, "batches": 1, "layout": 6, "where": "device",
         "algorithm": "nonblockingpcgroups", "depth": -1},
        # the cost model over a batch's regions: features and predictions
        {"name": "features_64m", "kind": "features", "bytes": (64 << 20) - 4099, "region": 1 << 14,
         "window": 1024, "bf16": False},
    ]


def _match(name, rules, patterns, num_seg, seg_len, algorithm, depth, groups, where="device",
           rules_seed=11):
    c = {"kind": "match", "rules": rules, "patterns": patterns, "num_seg": num_seg,
         "seg_len": seg_len, "algorithm": algorithm, "depth": depth, "groups": groups,
         "where": where, "rules_seed": rules_seed}
    return dict(c, name=name) if name else c


def draw(rng):
    u = rng.random()
    if u < 0.10:
        return {"kind": "features", "bytes": _log(rng, 40000, 60 << 20), "region": 1 << 14,
                "window": rng.choice([512, 1000, 1024]), "bf16": rng.random() < 0.3}
    if u < 0.30:
        return {"kind": "batch", "rules": rng.randint(2, 8), "scale": round(rng.uniform(0.2, 1.0), 3),
                "law": rng.choice(["lognormal", "loguniform"]), "streams": _log(rng, 1, 300),
                "batches": rng.choice([1, 1, 2, 3]), "layout": rng.randint(10, 1 << 20),
                "where": rng.choice(["device", "device", "pinned"]),
                "algorithm": rng.choice(["nonblockingpcgroups", "nonblockingpcgroups",
                                         "nonblockingallgroups"]),
                "depth": rng.choice([-1, -1, 3])}
    rules = rng.choice(["literal", "literal", "hamming", "hamming", "levenshtein", "dotstar", "mix",
                        "motif"])
    deep = rng.random() < 0.7  # automatic table depth; else the reference's options
    if deep:
        algorithm, depth = rng.choice(["nonblockingpcgroups", "nonblockingallgroups"]), -1
        most = {"literal": 1500, "hamming": 1000, "levenshtein": 300, "dotstar": 1500, "mix": 2000,
                "motif": 500}[rules]
        total = _log(rng, 64, 20 << 20)
        total = min(total, 6000000) if rules == "motif" else total
    elif rules == "literal":
        algorithm, depth = rng.choice([("blockinggroups", 0), ("NAPgroups", 0),
                                       ("nonblockinggroups", 0), ("nonblockingr1groups", 0),
                                       ("nonblockingallgroups", 3)])
        most, total = 64, _log(rng, 64, 1 << 20)
    else:
        algorithm, depth = rng.choice([("nonblockinggroups", 0), ("nonblockingr1groups", 0),
                                       ("nonblockingpcgroups", 2), ("nonblockingallgroups", 3),
                                       ("nonblockingallgroups", 0)])
        most, total = {"dotstar": 200, "mix": 100, "motif": 100}.get(rules, 50), _log(rng, 64, 1 << 20)
    patterns = _log(rng, 5, most)
    num_seg = rng.choice([1, 1, 2, 5, 16, 31])
    seg_len = max(64, total // num_seg)
    return _match(None, rules, patterns, num_seg, seg_len, algorithm, depth,
                  rng.choice([1, 1, 3, 10]),
                  where=rng.choice(["device", "device", "pinned"] if total >= 1 << 20 else
                                   ["device", "device", "pinned", "bytes"]),
                  rules_seed=rng.randint(1, 1 << 20))


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# ---- rule sets ----------------------------------------------------------------

def _rules(kind, patterns, seed):
    """(ANML, [sample inputs with planted occurrences])."""
    kw = dict(seed=seed, n_patterns=patterns, input_len=256 * SAMPLE_EVERY, plant_every=SAMPLE_EVERY)
    if kind == "literal":
        anml, data = workloads.literal_set(**kw)
    elif kind == "hamming":
        anml, data = workloads.hamming_set(**kw)
    elif kind == "motif":  # 8-mers with at most one substitution
        anml, data = workloads.hamming_set(k=8, d=1, **kw)
    elif kind == "levenshtein":
        anml, data = workloads.levenshtein_set(**kw)
    elif kind == "dotstar":
        anml, data = workloads.dotstar_set(**kw)
    else:  # the high-frontier mix: a fifth edit distance, the rest dot-star
        rng = np.random.default_rng(seed)
        w = workloads.AnmlWriter("mix")
        kw.pop("seed")
        kw.update(writer=w, rng=rng)
        _, dna = workloads.levenshtein_set(**dict(kw, n_patterns=max(1, patterns // 5)))
        _, text = workloads.dotstar_set(**dict(kw, n_patterns=max(1, patterns - patterns // 5)))
        return w.text(), [dna, text]
    return anml, [data]


class _Law:
    """Symbol law and planted occurrences of one sample input, on the GPU."""

    def __init__(self, sample):
        hist = np.bincount(sample, minlength=256).astype(np.float64)
        self.symbols = torch.from_numpy(np.flatnonzero(hist).astype(np.uint8)).cuda()
        cdf = np.cumsum(hist[hist > 0] / hist.sum())
        self.cdf = torch.from_numpy(cdf.astype(np.float32)).cuda()
        at = np.arange(SAMPLE_EVERY // 2, len(sample) - OCC, SAMPLE_EVERY)
        self.occ = torch.from_numpy(sample[at[:, None] + np.arange(OCC)]).cuda()

    def bytes(self, n, gen, every):
        out = torch.empty(n, dtype=torch.uint8, device="cuda")
        for a in range(0, n, 4 << 20):
            m = min(4 << 20, n - a)
            u = torch.rand(m, generator=gen, device="cuda")
            k = torch.searchsorted(self.cdf, u).clamp_(max=len(self.symbols) - 1)
            out[a:a + m] = self.symbols[k]
        if n >= OCC:  # one occurrence per `every` bytes, eight or so in short inputs
            every = min(n, every, max(64, n // 8))
            at = torch.arange(n // every, device="cuda") * every
            at += torch.randint(every - OCC + 1, (len(at),), generator=gen, device="cuda")
            pick = torch.randint(len(self.occ), (len(at),), generator=gen, device="cuda")
            out[at[:, None] + torch.arange(OCC, device="cuda")] = self.occ[pick]
        return out


@functools.lru_cache(maxsize=2)
def _handle(rules, patterns, seed, groups, depth):
    """What a program loads once: tables, an engine and the inputs' laws."""
    anml, samples = _rules(rules, patterns, seed)
    g = nb.Groups(nb.Nfa.from_string(anml), group_num=groups)
    return nb.Tables(g, device=0, precompute_depth=depth), nb.Engine(0), [_Law(s) for s in samples]


@functools.lru_cache(maxsize=1)
def _batch_handle(rules, scale, depth):
    sizes = {"literal": (200, 1500), "hamming": (20, 200), "levenshtein": (20, 150),
             "dotstar": (150, 1200)}
    tables, laws = [], []
    for i in range(rules):
        kind = KINDS[i % 4]
        anml, samples = _rules(kind, max(1, int(scale * sizes[kind][i // 4])), 100 + i)
        g = nb.Groups(nb.Nfa.from_string(anml), group_num=1)
        tables.append(nb.Tables(g, device=0, precompute_depth=depth))
        laws.append(_Law(samples[0]))
    return nb.TableSet(tables), nb.Engine(0), laws


def _layout(case):
    """Per batch of a batch case: (lengths, rule set of each stream), from the case alone."""
    r = random.Random(case["layout"])
    out = []
    for _ in range(case["batches"]):
        n = case["streams"] if case["batches"] == 1 else r.randint(1, case["streams"])
        if case["law"] == "lognormal":
            lens = [int(min(4 << 20, max(64, r.lognormvariate(math.log(65536), 1.5)))) for _ in range(n)]
        else:
            lens = [_log(r, 1 << 10, 4 << 20) for _ in range(n)]
        out.append((lens, [r.randrange(case["rules"]) for _ in range(n)]))
    return out


# ---- preparing and running ----------------------------------------------------------

def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if case["kind"] == "features":
        return _prepare_features(case, seed, gen)
    if case["kind"] == "batch":
        ts, engine, laws = _batch_handle(case["rules"], case["scale"], case["depth"])
        batches = []
        for lens, nfas in _layout(case):
            data = torch.cat([laws[k].bytes(n, gen, 16 << 10) for n, k in zip(lens, nfas)])
            offsets = np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.int64)
            room = sum(lens) // 128 + 16384
            batches.append((_place(data, case["where"]), offsets, np.array(lens, np.int64),
                            np.array(nfas, np.int64), np.full(room, -1, np.int64),
                            np.full(room, -1, np.int32)))
        return {"kind": "batch", "tables": ts, "engine": engine, "batches": batches,
                "algorithm": case["algorithm"]}
    tables, engine, laws = _handle(case["rules"], case["patterns"], case["rules_seed"],
                                   case["groups"], case["depth"])
    n = case["num_seg"] * case["seg_len"]
    part = [n // len(laws)] * len(laws)
    part[-1] += n - sum(part)
    data = torch.cat([law.bytes(m, gen, 64 << 10) for law, m in zip(laws, part)])
    room = n // 64 + 4096 + (n * case["patterns"] // 2048 if case["rules"] == "motif" else 0)
    return {"kind": "match", "tables": tables, "engine": engine, "data": _place(data, case["where"]),
            "reports": np.full(room, -1, np.int64),
            "num_seg": case["num_seg"], "seg_len": case["seg_len"], "algorithm": case["algorithm"]}


def _place(data, where):
    if where == "bytes":
        return data.cpu().numpy().tobytes()
    return data.cpu().pin_memory() if where == "pinned" else data


def _prepare_features(case, seed, gen):
    data = _text(case, gen)
    model = cost_model.LearnedModel(device=0, in_dim=258)
    params, model.mu, model.sd = _model_values(seed)
    model.set_params(params)
    rs, ra, rl = cost_model.regions_of([0], [case["bytes"]], case["region"])
    return {"kind": "features", "data": data, "offsets": np.zeros(1, np.int64), "regions": (rs, ra, rl),
            "window": case["window"], "model": model, "bf16": case["bf16"]}


def _text(case, gen):
    """Printable bytes whose symbol law changes from region to region."""
    n, region = case["bytes"], case["region"]
    out = torch.empty(n, dtype=torch.uint8, device="cuda")
    step = 256 * region
    for a in range(0, n, step):
        m = min(step, n - a)
        u = torch.rand(m, generator=gen, device="cuda")
        e = torch.rand(-(-m // region), generator=gen, device="cuda").repeat_interleave(region)[:m]
        out[a:a + m] = (32 + 95 * u ** (1 + 3 * e)).clamp_(max=126).to(torch.uint8)
    return out


def _model_values(seed):
    """Parameters in the model's layout (W1, b1, W2, b2, w3, b3) and its normalisation."""
    r = np.random.default_rng(seed)
    p = np.concatenate([r.normal(0, math.sqrt(2 / 258), 258 * 64), r.normal(0, 0.1, 64),
                        r.normal(0, math.sqrt(2 / 64), 64 * 64), r.normal(0, 0.1, 64),
                        r.normal(0, 0.125, 64), r.normal(0, 0.1, 1)]).astype(np.float32)
    return p, r.uniform(0, 0.02, 258).astype(np.float32), r.uniform(0.02, 0.1, 258).astype(np.float32)


def run(state):
    if state["kind"] == "features":
        x = cost_model.byte_features(state["data"], state["offsets"], *state["regions"],
                                     window=state["window"])
        return {"x": x, "y": state["model"].predict_log(x, bf16=state["bf16"])}
    engine = state["engine"]
    if state["kind"] == "match":
        engine.match_async(state["tables"], state["data"], state["num_seg"], state["seg_len"],
                           algorithm=state["algorithm"])
        engine.sync()
        out = state["reports"]
        n = nb.lib().ngap_results_copy(engine._h, out.ctypes.data, len(out))
        _all_copied(engine, n)
        return out
    for data, offsets, lengths, nfas, reports, streams in state["batches"]:
        nb.batch_match_async(engine, state["tables"], data, offsets, lengths, nfas,
                             algorithm=state["algorithm"])
        engine.sync()
        n = ctypes.c_uint64()
        nb.lib().ngap_batch_results(engine._h, reports.ctypes.data, streams.ctypes.data,
                                    len(reports), ctypes.byref(n))
        _all_copied(engine, n.value)
    return [(b[4], b[5]) for b in state["batches"]]


def _all_copied(engine, n):
    if n != engine.counts()[1]:
        raise RuntimeError("the result buffer is too small")


def work(case):
    """Input read once and results written once; matching is integer work."""
    if case["kind"] == "features":
        n = -(-case["bytes"] // case["region"])
        mlp = 2 * (258 * 64 + 64 * 64 + 64)
        return {"bytes": case["bytes"] + 4 * n * (258 + 1), "flops": float(n * mlp)}
    if case["kind"] == "batch":
        total = sum(sum(lens) for lens, _ in _layout(case))
        return {"bytes": total + 12 * (total >> 14), "flops": 0.0}
    total = case["num_seg"] * case["seg_len"]
    # reports: the planted occurrences; motifs match by chance at 25 of 4^8 positions each
    reports = total * case["patterns"] * 25 / 65536 if case["rules"] == "motif" else total / 65536
    return {"bytes": total + 8 * int(reports), "flops": 0.0}


def exact(case, seed):
    """Features and predictions in 64 bits; reports are whole numbers and have none."""
    if case["kind"] != "features":
        return None
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    data = _text(case, gen)
    region, window = case["region"], case["window"]
    rows = []
    for a in range(0, case["bytes"], region):
        d = data[a:a + region].long()
        hist = torch.bincount(d, minlength=256).double() / len(d)
        k = max(1, len(d) // window)
        w = min(window, len(d))
        ids = torch.arange(k, device="cuda").repeat_interleave(w) * 256 + d[:k * w]
        q = torch.bincount(ids, minlength=256 * k).double().view(k, 256) / w
        h = -(q * torch.log2(q.clamp(min=1e-300))).sum(1)
        rows.append(torch.cat([hist, (h.mean() / 8)[None], (h.max() / 8)[None]]))
    x = torch.stack(rows)
    p, mu, sd = (torch.from_numpy(v).double().cuda() for v in _model_values(seed))
    w1, b1, w2, b2, w3, b3 = torch.split(p, [258 * 64, 64, 64 * 64, 64, 64, 1])
    h = torch.relu(((x - mu) / sd) @ w1.view(258, 64) + b1)
    h = torch.relu(h @ w2.view(64, 64) + b2)
    return {"x": x.cpu().numpy(), "y": (h @ w3 + b3).cpu().numpy()}
