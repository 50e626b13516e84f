"""Workloads of the batched B+tree, through its public entry points.

A case is a dict of plain values; `listed()` names the standing ones, `draw`
gives others of the same ranges.  Its "kind" is what a program does with a
tree:

  search  bt_search_batch: point lookups of a read-only tree
  mixed   batches of GETs and writes.  Half of the batches INSERT fresh keys
          beside their GETs, the other half DELETE those keys again (entries
          that expire), so that every pass meets the same key set.  With Zipf
          keys the writes are updates of stored keys instead, hot ones first.
          "call" is how the batches are given: "each" (one call per batch),
          "many" (one call for all of them) or "host" (page-locked host
          buffers, three batches in flight)
  range   range scans
  load    a bulk build, one batch of 95 % GETs and 5 % INSERTs, the sorted
          contents: what the reference's program does with its two files
  grow    an empty tree filled by INSERT batches, the sorted contents

Inputs come from the seed alone.  Keys are int64 tensors in [0, 2^62), all
different from one index to the next; a value is its key under a constant.
"""
import torch

import eirene_b200 as E

MASK62 = (1 << 62) - 1
VALUE = 0x1E3779B97F4A7C15
# bytes a request cannot do without: its leaf's keys and one value sector; a
# write also puts its leaf row back
READ, WRITE = 288, 512
DEV = "cuda:0"


def listed():
    return [
        # a handful of lookups between other work of a program: all latency
        {"name": "search_100", "kind": "search", "tree": 1 << 20, "n": 100, "dist": "uniform", "learned": False},
        # a full batch of lookups on a tree far larger than L2, odd size
        {"name": "search_plain", "kind": "search", "tree": 1 << 25, "n": (1 << 22) - 5, "dist": "uniform",
         "learned": False},
        # the same through the trained leaf predictor, skewed keys
        {"name": "search_learned", "kind": "search", "tree": 1 << 25, "n": 1 << 22, "dist": "normal",
         "learned": True},
        # an interactive service's small batches
        {"name": "mixed_1000", "kind": "mixed", "tree": 1 << 20, "n": 1000, "batches": 2, "write": 5, "mode": "merge",
         "call": "each", "dist": "uniform", "learned": False},
        # the headline: 95/5 batches of 2^22 on 2^26 keys, trained predictor, several batches a call
        {"name": "mixed_headline", "kind": "mixed", "tree": 1 << 26, "n": 1 << 22, "batches": 4, "write": 5,
         "mode": "merge", "call": "many", "dist": "uniform", "learned": True},
        # write-heavy ingest
        {"name": "mixed_50_50", "kind": "mixed", "tree": 1 << 24, "n": 1 << 20, "batches": 2, "write": 50,
         "mode": "merge", "call": "each", "dist": "uniform", "learned": False},
        # hot keys: GETs and updates by a Zipf law, the default insert engine
        {"name": "mixed_zipf", "kind": "mixed", "tree": 1 << 22, "n": (1 << 18) + 1, "batches": 2, "write": 20,
         "mode": "sorted", "call": "each", "dist": "zipf", "learned": False},
        # concurrent transactions (the reference's v39 meaning)
        {"name": "mixed_stm", "kind": "mixed", "tree": 1 << 23, "n": 1 << 20, "batches": 2, "write": 5, "mode": "stm",
         "call": "each", "dist": "uniform", "learned": False},
        # requests and answers in host memory
        {"name": "mixed_host", "kind": "mixed", "tree": 1 << 24, "n": 1 << 20, "batches": 4, "write": 5,
         "mode": "merge", "call": "host", "dist": "uniform", "learned": False},
        # pages of neighbouring keys
        {"name": "range_100", "kind": "range", "tree": 1 << 24, "n": 20000, "span": 100, "max_per": 128,
         "dist": "uniform"},
        # 2^20 keys loaded, one 2^20 batch, read back
        {"name": "load_query", "kind": "load", "tree": 1 << 20, "n": 1 << 20, "dist": "uniform"},
        # the reference program's own build: P lines in batches of 1,310,720
        {"name": "grow_insert", "kind": "grow", "tree": (1 << 23) - 1, "n": 1310720, "dist": "uniform"},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["search", "search", "mixed", "mixed", "mixed", "mixed", "range", "load", "grow"])
    tree = _log(rng, 1 << 16, 1 << 24)
    if kind == "search":
        return {"kind": kind, "tree": tree, "n": _log(rng, 20, 1 << 22), "dist": rng.choice(["uniform", "normal"]),
                "learned": rng.random() < 0.5}
    if kind == "mixed":
        call = rng.choice(["each", "each", "many", "host"])
        dist = rng.choice(["uniform", "uniform", "normal", "zipf"])
        mode = rng.choice(["merge", "merge", "sorted", "stm"])
        if mode == "stm":  # answers that do not depend on the order: no key twice
            call, dist = rng.choice(["each", "host"]), "uniform"
        return {"kind": kind, "tree": tree, "n": min(_log(rng, 100, 1 << 21), tree // 2), "batches": rng.choice([2, 4]),
                "write": rng.choice([1, 5, 5, 20, 50]), "mode": mode, "call": call, "dist": dist,
                "learned": rng.random() < 0.3}
    if kind == "range":
        span = _log(rng, 1, 1000)
        return {"kind": kind, "tree": tree, "n": _log(rng, 50, 20000), "span": span,
                "max_per": rng.choice([span + span // 4 + 8, max(1, span // 2)]), "dist": "uniform"}
    if kind == "load":
        return {"kind": kind, "tree": tree, "n": _log(rng, 1000, 1 << 21), "dist": rng.choice(["uniform", "normal"])}
    return {"kind": kind, "tree": min(tree, 1 << 22), "n": _log(rng, 1 << 14, 1 << 20),
            "dist": rng.choice(["uniform", "normal"])}


# ---------------------------------------------------------------- inputs ----
class _Keys:
    """Keys by index (see the module's text), of one law and one seed."""

    def __init__(self, dist, seed):
        self.normal = dist == "normal"
        self.seed = seed
        self.gen = torch.Generator(device=DEV)
        self.gen.manual_seed(seed)

    def ints(self, lo, hi, n):
        return torch.randint(lo, hi, (n,), device=DEV, generator=self.gen)

    def zipf(self, hi, n):
        # ranks 0 .. hi - 1 with a weight of about 1 / (rank + 1)
        u = torch.rand(n, device=DEV, generator=self.gen, dtype=torch.float64)
        return (float(hi) ** u).long().clamp_(1, hi) - 1

    def keys(self, idx):
        if self.normal:  # about Normal(2^61, 2^57), the low bits from the index
            low = (idx * 0x2545F49 + self.seed % (1 << 27)) & ((1 << 27) - 1)
            # the same index always gives the same key: its deviate comes from the mixed index
            u = ((self._mix(idx).double() + 0.5) / float(1 << 62)).clamp_(1e-12, 1 - 1e-12)
            z = torch.special.ndtri(u)
            return (((1 << 34) + (z * (1 << 30))).long().clamp_(0, (1 << 35) - 1) << 27) | low
        return self._mix(idx)

    def _mix(self, idx):
        x = (idx + (self.seed * 0x632BE59BD9B4E5 & MASK62)) & MASK62
        x = (x * 0x2545F4914F6CDD1D) & MASK62
        x = x ^ (x >> 31)
        x = (x * 0x1B873593CC9E2D51) & MASK62
        return x ^ (x >> 29)


def _batches(case, K):
    """[(keys, vals, ops)] of a mixed case, and the tree's keys."""
    N, n, m = case["tree"], case["n"], case["batches"]
    w = max(1, n * case["write"] // 100)
    half = m // 2
    out = []
    writes = []
    for b in range(m):
        where = torch.randperm(n, device=DEV, generator=K.gen)
        ops = torch.full((n,), E.OP_GET, dtype=torch.uint8, device=DEV)
        idx = torch.empty(n, dtype=torch.int64, device=DEV)
        g = n - w
        if case["dist"] == "zipf":
            gets, put, op = K.zipf(N, g), K.zipf(N, w), E.OP_INSERT
        else:
            # GETs: half of them stored keys, half keys that never are
            gets = torch.where(K.ints(0, 2, g) == 0, K.ints(0, N, g), N + half * w + K.ints(0, 1 << 25, g))
            if b < half:
                put, op = N + b * w + torch.arange(w, device=DEV), E.OP_INSERT
                writes.append(put)
            else:
                put, op = writes[b - half][torch.randperm(w, device=DEV, generator=K.gen)], E.OP_DELETE
        idx[where[:g]] = gets
        idx[where[g:]] = put
        ops[where[g:]] = op
        keys = K.keys(idx)
        out.append((keys, (keys ^ VALUE) + b if case["dist"] == "zipf" else keys ^ VALUE, ops))
    return out


def _inputs(case, seed):
    K = _Keys(case["dist"], seed)
    N, n = case["tree"], case["n"]
    d = {"tree": K.keys(torch.arange(N, device=DEV)), "batches": []}
    kind = case["kind"]
    if kind == "search":
        d["q"] = K.keys(torch.where(K.ints(0, 2, n) == 0, K.ints(0, N, n), N + K.ints(0, 1 << 25, n)))
    elif kind == "mixed":
        d["batches"] = _batches(case, K)
    elif kind == "range":
        step = MASK62 // N
        d["lo"] = K.ints(0, MASK62, n)
        d["hi"] = d["lo"] + K.ints(1, 2 * case["span"] + 1, n) * step
    elif kind == "load":
        w = max(1, n // 20)
        idx = torch.cat([torch.where(K.ints(0, 2, n - w) == 0, K.ints(0, N, n - w), N + w + K.ints(0, 1 << 25, n - w)),
                         N + torch.arange(w, device=DEV)])
        ops = torch.full((n,), E.OP_GET, dtype=torch.uint8, device=DEV)
        ops[n - w:] = E.OP_INSERT
        at = torch.randperm(n, device=DEV, generator=K.gen)
        keys = K.keys(idx[at])
        d["batches"] = [(keys, keys ^ VALUE, ops[at])]
    else:  # grow: the keys in their drawn order, batch by batch
        for a in range(0, N, n):
            k = d["tree"][a:a + n]
            d["batches"].append((k, k ^ VALUE, torch.full_like(k, E.OP_INSERT, dtype=torch.uint8)))
    return d


# ------------------------------------------------------------------- run ----
MODES = {"merge": E.MODE_SORTED | E.MODE_MERGE_ENGINE, "sorted": E.MODE_SORTED, "stm": E.MODE_STM}


def prepare(case, seed):
    d = _inputs(case, seed)
    kind, n = case["kind"], case["n"]
    room = case["tree"] + sum(int(b[0].numel()) for b in d["batches"]) // 2 + 4096
    tree = E.BTree(max_keys=room, max_batch=max(n, 1024))
    s = {"case": case, "tree": tree, "batches": d["batches"]}
    if kind in ("search", "mixed", "range"):
        tree.bulk_build(d["tree"], d["tree"] ^ VALUE)
        if case.get("learned"):
            tree.retrain()
            tree.set_descent(True)
    if kind == "load":
        s["keys"], s["vals"] = d["tree"], d["tree"] ^ VALUE
    if kind == "grow":
        s["none"] = torch.empty(0, dtype=torch.int64, device=DEV)
    if kind == "search":
        s["q"] = d["q"]
        s["out"] = (torch.empty_like(d["q"]), torch.empty_like(d["q"], dtype=torch.uint8))
    if kind == "range":
        s["lo"], s["hi"] = d["lo"], d["hi"]
    s["mode"] = MODES[case.get("mode", "merge")]
    if case.get("call") == "host":
        pin = lambda t: t.cpu().pin_memory()  # noqa: E731
        s["host"] = [(pin(k), pin(o), pin(v[o == E.OP_INSERT])) for k, v, o in d["batches"]]
        s["outs"] = [(torch.empty(k.numel(), dtype=torch.int64, pin_memory=True),
                      torch.empty(k.numel(), dtype=torch.uint8, pin_memory=True)) for k, _, _ in d["batches"]]
        s["batches"] = []
    else:
        s["outs"] = [(torch.empty_like(k), torch.empty_like(o)) for k, _, o in d["batches"]]
    return s


def run(s):
    case, tree, mode = s["case"], s["tree"], s["mode"]
    kind = case["kind"]
    if kind == "search":
        tree.search(s["q"], *s["out"])
        return s["out"]
    if kind == "range":
        return tree.range(s["lo"], s["hi"], case["max_per"])
    if kind == "load":
        tree.bulk_build(s["keys"], s["vals"])
    elif kind == "grow":
        tree.bulk_build(s["none"], s["none"])
    if case.get("call") == "host":
        tickets = []
        for i, (k, o, v) in enumerate(s["host"]):
            tickets.append(tree.submit_host_packed(k, o, v, *s["outs"][i], mode=mode))
            if i >= 2:
                tree.wait_host(tickets[i - 2])
        for t in tickets[-2:]:
            tree.wait_host(t)
    elif case.get("call") == "many":
        tree.execute_many(s["batches"], s["outs"], mode=mode)
    else:
        for (k, v, o), (ov, os) in zip(s["batches"], s["outs"]):
            tree.execute(k, v, o, ov, os, mode=mode)
    if kind in ("load", "grow"):
        return s["outs"], tree.dump()
    return s["outs"]


# ---------------------------------------------------------- work, exact ----
def work(case):
    """Requests and answers once, a leaf's keys and a value sector per request
    (no more than the leaves there are), a leaf row written per write."""
    N, n, kind = case["tree"], case["n"], case["kind"]
    leaf_keys = 24
    leaves = N / leaf_keys
    if kind == "search":
        b = n * 17 + min(n * 256, leaves * 256) + n * 32
    elif kind == "range":
        b = n * (20 + 16 * case["max_per"]) + min(n * (case["span"] / leaf_keys + 1), leaves) * 512
    elif kind == "mixed":
        w = max(1, n * case["write"] // 100)
        b = case["batches"] * (n * 18 + 8 * w + min(n, leaves) * 256 + (n - w) * 32 + min(w, leaves) * (256 + WRITE))
    elif kind == "load":
        w = max(1, n // 20)
        b = N * 16 + leaves * 512 + n * 18 + 8 * w + min(n, leaves) * 256 + n * 32 + min(w, leaves) * (256 + WRITE)
        b += leaves * 512 + (N + w) * 16
    else:
        b = N * 26 + leaves * 512 + leaves * 512 + N * 16
        for a in range(0, N, n):  # every batch meets the leaves that the ones before it left
            b += min(min(n, N - a), a / leaf_keys) * 2 * WRITE
    return {"bytes": float(b), "flops": 0.0}


class _Plain:
    """The tree as two sorted tensors."""

    def __init__(self, keys):
        self.k = torch.sort(keys)[0]
        self.v = self.k ^ VALUE

    def get(self, q):
        if self.k.numel() == 0:
            return torch.zeros_like(q, dtype=torch.bool), torch.zeros_like(q)
        at = torch.searchsorted(self.k, q).clamp_(max=self.k.numel() - 1)
        hit = self.k[at] == q
        return hit, torch.where(hit, self.v[at], 0)

    def batch(self, keys, vals, ops):
        """Per key in request order; across keys the contents before the batch."""
        n = keys.numel()
        sk, order = torch.sort(keys, stable=True)
        so, sv = ops[order], vals[order]
        pos = torch.arange(n, device=keys.device)
        head = torch.ones(n, dtype=torch.bool, device=keys.device)
        head[1:] = sk[1:] != sk[:-1]
        start = torch.cummax(torch.where(head, pos, -1), 0)[0]
        last = torch.cummax(torch.where(so != E.OP_GET, pos, -1), 0)[0]
        before = torch.cat([last.new_full((1,), -1), last[:-1]])
        own = before >= start
        hit, val = self.get(sk)
        at = before.clamp(min=0)
        hit = torch.where(own, so[at] == E.OP_INSERT, hit)
        val = torch.where(hit, torch.where(own, sv[at], val), 0)
        out_v, out_s = torch.empty_like(val), torch.empty_like(ops)
        out_v[order], out_s[order] = val, hit.to(torch.uint8)
        # each key's last write
        tail = torch.ones_like(head)
        tail[:-1] = head[1:]
        w = tail & (last >= start)
        wk, wo, wv = sk[w], so[last[w]], sv[last[w]]
        if wk.numel():
            keep = ~torch.isin(self.k, wk, assume_unique=True) if self.k.numel() else self.k == 0
            k = torch.cat([self.k[keep], wk[wo == E.OP_INSERT]])
            v = torch.cat([self.v[keep], wv[wo == E.OP_INSERT]])
            self.k, p = torch.sort(k)
            self.v = v[p]
        return out_v, out_s


def exact(case, seed):
    """What run() answers on a new state, by sorting and searching in torch."""
    d = _inputs(case, seed)
    kind = case["kind"]
    t = _Plain(d["tree"] if kind != "grow" else d["tree"][:0])
    if kind == "search":
        hit, val = t.get(d["q"])
        return val, hit.to(torch.uint8)
    if kind == "range":
        a = torch.searchsorted(t.k, d["lo"])
        b = torch.searchsorted(t.k, d["hi"], right=True)
        at = a[:, None] + torch.arange(case["max_per"], device=a.device)
        there = at < b[:, None]
        at = at.clamp_(max=t.k.numel() - 1)
        return (b - a).to(torch.int32), torch.where(there, t.k[at], 0), torch.where(there, t.v[at], 0)
    outs = [t.batch(*x) for x in d["batches"]]
    return (outs, (t.k, t.v)) if kind in ("load", "grow") else outs
