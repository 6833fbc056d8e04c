"""The timed work of this library: what its users have it do, from one small call to whole shards.

Every case goes through a public entry point of ``B200Tokenizer``: ``encode_device`` (rows already
on the GPU), the Hugging Face style call (a list of strings) or ``encode_host`` (host arrays in and
out).  A case names a tokenizer, how many rows it takes and how long they are, and the layout of the
result.  All outputs are whole numbers and have to stay the same.

Inputs are seeded synthetic DNA: uniform bases with runs of N for the per-character and k-mer
tokenizers, soft-masked runs for the byte-level one, and order-3 Markov chains (the chains the two
BPE vocabularies were trained on) for BPE, which is where its token lengths come from.
"""
import functools
import gzip
import itertools
import json
import math
import os

import numpy as np
import torch

from dnatok_b200 import synth
from dnatok_b200.tables import Specials, TokenizerSpec, bpe_spec_from_json
from dnatok_b200.tokenizer import B200Tokenizer

GOLDEN = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tests", "golden")


def _case(name, tok, via, layout, rows, lo, hi, width=0, special=False, left=False, ids=64, mask=64):
    """rows of lo..hi bp (log-uniform); layout: "width" (padded or cut to ``width`` tokens), "longest" or "ragged";
    ids / mask: bits of an element, mask 0 for none."""
    return {"name": name, "tok": tok, "via": via, "layout": layout, "rows": rows, "lo": lo, "hi": hi, "width": width,
            "special": special, "left": left, "ids": ids, "mask": mask}


def listed():
    return [
        # an interactive call: a handful of sequences as Python strings, tensors back
        _case("call_char", "char", "call", "longest", 64, 200, 1024, special=True),
        # a shard of training windows with fixed width, buffers kept by the loop: the benchmark's headline shape
        _case("kmer6_windows", "kmer6", "device", "width", 32768, 6000, 6000, width=1000),
        # inference batches of uneven records, padded on the left to the longest (the plug-in's default side)
        _case("kmer6_longest_left", "kmer6", "device", "longest", 6001, 500, 8000, left=True),
        # contigs: few rows, each of them long
        _case("kmer6_contigs", "kmer6", "device", "ragged", 15, 300000, 1048576, ids=32),
        # a tokenizer whose windows with an N give runs of ids: the table of all 5^k windows
        _case("kmer5_table", "kmer5t", "device", "longest", 8190, 500, 4000),
        # reads of very different lengths, flat ids and offsets (a packed data set)
        _case("char_reads_ragged", "char", "device", "ragged", 16384, 150, 10000, special=True),
        # byte-level model, whole windows of a chromosome, ids only
        _case("byte_chromosome", "byte", "device", "longest", 64, 1048576, 1048576, ids=32, mask=0),
        # BPE, fixed-length records with [CLS] .. [SEP], model width 512
        _case("bpe4k_records", "bpe4k", "device", "width", 16384, 1024, 1024, width=512, special=True),
        # BPE, short sequencing reads, compact types
        _case("bpe4k_short_reads", "bpe4k", "device", "longest", 65536, 50, 300, special=True, ids=32, mask=8),
        # BPE, long-read data set, flat ids
        _case("bpe32k_reads_ragged", "bpe32k", "device", "ragged", 8192, 150, 10000),
        # BPE over assembled contigs
        _case("bpe4k_contigs", "bpe4k", "device", "ragged", 33, 40000, 400000),
        # host arrays in, host arrays out (a data-preparation job)
        _case("kmer6_host", "kmer6", "host", "width", 4096, 6000, 6000, width=1000),
    ]


def draw(rng):
    """One more case of these ranges: sizes spread over their logarithm, odd ones among them, no larger than the listed
    case of the same family."""
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    def bits():
        return {"ids": rng.choice([32, 64]), "mask": rng.choice([0, 8, 32, 64])}

    fam = rng.choice(["call", "kmer", "contigs", "table", "ragged", "byte", "bpe", "bpe_short", "bpe_ragged", "bpe_contigs", "host"])
    special, left = rng.random() < 0.5, rng.random() < 0.4
    if fam == "call":
        lo = log(30, 300)
        return _case("", rng.choice(["char", "kmer6", "bpe4k"]), "call", "longest", log(4, 256), lo, lo + log(1, 1500), special=special)
    if fam == "kmer":
        length = log(100, 6000)
        rows = log(500, 32768)
        if rng.random() < 0.5:
            return _case("", "kmer6", "device", "width", rows, length, length + rng.randint(0, 40), width=max(8, length // 6 + rng.randint(-9, 9)),
                         left=left, **bits())
        return _case("", "kmer6", "device", "longest", max(1, rows // 5), length, 2 * length, left=left, **bits())
    if fam == "contigs":
        lo = log(50000, 700000)
        return _case("", "kmer6", "device", "ragged", log(1, 15), lo, lo + log(10, 300000), ids=rng.choice([32, 64]))
    if fam == "table":
        lo = log(100, 1500)
        return _case("", "kmer5t", "device", "longest", log(300, 8190), lo, lo + log(1, 2500), left=left, **bits())
    if fam == "ragged":
        lo = log(100, 600)
        return _case("", rng.choice(["char", "byte"]), "device", "ragged", log(200, 16384), lo, lo + log(10, 9000), special=special,
                     ids=rng.choice([32, 64]))
    if fam == "byte":
        length = log(5000, 1048576)
        return _case("", "byte", "device", "longest", log(1, 64), length, length + rng.randint(0, 3), left=left, **bits())
    if fam == "bpe":
        length = log(300, 1024)
        return _case("", rng.choice(["bpe4k", "bpe32k"]), "device", "width", log(200, 10000), max(1, length - rng.randint(0, 200)), length,
                     width=max(64, length // 3), special=special, left=left, **bits())
    if fam == "bpe_short":
        lo = log(20, 150)
        return _case("", rng.choice(["bpe4k", "bpe32k"]), "device", "longest", log(500, 40000), lo, lo + log(1, 160), special=special, left=left,
                     **bits())
    if fam == "bpe_ragged":
        lo = log(150, 2000)
        return _case("", rng.choice(["bpe4k", "bpe32k"]), "device", "ragged", log(100, 5000), lo, lo + log(10, 8000), special=special,
                     ids=rng.choice([32, 64]))
    if fam == "bpe_contigs":
        lo = log(33000, 250000)
        return _case("", rng.choice(["bpe4k", "bpe32k"]), "device", "ragged", log(4, 33), lo, lo + log(10, 150000), ids=rng.choice([32, 64]))
    length = log(1000, 6000)
    return _case("", "kmer6", "host", "width", log(200, 4096), length, length, width=max(8, length // 6), **bits())


# ------------------------------------------------------------------ tokenizers (kept, as a program keeps them)

@functools.lru_cache(maxsize=None)
def _spec(kind):
    if kind == "byte":
        return TokenizerSpec("char", Specials(1, 0, -1, -1), 512, np.arange(256, dtype=np.int32))
    if kind in ("bpe4k", "bpe32k"):
        with gzip.open(os.path.join(GOLDEN, {"bpe4k": "bpe4096", "bpe32k": "bpe32000"}[kind] + ".tokenizer.json.gz"), "rt") as f:
            return bpe_spec_from_json(json.load(f))
    lut = np.full(256, 1, np.int32)
    if kind == "char":
        for i, c in enumerate("ACGTN"):
            lut[ord(c)] = 5 + i
        return TokenizerSpec("char", Specials(0, 1, 2, 3), 10, lut)
    k = 5 if kind == "kmer5t" else 6
    for i, c in enumerate("ACGTN"):
        lut[ord(c)] = 5 + 4 ** k + i
    if kind == "kmer6":
        return TokenizerSpec("kmer", Specials(0, 1, 2, 3), 10 + 4 ** k, lut, k=k, kmer_ids=np.arange(5, 5 + 4 ** k, dtype=np.int32))
    # every window over ACGTN: a clean one is one id, any other gives its letters one by one, a run of N as one token
    table, offsets, ids, n_clean = [], [0], [], 0
    for win in itertools.product("ACGTN", repeat=k):
        if "N" not in win:
            table.append(5 + n_clean)
            n_clean += 1
            continue
        table.append(-len(offsets))
        ids += [int(lut[ord(c)]) for i, c in enumerate(win) if c != "N" or i == 0 or win[i - 1] != "N"]
        offsets.append(len(ids))
    return TokenizerSpec("kmer", Specials(0, 1, 2, 3), 10 + 4 ** k, lut, k=k, kmer_table5=np.array(table, np.int32),
                         kmer_run_offsets=np.array(offsets, np.int32), kmer_run_ids=np.array(ids, np.int32))


@functools.lru_cache(maxsize=None)
def _tokenizer(kind, left):
    tok = B200Tokenizer(_spec(kind))
    tok.padding_side = "left" if left else "right"
    return tok


# ------------------------------------------------------------------ inputs

# The width of a batch padded to its longest row and the size of a flat result follow from the row lengths, from where the
# Ns are and, for BPE, from the text itself.  They belong to the case: the seed draws the bases between the Ns, and for BPE
# without a fixed width the order of the rows.

def _lengths(case):
    rng = np.random.default_rng([11, case["rows"], case["lo"], case["hi"]])
    lo, hi = case["lo"], case["hi"]
    return np.clip(np.floor(np.exp(rng.uniform(np.log(lo), np.log(hi + 1), size=case["rows"]))), lo, hi).astype(np.int64)


def _uniform(total, seed):
    """ACGT with runs of 1..50 N on about half a percent of the positions; where the runs are depends on the size alone."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    letters = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device="cuda")
    x = letters[torch.randint(0, 4, (total,), generator=g, device="cuda", dtype=torch.uint8).to(torch.int32)]
    g.manual_seed(total)
    n = max(1, total // 5000)
    start = torch.randint(0, total, (n,), generator=g, device="cuda")
    run = torch.randint(1, 51, (n,), generator=g, device="cuda")
    where = (start[:, None] + torch.arange(50, device="cuda")).clamp_(max=total - 1)
    x[where[torch.arange(50, device="cuda") < run[:, None]]] = ord("N")
    return x


def _soft_masked(total, seed):
    """Alternating upper- and lower-case stretches of a few hundred bp, single Ns."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = _uniform(total, seed + 1)
    flips = torch.zeros(total, dtype=torch.int32, device="cuda")
    flips[torch.randint(0, total, (max(1, total // 375),), generator=g, device="cuda")] = 1
    x[(torch.cumsum(flips, 0) & 1) > 0] |= 0x20
    return x


@functools.lru_cache(maxsize=None)
def _chain(kind):
    return torch.from_numpy(np.cumsum(synth.config3_chain() if kind == "bpe4k" else synth.config5_chain(), axis=1)).float().cuda()


def _markov(kind, total, seed):
    """Order-3 chains of 1,024 bp, laid end to end."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    steps = 1024 if total > 4096 else 64
    n = -(-total // steps)
    cum = _chain(kind)[:, :3].contiguous()
    ctx = torch.randint(0, 64, (n,), generator=g, device="cuda")
    out = torch.empty((steps, n), dtype=torch.uint8, device="cuda")
    for t in range(steps):
        nxt = (torch.rand(n, 1, generator=g, device="cuda") >= cum[ctx]).sum(1)
        out[t] = nxt
        ctx = ((ctx << 2) | nxt) & 63
    letters = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device="cuda")
    return letters[out.t().reshape(-1)[:total].to(torch.int32)]


def _starts(lens):
    offsets = np.zeros(len(lens) + 1, dtype=np.int64)
    np.cumsum(lens, out=offsets[1:])
    return offsets


def _batch(case, seed):
    """Packed bytes on the GPU and row offsets."""
    lens = _lengths(case)
    offsets = _starts(lens)
    total = int(offsets[-1])
    if case["tok"] in ("bpe4k", "bpe32k"):
        if case["layout"] == "width":
            return _markov(case["tok"], total, seed), offsets
        pool = _markov(case["tok"], total, case["rows"])
        order = np.random.default_rng([13, seed]).permutation(len(lens))
        moved = _starts(lens[order])
        shift = torch.from_numpy(offsets[:-1][order] - moved[:-1]).cuda()
        src = torch.repeat_interleave(shift, torch.from_numpy(lens[order]).cuda()) + torch.arange(total, device="cuda")
        return pool[src], moved
    return (_soft_masked(total, seed) if case["tok"] == "byte" else _uniform(total, seed)), offsets


def prepare(case, seed):
    d_bytes, offsets = _batch(case, seed)
    tok = _tokenizer(case["tok"], case["left"])
    ids_t = {32: torch.int32, 64: torch.int64}[case["ids"]]
    mask_t = {0: None, 8: torch.uint8, 32: torch.int32, 64: torch.int64}[case["mask"]]
    st = {"case": case, "tok": tok, "offsets": offsets}
    fmt = {"add_special_tokens": case["special"], "return_attention_mask": mask_t is not None and case["layout"] != "ragged"}
    if case["layout"] == "width":
        fmt.update(padding="max_length", max_length=case["width"], truncation=True)
    else:
        fmt.update(padding="longest" if case["layout"] == "longest" else False)
    st["fmt"] = fmt
    if case["via"] == "call":
        st["text"] = synth.rows_to_strings(d_bytes.cpu().numpy(), offsets)
    elif case["via"] == "host":
        # pinned host arrays the job keeps
        st["flat"] = d_bytes.cpu().pin_memory().numpy()
        n = case["rows"] * case["width"]
        st["out_ids"] = torch.empty(n, dtype=ids_t).pin_memory().numpy()
        st["out_mask"] = torch.empty(n, dtype=mask_t).pin_memory().numpy() if mask_t is not None else None
        fmt.update(ids_dtype=st["out_ids"].dtype, out_ids=st["out_ids"])
        if mask_t is not None:
            fmt.update(mask_dtype=st["out_mask"].dtype, out_mask=st["out_mask"])
    else:
        st["d_bytes"], st["d_offsets"] = d_bytes, torch.from_numpy(offsets).cuda()
        fmt.update(ids_dtype=ids_t)
        if mask_t is not None:
            fmt.update(mask_dtype=mask_t)
        if case["layout"] == "width":
            # a training loop keeps its output tensors and does not read the status words back every step
            shape = (case["rows"], case["width"])
            st["out"] = {"input_ids": torch.empty(shape, dtype=ids_t, device="cuda")}
            if mask_t is not None:
                st["out"]["attention_mask"] = torch.empty(shape, dtype=mask_t, device="cuda")
            fmt.update(out=st["out"], check=False)
    return st


def run(state):
    tok, via = state["tok"], state["case"]["via"]
    if via == "call":
        return dict(tok(state["text"], return_tensors="pt", **state["fmt"]))
    if via == "host":
        return dict(tok.encode_host((state["flat"], state["offsets"]), **state["fmt"]))
    return dict(tok.encode_device(state["d_bytes"], state["d_offsets"], host_offsets=state["offsets"], **state["fmt"]))


# ------------------------------------------------------------------ floors

# bp per token: one for the per-character tables, k for k-mers, and what the two BPE vocabularies reach on their chains
_BP_PER_TOKEN = {"char": 1.0, "byte": 1.0, "kmer6": 6.0, "kmer5t": 5.0, "bpe4k": 5.6, "bpe32k": 5.4}


def work(case):
    """Every input byte once, every element of the returned ids and mask once (with offsets where rows are ragged).  A row
    cut at ``width`` tokens needs the bytes under those tokens only."""
    lens = _lengths(case).astype(np.float64)
    per = _BP_PER_TOKEN[case["tok"]]
    special = 2 if case["special"] and case["tok"] != "byte" else 0
    tokens = np.ceil(lens / per) + special
    rows = len(lens)
    if case["layout"] == "ragged":
        out = tokens.sum() * case["ids"] / 8 + 8 * (rows + 1)
        read = lens.sum()
    else:
        width = case["width"] if case["layout"] == "width" else tokens.max()
        out = rows * width * (case["ids"] + case["mask"]) / 8
        read = np.minimum(lens, width * per).sum()
    return {"bytes": float(read + out + 8 * (rows + 1) + 4 * rows), "flops": 0.0}


def tolerance(case):
    return "exact"
