"""Tokenizers the fast k-mer form cannot express, through the complete window table (rows the reference
covers with its 5**k table and multi-token expansion, src/dna_tokenizer.py:743-822 and :1896-1953), and
per-character tokenizers whose first-position ids differ (:527-631, :1779-1820).  The tokenizers below are
re-creations of the shapes the reference's own tests use (tests/test_kmer_bytes_fallback.py:8-59: two
tokens for every window holding N, tail dropped; tests/test_ids_path_equivalence.py:310-345: k = 4, every
window one token, tail per character); the live tokenizer object is the oracle."""
import numpy as np
import pytest

from dnatok_b200 import tables

torch = pytest.importorskip("torch")


class TwoTokensForN:
    """k-mer tokenizer: clean windows get ids in order of first use, a window holding N gives the pair
    (97, 98), characters left over after the last whole window give nothing."""

    def __init__(self, k=3):
        self.k, self.pad_token_id, self.padding_side, self.seen = k, 0, "right", {}

    def _one(self, text):
        out = []
        for i in range(0, len(text) - self.k + 1, self.k):
            w = text[i:i + self.k]
            if "N" in w:
                out += [97, 98]
            else:
                out.append(self.seen.setdefault(w, len(self.seen) + 1))
        return out

    def __call__(self, texts, add_special_tokens=False, **kw):
        return {"input_ids": [self._one(t) for t in ([texts] if isinstance(texts, str) else texts)]}


class SumOfLetters:
    """k-mer tokenizer: a whole window is one token whose id is 100 + the sum of its letters' values
    (many windows share an id, windows with N included); the tail goes letter by letter."""

    def __init__(self, k=4):
        self.k, self.pad_token_id, self.value = k, 0, {"A": 1, "C": 2, "G": 3, "T": 4, "N": 5}

    def _one(self, text):
        out, i = [], 0
        while i < len(text):
            w = text[i:i + self.k]
            out += [100 + sum(self.value.get(c, 0) for c in w)] if len(w) == self.k else [self.value.get(c, 0) for c in w]
            i += len(w)
        return out

    def __call__(self, texts, add_special_tokens=False, **kw):
        return {"input_ids": [self._one(t) for t in ([texts] if isinstance(texts, str) else texts)]}


class FirstLetterDiffers:
    """One token per character; a character's id at the start of a sequence is 50 higher than later on."""

    def __init__(self):
        self.pad_token_id, self.unk_token_id = 0, 1
        self.later = {c: 10 + i for i, c in enumerate("ACGTNacgtn")}

    def _one(self, text):
        return [self.later.get(c, 1) + (50 if i == 0 else 0) for i, c in enumerate(text)]

    def __call__(self, texts, add_special_tokens=False, **kw):
        return {"input_ids": [self._one(t) for t in ([texts] if isinstance(texts, str) else texts)]}


def _strings(rng, n, lo, hi, alphabet="ACGTN", p=(0.23, 0.23, 0.23, 0.23, 0.08)):
    return ["".join(rng.choice(list(alphabet), size=int(k), p=p)) for k in rng.integers(lo, hi, size=n)]


@pytest.mark.parametrize("make", [TwoTokensForN, SumOfLetters])
def test_window_table_discovery_cpu(make):
    tok = make()
    spec = tables.spec_from_tokenizer(tok)
    assert spec.kind == "kmer" and spec.k == tok.k and spec.kmer_table5 is not None and len(spec.kmer_table5) == 5 ** tok.k
    assert spec.kmer_tail_singles == isinstance(tok, SumOfLetters)
    rng = np.random.default_rng(1)
    for s in _strings(rng, 200, 0, 90):
        assert tables.expected_kmer_table_ids(s, spec) == tok(s)["input_ids"][0]


def test_start_table_discovery_cpu():
    spec = tables.spec_from_tokenizer(FirstLetterDiffers())
    assert spec.kind == "char" and spec.start_lut256 is not None
    assert spec.start_lut256[ord("A")] == 60 and spec.lut256[ord("A")] == 10 and spec.lut256[ord("x")] == 1


@pytest.mark.gpu
@pytest.mark.parametrize("make", [TwoTokensForN, SumOfLetters])
@pytest.mark.parametrize("ids_dtype", ["int64", "int32"])
def test_window_table_tokenizers_on_gpu(make, ids_dtype):
    from dnatok_b200.tokenizer import B200Tokenizer
    live = make()
    tok = B200Tokenizer.from_hf(live)
    rng = np.random.default_rng(7)
    strs = _strings(rng, 300, 0, 400) + ["", "N" * 50, "ACG" * 200 + "NN", "A" * live.k, "A" * (live.k - 1), "ACGTN" * 333]
    want = [live(s)["input_ids"][0] for s in strs]
    from dnatok_b200.pack import pack_strings
    flat, offs = pack_strings(strs)
    d_b = torch.from_numpy(flat.copy()).cuda() if flat.size else torch.empty(0, dtype=torch.uint8, device="cuda")
    d_o = torch.from_numpy(offs).cuda()
    dt = getattr(torch, ids_dtype)
    # ragged
    enc = tok.encode_device(d_b, d_o, host_offsets=offs, padding=False, add_special_tokens=False, ids_dtype=dt)
    ids, oo = enc["input_ids"].cpu().numpy(), enc["offsets"].cpu().numpy()
    for i, w in enumerate(want):
        assert ids[oo[i]:oo[i + 1]].tolist() == w, "row %d %r" % (i, strs[i][:40])
    # padded to the longest, both sides, with mask
    for side in ("right", "left"):
        tok.padding_side = side
        enc = tok.encode_device(d_b, d_o, host_offsets=offs, padding="longest", add_special_tokens=False, ids_dtype=dt)
        ids, mask = enc["input_ids"].cpu().numpy(), enc["attention_mask"].cpu().numpy()
        width = max(len(w) for w in want)
        assert ids.shape == (len(strs), width)
        for i, w in enumerate(want):
            row = ([0] * (width - len(w)) + w) if side == "left" else (w + [0] * (width - len(w)))
            m = ([0] * (width - len(w)) + [1] * len(w)) if side == "left" else ([1] * len(w) + [0] * (width - len(w)))
            assert ids[i].tolist() == row and mask[i].tolist() == m, (side, i)
    # truncation to 20 tokens
    tok.padding_side = "right"
    enc = tok.encode_device(d_b, d_o, host_offsets=offs, padding="max_length", max_length=20, truncation=True,
                            add_special_tokens=False, ids_dtype=dt)
    ids = enc["input_ids"].cpu().numpy()
    for i, w in enumerate(want):
        assert ids[i].tolist() == (w[:20] + [0] * max(0, 20 - len(w)))
    # the HF call surface
    got = tok(strs[:50], add_special_tokens=False)["input_ids"]
    assert [list(g) for g in got] == want[:50]


@pytest.mark.gpu
def test_start_table_tokenizer_on_gpu():
    from dnatok_b200.tokenizer import B200Tokenizer
    live = FirstLetterDiffers()
    tok = B200Tokenizer.from_hf(live)
    rng = np.random.default_rng(9)
    strs = _strings(rng, 200, 0, 700, alphabet="ACGTNacx", p=(0.2, 0.2, 0.2, 0.2, 0.05, 0.05, 0.05, 0.05)) + ["", "A", "xA", "N" * 4097]
    want = [live(s)["input_ids"][0] for s in strs]
    got = tok(strs, add_special_tokens=False)["input_ids"]
    assert [list(g) for g in got] == want
    for side in ("right", "left"):
        tok.padding_side = side
        enc = tok(strs, padding=True, add_special_tokens=False, return_tensors="np")
        width = max(len(w) for w in want)
        for i, w in enumerate(want):
            row = ([0] * (width - len(w)) + w) if side == "left" else (w + [0] * (width - len(w)))
            assert enc["input_ids"][i].tolist() == row, (side, i)
    tok.padding_side = "right"
    enc = tok(strs, padding="max_length", max_length=33, truncation=True, add_special_tokens=False, return_tensors="np")
    for i, w in enumerate(want):
        assert enc["input_ids"][i].tolist() == w[:33] + [0] * max(0, 33 - len(w))


def _windows_spec(k, seed, runs):
    """A synthetic tokenizer given window by window: clean windows one id each, the others `runs` ids at most (no more than
    k: a row never has more tokens than bytes)."""
    import itertools
    from dnatok_b200.tables import Specials, TokenizerSpec
    rng = np.random.default_rng(seed)
    lut = np.full(256, 1, np.int32)
    for i, c in enumerate("ACGTN"):
        lut[ord(c)] = 5 + i
    table, offsets, ids = [], [0], []
    for win in itertools.product("ACGTN", repeat=k):
        if "N" not in win or runs == 1:
            table.append(int(rng.integers(10, 5000)))
        else:
            table.append(-len(offsets))
            ids += rng.integers(5000, 9000, size=int(rng.integers(1, runs + 1))).tolist()
            offsets.append(len(ids))
    return TokenizerSpec("kmer", Specials(0, 1, 2, 3), 9000, lut, k=k, kmer_table5=np.array(table, np.int32),
                         kmer_run_offsets=np.array(offsets, np.int32), kmer_run_ids=np.array(ids, np.int32))


@pytest.mark.gpu
@pytest.mark.parametrize("k,runs", [(1, 1), (2, 1), (2, 2), (3, 3), (4, 2), (5, 5), (6, 6), (7, 2), (8, 8)])
@pytest.mark.parametrize("tail", [True, False])
def test_clean_window_tables_in_the_row_encoder(k, runs, tail):
    """Rows around the chunks of 64 and 256 windows and the 16-byte chunks of the sizing pass, an odd start of the buffer,
    windows with Ns at every place, truncation inside a run."""
    from dnatok_b200.tokenizer import B200Tokenizer
    spec = _windows_spec(k, 3 * k + runs, runs)
    spec.kmer_tail_singles = tail
    tok = B200Tokenizer(spec)
    rng = np.random.default_rng(k)
    lens = [0, 1, k - 1, k, k + 1, 15, 16, 17, 63 * k, 64 * k, 64 * k + 1, 65 * k - 1, 256 * k, 257 * k + 1, 512 * k, 2049 * k + k - 1]
    lens += rng.integers(0, 700 * k, size=40).tolist()
    strs = []
    for i, n in enumerate(lens):
        x = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, size=n)].copy()
        x[rng.random(n) < (0.0, 0.002, 0.2)[i % 3]] = ord("N")
        if n > 40 and i % 4 == 0:
            x[n // 3:n // 3 + 30] = ord("x")
        strs.append(x.tobytes().decode())
    want = [tables.expected_kmer_table_ids(s, spec) for s in strs]
    data = "".join(strs).encode()
    offs = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    d_b = torch.zeros(len(data) + 3, dtype=torch.uint8, device="cuda")[3:]
    d_b.copy_(torch.from_numpy(np.frombuffer(data, np.uint8).copy()))
    d_o = torch.from_numpy(offs).cuda()
    enc = tok.encode_device(d_b, d_o, host_offsets=offs, padding=False, add_special_tokens=False, ids_dtype=torch.int32)
    ids, oo = enc["input_ids"].cpu().numpy(), enc["offsets"].cpu().numpy()
    for i, w in enumerate(want):
        assert ids[oo[i]:oo[i + 1]].tolist() == w, "row %d (%d bytes)" % (i, lens[i])
    for side in ("right", "left"):
        tok.padding_side = side
        for kw, cut in ((dict(padding="longest"), None), (dict(padding="max_length", max_length=131, truncation=True), 129)):
            enc = tok.encode_device(d_b, d_o, host_offsets=offs, add_special_tokens=True, **kw)
            got, mask = enc["input_ids"].cpu().numpy(), enc["attention_mask"].cpu().numpy()
            for i, w in enumerate(want):
                row = [2] + w[:cut] + [3]
                pad = [0] * (got.shape[1] - len(row))
                assert got[i].tolist() == (pad + row if side == "left" else row + pad), (side, kw, i)
                assert mask[i].sum() == len(row) and enc["lengths"][i].item() == len(row)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["kmer6", "table"])
def test_sizing_of_a_row_whose_device_offsets_decrease(kind):
    """The host offsets are right, the device's step back: such a row is empty, whatever its (negative) length modulo k."""
    import helpers as H
    from dnatok_b200.tokenizer import B200Tokenizer
    rng = np.random.default_rng(31)
    lens = rng.integers(40, 90, size=1301)
    offs = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    flat = np.frombuffer(b"ACGTN", np.uint8)[rng.choice(5, size=int(offs[-1]), p=[.24, .24, .24, .24, .04])]
    bad = offs.copy()
    at = np.arange(3, 1290, 29)
    bad[at + 1] = bad[at] - np.arange(len(at)) % 14
    spec = H.spec("kmer6") if kind == "kmer6" else _windows_spec(5, 19, 3)
    tok = B200Tokenizer(spec)
    tok.padding_side = "left"
    texts = [flat[bad[i]:bad[i + 1]].tobytes().decode() if bad[i + 1] > bad[i] else "" for i in range(len(lens))]
    if kind == "kmer6":
        o2 = np.concatenate([[0], np.cumsum([len(t) for t in texts])]).astype(np.int64)
        want = [w.tolist() for w in H.oracle_rows("kmer6", np.frombuffer("".join(texts).encode(), np.uint8), o2)]
    else:
        want = [tables.expected_kmer_table_ids(t, spec) for t in texts]
    enc = tok.encode_device(torch.from_numpy(flat.copy()).cuda(), torch.from_numpy(bad).cuda(), host_offsets=offs, padding="longest",
                            add_special_tokens=True)
    got, n = enc["input_ids"].cpu().numpy(), enc["lengths"].cpu().numpy()
    sp = spec.specials
    for i, w in enumerate(want):
        row = ([sp.cls_id] if sp.cls_id >= 0 else []) + w + ([sp.sep_id] if sp.sep_id >= 0 else [])
        assert n[i] == len(row), i
        assert got[i].tolist() == [sp.pad_id] * (got.shape[1] - len(row)) + row, i
