"""BPE words whose first round runs on the letters: lengths around the places where a lane owns four, 30, 31 or 32 of them,
bytes that are no letter at the lanes' borders, merge tables that must not take that route."""
import numpy as np
import pytest

import helpers as H
from dnatok_b200 import _cabi, synth
from dnatok_b200.tables import Specials, TokenizerSpec
from dnatok_b200.tokenizer import B200Tokenizer
from oracle import oracle

pytestmark = pytest.mark.gpu


def batch(lens, seed, aliens=b"Nnax-"):
    rng = np.random.default_rng(seed)
    offs = np.zeros(len(lens) + 1, dtype=np.int64)
    np.cumsum(lens, out=offs[1:])
    flat = synth.config3(batch=-(-int(offs[-1]) // 256), length=256, seed=seed).reshape(-1)[:int(offs[-1])].copy()
    for i, n in enumerate(lens):
        lane = max(1, -(-n // 32))                              # letters of a lane
        at = np.arange(0, n, lane)
        if i % 3 == 1 and n:
            flat[offs[i] + at] = ord("N")                       # the first letter of every lane
        if i % 3 == 2 and n:
            flat[offs[i] + np.minimum(at + lane - 1, n - 1)] = np.frombuffer(aliens, np.uint8)[rng.integers(0, len(aliens), size=len(at))]
        if i % 7 == 3:
            flat[offs[i]:offs[i + 1]] = ord("ACGT"[i % 4])
    return flat, offs


def check(tok, want, flat, offs):
    import torch
    enc = tok.encode_device(torch.from_numpy(flat).cuda(), torch.from_numpy(offs).cuda(), host_offsets=offs, padding=False,
                            add_special_tokens=False)
    assert np.array_equal(np.diff(enc["offsets"].cpu().numpy()), [len(w) for w in want])
    assert np.array_equal(enc["input_ids"].cpu().numpy(), np.concatenate(want))


LENS = sorted(set([1, 2, 31, 32, 33, 95, 96, 97, 98, 127, 128, 129] + list(range(925, 1025, 3)) + [991, 992, 993, 1023, 1024]))


@pytest.mark.parametrize("smem", [1, 0])
@pytest.mark.parametrize("name", ["bpe4096", "bpe32000"])
def test_lane_borders(name, smem):
    flat, offs = batch(LENS * 3, 9)
    L = _cabi.lib()
    _cabi.check(L.dnatok_set_option(b"bpe_smem_table", smem))
    _cabi.check(L.dnatok_set_option(b"bpe_team_warps", 1))
    try:
        check(B200Tokenizer(H.spec(name)), H.oracle_rows(name, flat, offs), flat, offs)
    finally:
        _cabi.check(L.dnatok_set_option(b"bpe_smem_table", 1))
        _cabi.check(L.dnatok_set_option(b"bpe_team_warps", 0))


@pytest.mark.parametrize("kind", ["few_pairs", "lower_case_as_upper", "other_byte_merges"])
def test_tables_off_the_beaten_track(kind):
    lut = np.full(256, 9, np.int32)
    for i, c in enumerate(b"ACGT"):
        lut[c] = i
    merges = {"few_pairs": [(0, 1, 10), (10, 2, 11), (3, 3, 12), (12, 12, 13)],
              "lower_case_as_upper": [(0, 0, 10), (1, 0, 11), (10, 11, 12), (2, 3, 13)],
              "other_byte_merges": [(0, 4, 10), (1, 2, 11), (4, 4, 12), (11, 10, 13), (3, 0, 14)]}[kind]
    if kind == "lower_case_as_upper":
        lut[ord("a")] = 0
    if kind == "other_byte_merges":
        lut[ord("N")] = 4
    a, b, o = (np.array(x, np.int32) for x in zip(*merges))
    spec = TokenizerSpec("bpe", Specials(0, 9), 20, lut, merge_a=a, merge_b=b, merge_out=o)
    flat, offs = batch(LENS, 4)
    ids, counts = oracle.encode_ragged("bpe", flat, offs, lut256=lut, k=0, kmer_ids=None, table=oracle.BpeTable(a, b, o), threads=4)
    L = _cabi.lib()
    _cabi.check(L.dnatok_set_option(b"bpe_team_warps", 1))
    try:
        check(B200Tokenizer(spec), oracle.rows(ids, offs, counts), flat, offs)
    finally:
        _cabi.check(L.dnatok_set_option(b"bpe_team_warps", 0))
