"""BPE words beyond 32,768 bytes, merged in overlapping windows: lengths around the places where a word gets one window
more, repeats that leave a border without a common token (mended, or left to the general kernel), every output layout."""
import numpy as np
import pytest

import helpers as H
from dnatok_b200 import _cabi, synth
from dnatok_b200.tokenizer import B200Tokenizer

pytestmark = pytest.mark.gpu

WIN, OVERLAP = 1024, 128
STEP = WIN - OVERLAP


def words():
    edge = OVERLAP + 37 * STEP                    # exactly 37 windows, the last one full
    lens = [edge, edge + 1, edge + STEP - 1, edge + STEP, 32769, 65536]
    out = [bytes(synth.config3(batch=1, length=n, seed=n)[0]) for n in lens]
    w = bytearray(synth.config3(batch=1, length=40000, seed=5)[0])
    w[STEP - 300:STEP + 500] = b"A" * 800         # a repeat across the first border
    out.append(bytes(w))
    w = bytearray(synth.config3(batch=1, length=40000, seed=6)[0])
    w[2 * STEP:2 * STEP + OVERLAP] = b"N" * OVERLAP   # an overlap of single-letter tokens
    w[-1] = ord("x")                              # a byte outside the alphabet
    out.append(bytes(w))
    return out + [b"AC" * 20001, b"", b"ACGTTGCA" * 3, bytes(synth.config3(batch=1, length=5000, seed=7)[0])]


@pytest.fixture(params=["auto", "one_warp", "table_in_global"])
def mode(request):
    L = _cabi.lib()
    opts = {"auto": [], "one_warp": [("bpe_team_warps", 1, 0)], "table_in_global": [("bpe_smem_table", 0, 1)]}[request.param]
    for name, value, _ in opts:
        _cabi.check(L.dnatok_set_option(name.encode(), value))
    yield request.param
    for name, _, back in opts:
        _cabi.check(L.dnatok_set_option(name.encode(), back))


@pytest.mark.parametrize("name", ["bpe4096", "bpe32000"])
def test_window_borders_ragged(name, mode):
    import torch
    flat, offs = H.pack_strs(words())
    tok = B200Tokenizer(H.spec(name))
    want = H.oracle_rows(name, flat, offs)
    for hint in (offs, None):
        enc = tok.encode_device(torch.from_numpy(flat).cuda(), torch.from_numpy(offs).cuda(), host_offsets=hint, padding=False,
                                add_special_tokens=False)
        ids, oo = enc["input_ids"].cpu().numpy(), enc["offsets"].cpu().numpy()
        for i in range(len(offs) - 1):
            assert np.array_equal(ids[oo[i]:oo[i + 1]], want[i]), "word %d (%d bytes)" % (i, offs[i + 1] - offs[i])


@pytest.mark.parametrize("left", [False, True])
@pytest.mark.parametrize("width", [700, 9000, 40000])     # cut in the first window, cut in the middle, wide enough
def test_window_borders_padded(left, width):
    import torch
    flat, offs = H.pack_strs(words())
    tok = B200Tokenizer(H.spec("bpe4096"))
    tok.padding_side = "left" if left else "right"
    want_ids, want_mask = H.oracle_batch("bpe4096", flat, offs, padding="max_length", max_length=width, truncation=True, pad_left=left)
    enc = tok.encode_device(torch.from_numpy(flat).cuda(), torch.from_numpy(offs).cuda(), host_offsets=offs, padding="max_length",
                            max_length=width, truncation=True)
    assert np.array_equal(enc["input_ids"].cpu().numpy(), want_ids)
    assert np.array_equal(enc["attention_mask"].cpu().numpy(), want_mask)


def left_words(tok, scratch, n_rows, total):
    """Words of the last encode that the windows left to the general kernel: a counter behind the merged tokens and the rows'
    counts, both padded to 256 bytes (bpe_scratch_layout)."""
    at = -(-(2 * total + 16) // 256) * 256 + -(-(4 * n_rows + 4) // 256) * 256
    import torch
    return int(scratch[at:at + 64].view(torch.int32)[8])


UNITS = [b"A", b"AC", b"ACG", b"AAC", b"TTAGGG", b"GATA", b"ACGTTGCAAC"]


def repeat_words(seed, lengths, per_word):
    """Words of 40,000 to 70,000 bp with tandem repeats of the given lengths at odd places, some of them side by side."""
    rng = np.random.default_rng(seed)
    out = []
    for i, n in enumerate(lengths):
        w = bytearray(synth.config3(batch=1, length=40000 + int(rng.integers(0, 30000)), seed=seed + i)[0])
        for k in range(per_word):
            unit = UNITS[int(rng.integers(len(UNITS)))]
            at = int(rng.integers(0, len(w) - n)) if k or i % 4 else (0 if i % 8 else len(w) - n)
            w[at:at + n] = (unit * (n // len(unit) + 1))[:n]
        out.append(bytes(w))
    return out


@pytest.mark.parametrize("name", ["bpe4096", "bpe32000"])
@pytest.mark.parametrize("lengths,per_word,most_left", [([129, 140, 200, 255, 300, 500, 700, 900] * 2, 6, 0), ([1000, 1100, 1792, 2000, 2816, 3000] * 2, 3, 0),
                                                        ([5000, 9000, 11648, 20000], 1, 0), ([31000, 33000, 40000], 1, 3)])
def test_repeats_across_borders(name, lengths, per_word, most_left):
    """Repeats longer than the overlap, taken up out of phase by the windows of either side: the border is mended, and only
    repeats that no piece spans leave the word to the general kernel."""
    import torch
    from dnatok_b200 import _cabi as C
    flat, offs = H.pack_strs(repeat_words(300 + len(lengths), lengths, per_word))
    tok = B200Tokenizer(H.spec(name))
    want = H.oracle_rows(name, flat, offs)
    B, total = len(offs) - 1, int(offs[-1])
    d_b, d_o = torch.from_numpy(flat).cuda(), torch.from_numpy(offs).cuda()
    C.check(C.lib().dnatok_set_row_bytes_hint(tok.handle.ptr, int(np.diff(offs).min()), int(np.diff(offs).max())))
    scratch = torch.empty(C.lib().dnatok_scratch_bytes(tok.handle.ptr, B, total), dtype=torch.uint8, device="cuda")
    enc = tok.encode_device(d_b, d_o, host_offsets=offs, padding=False, add_special_tokens=False, scratch=scratch)
    ids, oo = enc["input_ids"].cpu().numpy(), enc["offsets"].cpu().numpy()
    for i in range(B):
        assert np.array_equal(ids[oo[i]:oo[i + 1]], want[i]), "word %d (%d bytes)" % (i, offs[i + 1] - offs[i])
    assert left_words(tok, scratch, B, total) <= most_left
    for left, width in ((False, 9000), (True, 30000)):
        tok.padding_side = "left" if left else "right"
        want_ids, want_mask = H.oracle_batch(name, flat, offs, padding="max_length", max_length=width, truncation=True, pad_left=left)
        enc = tok.encode_device(d_b, d_o, host_offsets=offs, padding="max_length", max_length=width, truncation=True)
        assert np.array_equal(enc["input_ids"].cpu().numpy(), want_ids)
        assert np.array_equal(enc["attention_mask"].cpu().numpy(), want_mask)
