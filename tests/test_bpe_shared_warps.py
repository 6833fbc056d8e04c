"""BPE rows that share a warp: batches of more short rows than one wave of warps holds, row lengths around the largest
that two, four or eight rows on a warp allow, taken as they come (all rows short) and binned by length."""
import numpy as np
import pytest

import helpers as H
from dnatok_b200 import _cabi, synth
from dnatok_b200.tokenizer import B200Tokenizer

pytestmark = pytest.mark.gpu


def batch(rows, lens, seed):
    """rows rows whose lengths are drawn from `lens`."""
    rng = np.random.default_rng(seed)
    n = rng.choice(np.asarray(lens), size=rows).astype(np.int64)
    offs = np.zeros(rows + 1, dtype=np.int64)
    np.cumsum(n, out=offs[1:])
    flat = synth.config3(batch=-(-int(offs[-1]) // 256) or 1, length=256, seed=seed).reshape(-1)[:int(offs[-1])].copy()
    flat[rng.random(flat.size) < 0.002] = ord("N")
    for r in rng.integers(0, rows, size=40):                    # homopolymers
        flat[offs[r]:offs[r + 1]] = ord("A")
    return flat, offs


CASES = [
    # rows, lengths: (one wave holds 4,736 warps)
    (4737, [0, 1, 255, 256]),            # two rows per warp as they come, an odd row left over
    (9475, [512, 511, 0]),               # two per warp, the longest that fit
    (9475, [1, 2, 31, 128, 256]),        # four per warp
    (19001, [0, 1, 4, 33, 127, 128]),    # eight per warp
    (20003, [20, 128, 129, 256, 257, 512, 513, 20, 20, 20, 20, 20, 20]),   # binned
    (15001, [60, 60, 60, 60, 60, 60, 1024, 0]),                            # binned, full rows among them
]


@pytest.mark.parametrize("smem", [1, 0])
@pytest.mark.parametrize("name", ["bpe4096", "bpe32000"])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_rows_sharing_a_warp(name, case, smem):
    import torch
    rows, lens = CASES[case]
    flat, offs = batch(rows, lens, 40 + case)
    tok = B200Tokenizer(H.spec(name))
    want = H.oracle_rows(name, flat, offs)
    d_b, d_o = torch.from_numpy(flat).cuda(), torch.from_numpy(offs).cuda()
    L = _cabi.lib()
    _cabi.check(L.dnatok_set_option(b"bpe_smem_table", smem))
    try:
        enc = tok.encode_device(d_b, d_o, host_offsets=offs, padding=False, add_special_tokens=False)
        ids, oo = enc["input_ids"].cpu().numpy(), enc["offsets"].cpu().numpy()
        assert np.array_equal(np.diff(oo), [len(w) for w in want])
        assert np.array_equal(ids, np.concatenate(want))
        tok.padding_side = "left" if case % 2 else "right"
        width = 40
        want_ids, want_mask = H.oracle_batch(name, flat, offs, padding="max_length", max_length=width, truncation=True,
                                             pad_left=bool(case % 2), id_dtype=np.int32, mask_dtype=np.uint8)
        enc = tok.encode_device(d_b, d_o, host_offsets=offs, padding="max_length", max_length=width, truncation=True,
                                ids_dtype=torch.int32, mask_dtype=torch.uint8)
        assert np.array_equal(enc["input_ids"].cpu().numpy(), want_ids)
        assert np.array_equal(enc["attention_mask"].cpu().numpy(), want_mask)
    finally:
        _cabi.check(L.dnatok_set_option(b"bpe_smem_table", 1))


@pytest.mark.parametrize("longest", [256, 300])
def test_a_row_longer_than_the_hint_is_flagged(longest):
    """Rows that share a warp, taken as they come, one of them longer than the bounds said."""
    import ctypes
    import torch
    flat, offs = batch(9475, [100, longest], 77)
    tok = B200Tokenizer(H.spec("bpe4096"))
    L = _cabi.lib()
    B, total = len(offs) - 1, int(offs[-1])
    lens = np.diff(offs)
    _cabi.check(L.dnatok_set_row_bytes_hint(tok.handle.ptr, 1, 255))
    d_b, d_o = torch.from_numpy(flat).cuda(), torch.from_numpy(offs).cuda()
    fmt = tok._format(id_bits=32, mask_bits=0, add_special=False, max_tokens=0, out_stride=256)
    ids = torch.zeros((B, 256), dtype=torch.int32, device="cuda")
    lengths, status = (torch.full((B,), -1, dtype=torch.int32, device="cuda") for _ in range(2))
    scratch = torch.empty(L.dnatok_scratch_bytes(tok.handle.ptr, B, total), dtype=torch.uint8, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    _cabi.check(L.dnatok_encode(tok.handle.ptr, p(d_b), p(d_o), B, total, ctypes.byref(fmt), p(ids), None, p(lengths), None, p(status),
                                p(scratch), scratch.numel(), None))
    torch.cuda.synchronize()
    # 256-byte rows still fit what the launch was sized for; longer ones are reported and left empty
    over = lens > 256
    st, ln, out = status.cpu().numpy(), lengths.cpu().numpy(), ids.cpu().numpy()
    assert np.array_equal(st, np.where(over, _cabi.ROW_OUTSIDE_HINT, 0))
    want = H.oracle_rows("bpe4096", flat, offs)
    assert np.array_equal(ln, [0 if over[i] else len(want[i]) for i in range(B)])
    for i in range(0, B, 97):
        assert out[i, :ln[i]].tolist() == ([] if over[i] else want[i].tolist())


@pytest.mark.parametrize("rows,lens", [(4737, [100, 250]), (9475, [30, 100]), (19001, [20, 50]), (20003, [20] * 12 + [400])])
def test_a_row_whose_device_offsets_decrease_comes_out_empty(rows, lens):
    """Two, four or eight rows per warp as they come, and binned: the host offsets are right, the device's step back."""
    import torch
    flat, offs = batch(rows, lens, 90 + rows)
    bad = offs.copy()
    at = np.arange(5, rows - 3, rows // 37)
    bad[at + 1] = bad[at] - 7                                  # row `at` ends before it begins, the next one starts there
    texts = [flat[bad[i]:bad[i + 1]] if bad[i + 1] > bad[i] else flat[:0] for i in range(rows)]
    offs2 = np.concatenate([[0], np.cumsum([len(t) for t in texts])]).astype(np.int64)
    want_ids, want_mask = H.oracle_batch("bpe4096", np.concatenate(texts), offs2, padding="max_length", max_length=60, truncation=True)
    tok = B200Tokenizer(H.spec("bpe4096"))
    enc = tok.encode_device(torch.from_numpy(flat).cuda(), torch.from_numpy(bad).cuda(), host_offsets=offs, padding="max_length",
                            max_length=60, truncation=True)
    assert np.array_equal(enc["input_ids"].cpu().numpy(), want_ids)
    assert np.array_equal(enc["attention_mask"].cpu().numpy(), want_mask)
