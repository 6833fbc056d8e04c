"""Output stages of the one-token-per-element paths against the checker: ragged output around the spans a warp takes, and
short padded rows around the places where a vector crosses rows; unaligned sources and outputs."""
import ctypes

import numpy as np
import pytest

import helpers as H
from dnatok_b200 import _cabi
from dnatok_b200.tokenizer import B200Tokenizer

pytestmark = pytest.mark.gpu

SPAN = 1024


def batch(lens, seed):
    rng = np.random.default_rng(seed)
    offs = np.zeros(len(lens) + 1, dtype=np.int64)
    np.cumsum(lens, out=offs[1:])
    return np.frombuffer(b"ACGTN", dtype=np.uint8)[rng.integers(0, 5, size=int(offs[-1]))], offs


def encode(tok, flat, offs, *, shift, special, bits, stride=0, mask_bits=0, max_tokens=0, left=False):
    """dnatok_encode with the bytes at an odd address and the ids one element past a 16-byte boundary."""
    import torch
    L = _cabi.lib()
    B, total = len(offs) - 1, len(flat)
    buf = torch.zeros(total + 8, dtype=torch.uint8, device="cuda")
    buf[shift:shift + total] = torch.from_numpy(flat).cuda()
    d_off = torch.from_numpy(offs).cuda()
    fmt = _cabi.Format(bits, mask_bits, int(special), int(left), max_tokens, stride)
    n = B * stride if stride else int(L.dnatok_max_tokens(tok.handle.ptr, B, total, ctypes.byref(fmt)))
    ids = torch.full((n + 4,), -7, dtype={32: torch.int32, 64: torch.int64}[bits], device="cuda")
    one = shift % 2
    mask = torch.full((n + 4,), 9, dtype={0: torch.uint8, 8: torch.uint8, 32: torch.int32, 64: torch.int64}[mask_bits], device="cuda")
    lengths, status = (torch.full((max(B, 1),), -1, dtype=torch.int32, device="cuda") for _ in range(2))
    out_off = torch.zeros(B + 1, dtype=torch.int64, device="cuda")
    need = L.dnatok_scratch_bytes(tok.handle.ptr, B, total)
    scratch = torch.empty(max(need, 1), dtype=torch.uint8, device="cuda")
    p = lambda t, k=0: ctypes.c_void_p(t.data_ptr() + k * t.element_size())
    _cabi.check(L.dnatok_encode(tok.handle.ptr, p(buf, shift), p(d_off), B, total, ctypes.byref(fmt), p(ids, one),
                                p(mask, one) if mask_bits else None, p(lengths), p(out_off), p(status), p(scratch), need, None))
    torch.cuda.synchronize()
    got, m = ids.cpu().numpy(), mask.cpu().numpy()
    assert np.all(got[:one] == -7) and np.all(got[n + one:] == -7)       # nothing beside the output is touched
    return got[one:n + one], m[one:n + one], lengths.cpu().numpy()[:B], out_off.cpu().numpy(), status.cpu().numpy()[:B]


LENS = {
    "empty_rows": [0] * 70 + [1] + [0] * 40 + [5, 0, 0, 3000] + [0] * 33 + [2],
    "span_edges": [SPAN - 1, 1, SPAN, SPAN + 1, 2 * SPAN - 3, 2, 15, 16, 17, 4 * SPAN],
    "short_rows": list(range(0, 40)) * 60,
    "one_long": [100003],
}


@pytest.mark.parametrize("name", ["char", "byte", "bpe4096"])
@pytest.mark.parametrize("rows", sorted(LENS))
@pytest.mark.parametrize("special,bits,shift", [(True, 64, 0), (False, 32, 1), (True, 32, 6), (False, 64, 3)])
def test_ragged(name, rows, special, bits, shift):
    flat, offs = batch(LENS[rows], 3)
    tok = B200Tokenizer(H.spec(name))
    got, _, lengths, oo, status = encode(tok, flat, offs, shift=shift, special=special, bits=bits)
    sp = tok.spec.specials
    head, tail = ([sp.cls_id] if special and sp.cls_id >= 0 else []), ([sp.sep_id] if special and sp.sep_id >= 0 else [])
    want = [np.concatenate([head, w, tail]).astype(np.int64) for w in H.oracle_rows(name, flat, offs)]
    assert np.array_equal(np.diff(oo), [len(w) for w in want]) and np.array_equal(lengths, np.diff(oo)) and not status.any()
    assert np.array_equal(got[:oo[-1]], np.concatenate(want))


@pytest.mark.parametrize("name", ["char", "byte", "bpe4096"])
@pytest.mark.parametrize("left", [False, True])
@pytest.mark.parametrize("stride,bits,mask_bits,shift", [(2, 32, 8, 0), (3, 64, 64, 1), (17, 32, 8, 3), (31, 64, 32, 2), (128, 64, 8, 0),
                                                         (320, 32, 64, 5)])
@pytest.mark.parametrize("many", [False, True])
def test_short_padded_rows(name, left, stride, bits, mask_bits, shift, many):
    lens = (list(range(0, 45)) + [300, 0, 5000]) * (300 if many else 3)
    if many and stride < 31:
        lens = lens * 4
    flat, offs = batch(lens, 5)
    tok = B200Tokenizer(H.spec(name))
    got, mask, lengths, _, status = encode(tok, flat, offs, shift=shift, special=True, bits=bits, stride=stride, mask_bits=mask_bits,
                                           max_tokens=stride, left=left)
    ids_t, mask_t = {32: np.int32, 64: np.int64}[bits], {8: np.uint8, 32: np.int32, 64: np.int64}[mask_bits]
    want_ids, want_mask = H.oracle_batch(name, flat, offs, padding="max_length", max_length=stride, truncation=True, pad_left=left,
                                         id_dtype=ids_t, mask_dtype=mask_t)
    assert np.array_equal(got.reshape(-1, stride), want_ids)
    assert np.array_equal(mask.reshape(-1, stride), want_mask)
    assert np.array_equal(lengths, want_mask.sum(1)) and not status.any()


@pytest.mark.parametrize("name", ["char", "byte"])
@pytest.mark.parametrize("left", [False, True])
@pytest.mark.parametrize("bits,stride", [(32, 17), (64, 40)])
def test_short_rows_read_the_stated_buffer_only(name, left, bits, stride):
    """Rows that end behind total_bytes (the letters there belong to the same allocation, but not to the call) read zeros from
    there on, and a row whose offsets decrease is empty: as the span kernel has it for long rows."""
    import torch
    L = _cabi.lib()
    flat, offs = batch([23, 5, 0, 31, 12, 3, 40, 9] * 30, 8)
    total = int(offs[-1]) - 30
    bad = offs.copy()
    bad[50] = bad[49] - 4
    seen = flat.copy()
    seen[total:] = 0
    texts = [seen[bad[i]:bad[i + 1]] if bad[i + 1] > bad[i] else seen[:0] for i in range(len(bad) - 1)]
    lens = np.array([len(t) for t in texts])
    want_ids, want_mask = H.oracle_batch(name, np.concatenate(texts), np.concatenate([[0], np.cumsum(lens)]).astype(np.int64),
                                         padding="max_length", max_length=stride, truncation=True, pad_left=left,
                                         id_dtype={32: np.int32, 64: np.int64}[bits], mask_dtype=np.uint8)
    tok = B200Tokenizer(H.spec(name))
    B = len(texts)
    buf = torch.zeros(len(flat) + 4096, dtype=torch.uint8, device="cuda")
    buf[:len(flat)] = torch.from_numpy(flat).cuda()
    d_off = torch.from_numpy(bad).cuda()
    ids = torch.full((B, stride), -7, dtype={32: torch.int32, 64: torch.int64}[bits], device="cuda")
    mask = torch.full((B, stride), 9, dtype=torch.uint8, device="cuda")
    lengths, status = (torch.full((B,), -1, dtype=torch.int32, device="cuda") for _ in range(2))
    fmt = _cabi.Format(bits, 8, 1, int(left), stride, stride)
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    _cabi.check(L.dnatok_encode(tok.handle.ptr, p(buf), p(d_off), B, total, ctypes.byref(fmt), p(ids), p(mask), p(lengths), None, p(status),
                                None, 0, None))
    torch.cuda.synchronize()
    assert np.array_equal(ids.cpu().numpy(), want_ids)
    assert np.array_equal(mask.cpu().numpy(), want_mask)
    assert np.array_equal(lengths.cpu().numpy(), want_mask.sum(1)) and not status.any()
