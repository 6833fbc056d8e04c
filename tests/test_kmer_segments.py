"""Ragged k-mer encodes of few or long rows: dnatok_encode hands the segments' places from its sizing pass to its encoder,
dnatok_prepare + dnatok_write settle them again by looking back."""
import copy
import ctypes

import numpy as np
import pytest

import helpers as H
from dnatok_b200 import _cabi
from dnatok_b200.tables import Specials
from dnatok_b200.tokenizer import B200Tokenizer

pytestmark = pytest.mark.gpu

SEG = 256 * 6                                                   # bytes of a segment of six-mers
LENS = {"edges": [0, 5, SEG - 1, SEG, SEG + 1, 2 * SEG, 9 * SEG + 3, 0, 17], "one": [70 * SEG + 5],
        "uneven": [100003] + [40] * 50 + [33 * SEG - 2, 256 * SEG], "many_segments": [300 * SEG, 257 * SEG + 1, 12]}


@pytest.mark.parametrize("lens", sorted(LENS))
@pytest.mark.parametrize("hint", ["none", "exact", "low"])      # low: rows beyond it finish in their last segment
@pytest.mark.parametrize("special,bits,cut", [(False, 32, 0), (True, 64, 0), (True, 32, 1000)])
def test_places_from_the_sizing_pass(lens, hint, special, bits, cut):
    import torch
    L = _cabi.lib()
    rng = np.random.default_rng(len(lens) + cut)
    offs = np.concatenate([[0], np.cumsum(LENS[lens])]).astype(np.int64)
    B, total = len(offs) - 1, int(offs[-1])
    flat = np.frombuffer(b"ACGTN", np.uint8)[rng.choice(5, size=total, p=[.249, .249, .249, .249, .004])]
    spec = copy.copy(H.spec("kmer6"))
    spec.specials = Specials(0, 1, 2, 3)
    tok = B200Tokenizer(spec)
    lo, hi = {"none": (0, 0), "exact": (0, max(LENS[lens])), "low": (0, 2 * SEG)}[hint]
    _cabi.check(L.dnatok_set_row_bytes_hint(tok.handle.ptr, lo, hi))
    fmt = _cabi.Format(bits, 0, int(special), 0, cut, 0)
    d_b, d_o = torch.from_numpy(flat.copy()).cuda(), torch.from_numpy(offs).cuda()
    n = int(L.dnatok_max_tokens(tok.handle.ptr, B, total, ctypes.byref(fmt)))
    need = L.dnatok_scratch_bytes(tok.handle.ptr, B, total)
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    sp = tok.spec.specials
    head, tail = ([x] if special and x >= 0 else [] for x in (sp.cls_id, sp.sep_id))
    keep = cut - len(head) - len(tail) if cut else None
    want = [np.concatenate([head, w[:keep], tail]).astype(np.int64) for w in H.oracle_rows("kmer6", flat, offs)]
    for call in ("encode", "prepare_write"):
        ids = torch.full((n + 1,), -7, dtype={32: torch.int32, 64: torch.int64}[bits], device="cuda")
        lengths, status = (torch.full((B,), -1, dtype=torch.int32, device="cuda") for _ in range(2))
        out_off = torch.zeros(B + 1, dtype=torch.int64, device="cuda")
        scratch = torch.full((need,), 255, dtype=torch.uint8, device="cuda")     # what a call before left there
        batch = (tok.handle.ptr, p(d_b), p(d_o), B, total, ctypes.byref(fmt))
        work = (p(status), p(scratch), need, None)
        if call == "encode":
            _cabi.check(L.dnatok_encode(*batch, p(ids), None, p(lengths), p(out_off), *work))
        else:
            _cabi.check(L.dnatok_prepare(*batch, p(lengths), *work))
            _cabi.check(L.dnatok_scan_lengths(p(lengths), B, p(out_off), None))
            _cabi.check(L.dnatok_write(*batch, p(lengths), p(out_off), p(ids), None, *work))
        torch.cuda.synchronize()
        oo = out_off.cpu().numpy()
        assert np.array_equal(np.diff(oo), [len(w) for w in want]) and not status.any(), call
        got = ids.cpu().numpy()
        assert np.array_equal(got[:oo[-1]], np.concatenate(want)) and np.all(got[n:] == -7), call
