"""dnatok_row_summary and dnatok_offset_bounds: what encode_device waits for."""
import ctypes
import threading

import numpy as np
import pytest

import helpers as H
from dnatok_b200 import _cabi


@pytest.mark.parametrize("lens,want", [([], (0, 0)), ([5], (5, 5)), ([3, 0, 9, 4], (0, 9))])
def test_offset_bounds(lens, want):
    offs = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    lo, hi = ctypes.c_int64(-1), ctypes.c_int64(-1)
    _cabi.check(_cabi.lib().dnatok_offset_bounds(_cabi.np_ptr(offs), len(lens), ctypes.byref(lo), ctypes.byref(hi)))
    assert (lo.value, hi.value) == want


@pytest.mark.gpu
def test_row_summary_sizes_and_threads():
    """Around the rows of one block, every pointer left out in turn, and from several threads and streams at once."""
    import torch
    L = _cabi.lib()
    handle = _cabi.Handle(H.spec("char"))
    errors = []

    def work(seed):
        try:
            stream = torch.cuda.Stream()
            rng = np.random.default_rng(seed)
            for n in [0, 1, 255, 4095, 4096, 4097, 100003]:
                lens, st = rng.integers(0, 1 << 30, size=n).astype(np.int32), np.zeros(n, np.int32)
                st[rng.integers(0, n, size=3) if n else []] = [1, 4, 16] if n else []
                with torch.cuda.stream(stream):
                    d_l, d_s = torch.from_numpy(lens).cuda(), torch.from_numpy(st).cuda()
                    word = torch.tensor([seed * 1000003 + n], device="cuda")
                for a, b, w in [(1, 1, 1), (0, 1, 1), (1, 0, 1), (1, 1, 0)]:
                    out = (ctypes.c_int64 * 3)()
                    _cabi.check(L.dnatok_row_summary(handle.ptr, d_l.data_ptr() if a and n else None, d_s.data_ptr() if b and n else None, n,
                                                     word.data_ptr() if w else None, ctypes.addressof(out), stream.cuda_stream))
                    assert out[0] == (int(lens.max()) if a and n else 0)
                    assert out[1] == (int(np.bitwise_or.reduce(st)) if b and n else 0)
                    assert out[2] == (seed * 1000003 + n if w else 0)
        except Exception as e:                                  # a thread's assertion has to reach the test
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


@pytest.mark.gpu
@pytest.mark.parametrize("waiting", [1, 3, 12])
def test_a_waiting_call_holds_up_no_other(waiting):
    """While threads wait for a busy stream, a call on the same handle and another stream returns; twelve are more than the
    eight sets of words the handle starts with, and every one of them gets its own result."""
    import time
    import torch
    L = _cabi.lib()
    handle = _cabi.Handle(H.spec("char"))
    lens = [torch.tensor([3, 9 + k, 4], dtype=torch.int32, device="cuda") for k in range(waiting + 1)]
    torch.cuda.synchronize()

    def summary(stream, k, out):
        _cabi.check(L.dnatok_row_summary(handle.ptr, lens[k].data_ptr(), None, 3, None, ctypes.addressof(out), stream.cuda_stream))

    outs = [(ctypes.c_int64 * 3)() for _ in lens]
    free, busy = torch.cuda.Stream(), torch.cuda.Stream()
    summary(free, waiting, outs[-1])                            # tables and words are there
    assert outs[-1][0] == 9 + waiting
    outs[-1][0] = 0
    done = torch.cuda.Event()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(1 << 30)                              # about half a second
        done.record()
    threads = [threading.Thread(target=summary, args=(busy, k, outs[k])) for k in range(waiting)]
    for t in threads:
        t.start()
    time.sleep(0.1)
    summary(free, waiting, outs[-1])
    still_busy = not done.query()
    for t in threads:
        t.join()
    assert still_busy or waiting > 8                            # an allocation may wait for the GPU, and others then for it
    assert [o[0] for o in outs] == [9 + k for k in range(waiting + 1)]


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["byte", "kmer6"])
def test_empty_rows_padded_to_the_longest(name):
    """Rows without a column: the words are defined all the same (the memory they come from held others before)."""
    import torch
    from dnatok_b200.tokenizer import B200Tokenizer
    tok = B200Tokenizer(H.spec(name))
    offs = np.zeros(6, np.int64)
    d_b, d_o = torch.empty(0, dtype=torch.uint8, device="cuda"), torch.from_numpy(offs).cuda()
    poison = [torch.full((k,), 5, dtype=torch.int32, device="cuda") for k in (1, 5, 64, 128) for _ in range(8)]
    del poison
    for hint in (offs, None):
        enc = tok.encode_device(d_b, d_o, host_offsets=hint, padding="longest", add_special_tokens=False)
        assert tuple(enc["input_ids"].shape) == (5, 0) and enc["lengths"].tolist() == [0] * 5
    if name == "byte":
        poison = [torch.full((k,), 5, dtype=torch.int32, device="cuda") for k in (1, 5, 64, 128) for _ in range(8)]
        del poison
        emb = tok.embed_device(d_b, d_o, torch.zeros((512, 8), device="cuda"), host_offsets=offs, add_special_tokens=False)
        assert tuple(emb["embeddings"].shape) == (5, 0, 8) and emb["lengths"].tolist() == [0] * 5
