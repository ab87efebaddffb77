"""The device page encoder (csrc/encode.cu) at the edges of its split: a page
is cut into parts of whole 1024-value mini-blocks, a warp a part, at most 128
parts a page; an RLE page keeps at most 4096 runs; the offsets of at most 4096
pages go through a pinned buffer.  Every page must be byte for byte the host
encoder's (pf_page_encode)."""
import numpy as np
import pytest
import torch

from pageflow_b200 import paged

pytestmark = pytest.mark.gpu


def _same(v, cuts):
    got, offs = paged.encode_pages_device(torch.from_numpy(v).cuda(), cuts)
    got = got.cpu().numpy()
    want = [paged.encode_page(v[a:b]) for a, b in zip(cuts[:-1], cuts[1:])]
    assert offs == list(np.concatenate([[0], np.cumsum([w.shape[0] for w in want])]))
    assert np.array_equal(got, np.concatenate(want))
    return {int(w[4]) for w in want}


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
@pytest.mark.parametrize("n", [1, 31, 33, 1023, 1024, 1025, 128 * 1024, 128 * 1024 + 1,
                               129 * 1024 + 7])
def test_page_lengths_at_the_edges_of_parts(n, dtype):
    rng = np.random.default_rng(n)
    for v in (rng.integers(-50, 1 << 20, n), np.cumsum(rng.integers(0, 9, n)),
              np.repeat(rng.integers(0, 1 << 30, n // 40 + 1), 40)[:n]):
        _same(v.astype(dtype), [0, n])
        _same(v.astype(dtype), [0, n // 3, n // 3, n])


@pytest.mark.parametrize("bits", [0, 1, 5, 8, 31, 32, 33, 48, 63, 64])
def test_every_field_width_class(bits):
    """A block's fields of 0 to 64 bits: whole, shared and split words."""
    rng = np.random.default_rng(bits)
    n = 3 * 1024 + 11
    v = rng.integers(0, 1 << 64, n, dtype=np.uint64) >> np.uint64(64 - bits) if bits else \
        np.zeros(n, np.uint64)
    v[::1024] = 0
    if bits:
        v[5::1024] = np.uint64((1 << bits) - 1)
    _same(v.view(np.int64) if bits == 64 else v.astype(np.int64), [0, n])
    _same(np.cumsum(v).view(np.int64), [0, n])


@pytest.mark.parametrize("runs", [1, 2, 1024, 1025, 4095, 4096, 4097])
def test_run_counts_at_the_rle_limit(runs):
    v = np.repeat((np.arange(runs) * 7919 % 100_003) << 30, 37).astype(np.int64)
    schemes = _same(v, [0, v.shape[0]])
    if runs >= 1024:   # fewer runs: a FOR page is the smaller one
        assert (3 in schemes) == (runs <= 4096)


def test_more_pages_than_the_pinned_buffer_holds():
    v = np.random.default_rng(3).integers(0, 1000, 4100 * 3 + 1).astype(np.int32)
    _same(v, list(range(0, 4100 * 3, 3)) + [v.shape[0]])
    _same(v[:4096 * 3], list(range(0, 4096 * 3 + 1, 3)))


def test_too_small_a_capacity_writes_nothing():
    import ctypes
    from pageflow_b200 import _native as N
    v = torch.arange(5000, dtype=torch.int64, device="cuda") * 977
    rows = N.arr(ctypes.c_int64, [0, 2500, 5000])
    out = torch.full((256,), 0xAB, dtype=torch.uint8, device="cuda")
    offs = (ctypes.c_int64 * 3)()
    ws = N.workspace(N.lib().pf_encode_pages_workspace(2), v.device)
    rc = N.lib().pf_encode_pages(v.data_ptr(), 8, rows, 2, out.data_ptr(), 256, offs,
                                 ws.data_ptr(), ws.numel(), N.stream_of(v.device))
    assert rc == N.PF_ENOSPACE
    assert int((out != 0xAB).sum()) == 0
