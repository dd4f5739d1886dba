"""The sort that takes one launch, and the first sizes beyond it, against a
stable sort."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from oncolytica_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["random", "equal", "descending", "values"])
@pytest.mark.parametrize("bits", [1, 8, 9, 17, 32])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 8191, 8193, 10007, 65535, 65536, 65537])
def test_small_sort_is_the_stable_sort(cuda, olc, n, bits, kind):
    import torch

    rng = np.random.default_rng(n + bits)
    k = rng.integers(0, 1 << bits, n, dtype=np.uint64).astype(np.uint32)
    if kind == "equal":
        k[:] = k[0]
    if kind == "descending":
        k = np.sort(k)[::-1].copy()
    v = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32) if kind == "values" else None
    order = np.argsort(k, kind="stable")
    dev = lambda a: torch.from_numpy(a.view(np.int32).copy()).to(cuda)  # noqa: E731
    kin, kout, vout = dev(k), dev(np.zeros_like(k)), dev(np.zeros_like(k))
    vin = dev(v) if v is not None else None
    nbytes = olc.olc_sort_scratch_bytes(n, bits)
    scratch = torch.full((nbytes,), 255, dtype=torch.uint8, device=cuda)
    ptr = lambda t: C.c_void_p(t.data_ptr()) if t is not None else None  # noqa: E731
    _lib.check(olc.olc_stage_sort_pairs(ptr(kin), ptr(vin), ptr(kout), ptr(vout), n, bits, ptr(scratch), nbytes, None))
    torch.cuda.synchronize()
    np.testing.assert_array_equal(kout.cpu().numpy().view(np.uint32), k[order])
    np.testing.assert_array_equal(vout.cpu().numpy().view(np.uint32), v[order] if v is not None else order)
    np.testing.assert_array_equal(kin.cpu().numpy().view(np.uint32), k)
    at = olc.olc_sort_status_offset()
    assert scratch[at:at + 4].cpu().numpy().view(np.uint32)[0] == 0


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("bits", [7, 16, 17, 32])
@pytest.mark.parametrize("n", [65537, 65552, 139265])
def test_sort_by_passes_counts_every_key(cuda, olc, n, bits, offset):
    """Keys at and off a 16-byte boundary, with a last thread's share that is not
    full, in runs of equal digits and in none."""
    import torch

    rng = np.random.default_rng(n + bits)
    k = np.sort(rng.integers(0, 1 << bits, n, dtype=np.uint64).astype(np.uint32))
    moved = rng.random(n) < 0.2
    k[moved] = rng.integers(0, 1 << bits, int(moved.sum()), dtype=np.uint64).astype(np.uint32)
    order = np.argsort(k, kind="stable")
    room = torch.zeros(n + 4, dtype=torch.int32, device=cuda)
    kin = room[offset:offset + n]
    kin.copy_(torch.from_numpy(k.view(np.int32).copy()))
    kout, vout = (torch.zeros(n, dtype=torch.int32, device=cuda) for _ in range(2))
    nbytes = olc.olc_sort_scratch_bytes(n, bits)
    scratch = torch.empty(nbytes, dtype=torch.uint8, device=cuda)
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    _lib.check(olc.olc_stage_sort_pairs(ptr(kin), None, ptr(kout), ptr(vout), n, bits, ptr(scratch), nbytes, None))
    torch.cuda.synchronize()
    np.testing.assert_array_equal(kout.cpu().numpy().view(np.uint32), k[order])
    np.testing.assert_array_equal(vout.cpu().numpy().view(np.uint32), order)


@pytest.mark.parametrize("n", [1, 16, 500, 4096])
def test_small_sort_among_other_work(cuda, olc, n):
    """One-pass sorts, back to back on several streams while other kernels hold the
    SMs: the cluster's CTAs start at different times, and none may write to another
    before it has started."""
    import torch

    rng = np.random.default_rng(n)
    k = rng.integers(0, 256, n, dtype=np.uint64).astype(np.uint32)
    order = np.argsort(k, kind="stable")
    kin = torch.from_numpy(k.view(np.int32).copy()).to(cuda)
    nbytes = olc.olc_sort_scratch_bytes(n, 8)
    streams = [torch.cuda.Stream() for _ in range(4)]
    runs = []
    noise = torch.zeros(1 << 24, device=cuda)
    torch.cuda.synchronize()
    for r in range(32):
        st = streams[r % 4]
        noise.add_(1.0)  # on the default stream, beside the sorts
        with torch.cuda.stream(st):
            out = [torch.full((n,), -1, dtype=torch.int32, device=cuda) for _ in range(2)]
            scratch = torch.empty(nbytes, dtype=torch.uint8, device=cuda)
            runs.append((out, scratch))
            _lib.check(olc.olc_stage_sort_pairs(C.c_void_p(kin.data_ptr()), None, C.c_void_p(out[0].data_ptr()),
                                                C.c_void_p(out[1].data_ptr()), n, 8, C.c_void_p(scratch.data_ptr()),
                                                nbytes, C.c_void_p(st.cuda_stream)))
    torch.cuda.synchronize()
    for out, _ in runs:
        np.testing.assert_array_equal(out[0].cpu().numpy().view(np.uint32), k[order])
        np.testing.assert_array_equal(out[1].cpu().numpy().view(np.uint32), order)


@pytest.mark.parametrize("offset", [0, 3])
@pytest.mark.parametrize("kind", ["equal", "runs", "random"])
@pytest.mark.parametrize("n", [65537, 262143, 262144, 262145, 262161])
def test_sorts_on_either_side_of_few_keys_per_thread(cuda, olc, n, kind, offset):
    """The counts with 4 and with 16 keys per thread, at and off a 16-byte boundary,
    where the last thread's share is not full."""
    import torch

    rng = np.random.default_rng(n)
    k = rng.integers(0, 1 << 30, n, dtype=np.uint64).astype(np.uint32)
    if kind == "equal":
        k[:] = k[0]
    if kind == "runs":
        k = np.sort(k)
    order = np.argsort(k, kind="stable")
    room = torch.zeros(n + 4, dtype=torch.int32, device=cuda)
    kin = room[offset:offset + n]
    kin.copy_(torch.from_numpy(k.view(np.int32).copy()))
    kout, vout = (torch.zeros(n, dtype=torch.int32, device=cuda) for _ in range(2))
    nbytes = olc.olc_sort_scratch_bytes(n, 30)
    scratch = torch.empty(nbytes, dtype=torch.uint8, device=cuda)
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    _lib.check(olc.olc_stage_sort_pairs(ptr(kin), None, ptr(kout), ptr(vout), n, 30, ptr(scratch), nbytes, None))
    torch.cuda.synchronize()
    np.testing.assert_array_equal(kout.cpu().numpy().view(np.uint32), k[order])
    np.testing.assert_array_equal(vout.cpu().numpy().view(np.uint32), order)
