"""CPU suite: the device scratch the Python mirror hands to products and convolutions, with a library that only records. What the calls
queue on a stream hand on in that scratch must not be mixed with another thread's."""
import contextlib
import threading
import time

import pytest
import torch

from dlf_b200 import gblas as gb
from dlf_b200 import gdnn


class _Library:
    """Stands in for the C entries of a product that needs `need` bytes of scratch."""

    def __init__(self, need, seconds=0.0):
        self.need, self.seconds = need, seconds
        self.guard, self.inside, self.most, self.calls = threading.Lock(), {}, 0, []

    def dlf_b200_gemm_scratch_bytes(self, *args):
        return self.need

    def dlf_b200_gemm_workspace_bytes(self, *args):
        return 16

    def dlf_b200_conv2d_workspace_bytes(self, *args):
        return self.need

    def dlf_b200_gemm_ex(self, *args):
        ws, ws_bytes, stream = (getattr(a, "value", a) for a in args[-3:])
        with self.guard:
            self.inside[ws] = self.inside.get(ws, 0) + 1
            self.most = max(self.most, self.inside[ws])
            self.calls.append((ws, ws_bytes, stream))
        time.sleep(self.seconds)  # ctypes gives other threads their turn here
        with self.guard:
            self.inside[ws] -= 1
        return 0

    dlf_b200_conv2d_fused = dlf_b200_gemm_ex


class _Stream:
    def __init__(self, handle):
        self.cuda_stream = handle


class _Matrix:
    """A device operand, as far as the call looks at it."""
    dtype, device, is_cuda, address, offset = torch.float32, torch.device("cpu"), True, 4096, 0

    def numel(self):
        return 1 << 20


@pytest.fixture
def product(monkeypatch, built_lib):  # (a failed call asks the real library for its text)
    def install(**kw):
        library = _Library(**kw)
        monkeypatch.setattr(gb, "lib", lambda: library)
        monkeypatch.setattr(gdnn, "lib", lambda: library)
        monkeypatch.setattr(gdnn, "_ptr", lambda buf: buf.data_ptr())
        monkeypatch.setattr(gb, "_GEMM_WORKSPACES", {})
        monkeypatch.setattr(gdnn, "_WORKSPACES", {})
        monkeypatch.setattr(torch.cuda, "stream", lambda stream: contextlib.nullcontext())
        monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
        monkeypatch.setattr(torch.Tensor, "record_stream", lambda self, stream: None)
        return library

    return install


def _call(handle):
    gb._gemm(gb.Layout.RowMajor, gb.Transpose.NoTrans, gb.Transpose.NoTrans, 33, 35, 37, 1.0, _Matrix(), 37, _Matrix(), 35,
             0.0, _Matrix(), 35, queue=_Stream(handle))


def _convolve(handle):
    f = gdnn.Filter2D((1, 4, 3, 3), (4, 4, 1, 1))
    gdnn.conv2d_filter(torch.zeros(36), torch.zeros(16), torch.zeros(36), f, queue=_Stream(handle))


def _threads(*handles, call=_call):
    ts = [threading.Thread(target=lambda h=h: [call(h) for _ in range(5)]) for h in handles]
    for t in ts:
        t.start()
    for t in ts:
        t.join()


@pytest.mark.parametrize("call", [_call, _convolve], ids=["product", "convolution"])
def test_threads_on_one_stream_queue_one_after_the_other(product, call):
    library = product(need=1000, seconds=0.01)
    _threads(7, 7, 7, call=call)
    assert len(library.calls) == 15 and len({ws for ws, _, _ in library.calls}) == 1
    assert library.most == 1


def test_threads_on_their_own_streams_do_not_wait_for_each_other(product):
    library = product(need=1000, seconds=0.02)
    start = time.perf_counter()
    _threads(1, 2, 3, 4, 5, 6)
    assert time.perf_counter() - start < 6 * 5 * 0.02  # what they would take in turn
    assert len({ws for ws, _, _ in library.calls}) == 6 and library.most == 1


def test_a_call_that_fails_leaves_the_stream_usable(product):
    library = product(need=1000)
    library.dlf_b200_gemm_ex = lambda *args: -30
    with pytest.raises(gb.BLASError):
        _call(1)
    del library.dlf_b200_gemm_ex
    _call(1)


def test_a_callers_scratch_needs_no_lock_and_only_what_the_plain_product_uses(product):
    library = product(need=1000)
    own = torch.empty(64, dtype=torch.uint8)
    with gb.scratch(own):
        _call(1)
    assert library.calls == [(own.data_ptr(), 64, 1)] and not gb._GEMM_WORKSPACES
    with gb.scratch(torch.empty(8, dtype=torch.uint8)), pytest.raises(gb.BLASError):
        _call(1)


def test_scratch_for_copies_of_large_operands_is_not_kept(product):
    library = product(need=100 << 20)
    _call(1)
    assert library.calls[0][1] == 100 << 20
    assert all(e.buffer is None for e in gb._GEMM_WORKSPACES.values())
    library.need = 1000
    _call(1)
    assert [e.buffer.numel() for e in gb._GEMM_WORKSPACES.values()] == [1000]


@pytest.mark.parametrize("call,table", [(_call, lambda: gb._GEMM_WORKSPACES), (_convolve, lambda: gdnn._WORKSPACES)],
                         ids=["product", "convolution"])
def test_a_captured_call_neither_uses_nor_leaves_kept_scratch(product, monkeypatch, call, table):
    library = product(need=1000)
    call(1)
    kept = [e.buffer for e in table().values()]
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    library.need = 2000
    call(1)
    assert library.calls[0][0] == kept[0].data_ptr() and library.calls[1][0] != kept[0].data_ptr()
    assert [e.buffer for e in table().values()] == kept


def test_a_product_runs_without_scratch_where_the_device_has_no_room(product, monkeypatch):
    library = product(need=100 << 20)

    def full(*args, **kw):
        raise torch.OutOfMemoryError

    monkeypatch.setattr(torch, "empty", full)
    _call(1)
    assert library.calls == [(None, 0, 1)]
