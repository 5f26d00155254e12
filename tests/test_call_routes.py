"""Which C calls the Python entry points make, with which arguments, checked without a GPU.

Fake tensors (device, shape and strides, no memory) go through the real entry points and a stand-in library records the
calls, so rules about routes and flags are tested on the CPU, among them those whose breach would be a race on the device.
"""

import contextlib
import warnings

import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

from gaudi_kernels_b200 import _lib, block_fp8_gemm, fp8_codec, row_parallel, sharded


class _Recorder:
    """Stands for libbfp8.so: every function succeeds and is noted as (name, arguments)."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def call(*args):
            self.calls.append((name, args))
            return 0
        return call

    def named(self, name):
        return [args for n, args in self.calls if n == name]


def _raw_stream(index):
    if not isinstance(index, int):
        raise RuntimeError("a device index is required, as the real function does")
    return 7


@pytest.fixture
def lib(monkeypatch):
    rec = _Recorder()
    monkeypatch.setattr(_lib, "load", lambda: rec)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", _raw_stream)
    with warnings.catch_warnings(), FakeTensorMode():
        warnings.simplefilter("ignore")                      # a fake tensor's data pointer is 0, and warns about it
        yield rec


def _operands(m, k, n):
    groups = (k + 127) // 128
    a = torch.empty((m, k), dtype=torch.uint8, device="cuda:0")
    sa = torch.empty_strided((m, groups), (1, m), device="cuda:0")
    w = torch.empty((n, k), dtype=torch.uint8, device="cuda:0")
    ws = torch.empty(((n + 127) // 128, groups), device="cuda:0")
    return a, sa, w, ws


EX_SCHEDULE = 18                                             # position of `schedule` in bfp8_gemm_block128_ex


@pytest.mark.parametrize("m", [1, 64, 128, 129])
@pytest.mark.parametrize("k,schedule", [(1000, 0), (1003, 1), (1024, 0), (1008, 1)])
def test_a_padded_copy_of_the_weight_is_declared_fresh(lib, m, k, schedule):
    # K that is not a multiple of 16: the GEMM reads a copy which a kernel enqueued just before it writes; a weight declared
    # at rest is read before that kernel has ended, so the copy must never be taken for one
    a, sa, w, ws = _operands(m, k, 256)
    status = torch.empty(4, dtype=torch.int32, device="cuda:0")
    block_fp8_gemm.gemm_block_fp8(a, sa, w, ws, check=False, status=status, schedule=schedule)
    copied = len(lib.named("bfp8_repitch_codes"))
    assert copied == (1 if k % 16 else 0)
    (args,) = lib.named("bfp8_gemm_block128_ex")
    assert args[EX_SCHEDULE] == schedule | (_lib.SCHEDULE_FRESH_WEIGHT if copied else 0)


@pytest.mark.parametrize("k", [1000, 1024])
@pytest.mark.parametrize("native_half", [True, False])
def test_reference_declares_its_weight_fresh(lib, monkeypatch, k, native_half):
    # the weight is uploaded and re-encoded by the call itself
    monkeypatch.setattr(block_fp8_gemm, "_read_status", lambda buf: (0, 0))
    x = torch.empty((3, k), dtype=torch.bfloat16, device="cuda:0")
    w = torch.empty((256, k), dtype=torch.float8_e4m3fn, device="cuda:0")
    s = torch.empty((2, (k + 127) // 128), device="cuda:0")
    block_fp8_gemm.reference(x, w, s, native_half=native_half)
    (args,) = lib.named("bfp8_gemm_block128_ex")
    assert args[EX_SCHEDULE] == _lib.SCHEDULE_FRESH_WEIGHT


@pytest.mark.parametrize("m,schedule", [(1, 0), (128, 0), (129, 1), (300, 1)])
def test_column_slices_add_k_blocks_in_order(lib, m, schedule):
    # a narrow slice has few tiles, which the automatic schedule may sum in slices of K: other bits than the whole product
    a, sa, w, ws = _operands(m, 4096, 1024)
    sharded.gemm_sharded(a, sa, w[256:512], ws[2:4])
    (args,) = lib.named("bfp8_gemm_block128_ex")
    assert args[EX_SCHEDULE] == schedule


@pytest.mark.parametrize("words", [3, 4, 8])
def test_status_buffers_of_any_length(words):
    # a caller's own status buffer needs the three words that are read; what follows them does not matter
    buf = torch.full((words,), -1, dtype=torch.int32)
    buf[:3] = torch.tensor([-2, 1, _lib.STATUS_BAD_SCALE], dtype=torch.int32)
    assert fp8_codec._read_status(buf) == ((1 << 32) | 0xFFFFFFFE, _lib.STATUS_BAD_SCALE)
    assert not block_fp8_gemm.wait_timed_out(buf)
    buf[2] |= _lib.STATUS_WAIT_TIMEOUT
    assert block_fp8_gemm.wait_timed_out(buf)


class _Exchange:
    """The parts of a PeerExchange that gemm_k_sharded uses, for a device named without an index."""

    world, rank, nbytes, ptrs = 2, 0, 1 << 20, [0, 0]
    device = torch.device("cuda")

    def __init__(self, lib):
        self.lib = lib
        self.status = torch.empty(4, dtype=torch.int32, device="cuda:0")

    def barrier(self):
        pass


def test_row_parallel_gemm_on_a_device_without_an_index(lib, monkeypatch):
    # PeerExchange takes "cuda" for the current device; the decode bucket's workspace is kept per stream of that device
    monkeypatch.setattr(torch.cuda, "device", lambda dev: contextlib.nullcontext())
    monkeypatch.setattr(block_fp8_gemm, "_workspaces", {})
    monkeypatch.setattr(_Recorder, "bfp8_gemm_block128_workspace_bytes", lambda self, m, n, k: 1024, raising=False)
    a, sa, w, ws = _operands(8, 1024, 256)
    row_parallel.gemm_k_sharded(a, sa, w, ws, _Exchange(lib))
    assert len(lib.named("bfp8_gemm_block128_push")) == 1
    assert list(block_fp8_gemm._workspaces) == [(None, 7)]


@pytest.mark.parametrize("rows,schedule", [(3, 0), (200, 1)])
def test_reference_sharded_declares_its_weight_fresh(lib, monkeypatch, rows, schedule):
    class Enqueued(Exception):
        pass

    def all_reduce(*args, **kwargs):                         # the exchange of the status bits: every kernel is enqueued
        raise Enqueued

    monkeypatch.setattr(torch.cuda, "device", lambda dev: contextlib.nullcontext())
    monkeypatch.setattr(sharded.dist, "get_world_size", lambda group=None: 1)
    monkeypatch.setattr(sharded.dist, "all_gather_into_tensor", lambda *args, **kwargs: None)
    monkeypatch.setattr(sharded.dist, "all_reduce", all_reduce)
    x = torch.empty((rows, 1024), dtype=torch.bfloat16, device="cuda:0")
    w = torch.empty((256, 1024), dtype=torch.float8_e4m3fn, device="cuda:0")
    with pytest.raises(Enqueued):
        sharded.reference_sharded(x, w, torch.empty((2, 8), device="cuda:0"))
    (args,) = lib.named("bfp8_gemm_block128_ex")
    assert args[EX_SCHEDULE] == schedule | _lib.SCHEDULE_FRESH_WEIGHT
