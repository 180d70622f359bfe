"""Uploads of plan tables (mvd::upload_table) inside an allocation scope: the table that lands on the
device is the one that was passed, whatever becomes of its memory before the stream gets there."""
import ctypes

import pytest

from spim_registration_gb300 import native

pytestmark = pytest.mark.gpu


def test_scoped_upload_does_not_read_its_source_after_it_returns():
    """A page-locked source, so that the copy surely waits for the busy stream."""
    torch = pytest.importorskip("torch")
    lib = native.load()
    upload = lib._ZN3mvd12upload_tableEPvPKvm           # mvd::upload_table(void*, const void*, size_t)
    begin = lib._ZN3mvd10AllocScopeC1EP11CUstream_st    # mvd::AllocScope::AllocScope(cudaStream_t)
    end = lib._ZN3mvd10AllocScopeD1Ev                   # mvd::AllocScope::~AllocScope()
    upload.argtypes, upload.restype = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t], None
    begin.argtypes, begin.restype = [ctypes.c_void_p, ctypes.c_void_p], None
    end.argtypes, end.restype = [ctypes.c_void_p], None
    want = torch.arange(5000, dtype=torch.int32)
    src, dst = want.clone().pin_memory(), torch.zeros(5000, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    scope = ctypes.create_string_buffer(256)  # room for an AllocScope
    begin(scope, s.cuda_stream)
    try:
        with torch.cuda.stream(s):
            torch.cuda._sleep(20_000_000)
        upload(dst.data_ptr(), src.data_ptr(), 4 * 5000)
        src.fill_(-1)
    finally:
        end(scope)
    s.synchronize()
    assert torch.equal(dst.cpu(), want)
