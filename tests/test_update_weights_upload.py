"""A weight update whose map upload fails must not leave an unwritten map behind (CPU, on a fake CUDA runtime).

The library's objects are linked against a runtime whose device memory is host memory, whose kernels do nothing and whose
next host-to-device copy of a given size fails on request. A host-built handle uploads the stored index of every arc with
its first update; when that copy fails, the update must fail, and the next one must upload the map again before any
kernel looks at it.
"""

from __future__ import annotations

import ctypes as C
import glob
import os
import shutil
import subprocess

import numpy as np
import pytest

import neurograph_b200 as ngx
from neurograph_b200 import build

FAKE = r"""
#include <stddef.h>
#include <stdlib.h>
#include <string.h>
typedef int err;
static size_t fail_size = 0;      /* the next host-to-device copy of this size fails */
static int copies_of_size = 0;    /* host-to-device copies of the watched size that succeeded */
static size_t watched = 0;
void fake_fail_copy(size_t bytes) { fail_size = bytes; watched = bytes; copies_of_size = 0; }
void fake_watch_copy(size_t bytes) { watched = bytes; copies_of_size = 0; }
int fake_copies(void) { return copies_of_size; }
err cudaMalloc(void** p, size_t n) { *p = calloc(1, n ? n : 1); return *p ? 0 : 2; }
err cudaFree(void* p) { free(p); return 0; }
err cudaFreeAsync(void* p, void* s) { (void)s; free(p); return 0; }
err cudaHostAlloc(void** p, size_t n, unsigned f) { (void)f; return cudaMalloc(p, n); }
err cudaFreeHost(void* p) { free(p); return 0; }
err cudaHostGetDevicePointer(void** d, void* h, unsigned f) { (void)f; *d = h; return 0; }
err cudaMemcpy(void* d, const void* s, size_t n, int kind) { (void)kind; memcpy(d, s, n); return 0; }
err cudaMemcpyAsync(void* d, const void* s, size_t n, int kind, void* st) {
    (void)st;
    if (kind == 1 && n == fail_size) { fail_size = 0; return 1; }
    if (kind == 1 && n == watched) { ++copies_of_size; }
    memcpy(d, s, n);
    return 0;
}
err cudaMemsetAsync(void* d, int v, size_t n, void* st) { (void)st; memset(d, v, n); return 0; }
err cudaGetDeviceCount(int* n) { *n = 1; return 0; }
err cudaGetDevice(int* d) { *d = 0; return 0; }
err cudaDeviceGetAttribute(int* v, int attr, int dev) { (void)dev; *v = attr == 75 ? 10 : 148; return 0; }
err cudaStreamCreateWithFlags(void** s, unsigned f) { (void)f; *s = NULL; return 0; }
err cudaMemGetInfo(size_t* f, size_t* t) { *f = *t = (size_t)1 << 36; return 0; }
err cudaFuncGetAttributes(int* attr, const void* f) { (void)f; memset(attr, 0, 64); attr[6] = 1024; attr[8] = attr[9] = 100; return 0; }
const char* cudaGetErrorString(err e) { (void)e; return "fake error"; }
void** __cudaRegisterFatBinary(void* f) { static void* h; (void)f; return &h; }
"""
# the other runtime entry points the objects refer to: they report success and do nothing
STUB = "int %s() { return 0; }\n"


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    objects = sorted(glob.glob(os.path.join(build.LIB_DIR, "obj", "*.o")))
    if not build.up_to_date() or len(objects) != len(build.sources()) or shutil.which("gcc") is None or shutil.which("nm") is None:
        pytest.skip("the library's objects are not built here")
    out = tmp_path_factory.mktemp("fake")
    names = subprocess.run(["nm", "-u", *objects], check=True, capture_output=True, text=True).stdout.split()
    names = {x for x in names if x.startswith(("cuda", "__cuda"))}
    source = FAKE + "".join(STUB % x for x in sorted(names) if f" {x}(" not in FAKE)
    (out / "fake.c").write_text(source)
    lib = str(out / "libngx_fake.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-w", "-o", lib, str(out / "fake.c"), *objects, "-Wl,-Bsymbolic,--no-undefined", "-lstdc++",
                    "-lm", "-lpthread"], check=True)
    return C.CDLL(lib)


def test_a_failed_upload_is_repeated(fake):
    n = 5
    rp, col, w = np.arange(n + 1, dtype=np.int64) * 2, np.array([1, 2, 2, 3, 3, 4, 4, 0, 0, 1], np.int32), np.arange(1.0, 11.0)
    fake.fake_fail_copy.argtypes = [C.c_size_t]
    fake.ngx_graph_create_ex.argtypes = [C.c_void_p, C.c_int, C.c_int, C.POINTER(C.c_void_p)]
    fake.ngx_graph_update_weights.argtypes = [C.c_void_p, C.c_void_p]
    fake.ngx_graph_destroy.argtypes = [C.c_void_p]
    fake.ngx_last_error.restype = C.c_char_p
    csr, keep = ngx._csr_struct(n, rp, col, w)
    handle = C.c_void_p()
    on_host = 1
    assert fake.ngx_graph_create_ex(C.byref(csr), 0, on_host, C.byref(handle)) == 0, fake.ngx_last_error()
    new = np.arange(2.0, 12.0)
    fake.fake_fail_copy(4 * w.size)
    assert fake.ngx_graph_update_weights(handle, new.ctypes.data) != 0
    assert fake.fake_copies() == 0
    assert fake.ngx_graph_update_weights(handle, new.ctypes.data) == 0, fake.ngx_last_error()
    assert fake.fake_copies() == 1  # the map went up before the kernels
    assert fake.ngx_graph_update_weights(handle, new.ctypes.data) == 0
    assert fake.fake_copies() == 1  # and is kept
    fake.ngx_graph_destroy(handle)
    del keep
