"""A batch of one graph takes its sources from the graph's order (CPU, on a fake CUDA runtime).

One graph is built on the device, where its all-sources order is computed on first use. The batch run must ask for it and
upload one id per source: without it the tiles would take whatever is in the buffer for vertices.
"""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import neurograph_b200 as ngx
from test_update_weights_upload import fake  # noqa: F401  (fixture)


@pytest.mark.parametrize("task", [0, 1, 2])
def test_sources_are_uploaded(fake, task):  # noqa: F811
    n = 37
    csr, keep = ngx._csr_struct(n, np.zeros(n + 1, np.int64), np.zeros(0, np.int32), np.zeros(0))
    fake.fake_fail_copy.argtypes = [C.c_size_t]
    fake.ngx_batch_create.argtypes = [C.c_void_p, C.c_int64, C.c_int, C.POINTER(C.c_void_p)]
    fake.ngx_batch_run.argtypes = [C.c_void_p] * 6
    fake.ngx_graph_destroy.argtypes = [C.c_void_p]
    handle = C.c_void_p()
    fake.ngx_last_error.restype = C.c_char_p
    assert fake.ngx_batch_create(C.byref(csr), 1, 0, C.byref(handle)) == 0, fake.ngx_last_error()
    opts = ngx._BatchOpts(task, 0, 0.0, 0, 0, 0.0, 0, 0, 0)
    result, *keep_result = ngx.Graph._result_struct(0, False, n)
    bc = np.zeros(n)
    fake.fake_watch_copy(C.c_size_t(4 * n))
    fake.ngx_batch_run(handle, C.byref(opts), C.byref(result), bc.ctypes.data, bc.ctypes.data, bc.ctypes.data)  # no kernel runs: an error
    assert fake.fake_copies() == 1
    fake.ngx_graph_destroy(handle)
    del keep, keep_result
