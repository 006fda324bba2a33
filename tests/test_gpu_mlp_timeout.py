"""A training epoch after a GEMM's wait has run out: the call reports it and the
network's parameters stay as they were, to the last bit.

The time-out flag is the device word that such a wait sets; the test sets it the same
way, through the library's own buffer table, and mq_mlp_init clears it."""
import ctypes

import numpy as np
import pytest

from myqc_gb300._lib import MyQCError
from myqc_gb300.session import Context

pytestmark = pytest.mark.gpu


def test_parameters_after_a_time_out():
    rng = np.random.default_rng(0)
    n, nin, width, nout = 4096, 64, 256, 25
    ctx = Context(0)
    try:
        ctx.mlp_init(nin, width, nout)
        ctx.mlp_set_data(rng.standard_normal((n, nin), dtype=np.float32), rng.standard_normal((n, nout), dtype=np.float32),
                         np.ones((n, nout), dtype=np.float32))
        ctx.mlp_set_params(0.05 * rng.standard_normal(nin * width + width * width + width * nout + 2 * width + nout)
                           .astype(np.float32))
        ctx.mlp_train_epoch(1024, 1e-3, 1)
        before = ctx.mlp_get_params()
        buf = ctx.L["_ZN2mq3bufEP6mq_ctxPKcm"]  # mq::buf(mq_ctx *, const char *, size_t)
        buf.restype, buf.argtypes = ctypes.c_void_p, [ctypes.c_void_p, ctypes.c_char_p, ctypes.c_size_t]
        flag = buf(ctx.h, b"mlp_err", 64)
        driver = ctypes.CDLL("libcuda.so.1")
        driver.cuMemsetD32_v2.argtypes = [ctypes.c_uint64, ctypes.c_uint, ctypes.c_size_t]
        assert driver.cuMemsetD32_v2(flag, 3, 1) == 0
        with pytest.raises(MyQCError, match="timed out"):
            ctx.mlp_train_epoch(1024, 1e-3, 2)
        assert np.array_equal(ctx.mlp_get_params(), before)
        ctx.mlp_init(nin, width, nout)
        ctx.mlp_set_params(before)
        ctx.mlp_set_data(rng.standard_normal((n, nin), dtype=np.float32), rng.standard_normal((n, nout), dtype=np.float32),
                         np.ones((n, nout), dtype=np.float32))
        assert np.isfinite(ctx.mlp_train_epoch(1024, 1e-3, 3))
        assert not np.array_equal(ctx.mlp_get_params(), before)
    finally:
        ctx.close()
