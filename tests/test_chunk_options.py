"""n2b_options.chunk, its steps and its block, is checked on the host, by the size query already."""

import ctypes

import pytest

from naer2_b200 import _lib


@pytest.mark.parametrize("kw, msg", [(dict(chunk=-1), "chunk < 0"), (dict(chunk=48 << 16), "block"),
                                     (dict(chunk=512 << 16 | 3), "block"), (dict(chunk=7 | 64 << 16), None)])
def test_chunk_options(kw, msg):
    lib = _lib.load()
    p = _lib.Population()
    p.model, p.n, p.acc_depth, p.shift = _lib.MODEL_LIF_DELTA, 100, 16, 40
    p.v = p.ref = p.acc = 0x1000  # never dereferenced by the host
    opt, n = _lib.Options(block=128, device=0, persistent=1, **kw), ctypes.c_size_t()
    rc = lib.n2b_workspace_bytes((_lib.Population * 1)(p), 1, (_lib.Connection * 1)(), 0, ctypes.byref(opt), ctypes.byref(n))
    if msg is None:
        assert rc == 0 and n.value > 0
    else:
        assert rc != 0 and msg in lib.n2b_last_error().decode()
