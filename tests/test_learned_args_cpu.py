"""The learned coder's entries without a model: refused before anything reads it."""
import ctypes

import numpy as np
import pytest

from pentago_b200 import capi


@pytest.mark.parametrize("entry", ["pg_rans_learned_encode", "pg_rans_learned_decode", "pg_learned_freqs"])
def test_no_model_is_refused(entry):
    L, some = capi.lib(), capi.ptr(np.zeros(64, np.int64))
    refs = (capi.pg_block_ref_t * 1)()
    if entry == "pg_learned_freqs":
        rc = L.pg_learned_freqs(None, refs, 1, some, some, some, 1, some, None)
    else:
        rc = getattr(L, entry)(None, refs, 1, *[some] * (len(getattr(L, entry).argtypes) - 4), None)
    assert rc == capi.PG_ERR_ARG
    assert b"model" in ctypes.cast(L.pg_last_error(), ctypes.c_char_p).value
