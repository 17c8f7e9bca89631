"""Cache.infer hands its ids over as one typed array where it can: what the library sees is what the conversion element by
element gives, for every kind of sequence and number, and what was refused is refused."""
import ctypes as C
from unittest import mock

import numpy as np
import pytest


def _seen(pkg, ids, max_seq=16):
    engine = __import__("sys").modules[pkg.Cache.__module__]
    cache = pkg.Cache.__new__(pkg.Cache)
    cache.max_seq, cache.model, cache._d_tokens, cache.ptr = max_seq, mock.Mock(), None, None
    cache._x, cache._tokens = engine.TensorStruct(), (C.c_int * (max_seq + 2))()
    got = []
    with mock.patch.object(engine, "lib") as lib:
        lib.inference.side_effect = lambda m, x, d, tokens, ptr: got.extend(tokens) or 0
        cache.infer(ids)
    return got


@pytest.mark.parametrize("ids", [[5], [1, 2, 3], (1, 2, 3), [0, -1, 2 ** 31 - 1], [2 ** 31, -2 ** 31 - 1, 2 ** 32 + 7], [1.0, 2.9], [True, False],
                                 [np.int64(7), np.int32(8)], np.arange(4), np.arange(4, dtype=np.int64), range(6), b"abc", ["12", 3], list(range(17)), []])
def test_ids_reach_the_library_as_before(pkg, ids):
    n = len(ids)
    want = (C.c_int * 18)()
    want[0] = n + 1
    want[1:n + 1] = [int(t) for t in ids]
    assert _seen(pkg, ids) == list(want)


def test_more_ids_than_rows_are_refused(pkg):
    with pytest.raises(ValueError):
        _seen(pkg, list(range(18)))
