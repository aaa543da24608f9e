"""What a caller of the eigensolver is told: the device's status word keeps the first
failure, and its code and message reach the caller.  The words are injected on the
host; no kernel runs."""
import ctypes

import pytest


@pytest.mark.parametrize("word,code,text", [(0, 0, None), (4, 4, b"wait"), (6, 6, b"inverse iteration"),
                                            (99, 6, b"inverse iteration")])
def test_status_word_to_return_code(word, code, text):
    from mopac_gpu_b200._lib import lib
    L = lib()
    L.mb_eigh_status.argtypes, L.mb_eigh_status.restype = [ctypes.c_int], ctypes.c_int
    assert L.mb_eigh_status(word) == code
    if text:
        assert text in L.mb_last_error()
