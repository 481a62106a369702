"""The features per work item of the 16-bit SpMM: the rule's decision, and that
saving and restoring every option leaves it in force."""
import ctypes

import pytest

KEYS = (b"spmm_fc", b"spmm_stages", b"spmm_fp8", b"spmm_gather", b"spmm_tf32")


@pytest.fixture
def lib():
    from att_gb300 import _lib, builder
    builder.build()
    return _lib.load()


def _read(lib):
    got = {}
    for k in KEYS:
        v = ctypes.c_int(0)
        assert lib.att_get_option(k, ctypes.byref(v)) == 0
        got[k] = v.value
    return got


def _rule(lib):
    many, few = 4096, 4095
    return {(F, p): lib.att_spmm_item_features(F, p) for F in (8, 32, 33, 64, 65, 128, 129, 192, 193, 256, 320)
            for p in (0, few, many, 1 << 40)}


EXPECTED = {8: (32, 32), 32: (32, 32), 33: (64, 64), 64: (64, 64), 65: (64, 128), 128: (64, 128), 129: (64, 64),
            192: (64, 64), 193: (64, 128), 256: (64, 128), 320: (64, 64)}


def test_rule(lib):
    for (F, parts), width in _rule(lib).items():
        assert width == EXPECTED[F][parts >= 4096], (F, parts)


def test_saving_and_restoring_keeps_the_rule(lib):
    before = _rule(lib)
    old = _read(lib)
    assert old[b"spmm_fc"] == 64
    try:
        assert lib.att_set_option(b"spmm_fc", 128) == 0
        assert lib.att_spmm_item_features(128, 1) == 128 and lib.att_spmm_item_features(192, 1) == 128
    finally:
        for k, v in old.items():
            assert lib.att_set_option(k, v) == 0
    assert _rule(lib) == before and _read(lib) == old


@pytest.mark.parametrize("width", [64, 128])
def test_a_threads_width_is_taken_as_it_is(lib, width):
    assert lib.att_set_thread_option(b"spmm_fc", width) == 0
    try:
        assert {lib.att_spmm_item_features(F, p) for F in (72, 128, 192, 256) for p in (1, 1 << 20)} == {width}
    finally:
        assert lib.att_set_thread_option(b"spmm_fc", -1) == 0
    assert lib.att_spmm_item_features(128, 4096) == 128 and lib.att_spmm_item_features(128, 4095) == 64
    assert lib.att_set_option(b"spmm_fc", 0) == 1 and lib.att_set_thread_option(b"spmm_fc", 0) == 1
