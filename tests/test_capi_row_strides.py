"""Entry points that take the distance of a query's rows refuse one that is shorter than a row, before any pointer is used."""
import ctypes

import pytest

H, L, P = 2, 1, 4


def _calls(rows):
    from dfa3d_b200 import _lib
    lib, p = _lib.load(), ctypes.byref(_lib.Problem(1, 16, H, 32, 8, L, 5, P, 0, 0, 0))
    yield lambda maps: lib.dfa3d_attn3d_forward_rows(p, 1, 2, *rows(maps), *([None] * 12)), 1, lib
    yield lambda maps: lib.dfa3d_attn3d_backward_rows(p, 1, 2, *rows(maps), *([None] * 16)), 1, lib
    yield lambda maps: lib.dfa3d_attn2d_forward(p, maps, *rows(maps), *([None] * 8)), 2, lib
    yield lambda maps: lib.dfa3d_attn2d_backward(p, maps, *rows(maps), *([None] * 11)), 2, lib


@pytest.mark.parametrize("offsets_less,logits_less", [(1, 0), (0, 1), (10 ** 6, 0), (0, 10 ** 6)])
def test_rows_that_overlap_are_refused(lib_built, offsets_less, logits_less):
    rows = lambda maps: (2 * H * L * P * maps - offsets_less, H * L * P * maps - logits_less)
    for call, maps, lib in _calls(rows):
        assert call(maps) == -1 and b"offsets_row and logits_row" in lib.dfa3d_last_error()


@pytest.mark.parametrize("extra", [None, 0, 8])
def test_rows_that_do_not_are_accepted(lib_built, extra):
    rows = lambda maps: (0, 0) if extra is None else (2 * H * L * P * maps + extra, H * L * P * maps + extra)
    for call, maps, lib in _calls(rows):
        assert call(maps) == -1 and b"is null" in lib.dfa3d_last_error()
