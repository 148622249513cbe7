"""Tile heights of a structure that is not tuned (host rule, no GPU): by the
waves of CTAs that the tallest tiles of its plan fill, on both sides of every line."""
import ctypes

import pytest

N_SM = 152
WAVE = 4 * N_SM     # two tiles per CTA, two CTAs per SM


@pytest.mark.parametrize("tall,rows", [(0, 0), (8 * WAVE - 1, 0), (8 * WAVE, 128), (16 * WAVE - 1, 128), (16 * WAVE, 256),
                                       (25 * WAVE - 1, 256), (25 * WAVE, 512), (10 ** 9, 512)])
def test_single_vector(library, tall, rows):
    f = library.h2g_default_tile_rows
    f.argtypes = [ctypes.c_longlong, ctypes.c_int, ctypes.c_int]
    assert f(tall, N_SM, 0) == rows
    assert f(2 * tall, 2 * N_SM, 0) == rows or tall % WAVE    # a matter of waves, not of tiles


@pytest.mark.parametrize("tall,rows", [(0, 0), (2 * WAVE - 1, 0), (2 * WAVE, 512), (10 ** 9, 512)])
def test_several_vectors(library, tall, rows):
    f = library.h2g_default_tile_rows
    f.argtypes = [ctypes.c_longlong, ctypes.c_int, ctypes.c_int]
    assert f(tall, N_SM, 1) == rows
