"""Which grids take the fused FFT passes and which the library's transform, on both sides of
every line of the rule (host code, no GPU calls).  Each line is where the timings of the two
cross; a grid on its wrong side is a call that got slower."""

import ctypes

import pytest


def fused(os_shape, shape=None, gram=False, lowrank=0, nseg=1):
    from pyfourier_b200 import _lib

    out = ctypes.c_int(-1)
    _lib.check(_lib.load().pfb_fft_route(len(os_shape), _lib.int_array(shape or os_shape), _lib.int_array(os_shape),
                                         int(gram), lowrank, nseg, ctypes.byref(out)))
    return out.value


def half(os_shape):
    return tuple(max(1, n // 2) for n in os_shape)


@pytest.mark.parametrize("os, want", [
    ((64,), 0),  # 1D
    ((1024, 1024), 1), ((1025, 64), 0), ((961, 16), 1), ((1, 1), 1),          # two stages
    ((735, 735), 1), ((768, 768), 1), ((770, 64), 0), ((1000, 1000), 0), ((64, 936), 0),  # three
    ((61 * 8, 61 * 8), 1), ((64, 561), 0), ((578, 64), 0), ((37 * 11, 60), 1),  # a prime to 64
    ((127, 127), 1), ((254, 254), 1), ((3 * 67, 64), 0), ((508, 508), 0), ((64, 131), 0),  # to 127, 2D
    ((64, 134, 64), 1), ((64, 83, 64), 0), ((96, 83, 96), 1), ((83, 64, 64), 0), ((64, 3 * 67, 64), 0),  # 3D
    ((107, 107, 96), 0), ((96, 96, 107), 1), ((37, 37, 10), 1), ((61, 61, 10), 0),  # two such axes
])
def test_nufft_grids(os, want):
    assert fused(os, half(os)) == want


@pytest.mark.parametrize("os, shape, want", [
    ((150, 167, 150), (100, 111, 100), 1), ((167, 150, 150), (111, 100, 100), 1),
    ((150, 150, 167), (100, 100, 111), 0),  # the x axis
    ((150, 167, 150), (120, 133, 120), 0),  # less than 1.5 times the image
    ((150, 173, 150), (100, 115, 100), 0), ((150, 334, 150), (100, 222, 100), 0), ((64, 167, 64), (42, 111, 42), 0),
])
def test_large_primes_on_an_outer_axis(os, shape, want):
    assert fused(os, shape) == want


@pytest.mark.parametrize("os, lowrank, want", [
    ((256, 256), 0, 1), ((256, 256), 4, 1), ((256, 256), 5, 1), ((256, 256), 6, 0), ((256, 256), 8, 0),
    ((64, 64), 0, 0), ((96, 96), 3, 1), ((384, 384), 4, 1), ((500, 500), 4, 0), ((512, 512), 0, 0),
    ((125, 125), 4, 0), ((243, 243), 4, 0), ((165, 165), 0, 1), ((272, 272), 4, 1), ((289, 289), 4, 0), ((97, 97), 0, 0),
    ((64, 64, 64), 0, 0), ((128, 128, 128), 4, 0),
])
def test_gram_grids_of_the_images_size(os, lowrank, want):
    assert fused(os, os, gram=True, lowrank=lowrank) == want


@pytest.mark.parametrize("os, lowrank, nseg, want", [
    ((512, 512), 0, 1, 1), ((512, 512), 4, 1, 1), ((440, 440), 8, 1, 1), ((512, 512), 8, 1, 0), ((1024, 1024), 3, 1, 1),
    ((1024, 1024), 4, 1, 0), ((96, 96, 96), 4, 1, 1), ((508, 508), 0, 1, 0),
])
def test_embedded_gram_grids(os, lowrank, nseg, want):
    assert fused(os, half(os), gram=True, lowrank=lowrank, nseg=nseg) == want


def test_segments_need_the_full_pipeline():
    # two segments: not in place, so the lines are the embedded ones
    assert fused((64, 64), (64, 64), gram=True, nseg=1) == 0
    assert fused((64, 64), (64, 64), gram=True, nseg=2) == 1


def test_bad_arguments():
    with pytest.raises(ValueError):
        fused((8, 8), (9, 8))
    with pytest.raises(ValueError):
        fused((8, 8, 8, 8))
