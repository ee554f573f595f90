"""How prompts are cut into token tiles and K slices (the choice needs no GPU)."""
import ctypes

import pytest

from atlasinfer_b200 import _capi, build

SMS = 148


@pytest.fixture(scope="module")
def lib():
    build.build()
    return _capi.load()


def plan(lib, m, n, k):
    tokens, slices = ctypes.c_int(), ctypes.c_int()
    _capi.check(lib.atlas_qlinear_gemm_plan(m, n, k, ctypes.byref(tokens), ctypes.byref(slices)), "atlas_qlinear_gemm_plan")
    return tokens.value, slices.value


def _slices_of_256(m, n, k):
    """K slices of tiles of 256 tokens, the rule that no other tile may undercut."""
    tiles, k_tiles, best, cost = -(-n // 128) * -(-m // 256), k // 64, 1, None
    for s in range(1, 17):
        if s > 1 and k_tiles // s < 8:
            break
        us = -(-tiles * s // SMS) * (0.4 * -(-k_tiles // s) + 7.0) + (2.5 + 2e-6 * s * m * n if s > 1 else 0.0)
        if cost is None or us < cost:
            best, cost = s, us
    return best


@pytest.mark.parametrize("k", [512, 640, 1024, 2048, 2176, 4096, 4224, 5120, 8192, 11008, 14336])
def test_sums_are_never_longer_than_with_tiles_of_256(k, lib):
    for n in (512, 1000, 1024, 2048, 3072, 4096, 5120, 6144, 8192, 10240, 11008, 12288, 14336, 16384, 22016, 28672):
        for m in (129, 160, 192, 200, 256, 257, 300, 301, 320, 384, 385, 500, 512, 600, 769, 1000, 1024, 1152, 1500, 1536, 2048):
            tokens, slices = plan(lib, m, n, k)
            assert slices >= _slices_of_256(m, n, k), (m, n, k, tokens, slices)


def test_only_prompts_have_a_plan(lib):
    two = ctypes.c_int(), ctypes.c_int()
    ask = lambda *a: lib.atlas_qlinear_gemm_plan(*a, ctypes.byref(two[0]), ctypes.byref(two[1]))  # noqa: E731
    assert ask(128, 4096, 4096) == _capi.ERR_UNSUPPORTED
    assert ask(0, 4096, 4096) == _capi.ERR_BAD_ARGUMENT and ask(300, 4096, 100) == _capi.ERR_BAD_ARGUMENT
