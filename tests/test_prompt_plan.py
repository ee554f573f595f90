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


# (rows, output features, input features) for every token tile, without and with K slices, with every number of pipeline
# stages modulo the barriers of its code ring (six for tiles of 320, else four) and a whole or half last stage of a slice.
RUNS = {
    160: [(129, 1000, 512), (129, 1000, 448), (129, 1000, 640), (129, 1000, 576), (129, 1000, 768), (129, 1000, 704),
          (129, 1000, 384), (129, 1000, 320), (129, 1000, 1024), (160, 4000, 2880), (129, 1000, 1216), (129, 1000, 1088),
          (129, 1000, 1472), (129, 1000, 1344), (320, 2048, 2624), (257, 1000, 5824)],
    192: [(177, 5500, 1024), (177, 11008, 448), (177, 9400, 640), (177, 9400, 576), (177, 8192, 768), (177, 8192, 704),
          (177, 11008, 384), (177, 8192, 832), (192, 9400, 3008), (177, 9400, 2880), (177, 5500, 1920), (192, 4000, 1664),
          (1150, 1000, 2240), (177, 5500, 1984), (384, 4000, 2752), (350, 4000, 2624)],
    224: [(200, 22016, 512), (200, 22016, 448), (200, 22016, 640), (200, 22016, 576), (769, 13000, 768), (769, 13000, 704),
          (200, 11008, 384), (177, 11008, 320), (224, 8192, 3072), (200, 8192, 2880), (200, 4000, 1792), (200, 4000, 1728),
          (200, 5500, 2176), (200, 5500, 2048), (200, 8192, 2816), (224, 5500, 2368)],
    256: [(200, 11008, 512), (200, 11008, 448), (200, 9400, 640), (200, 11008, 576), (200, 9400, 768), (200, 9400, 704),
          (500, 5500, 384), (500, 5500, 320), (177, 1000, 2048), (200, 1000, 8512), (177, 1000, 2368), (177, 1000, 2112),
          (177, 2048, 1472), (177, 2048, 1344), (200, 2048, 3584), (200, 1000, 5824)],
    320: [(257, 11008, 768), (257, 11008, 704), (257, 11008, 896), (257, 11008, 832), (257, 11008, 1024), (257, 11008, 960),
          (257, 11008, 384), (257, 11008, 320), (257, 11008, 512), (257, 11008, 448), (257, 11008, 640), (257, 11008, 576),
          (257, 4000, 5952), (257, 4000, 5696), (257, 4000, 6464), (257, 4000, 6208), (257, 4000, 4032), (257, 4000, 3776),
          (257, 4000, 4416), (257, 4000, 4160), (257, 4000, 4928), (257, 4000, 4672), (257, 4000, 5440), (257, 4000, 5184)],
    384: [(350, 11008, 512), (350, 11008, 448), (350, 11008, 640), (350, 11008, 576), (350, 11008, 768), (350, 11008, 704),
          (350, 11008, 384), (350, 11008, 320), (350, 4000, 6080), (350, 5500, 4288), (350, 4000, 6464), (350, 4000, 6336),
          (350, 4000, 6976), (350, 4000, 6720), (350, 5500, 4224), (350, 4000, 7232)],
}


@pytest.mark.parametrize("tokens", sorted(RUNS))
def test_runs_cover_the_tile(tokens, lib):
    seen, ring = set(), 6 if tokens == 320 else 4
    for m, n, k in RUNS[tokens]:
        chosen, slices = plan(lib, m, n, k)
        k_tiles = -(-(k // 64) // slices)
        seen.add((chosen, slices > 1, -(-k_tiles // 2) % ring, k_tiles % 2))
    assert seen == {(tokens, sliced, stages, odd) for sliced in (False, True) for stages in range(ring) for odd in (0, 1)}
