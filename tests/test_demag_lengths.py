"""The rule for the transform lengths of a mesh (maf_demag_lengths, host only): every axis is
at its own doubled length or at the next one with compile-time kernels, all axes or none
but for x on 3-D meshes, on both sides of each of the rule's lines."""
import pytest

M = pytest.importorskip("magnumaf")

X = [2 * n for n in (16, 32, 64, 96, 128, 192, 256, 384, 512, 768, 1024, 1536, 2048)]
Y2 = [16, 32, 64, 96, 128, 192, 256, 384, 512, 768, 1024, 1536, 2048]
Y3 = Y2 + [4096]
Z = [8, 16, 32, 64, 96, 128]


def _next(lengths, n):
    return min((v for v in lengths if v >= n), default=None)


@pytest.mark.parametrize("nz", [1, 2, 3, 4, 9, 16, 20, 33, 48, 64, 65])
def test_lengths_are_own_or_the_next_compile_time_ones(nz):
    for nx in list(range(1, 40)) + [96, 97, 260, 520, 1024, 1040, 1300, 2048, 2049]:
        for ny in list(range(1, 20)) + [64, 65, 260, 520, 1024, 1025, 1040, 1300, 2048, 2049]:
            own = (2 * nx, 2 * ny, 1 if nz == 1 else 2 * nz)
            pad = (_next(X, 2 * nx), _next(Y2 if nz == 1 else Y3, 2 * ny - 1), 1 if nz == 1 else _next(Z, 2 * nz - 1))
            got = M.DemagField.lengths(nx, ny, nz)
            if None in pad:
                assert got == own
                continue
            assert got[1:] == pad[1:] and got[0] in (own[0], pad[0])
            if nz == 1 or (pad[0] // 2 + 1) * pad[1] * pad[2] <= 65536:
                assert got == pad
            elif got[0] != pad[0]:
                assert pad[0] // 2 + 1 > 1.25 * (nx + 1)


@pytest.mark.parametrize("shape,lengths", [
    ((100, 25, 1), (256, 64, 1)), ((1, 13, 1), (32, 32, 1)), ((130, 1040, 1), (260, 2080, 1)),  # no y length
    ((512, 512, 16), (1024, 1024, 32)), ((125, 75, 40), (256, 192, 96)), ((100, 100, 65), (200, 200, 130)),
    ((10, 500, 30), (32, 1024, 64)), ((9, 500, 30), (18, 1024, 64)),  # x's spectrum 1.55 and 1.7 times as long
    ((1, 128, 4), (32, 256, 8)), ((1, 256, 4), (2, 512, 8)),  # up to 2^16 values and more
    ((600, 1024, 9), (1536, 2048, 32)), ((600, 1040, 9), (1200, 4096, 32)),  # beside 2048 and 4096 points
    ((1300, 1300, 4), (3072, 4096, 8)), ((1040, 1040, 9), (2080, 4096, 32)),
])
def test_lengths_on_both_sides_of_the_lines(shape, lengths):
    assert M.DemagField.lengths(*shape) == lengths


def test_lengths_reject_empty_meshes():
    with pytest.raises(M.MafError):
        M.DemagField.lengths(0, 4, 4)
