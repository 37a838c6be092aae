"""ERI batches in loop-length order (GPU tests).

pfk_eri_batch_run works on windows of 2^14 listed quartets in the order of
their loop lengths and writes every block to its listed place; the parts of a
range that do not fill a window run as listed.  Any range gives the bits of
the whole list's run (a quartet's arithmetic does not depend on its
neighbours)."""
import numpy as np
import pytest

from helpers import pfk

pytestmark = pytest.mark.gpu

W = 1 << 14


@pytest.mark.parametrize("cls,engine", [((0, 0, 0, 0), "os"), ((1, 0, 1, 0), "rys"), ((2, 0, 2, 1), "rys"),
                                        ((3, 3, 3, 3), "rys")])
def test_ranges_agree(cls, engine):
    torch = pytest.importorskip("torch")
    P = pfk()
    la, lb, lc, ld = cls
    big = sum(cls) < 12
    n = 2 * W + 100 if big else 40
    bra_first = (la, lb) >= (lc, ld)
    sh, pairs, quartets = P.workloads.eri_class_quartets(*(cls if bra_first else (lc, ld, la, lb)), n, seed=3)
    b = P.EriBatch(sh, pairs, quartets)

    def run(first, count):
        out = torch.full((count + 1, b.ncomp), 7.0, dtype=torch.float64, device="cuda:0")
        b.run(first, count, engine, "fp64", out.data_ptr())
        torch.cuda.synchronize()
        assert bool((out[count] == 7.0).all())          # nothing past the range
        return out[:count]
    whole = run(0, n)
    ranges = [(0, 1), (n - 1, 1), (5, 20)]
    if big:
        ranges += [(0, W), (0, W - 1), (1, W), (W, W), (W - 1, W + 2), (3, n - 3), (2 * W, 100), (2 * W - 1, 101),
                   (W + 7, W)]
    for first, count in ranges:
        assert bool((run(first, count) == whole[first:first + count]).all()), (first, count)
    b.close()


@pytest.mark.parametrize("cls,engine", [((1, 1, 1, 1), "os"), ((2, 0, 2, 0), "rys"), ((2, 1, 1, 1), "rys"),
                                        ((2, 2, 2, 1), "rys"), ((3, 0, 1, 0), "rys"), ((3, 1, 2, 1), "rys")])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_around_one_wave(cls, engine, precision):
    """Ranges of up to one wave run as listed in builds of their own, longer
    ones in windows: the same bits on both sides of the line, which lies at a
    whole number of blocks per SM (148 SMs; a block holds 128 quartets or
    128 / team)."""
    torch = pytest.importorskip("torch")
    P = pfk()
    ncart = [(l + 1) * (l + 2) // 2 for l in cls]
    ncomp = int(np.prod(ncart))
    rest = ncomp // ncart[0]
    group = ncart[0] if rest <= 64 else ncart[0] * ncart[1]
    per = 128 if ncomp <= 81 else 128 // (1 << max(2, (group - 1).bit_length()))
    waves = [148 * per * b for b in (1, 2, 3, 4)]
    n = waves[-1] + W + 100
    sh, pairs, quartets = P.workloads.eri_class_quartets(*cls, n, seed=8)
    b = P.EriBatch(sh, pairs, quartets)
    assert b.ncomp == ncomp

    def run(first, count):
        out = torch.full((count + 1, ncomp), 7.0, dtype=torch.float64, device="cuda:0")
        b.run(first, count, engine, precision, out.data_ptr())
        torch.cuda.synchronize()
        assert bool((out[count] == 7.0).all())
        return out[:count]
    whole = run(0, n)
    for first, count in [(0, 1), (n - 77, 77)] + [(f, w + d) for w in waves for f, d in ((0, 0), (0, 1), (9, 0), (9, 1))]:
        assert bool((run(first, count) == whole[first:first + count]).all()), (first, count)
    b.close()
