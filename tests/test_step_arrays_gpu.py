"""What brings a captured step's arrays to the device (csrc/runtime.cu) against the same numbers laid out by hand."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("small,rows,widths,pitch", [(4, 0, [], 1), (8, 1, [1], 1), (116, 13, [8], 300), (260, 3, [1, 37, 5], 64),
                                                     (0, 5, [7] * 8, 9), (84, 100, [163], 163), (4, 2, [3] * 19, 4), (516, 64, [4096], 4100)])
def test_arrays_lie_where_they_belong(small, rows, widths, pitch):
    from atom_b200 import native

    n = small + rows * sum(widths)
    src = torch.randint(-2 ** 31, 2 ** 31 - 1, (n + 3,), dtype=torch.int32).pin_memory()
    ats = [small + 2 + k * (max(rows, 1) * pitch + 5) for k in range(len(widths))]
    dst = torch.full((small + 2 + len(widths) * (max(rows, 1) * pitch + 5) + 1,), -7, dtype=torch.int32)
    want, dev, at = dst.clone(), dst.cuda(), small
    want[:small] = src[:small]
    for a, w in zip(ats, widths):
        for r in range(rows):
            want[a + r * pitch:a + r * pitch + w] = src[at:at + w]
            at += w
    assert at == n
    native.step_arrays(dev, src, small, rows, widths, ats, [pitch] * len(widths))
    assert torch.equal(dev.cpu(), want)


def test_tables_beyond_the_array_are_refused():
    from atom_b200 import native

    src = torch.zeros(14, dtype=torch.int32).pin_memory()
    dev = torch.full((64,), -7, dtype=torch.int32, device="cuda:0")
    for small, rows, width, at, pitch in ((4, 2, 5, 55, 5), (65, 0, 1, 0, 1), (4, 2, 5, -1, 5), (4, 2, 5, 4, 4)):
        with pytest.raises((native.NativeError, AssertionError)):
            native.step_arrays(dev, src, small, rows, [width], [at], [pitch])
    assert bool((dev == -7).all())
