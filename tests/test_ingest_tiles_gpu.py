"""The Matrix-Market parser's tiles: lines that start, end or run on across the
4 KB tiles and the 256 staged bytes past them, text that does not start on a
16-byte boundary, a header longer than the first 4 KB read, and the errors."""
import numpy as np
import pytest

gv_b200 = pytest.importorskip("gv_b200")
pytestmark = pytest.mark.gpu


def _parse(text, shift, values):
    import torch
    buf = torch.zeros(shift + len(text), dtype=torch.uint8)
    buf[shift:] = torch.frombuffer(bytearray(text), dtype=torch.uint8)
    return gv_b200.mtx_parse(buf.cuda()[shift:], with_values=values)


@pytest.mark.parametrize("shift", [0, 1, 15])
@pytest.mark.parametrize("head", [0, 5000])   # bytes of comment before the size line
@pytest.mark.parametrize("pad", [0, 1, 300])  # blanks inside some lines: over the staged bytes for 300
def test_lines_across_tiles(shift, head, pad):
    rng = np.random.default_rng(pad + shift)
    k, n = 3000, 99_999
    s, d = rng.integers(1, n + 1, k), rng.integers(1, n + 1, k)
    w = rng.integers(1, 10_000, k)
    lines = [f"{a}{' ' * (1 + (pad if i % 3 == 0 else 0))}{b} 0.{c:04d}" for i, (a, b, c) in enumerate(zip(s, d, w))]
    for i in range(0, k, 50):
        lines[i] = ["%" + "x" * (i % 40), "", "   ", "\t\r"][(i // 50) % 4] + "\n" + " " + lines[i]
    text = "%%MatrixMarket matrix coordinate real general\n" + ("%" + "c" * head + "\n" if head else "")
    text += f"{n} {n} {k}\n" + "\n".join(lines)
    meta, src, dst, val = _parse(text.encode(), shift, True)
    assert meta["entries"] == k
    assert np.array_equal(src.cpu().numpy(), s - 1) and np.array_equal(dst.cpu().numpy(), d - 1)
    assert np.array_equal(val.cpu().numpy(), (w.astype(np.float64) / 10_000).astype(np.float32))


@pytest.mark.parametrize("line", ["7 8\n9", "1 x", "0 5", "5 100000", "3 4 nothing"])
def test_a_bad_line_is_refused(line):
    text = "%%MatrixMarket matrix coordinate real general\n99999 99999 3\n1 2 0.5\n" + line + "\n2 3 0.25\n"
    with pytest.raises(gv_b200.GvError):
        _parse(text.encode(), 0, True)


def test_empty_data_and_capacity():
    import torch
    meta, src, _, _ = _parse(b"%%MatrixMarket matrix coordinate pattern general\n5 5 0\n\n% end\n", 3, False)
    assert meta["rows"] == 5 and len(src) == 0
    text = b"%%MatrixMarket matrix coordinate pattern general\n5 5 1\n" + b"1 2\n" * 40  # more entries than stated
    with pytest.raises(gv_b200.GvError):
        _parse(text, 0, False)
