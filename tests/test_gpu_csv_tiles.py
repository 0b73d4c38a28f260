"""The device CSV reader at the edges of its tiles: texts that end around a multiple of 16 KB and of 16 bytes, lines
across tile borders, blocks of lines longer than the shared staging, more lines than the first room holds (empty
lines after the bounds), and lines left to the host beside group starts.  Against the host reader's binary files."""
import numpy as np
import pytest

import colo

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return colo.Context(0)


def _same(ctx, tmp_path, text):
    path = tmp_path / "d.csv"
    path.write_bytes(text.encode())
    colo.csv_to_binary(path, tmp_path / "host.colo", 1)
    colo.Dataset.from_csv(ctx, path, device=True).write_binary(tmp_path / "dev.colo")
    assert (tmp_path / "dev.colo").read_bytes() == (tmp_path / "host.colo").read_bytes()


def _text(lines, tail="\n"):
    return f"{len(lines)}\n" + "\n".join(lines) + "\n\n0,0,10,10" + tail


@pytest.mark.parametrize("size", [16384, 2 * 16384, 5 * 16384])
@pytest.mark.parametrize("off", [-17, -16, -15, -1, 0, 1, 15, 16, 17])
def test_text_sizes(ctx, tmp_path, size, off):
    lines = [f"{i * 7 // (size // 20)},{i}.5,{i % 10}.25" for i in range(size // 20)]
    body = len(_text(lines)) - len(f"{len(lines)}\n")
    lines[3] += "0" * (size + off - body)   # a line as long as it takes
    for tail in ("\n", ""):
        _same(ctx, tmp_path, _text(lines, tail))


@pytest.mark.parametrize("pad", [0, 40, 63, 64, 200])
def test_long_lines(ctx, tmp_path, pad):
    """Blocks of 256 lines on both sides of 16 KB."""
    _same(ctx, tmp_path, _text([f"{i // 300},{i}.125,{i % 17}.5," + "z" * pad for i in range(1100)]))


@pytest.mark.parametrize("empty", [0, 1, 70, 5000, 40000])
def test_more_lines_than_room(ctx, tmp_path, empty):
    _same(ctx, tmp_path, _text([f"{i // 3},{i}.5,1" for i in range(9)], "\n" * (empty + 1)))


@pytest.mark.parametrize("every", [1, 2, 300])
def test_host_lines_beside_group_starts(ctx, tmp_path, every):
    """Hexadecimal coordinates are read by the host; more than 256 groups, some starting with such a line."""
    _same(ctx, tmp_path, _text([f"{i // 2},{'0x10' if i % every == 0 else '4.5'},{i}" for i in range(1500)]))


@pytest.mark.parametrize("places", list(range(0, 14)))
def test_decimal_places(ctx, tmp_path, places):
    """Every number of decimal places converted in integers (up to eleven) and the first beyond: random digits, and
    values on, just below and just above the midpoint of two floats."""
    rng = np.random.default_rng(places)
    lines = []
    for i in range(4000):
        m = int(rng.integers(1, 1 << int(rng.integers(1, 54))))
        if i % 2:
            h = 2 * int(rng.integers(1 << 23, 1 << 24)) + 1            # 25 bits, the lowest set
            m = max(h * 10 ** places >> int(rng.integers(0, 3 * places + 25)), 1) + int(rng.integers(-1, 2))
            m = min(max(m, 1), (1 << 53) + 1)
        t = str(m).rjust(places + 1, "0")
        lines.append(f"{i // 500},{'-' if i % 3 == 0 else ''}{t[:len(t) - places]}.{t[len(t) - places:]},{m}e-{places}")
    _same(ctx, tmp_path, _text(lines))
