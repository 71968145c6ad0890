"""Host rules that choose launch shapes from sizes (csrc/launch_rules.h), compiled by the
host compiler and evaluated over their whole range: every rule ends, covers the grid and
keeps within the slots it is given."""
import pathlib
import shutil
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "zoomy-jax_b200" / "csrc"


@pytest.fixture(scope="module")
def evaluate(tmp_path_factory):
    """``evaluate(body, rows)``: a program that reads one line of integers per call of
    ``body`` (as ``a[]``) and prints what it prints."""
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no C++ compiler")

    def run(body, rows):
        d = tmp_path_factory.mktemp("rules")
        n = len(rows[0])
        (d / "rules.cpp").write_text(
            '#include <cstdio>\n#include "launch_rules.h"\nusing namespace zb;\n'
            f"int main() {{\n  long long a[{n}];\n  for (;;) {{\n"
            f"    for (int i = 0; i < {n}; ++i) if (std::scanf(\"%lld\", &a[i]) != 1) return 0;\n"
            f"    {body}\n  }}\n}}\n")
        subprocess.run([gxx, "-std=c++17", "-O2", "-I", str(CSRC), str(d / "rules.cpp"), "-o",
                        str(d / "rules")], check=True)
        text = "\n".join(" ".join(str(int(v)) for v in r) for r in rows)
        out = subprocess.run([str(d / "rules")], input=text, capture_output=True, text=True,
                             check=True, timeout=60).stdout
        return [[int(v) for v in line.split()] for line in out.splitlines()]

    return run


# (nx, ny) of a level on strips: square, tall, wide; wide ones with more strips than there
# are slots for partial sums, up to the largest level (2^31 cells)
LEVELS = [(800, 800), (1024, 1024), (2048, 2048), (46340, 46340), (10242, 64), (80004, 8),
          (64, 10242), (8, 80004), (8, 851968), (8, 852020), (8, 900000), (8, 1000000),
          (4, 500000), (6, 3000000), (8, 260000000), (4, 536870910), (536870910, 4)]


@pytest.mark.parametrize("nu", [1, 2, 3, 4])
def test_multigrid_strips(evaluate, nu):
    cols, parts = 64 - 2 * (2 * nu + 2), 4096
    got = evaluate("MgStrips s = mg_strips((int)a[0], (int)a[1], (int)a[2], a[3] != 0, (int)a[4]);"
                   ' std::printf("%d %d %d %d\\n", s.strips, s.rows, s.ctas, (int)s.dot);',
                   [(nx, ny, cols, dot, parts) for nx, ny in LEVELS for dot in (0, 1)])
    for k, (nx, ny) in enumerate(LEVELS):
        plain, with_dot = got[2 * k], got[2 * k + 1]
        for strips, rows, ctas, dot in (plain, with_dot):
            assert strips * cols >= ny > (strips - 1) * cols
            assert rows >= 4 and rows % 2 == 0
            assert 4 * ctas >= strips * -(-nx // rows) > 4 * (ctas - 1)
            assert not dot or ctas <= parts
        assert not plain[3]
        # the sums are left out only where full-height items do not fit
        assert with_dot[3] == (-(-with_dot[0] // 4) <= parts)
        if not with_dot[3] or plain[2] <= parts:
            assert with_dot[:3] == plain[:3]


# (16, 16) networks at 512 x 724^2 and 512 x 726^2 lie on both sides of 2^32 elements
PLANES = [(8, 64 * 32 ** 2), (24, 64 * 32 ** 2), (24, 512 * 256 ** 2), (16, 512 * 724 ** 2),
          (16, 512 * 726 ** 2), (24, 178956971), (8, 430000000), (16, 279000000)]


def test_plane_slices(evaluate):
    stride = 148 * 16 * 256    # a grid's threads
    got = evaluate('std::printf("%d\\n", plane_slice((int)a[0], a[1]));', PLANES)
    for (channels, pixels), (n,) in zip(PLANES, got):
        assert 1 <= n <= channels
        assert n * pixels + stride < 2 ** 32
        assert n == channels or (n + 1) * pixels > 2 ** 31


# widths on both sides of the first middle strip (58 columns), heights on both sides of the
# uniform list's limit; the tall narrow grids have boundary strips alone
GRIDS = [(nx, ny) for ny in (3, 28, 40, 56, 57, 58, 84, 300, 2048)
         for nx in (3, 5, 64, 500, 2048, 20000, 100000, 300000) if nx * ny < 2 ** 31] + [
             (700000000, 3), (3, 700000000), (4, 500000000)]


@pytest.mark.parametrize("f32", [0, 1])
def test_strip_rows(evaluate, f32):
    got = evaluate("StripRows r = strip_rows((int)a[0], (int)a[1], a[2] != 0);"
                   ' std::printf("%d %d %d %d\\n", r.sx, r.sxc, (int)r.single,'
                   " full_mid_strips((int)a[1]));", [(nx, ny, f32) for nx, ny in GRIDS])
    for (nx, ny), (sx, sxc, single, nmid) in zip(GRIDS, got):
        strips = -(-ny // 28)
        assert 1 <= sx <= 64 and sxc == 4
        assert nmid == max(0, (ny - 30) // 28 if ny >= 30 else 0)
        assert single == (nmid == 0 or strips * nx < 6 * 592)
        # boundary strips alone: never in shorter chunks than beside middle strips, and
        # few halo rows on a grid of many waves
        if nmid == 0 and strips * nx >= 6 * 592:
            assert sx >= (32 if strips * nx >= 200000 else 4)
