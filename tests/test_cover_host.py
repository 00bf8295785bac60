"""The column tiles of rows copied by the aligned 16-byte vectors that cover them: no byte behind a row is read."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "compressgnn_b200" / "csrc"

# Every width around several tiles, every row begin a unit allows, every tile of a row: the columns have to lie in the
# cover, and the cover -- all of it where ragged_whole_cover says so, else what is clipped to the tile -- in the row.
PROGRAM = r"""
#include <algorithm>
#include <cstdio>
#include "cgnn_cover.h"
int main() {
    for (int unit : {4, 8})
        for (int lpr : {4, 8, 16, 32}) {
            const int tile = cgnn::ragged_tile(lpr, unit);
            for (int64_t width = unit / 4; width <= (lpr == 32 ? 5 * tile + 8 : tile); width += unit / 4)
                for (int lead = 0; lead < 16; lead += unit)
                    for (int64_t col0 = 0; col0 < width; col0 += tile) {
                        // bytes from the row's first: the tile begins `lead` bytes behind a 16-byte boundary
                        const int64_t begin = 4 * col0, end = std::min<int64_t>(4 * (col0 + tile), 4 * width);
                        const int64_t cover = begin - lead + lpr * 16;
                        const int64_t read = cgnn::ragged_whole_cover(lpr, width, col0) ? cover : std::min(cover, end);
                        if (cover < end || read > 4 * width)
                            return printf("unit %d lanes %d width %lld lead %d column %lld\n", unit, lpr, (long long)width, lead,
                                          (long long)col0), 1;
                    }
        }
}
"""


def test_a_cover_stays_inside_its_row(tmp_path):
    source, program = tmp_path / "cover.cpp", tmp_path / "cover"
    source.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", f"-I{CSRC}", str(source), "-o", str(program)], check=True)
    found = subprocess.run([str(program)], stdout=subprocess.PIPE, text=True)
    assert found.returncode == 0, found.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
@pytest.mark.parametrize("width", [125, 126, 127, 128, 249, 250, 251, 252, 373, 376])
def test_rows_that_end_inside_a_cover(width, shift):
    """Widths a few columns beyond whole tiles, rows long enough for full stages, and the matrix ending where its last
    row does, against float64 sums; the bound is that of any order of a row's additions."""
    import torch
    from compressgnn_b200 import runtime as rt
    gen = torch.Generator(device="cuda").manual_seed(width)
    rows, src_rows, degree = 200, 150, 40
    flat = torch.randn(src_rows * width + shift, device="cuda", generator=gen)
    src = flat[shift:].view(src_rows, width)
    rowptr = torch.arange(rows + 1, device="cuda") * degree
    col = torch.randint(0, src_rows, (rows * degree,), device="cuda", generator=gen)
    col[::7] = src_rows - 1
    val = torch.randn(rows * degree, device="cuda", generator=gen)
    got = rt.spmm_func(rowptr, col, val, src, "rowbalance_rowcache", None)
    terms = (src[col].double() * val.double()[:, None]).view(rows, degree, width)
    bound = degree * 0.5 * torch.finfo(torch.float32).eps * terms.abs().sum(1) * (1 + 1e-3)
    assert bool(((got.double() - terms.sum(1)).abs() <= bound).all())
