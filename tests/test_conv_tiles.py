"""The row-tile convolution's shapes over every pair of widths that the
launcher accepts, from the header the launcher uses: where it is taken, its two
accumulators lie in the tensor memory that a CTA allocates, the CTAs resident
on an SM take no more than there is, and everything fits in shared memory."""
import os
import shutil
import subprocess

import pytest

from tests.conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include "conv_tiles.hpp"
int main() {
  using namespace swfwi;
  for (int cin = 16; cin <= 128; cin += 16)
    for (int cout = 16; cout <= 256; cout += 16)
      std::printf("%d %d %d %d %d %d %zu %zu\n", cin, cout, tg::fits(cin, cout) ? 1 : 0, tg::cols(cin, cout),
                  tmem_cols(2 * tg::cols(cin, cout)), tg::stages(cin, cout), tg::smem(cin, cout),
                  tg::launch_smem(cin, cout));
}
"""


@pytest.fixture(scope="module")
def shapes(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("conv")
    (d / "p.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Wextra", "-Werror", "-I",
                    os.path.join(ROOT, "swfwi_b200", "csrc"), str(d / "p.cpp"), "-o", str(d / "p")], check=True)
    text = subprocess.run([str(d / "p")], capture_output=True, text=True, check=True).stdout
    return [tuple(map(int, line.split())) for line in text.splitlines()]


def test_taken_shapes_fit(shapes):
    assert len(shapes) == 8 * 16
    for cin, cout, fits, cols, allocated, stages, need, smem in shapes:
        if not fits:
            continue
        assert cols % 16 == 0 and cols <= 256 and cout in (cols, 2 * cols)    # one MMA's columns
        assert 2 * cols <= allocated, (cin, cout)                             # two accumulators
        resident = (228 * 1024) // (smem + 1024)
        assert resident * allocated <= 512, (cin, cout, resident)
        assert stages >= 2 and need <= smem <= 227 * 1024, (cin, cout)


def test_the_networks_layers_take_row_tiles(shapes):
    taken = {(s[0], s[1]) for s in shapes if s[2]}
    for cin, cout in ((16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (128, 64), (96, 32), (48, 16),
                      (16, 48), (32, 96), (64, 128), (32, 16), (64, 32)):
        assert (cin, cout) in taken, (cin, cout)


def test_epilogue_leaves_by_a_vote():
    """Reads of tensor memory need whole warps: where the row-tile kernel's
    epilogue may leave its loop on a wait that gave up, the warp votes."""
    with open(os.path.join(ROOT, "swfwi_b200", "csrc", "precond.cu")) as f:
        text = f.read()
    at = text.index("// ---- epilogue")
    loop = text[at:text.index("tcgen05.ld.sync", at)]
    leaves = [line.strip() for line in loop.splitlines() if "break;" in line]
    assert leaves and all(line.startswith("if (__any_sync(0xffffffffu,") for line in leaves), leaves
