"""How the kernels that read planes in place cut their outputs into blocks (BlockTile in csrc/common.cuh), computed by its host code."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")

MAIN = """
#include <cstdio>
#include "common.cuh"
int main() {
  long long h, w, l;
  while (scanf("%lld %lld %lld", &h, &w, &l) == 3) {
    const sph::BlockTile t = sph::BlockTile::make(h, w, (int)l);
    printf("%d %d %d %u\\n", t.height, t.width, t.log_tx, t.blocks());
  }
}
"""


@pytest.fixture(scope="module")
def tiles(tmp_path_factory):
    nvcc = NVCC if os.path.exists(NVCC) else shutil.which("nvcc")
    if nvcc is None:
        pytest.skip("no CUDA compiler")
    d = tmp_path_factory.mktemp("tiles")
    (d / "main.cu").write_text(MAIN)
    csrc = os.path.join(ROOT, "spherical-package_b200", "csrc")
    subprocess.run([nvcc, "-std=c++17", "-I" + csrc, "-I" + os.path.join(ROOT, "include"), str(d / "main.cu"), "-o", str(d / "main")], check=True)

    def run(shapes):
        text = "".join("%d %d %d\n" % s for s in shapes)
        r = subprocess.run([str(d / "main")], input=text, capture_output=True, text=True, check=True)
        return [tuple(map(int, line.split())) for line in r.stdout.splitlines()]
    return run


def test_blocks_cover_the_outputs_and_are_filled(tiles):
    """Whatever the shape, one row and one column among them: every output has a thread, and beyond a few blocks four fifths of the threads
    have an output (16 x 16 tiles of a single row would have one in sixteen)."""
    sizes = (1, 2, 3, 4, 5, 7, 8, 9, 12, 15, 16, 17, 31, 33, 63, 64, 65, 66, 100, 129, 255, 257, 1000, 4097, 65536)
    shapes = [(h, w, l) for h in sizes for w in sizes for l in (4, 5, 6)]
    for (h, w, l), (th, tw, log_tx, blocks) in zip(shapes, tiles(shapes)):
        assert (th, tw, log_tx) == (1, h * w, 8) or (th, tw) == (h, w) and log_tx in (l, l - 1), (h, w, l)
        assert blocks == -(-tw // (1 << log_tx)) * -(-th // (256 >> log_tx))
        need = -(-h * w // 256)
        assert need <= blocks <= 1.25 * need + 8, (h, w, l, blocks)


def test_images_keep_their_tiles(tiles):
    shapes = [(1280, 64, 4), (5120, 256, 4), (512, 1024, 5), (128, 256, 6), (23, 46, 6), (33, 66, 6)]
    assert [t[2] for t in tiles(shapes)] == [4, 4, 5, 6, 6, 5]
