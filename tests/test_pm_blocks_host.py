"""How many blocks PhotonMap's gathers get (pm_eye_blocks in renderx_gb300/csrc/rx_internal.h): a
pixel per warp until there are 256 blocks per SM, so that no large part of the image waits for
the blocks that find no room at first."""
import os
import shutil
import subprocess

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "rx_internal.h"
int main(int argc, char** argv) {
  for (int k = 2; k < argc; k++) printf("%u\n", rx::pm_eye_blocks((uint32_t)strtoul(argv[k], nullptr, 10), atoi(argv[1])));
}
"""


def test_a_pixel_per_warp(tmp_path):
    csrc = os.path.join(ROOT, "renderx_gb300", "csrc")
    src, exe = tmp_path / "blocks.cu", tmp_path / "blocks"
    src.write_text(SOURCE)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-I",
                    os.path.join(ROOT, "include"), "-I", csrc, str(src), "-o", str(exe)], check=True)
    pixels = [1, 3, 4, 5, 10_000, 1 << 16, 4 * 256 * 152 - 1, 4 * 256 * 152, 4 * 256 * 152 + 1, 1 << 22, 2 ** 32 - 1]
    r = subprocess.run([str(exe), "152", *map(str, pixels)], capture_output=True, text=True, check=True)
    assert [int(x) for x in r.stdout.split()] == [min(-(-n // 4), 256 * 152) for n in pixels]
    assert "k_pm_eye<<<pm_eye_blocks(P.n_pixels, c->trace_cfg.sms), 128, " in open(os.path.join(csrc, "rx_vcm.cu")).read()
