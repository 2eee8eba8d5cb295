"""How many CTAs an inference over n records gets (infer_ctas in renderx_gb300/csrc/rx_guide.h,
which both evaluation entry points use): one per 128-row tile until every SM has one."""
import os
import shutil
import subprocess

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "rx_guide.h"
int main(int argc, char** argv) {
  for (int k = 2; k < argc; k++) printf("%u\n", rx::guide::infer_ctas((uint32_t)strtoul(argv[k], nullptr, 10), atoi(argv[1])));
}
"""


def test_tiles_spread_over_the_sms_first(tmp_path):
    src, exe = tmp_path / "ctas.cu", tmp_path / "ctas"
    src.write_text(SOURCE)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-I",
                    os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "renderx_gb300", "csrc"), str(src), "-o",
                    str(exe)], check=True)
    rows = [1, 127, 128, 129, 1000, 1024, 1025, 20_000, 152 * 128 - 1, 152 * 128, 152 * 128 + 1, 1 << 20, 2 ** 32 - 1]
    r = subprocess.run([str(exe), "152", *map(str, rows)], capture_output=True, text=True, check=True)
    assert [int(x) for x in r.stdout.split()] == [min(-(-n // 128), 152) for n in rows]
    entry = open(os.path.join(ROOT, "renderx_gb300", "csrc", "rx_guide.cu")).read().split('extern "C" rx_status ')
    for name in ("rx_guide_eval(", "rx_guide_eval_device("):
        (body,) = [e for e in entry if e.startswith(name)]
        assert "<<<rx::guide::infer_ctas(n, g->sms), " in body
