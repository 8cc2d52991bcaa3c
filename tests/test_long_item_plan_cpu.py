"""plan_long_items on the host: the SMs it takes from the paired launches are
fewer than the device has, whatever their number."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
PKG = os.path.join(ROOT, "swhybrid_b200")
CUDA = "/usr/local/cuda/include"

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "csrc/sw_engine.h"
#include "csrc/sw_registry.h"
int main(int argc, char** argv) {
    sw_ctx c;
    c.num_sms = atoi(argv[1]);
    c.max_smem = 232448;
    c.n_pairs = 2000;
    c.pair_prefix.push_back(0);
    for (int p = 0; p < c.n_pairs; ++p) {
        c.pair_ncols.push_back(p < 40 ? 30000u : 300u);
        c.pair_prefix.push_back(c.pair_cols_total += c.pair_ncols.back());
    }
    std::vector<uint32_t> qlen;
    for (int i = 0; i < 16; ++i) qlen.push_back(50u + 500u * i);
    std::vector<swb::QpLoad> loads(3);
    for (auto& l : loads) { l.sum_passes = 8; l.max_passes = 2; }
    const swb::LongItemPlan plan =
        swb::plan_long_items(&c, qlen, loads, *swb::find_qp(16, 64), 1.0, argc > 2 ? atoi(argv[2]) : -1);
    printf("%lld %d %zu\n", (long long)plan.n_long, plan.sms, plan.count());
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    lib = os.path.join(PKG, "libswb200.so")
    if not (shutil.which("g++") and os.path.isdir(CUDA) and os.path.exists(lib)):
        pytest.skip("needs g++, the CUDA headers and the built library")
    d = tmp_path_factory.mktemp("plan")
    (d / "main.cpp").write_text(SOURCE)
    exe = str(d / "main")
    out = subprocess.run(["g++", "-std=c++17", "-O1", "-I", PKG, "-I", CUDA, "-o", exe,
                          str(d / "main.cpp"), lib, "-Wl,-rpath," + PKG, "-L/usr/local/cuda/lib64",
                          "-lcudart"], capture_output=True, text=True)
    assert out.returncode == 0, out.stderr
    return exe


@pytest.mark.parametrize("sms", [2, 3, 16, 20, 72, 96, 97, 148])
def test_the_paired_launches_keep_an_sm(program, sms):
    out = subprocess.run([program, str(sms)], capture_output=True, text=True, check=True)
    n_long, taken, items = map(int, out.stdout.split())
    assert 0 <= taken < sms
    assert (n_long == 0) == (items == 0) == (taken == 0)


def test_given_pairs(program):
    out = subprocess.run([program, "148", "40"], capture_output=True, text=True, check=True)
    n_long, taken, items = map(int, out.stdout.split())
    # 16 queries of 50..7,550 residues: 16 / passes pipelines a block
    pipes = [16 // -(-q // (32 * r)) for q in range(50, 8000, 500)
             for r in [4 if q <= 2048 else 8 if q <= 4096 else 16]]
    assert n_long == 40 and 0 < taken <= 98 and items == sum(-(-40 // g) for g in pipes)
