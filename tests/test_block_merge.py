"""The block merge (subsets of the low terminals reduced together in registers):
its plan on the CPU, and whole tables against the oracle on the GPU."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "steiner_edge_linear_gb300", "csrc")
SMEM_BYTES = 224 * 1024  # emv_device.cu


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path_factory.mktemp("plan") / "block_merge_check")
    subprocess.run([gxx, "-O2", "-std=c++17", "-I", CSRC, os.path.join(ROOT, "tests", "block_merge_check.cpp"),
                    os.path.join(CSRC, "emv_plan.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("k,low", [(k, low) for k in range(6, 13) for low in (4, 5)])
def test_plan_forms_every_pair(checker, k, low):
    out = subprocess.run([checker, str(k), str(SMEM_BYTES), str(low)], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and out.stdout == f"ok k={k} block_levels={k - 2}\n", out.stdout + out.stderr


def test_plan_leaves_out_levels_that_do_not_fit(checker):
    """512 rows: of k = 12 only level 3 (220 minima, 12 + 66 staged rows)."""
    out = subprocess.run([checker, "12", str(64 * 1024)], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and out.stdout.startswith("ok k=12 block_levels=1"), out.stdout + out.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("n,k,wmax,bits", [(40037, 6, 100, 0), (40000, 8, 100, 0), (33001, 9, 1000, 32), (9001, 10, 9000, 0),
                                           (10007, 11, 100, 0), (10007, 11, 1000, 32), (4099, 12, 300, 0),
                                           (4128, 12, 1000, 32), (33, 12, 9, 0), (64, 12, 9, 0), (65, 12, 9, 32)])
def test_whole_tables(emv, orc, n, k, wmax, bits):
    """Odd and even table strides, ragged last blocks, 16- and 32-bit values."""
    csr = emv.Csr.from_stp(emv.StpInstance.regular(n, 4, 1, wmax, k, 17))
    want, cost = orc.emv_table(csr.n, csr.row_ptr, csr.col, csr.w, csr.terminals, threads=16)
    with emv.Solver(0) as s:
        s.set_value_bits(bits)
        res = s.solve(csr, table=True)
        assert res.cost == cost and np.array_equal(res.table, want)


SKIP_CHECK = r"""
#include <cstdio>
#include <cstdlib>
#include "emv_plan.h"
using namespace emv;
int main(int, char **argv)
{
    const int k = atoi(argv[1]);
    std::vector<uint32_t> xs, all, some, blocks;
    std::vector<int64_t> off;
    subset_levels(k, xs, off);
    std::vector<std::vector<HostGroup>> whole, part;
    std::vector<HostBlockLevel> block;
    plan_block_levels(k, BLOCK_LOW, xs, off, 224 * 1024, blocks, block);
    std::vector<bool> skip;
    for (const HostBlockLevel &L : block) skip.push_back(!L.phases.empty());
    plan_stream_levels(k, xs, off, 224 * 1024, all, whole);
    plan_stream_levels(k, xs, off, 224 * 1024, some, part, skip);
    for (int m = 2; m <= k; m++) {
        if (skip[m] != part[m].empty()) return printf("level %d\n", m), 1;
        if (skip[m]) continue;
        if (part[m].size() != whole[m].size()) return printf("groups of level %d\n", m), 1;
        for (size_t g = 0; g < part[m].size(); g++)
            for (size_t p = 0; p < part[m][g].phases.size(); p++) {
                const HostPhase &a = part[m][g].phases[p], &b = whole[m][g].phases[p];
                if (a.nrows != b.nrows || a.pairs_at % 4) return printf("phase of level %d\n", m), 1;
                for (int i = 0; i < a.nrows; i++)
                    if (some[a.rows_at + i] != all[b.rows_at + i]) return printf("rows of level %d\n", m), 1;
            }
    }
    printf("ok %d\n", some.size() * 4 < all.size());
}
"""


@pytest.mark.parametrize("k", [6, 9, 11])
def test_levels_with_a_block_merge_have_no_streamed_plan(tmp_path, k):
    """The streamed plan of the other levels is as without the omission, and
    the whole a fraction of the plan of all levels."""
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    src, exe = tmp_path / "skip.cpp", tmp_path / "skip"
    src.write_text(SKIP_CHECK)
    subprocess.run([gxx, "-O1", "-std=c++17", "-I", CSRC, str(src), os.path.join(CSRC, "emv_plan.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe), str(k)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout == "ok 1\n", out.stdout + out.stderr
