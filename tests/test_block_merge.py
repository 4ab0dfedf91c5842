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
