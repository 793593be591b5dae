"""A prediction reports a timed-out product whichever of its rows were discarded for it: k_take's blocks read the flag
at different moments, and what each acted on comes back behind the results (any_discarded, csrc/mlp.cu)."""
import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include "mlp.cu"
int main(int argc, char**)
{
    // host: one block of five has discarded its rows, each in turn; none
    const int n = 4 * kTakeRows + 1, blocks = take_blocks(n);
    float acted[5] = {};
    bool ok = blocks == 5 && !any_discarded(acted, n);
    for (float& a : acted) { a = 1.f; ok = ok && any_discarded(acted, n); a = 0.f; }
    float rows[n] = {};
    ok = ok && !maybe_discarded(rows, n);
    for (int b = 0; b < blocks; ++b) {
        for (int i = b * kTakeRows; i < n && i < (b + 1) * kTakeRows; ++i) rows[i] = NAN;
        ok = ok && maybe_discarded(rows, n);
        for (float& r : rows) r = 0.f;
    }
    if (argc > 1) {
        // device: the kernel with the flag down and up
        float *out, *y, h[n + 5];
        if (cudaMalloc(&out, (size_t)n * kOut * 4) || cudaMalloc(&y, sizeof h) || cudaMemset(out, 0, (size_t)n * kOut * 4)) return 2;
        for (int flag = 0; flag < 2; ++flag) {
            if (cudaMemcpyToSymbol(g_tc_error, &flag, sizeof flag)) return 2;
            k_take<<<blocks, kTakeRows>>>(out, n, y, y + n);
            if (cudaMemcpy(h, y, sizeof h, cudaMemcpyDeviceToHost)) return 2;
            for (int i = 0; i < n; ++i) ok = ok && (flag ? h[i] != h[i] : h[i] == 0.f);
            for (int b = 0; b < blocks; ++b) ok = ok && h[n + b] == (float)flag;
        }
    }
    std::puts(ok ? "ok" : "wrong");
    return 0;
}
"""


def _run(tmp_path, *args):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    (tmp_path / "status.cu").write_text(PROGRAM)
    exe = tmp_path / "status"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O1", "-std=c++17", "-I", str(ROOT / "include"),
                    "-I", str(ROOT / "rewl_simulator_gb300" / "csrc"), str(tmp_path / "status.cu"), "-o", str(exe)],
                   check=True, timeout=300)
    assert subprocess.run([str(exe), *args], check=True, timeout=120, capture_output=True, text=True).stdout.strip() == "ok"


def test_every_block_counts(tmp_path):
    _run(tmp_path)


@pytest.mark.gpu
def test_blocks_publish_what_they_acted_on(tmp_path):
    _run(tmp_path, "gpu")
