"""The buffer of the gradient reduction's partial sums holds what a launch writes, whatever number of
materials the parameters are set to after it was allocated."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include <cstdio>
#include <initializer_list>
#include "da_internal.h"
int main() {
    using namespace da;
    for (int ninst : {0, 1, 11, 12, 17, 24, 512, 70000})
        for (int mat = 1; mat <= DA_MAX_MATERIALS; ++mat) {
            // k_adj_reduce: kAdjReduceParts ranges of every output; k_adj_reduce_inst: the last member's
            // last output's last range
            const size_t nout = mat + 2;
            const size_t single = (size_t)kAdjReduceParts * (mat + 1 + DA_MAX_PILES);
            const size_t members = ninst ? (((size_t)(ninst - 1) * nout + nout - 1) * kAdjInstParts + kAdjInstParts) : 0;
            if (adj_part_doubles(ninst) < single || adj_part_doubles(ninst) < members) {
                printf("%d members, %d materials: %zu doubles\n", ninst, mat, adj_part_doubles(ninst));
                return 1;
            }
        }
    return 0;
}
"""


def test_partial_sums_fit_any_material_count(tmp_path):
    (tmp_path / "p.cpp").write_text(SRC)
    exe = str(tmp_path / "p")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-I" + os.path.join(cuda, "include"), "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "discrete_adjoint_b200", "csrc"), str(tmp_path / "p.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
