"""The block products' reduction refuses a symmetric plan: the partials of the symmetric kernels lack the self blocks and,
without torques, a factor 8 pi, so summing them as a block's would be silently wrong.  Calls the launch interface of
csrc/rpy_kernels.cuh directly; nothing is launched."""
import subprocess

from cufcm_fil_b200 import build

MAIN = r"""
#include "common.cuh"
#include "rpy_kernels.cuh"
#include <cstdio>
using namespace cufil;
int main() {
    int status[2];
    for (int c = 0; c < 2; ++c) {
        RpyBlockDesc d{};
        d.wall = c;
        d.vd = d.fd = 3;
        d.self_set = 1;
        d.nt = d.ns = 0;  // nothing to launch, were it accepted
        d.at = d.as = d.mu = 1.0f;
        const RpyPlan plan = rpy_plan_for(d, 148);
        if (!plan.sym) return 1;
        status[c] = rpy_launch_reduce_f32(d, plan, nullptr, nullptr, 6, kOutWrite, nullptr);
    }
    std::printf("%d", status[0] == CF_EINVAL && status[1] == CF_EINVAL);
}
"""


def test_symmetric_plans_are_refused(tmp_path):
    build.build()
    src, exe = tmp_path / "main.cu", tmp_path / "main"
    src.write_text(MAIN)
    objs = [str(build.BUILD / f"{n}.o") for n in ("rpy_kernels", "errors")]
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", str(build.CSRC), "-I",
                    str(build.INCLUDE), str(src), *objs, "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout == "1"
