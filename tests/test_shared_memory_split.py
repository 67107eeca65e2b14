"""The shared-memory split every kernel of a step asks for: room for the CTAs
that its launch bound makes resident, each with its own shared memory and the
1 KB the system takes, out of the SM's 228 KB; all of it for dual numbers, whose
kernels have no launch bound.  Checked at compile time by a translation unit of
static assertions over the kernels' own constants."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
HEAD = r'''
#include "tri_kernels.cuh"
using namespace zj;
constexpr bool fits(int percent, int ctas, size_t smem) {
    return percent >= 100 || (long long)percent * 228 * 1024 >= 100LL * ctas * (long long)(smem + 1024);
}
'''
QUAD = r'''
template <int P, typename T> constexpr bool quad() {
    static_assert(fits(phys_carveout<P, T>(), PhysMinBlocks<T>::value, stage_smem<P, T>()), "inviscid stage");
    static_assert(fits(ns_carveout<P, T>(), NSMinBlocks<T, P>::stage, stage_smem<P, T>()), "viscous stage");
    static_assert(fits(ns_carveout<P, T>(), LineShape<P, T>::MIN_BLOCKS, LineShape<P, T>::SMEM), "gradient");
    return true;
}
template <typename T> constexpr bool all() { return quad<1, T>() && quad<2, T>() && quad<3, T>() && quad<4, T>() && quad<5, T>(); }
static_assert(all<double>() && all<float>(), "");
'''
DUAL = r'''
template <int P> constexpr bool dual() { return phys_carveout<P, Dual>() == 100 && ns_carveout<P, Dual>() == 100; }
static_assert(dual<1>() && dual<2>() && dual<3>() && dual<4>() && dual<5>(), "dual numbers take the largest split");
'''


@pytest.mark.parametrize("body", [QUAD, DUAL], ids=["quad", "dual"])
def test_split_holds_the_resident_ctas(tmp_path, body):
    src = tmp_path / "split.cu"
    src.write_text(HEAD + body)
    r = subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-c", "-I",
                        os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "zhijian_b200", "csrc"),
                        str(src), "-o", str(tmp_path / "split.o")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
