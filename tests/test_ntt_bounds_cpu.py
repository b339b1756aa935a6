"""Bounds that the forward transforms assume for what they read, checked as the compiler of the kernels sees them."""
import os
import subprocess

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = """
#include "ntt_kernels.cuh"
using namespace b2;
template <class A> constexpr bool sources() {
    return src_bound<A, 0>() == A::B_CANON && src_bound<A, SRC_WORDS>() == A::B_WORDS && src_bound<A, SRC_CONV>() == A::B_BCONV &&
           src_bound<A, SRC_REM>() == A::B_CANON && src_bound<A, SRC_REM | SRC_NEAR>() == A::B_CANON &&
           src_bound<A, SRC_WORDS | SRC_REM>() == A::B_CANON + A::B_WORDS && src_bound<A, SRC_CONV | SRC_REM>() == A::B_CANON + A::B_BCONV;
}
static_assert(sources<ArithFp<false>>() && sources<ArithFp<true>>() && sources<ArithIntLazy>() && sources<ArithInt>());
// what the units stand for: sixteenths of q (FP64, primes of 41 to 50 bits), q (lazy integers)
static_assert(ArithFp<true>::B_CANON == 16 && ArithFp<true>::B_WORDS == 32 && ArithIntLazy::B_CANON == 1 && ArithIntLazy::B_WORDS == 2);
// canonical words of a 41- to 50-bit prime: two stages without a reduction
using F = ArithFp<true>;
static_assert(F::factor(src_bound<F, 0>()) == src_bound<F, 0>() && F::factor(ct_bound<F>(src_bound<F, 0>(), 1)) == ct_bound<F>(src_bound<F, 0>(), 1));
"""


def test_source_bounds(tmp_path):
    src = tmp_path / "bounds.cu"
    src.write_text(SOURCE)
    out = subprocess.run(["nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I" + os.path.join(_ROOT, "phantom-fhe_b200", "csrc"),
                          "-c", str(src), "-o", str(tmp_path / "bounds.o")], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
