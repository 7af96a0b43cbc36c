"""The library holds no kernel of the FP64 triangle for the operators that never take it: the
stretching and the adjoint go from the circle to several launches (plan_both64 with MULTI false)."""
import subprocess


def test_no_triangle_of_the_fp64_stretching_and_adjoint():
    from openonda_b200 import _lib, build

    build.build()
    names = subprocess.run(["nm", "-C", _lib.LIB_PATH], capture_output=True, text=True,
                           check=True).stdout.splitlines()
    lists = [s for s in names if "rot64_lists_kernel<" in s]
    assert any("OpStretchBoth" in s and "CircleLists" in s for s in lists)
    assert any("OpVelBoth" in s and "TriLists64" in s for s in lists)
    reached = ("OpVelBoth", "OpPseBoth", "OpVelStretchBoth", "OpLesStepBoth")
    for s in lists:
        if "TriLists64" in s:
            assert any(op in s for op in reached), s
