"""Source rules of the element-wise kernels."""
import os
import re

from iris_b200 import _native


def test_kernels_that_start_early_read_through_the_coherent_path():
    """These kernels are placed while the kernel that makes their inputs may still run, so nothing they read is constant
    for their whole lifetime: no pointer may promise that (``__restrict__`` lets the compiler read through the
    non-coherent path and lift a load over the grid dependency wait), and no load may ask for that path by name."""
    path = os.path.join(os.path.dirname(_native.__file__), "csrc", "kernels", "elementwise.cu")
    source = re.sub(r"//[^\n]*", "", open(path).read())
    kernels = re.findall(r"__global__[^;{]*?(\w+_kernel)\(([^{]*?)\)\s*\{(.*?)\n\}\n", source, re.S)
    assert {k[0] for k in kernels} == {"rmsnorm_kernel", "rmsnorm_reg_kernel", "add_rmsnorm_reg_kernel", "swiglu_kernel",
                                       "residual_add_kernel"}
    for name, params, body in kernels:
        assert "__restrict__" not in params, name
        assert not re.search(r"__ldg|__ldlu|ld\.global\.nc", body), name
        # nothing is read before the wait
        assert re.search(r"^\s*(constexpr[^;]*;|__shared__[^;]*;|\s)*begin\(\);", body), name
