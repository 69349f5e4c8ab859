"""Kernels that are launched while the one in front of them still writes (those that call griddep_wait) read nothing
past the coherent path: ``ld.global.nc`` wants data that nobody writes while the kernel lives."""
import os
import re

import tridist_b200

# behind the metadata kernel, which starts it when all kernels before are complete
BEHIND_ANOTHER = {"moe_dispatch_kernel"}


def test_early_kernels_read_coherently():
    ops = os.path.join(os.path.dirname(tridist_b200.__file__), "csrc", "ops")
    seen = set()
    for name in ("moe_a2a.cu", "elementwise.cu"):
        with open(os.path.join(ops, name)) as f:
            parts = re.split(r"__global__ void", f.read())[1:]
        for part in parts:
            kernel = re.search(r"(\w+_kernel)\(", part).group(1)
            body = part[:part.index("\n}\n")]
            if "griddep_wait()" in body:
                seen.add(kernel)
                assert "ld_global_nc" not in body or kernel in BEHIND_ANOTHER, kernel
    assert {"moe_route_dispatch_kernel", "moe_dispatch_kernel", "swiglu_kernel"} <= seen
